"""The ray design on a device that is nearly full: a plan without room for the whole volume's
accumulator (8 bytes a voxel) takes the slabs', with the same bits."""
import pytest

from conftest import small_cfg

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from recon_b200 import PROJECTOR_BACK, SIDDON_BP_RAY, Options, Plan  # noqa: E402

# 256^3: the accumulator takes 136 MB, the z-fastest copy of the image 68 MB, the slabs 67 MB,
# an image or a sensitivity 67 MB
CFG = small_cfg(Xdim=256, Ydim=256, Zdim=256, XVoxSize=0.25, YVoxSize=0.25, ZVoxSize=0.25, AxPixels=120, TAxPixels=110,
                AxPixDim=1.0, TAxPixDim=1.0, NumProj=12)
MB = 1 << 20


def _fill(leave):
    """Takes the device's free memory but for `leave` MB."""
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    if free < (leave + 64) * MB:
        pytest.skip("the device has too little free memory to begin with")
    return torch.empty((free - leave * MB) // (2 * MB) * (2 * MB), dtype=torch.uint8, device="cuda")


@pytest.mark.parametrize("leave", [
    170,  # less than the accumulator after the z-fastest copy
    230,  # room for the accumulator, then none for an iteration's sensitivity
])
def test_plan_without_room(leave):
    opts = Options(siddon_bp=SIDDON_BP_RAY)
    P = Plan(CFG, opts)
    gen = torch.Generator("cuda").manual_seed(331)
    y = torch.rand((P.nproj, P.nv, P.nu), device="cuda", generator=gen)
    want, out = P.bp_views(y), P.new_volume()
    assert P.last_kernel(PROJECTOR_BACK) == "bp_column_kernel"
    f = P.new_volume(1.0)
    g = P.fp_views(f) * (0.5 + y)
    P.mlem_prepare()
    expect = f.clone()
    P.mlem_iteration(g, expect)
    P.close()
    hold = _fill(leave)
    try:
        Q = Plan(CFG, opts)
        Q.bp_views(y, out=out)
        assert Q.last_kernel(PROJECTOR_BACK) == "bp_ray_kernel"
        assert torch.equal(out.view(torch.int32), want.view(torch.int32))
        if leave > 200:
            Q.mlem_prepare()
            Q.mlem_iteration(g, f)
            assert torch.equal(f.view(torch.int32), expect.view(torch.int32))
        Q.close()
    finally:
        del hold
        torch.cuda.empty_cache()
    R = Plan(CFG, opts)
    R.bp_views(y, out=out)
    assert R.last_kernel(PROJECTOR_BACK) == "bp_column_kernel"

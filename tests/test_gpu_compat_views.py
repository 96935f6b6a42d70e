"""COMPAT projections of one and of many views: the two take different routes through
memory (the caller's volume, a copy whose z runs fastest) and, for power-of-two voxel
sizes, products in place of divisions; every ray's sum is the same, bit for bit."""
import numpy as np
import pytest

from conftest import rel_l2, small_cfg

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from recon_b200 import ARITH_COMPAT, Options, Plan  # noqa: E402

GEOMS = {
    "pow2": small_cfg(),
    "pow2_unequal": small_cfg(XVoxSize=0.5, YVoxSize=2.0, ZVoxSize=0.25, Zdim=33, Xdim=41),
    "odd": small_cfg(Xdim=31, Ydim=45, Zdim=27, XVoxSize=0.7, YVoxSize=0.9, ZVoxSize=1.1, AxPixels=61, TAxPixels=75),
    "one_slice": small_cfg(Zdim=1, TAxPixels=3, AxPixels=9, NumProj=7, DeltaAng=51.0),
    "tilted": small_cfg(Dx=0.7, Dz=-0.4, Ry=803.0, M=1.2, xangle=0.02, yangle=-0.01, zangle=0.03),
}


def _bits(t):
    return t.view(torch.int32)


@pytest.mark.parametrize("name", list(GEOMS))
def test_views_equal_single_views(name):
    P = Plan(GEOMS[name], Options(arith=ARITH_COMPAT))
    gen = torch.Generator("cuda").manual_seed(301)
    vol = torch.rand(P.shape_vol, device="cuda", generator=gen)
    all_views = P.fp_views(vol)
    assert all_views.abs().sum() > 0
    for n in range(P.nproj):
        assert torch.equal(_bits(all_views[n]), _bits(P.fp_view(vol, P.angle(n)))), n
    # the back projections of all views in one rounding: each single view's image is
    # rounded to 2^-24 of its voxel, and adding them rounds as often again
    y = torch.rand((P.nproj, P.nv, P.nu), device="cuda", generator=gen) - 0.2
    total = sum(P.bp_view(y[n], P.angle(n)).double() for n in range(P.nproj))
    assert rel_l2(P.bp_views(y).cpu().numpy(), total.cpu().numpy()) < P.nproj * 2.0**-24
    assert torch.equal(P.bp_views(y[2:3], 2, 1), P.bp_view(y[2], P.angle(2)))
    some = sum(P.bp_view(y[n], P.angle(n)).double() for n in (1, 2, 3))
    assert rel_l2(P.bp_views(y[1:4], 1, 3).cpu().numpy(), some.cpu().numpy()) < 3 * 2.0**-24


@pytest.mark.parametrize("name", list(GEOMS))
def test_sums_equal_the_traced_steps(name):
    """A ray's projection is its traced steps' products, added in order in FP32 (the
    trace divides by the voxel size)."""
    P = Plan(GEOMS[name], Options(arith=ARITH_COMPAT))
    vol = torch.rand(P.shape_vol, device="cuda", generator=torch.Generator("cuda").manual_seed(302))
    flat = vol.cpu().numpy().ravel()
    for n in range(0, P.nproj, 3):
        img = P.fp_views(vol)[n].cpu().numpy().ravel()
        rays = np.arange(0, P.nu * P.nv, 7, dtype=np.int32)
        loop, _, _ = P.compat_trace(P.angle(n), rays[:1], 1)
        _, idx, length = P.compat_trace(P.angle(n), rays, loop + 1)
        acc = np.zeros(len(rays), np.float32)
        for k in range(loop + 1):
            acc += np.where(idx[:, k] >= 0, length[:, k] * flat[np.maximum(idx[:, k], 0)], np.float32(0)).astype(np.float32)
        assert np.array_equal(acc.view(np.uint32), img[rays].view(np.uint32)), n


def test_projections_on_two_streams():
    """Calls on two streams of one plan, whose copies of the volume share memory."""
    P = Plan(GEOMS["odd"], Options(arith=ARITH_COMPAT))
    gen = torch.Generator("cuda").manual_seed(303)
    vols = [torch.rand(P.shape_vol, device="cuda", generator=gen) for _ in range(2)]
    expect = [P.fp_views(v) for v in vols]
    streams = [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()
    outs = [[], []]
    for _ in range(8):
        for k, s in enumerate(streams):
            with torch.cuda.stream(s):
                outs[k].append(P.fp_views(vols[k]))
    torch.cuda.synchronize()
    for k in range(2):
        for o in outs[k]:
            assert torch.equal(_bits(o), _bits(expect[k]))

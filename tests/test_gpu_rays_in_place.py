"""The ray design's back projection of a sinogram read in place along detector columns (volumes
of more than 2^20 voxels, or many rays): against the slabs' kernel, whose sums are the same
integers.  Ranges of few rays take the one, of many the other, so that the sums of ranges,
each rounded once, bound the whole's: n roundings of parts no larger than the sum of their
magnitudes."""
import pytest

from conftest import small_cfg

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from recon_b200 import PROJECTOR_BACK, SIDDON_BP_RAY, Options, Plan  # noqa: E402

FINE = dict(AxPixels=256, TAxPixels=192, AxPixDim=0.375, TAxPixDim=0.375)
GEOMS = {
    "mirror": small_cfg(**FINE),
    "odd": small_cfg(Xdim=31, Ydim=45, Zdim=27, XVoxSize=0.7, YVoxSize=0.9, ZVoxSize=1.1, AxPixels=255, TAxPixels=191,
                     AxPixDim=0.3, TAxPixDim=0.4),
    "offset": small_cfg(Dx=0.7, Dz=-0.4, Ry=803.0, M=1.2, **FINE),
}


@pytest.mark.parametrize("name", list(GEOMS))
def test_columns_equal_slabs(name):
    P = Plan(GEOMS[name], Options(siddon_bp=SIDDON_BP_RAY))
    y = torch.rand((P.nproj, P.nv, P.nu), device="cuda", generator=torch.Generator("cuda").manual_seed(411)) - 0.25
    out = P.bp_views(y)
    assert P.last_kernel(PROJECTOR_BACK) == "bp_column_kernel"
    total, size = torch.zeros_like(out, dtype=torch.float64), torch.zeros_like(out, dtype=torch.float64)
    for n in range(0, P.nproj, 4):
        part = P.bp_views(y[n:n + 4].contiguous(), n, 4)
        assert P.last_kernel(PROJECTOR_BACK) == "bp_ray_kernel"
        total += part.double()
        size += part.double().abs()
    assert ((out - total).abs() <= 2 * 2.0**-24 * size + 1e-9).all()
    assert torch.equal(out, P.bp_views(y))
    bad = y.clone()
    bad[3, 5, 7] = float("nan")
    assert torch.isnan(P.bp_views(bad)).all()


def test_stretches_of_large_volumes():
    """One, three and all views of a volume for which the columns serve every call."""
    P = Plan(small_cfg(Xdim=140, Ydim=131, Zdim=62, XVoxSize=0.2, YVoxSize=0.2, ZVoxSize=0.3, AxPixels=120, TAxPixels=70,
                       AxPixDim=0.6, TAxPixDim=0.6), Options(siddon_bp=SIDDON_BP_RAY))
    y = torch.rand((P.nproj, P.nv, P.nu), device="cuda", generator=torch.Generator("cuda").manual_seed(412)) - 0.25
    out = P.bp_views(y).double()
    for step in (1, 3):
        total, size = torch.zeros_like(out), torch.zeros_like(out)
        for n in range(0, P.nproj, step):
            part = P.bp_views(y[n:n + step].contiguous(), n, step).double()
            assert P.last_kernel(PROJECTOR_BACK) == "bp_column_kernel"
            total += part
            size += part.abs()
        assert ((out - total).abs() <= (P.nproj // step + 1) * 2.0**-24 * size + 1e-9).all()

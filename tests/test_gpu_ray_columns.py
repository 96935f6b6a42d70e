"""The ray design's back projection along detector columns (bp_column_kernel), where its
dispatch and its edges are: mirrored and single rows, partial warps and tiles, rows much
closer and much further apart than voxels, single views at any angle, view ranges, and an
accumulator larger than L2 (taken 32 rows of every view at a time).

Against the FP64 oracle: products rounded to 2^-49 of the largest and exact sums leave the
FP32 rounding of the lengths (planes to about 4e-6 mm of a piece of the order of a voxel,
independent over a voxel's rays), 1e-6 relative L2 with room."""
import numpy as np
import pytest

from conftest import rel_l2, small_cfg

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from oracle import oracle as O  # noqa: E402
from recon_b200 import (FP_RAY_WALK, PROJECTOR_BACK, SIDDON_BP_GATHER, SIDDON_BP_RAY, SINO_BF16, Options,  # noqa: E402
                        Plan)
from recon_b200.configs import geom_dict  # noqa: E402

GEOMS = {
    "mirror": small_cfg(TAxPixels=70),
    "odd": small_cfg(Xdim=31, Ydim=45, Zdim=27, XVoxSize=0.7, YVoxSize=0.9, ZVoxSize=1.1, AxPixels=61, TAxPixels=75),
    "offset": small_cfg(Dx=0.7, Dz=-0.4, Ry=803.0, M=1.2),
    "dense": small_cfg(AxPixDim=0.4, TAxPixDim=0.35, AxPixels=160, TAxPixels=130, NumProj=6),
    "sparse": small_cfg(AxPixDim=3.1, TAxPixDim=3.3, AxPixels=34, TAxPixels=23),
    "one_voxel": small_cfg(Xdim=1, Ydim=1, Zdim=1, TAxPixels=3, AxPixels=5),
}


@pytest.mark.parametrize("name", list(GEOMS))
def test_sums(name):
    cfg = GEOMS[name]
    P = Plan(cfg, Options(siddon_bp=SIDDON_BP_RAY))
    assert P.forward_projector != FP_RAY_WALK and P.siddon_bp == SIDDON_BP_RAY
    g = O.Geom.from_dict(geom_dict(cfg))
    gen = torch.Generator("cuda").manual_seed(401)
    y = torch.rand((P.nproj, P.nv, P.nu), device="cuda", generator=gen) - 0.25
    ref = O.x_bp_all(g, P.nproj, np.float32(cfg["DeltaAng"]), y.cpu().numpy().astype(np.float64).ravel())
    out = P.bp_views(y)
    assert rel_l2(out.cpu().numpy(), ref) < 1e-6
    assert torch.equal(out, P.bp_views(y))
    assert P.count_projector_pairs(PROJECTOR_BACK) == P.count_intersections()
    # view by view, at plan angles (a range) and through the scratch slot: each rounded once
    total = sum(P.bp_views(y[n:n + 1].contiguous(), n, 1).double() for n in range(P.nproj))
    assert rel_l2(total.cpu().numpy(), out.cpu().numpy()) < P.nproj * 2.0**-24
    Q = Plan({**cfg, "NumProj": 0}, Options(siddon_bp=SIDDON_BP_RAY))
    for n in (0, 2):
        assert torch.equal(Q.bp_view(y[n].contiguous(), P.angle(n)), P.bp_view(y[n].contiguous(), P.angle(n)))


@pytest.mark.parametrize("name", ["mirror", "odd"])
@pytest.mark.parametrize("kw", [{}, {"sino": SINO_BF16}, {"fp_block": 12}, {"fp_rows": 32}])
def test_mlem_halves(name, kw):
    """The ratio's maxima per view survive being written in ranges and read in others."""
    P = Plan(GEOMS[name], Options(siddon_bp=SIDDON_BP_RAY, **kw))
    gen = torch.Generator("cuda").manual_seed(402)
    g = torch.rand((P.nproj, P.nv, P.nu), device="cuda", generator=gen) * 3
    g = g.bfloat16() if "sino" in kw else g
    P.mlem_prepare()
    f = torch.rand(P.shape_vol, device="cuda", generator=gen) + 0.5
    whole, parts, some = P.new_volume(), P.new_volume(), P.new_volume()
    P.mlem_forward(g, f)
    P.mlem_backward(whole)
    P.mlem_forward(g, 2 * f, 3, 4)  # written again below
    for a, n in ((0, 5), (5, P.nproj - 5)):
        P.mlem_forward(g, f, a, n)
    P.mlem_backward(parts)
    assert torch.equal(whole, parts)
    P.mlem_backward(some, 1, 6)
    P.mlem_backward(parts, 0, 1)
    some += parts
    P.mlem_backward(parts, 7, P.nproj - 7)
    some += parts
    assert rel_l2(some.cpu().numpy(), whole.cpu().numpy()) < 3 * 2.0**-24


def test_accumulator_beyond_l2():
    cfg = small_cfg(Xdim=250, Ydim=246, Zdim=248, XVoxSize=0.2, YVoxSize=0.2, ZVoxSize=0.2, AxPixels=150, TAxPixels=141,
                    AxPixDim=0.6, TAxPixDim=0.6, NumProj=40)
    P = Plan(cfg, Options(siddon_bp=SIDDON_BP_RAY))
    y = torch.rand((P.nproj, P.nv, P.nu), device="cuda", generator=torch.Generator("cuda").manual_seed(403))
    out = P.bp_views(y)  # 40 views: by rows
    parts = P.bp_views(y[:20].contiguous(), 0, 20).double() + P.bp_views(y[20:].contiguous(), 20, 20).double()  # by views
    assert rel_l2(out.cpu().numpy(), parts.cpu().numpy()) < 2 * 2.0**-24
    G = Plan(cfg, Options(siddon_bp=SIDDON_BP_GATHER))
    assert rel_l2(out.cpu().numpy(), G.bp_views(y).cpu().numpy()) < 2e-6

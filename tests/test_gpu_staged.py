"""Gather back projectors that stage their values in shared memory, at the sizes
where they can go wrong: tiles and columns that do not fill, several candidate rows
per voxel, a voxel column wider than one detector column, both stage sizes, one and
two chunks of slices, and non-finite input.

Against the FP64 oracle: each length is exact to FP32 rounding of its planes (about
4e-6 mm of a piece of the order of a voxel) and a voxel sums a few hundred products in
FP32, so 5e-6 relative L2 bounds both with room; the projector's pair count is exact.
"""
import numpy as np
import pytest

from conftest import rel_l2, small_cfg

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from oracle import oracle as O  # noqa: E402
from recon_b200 import PROJECTOR_BACK, SIDDON_BP_GATHER, Options, Plan  # noqa: E402
from recon_b200.configs import geom_dict  # noqa: E402

QUARTER = {
    # 10 x 10: 5 x 5 base columns on 4 x 4 tiles
    "partial_tiles": small_cfg(Xdim=10, Ydim=10, Zdim=40, TAxPixels=66, NumProj=8, DeltaAng=45.0),
    # 2 x 2: one base column, most of a tile's warps idle; two slices: one pair
    "one_column": small_cfg(Xdim=2, Ydim=2, Zdim=2, TAxPixels=6, AxPixels=10, NumProj=4, DeltaAng=90.0),
    # rows half a voxel apart and columns a third: two to three candidate rows, up to
    # five detector columns per voxel column
    "dense": small_cfg(Xdim=12, Ydim=12, Zdim=20, TAxPixels=96, AxPixels=120, TAxPixDim=0.8, AxPixDim=0.5, NumProj=8,
                       DeltaAng=45.0),
    # rows two voxels apart: voxels without a row
    "sparse": small_cfg(Xdim=16, Ydim=16, Zdim=34, TAxPixels=24, TAxPixDim=3.2, NumProj=12, DeltaAng=30.0),
    # 130 pairs: two chunks of 96 and 34 slices; a tall detector (the larger stage)
    "two_chunks": small_cfg(Xdim=12, Ydim=12, Zdim=260, ZVoxSize=0.25, TAxPixels=190, TAxPixDim=0.6, NumProj=8,
                            DeltaAng=45.0),
}


@pytest.mark.parametrize("name", list(QUARTER))
def test_quarter_sums(name):
    cfg = QUARTER[name]
    P = Plan(cfg, Options(siddon_bp=SIDDON_BP_GATHER))
    assert P.quarter_turns and P.mirror_pairs
    y = torch.rand((P.nproj, P.nv, P.nu), device="cuda", generator=torch.Generator("cuda").manual_seed(201))
    out = P.bp_views(y)
    ref = O.x_bp_all(O.Geom.from_dict(geom_dict(cfg)), P.nproj, np.float32(cfg["DeltaAng"]),
                     y.cpu().numpy().astype(np.float64).ravel())
    assert np.abs(ref).sum() > 0
    assert rel_l2(out.cpu().numpy(), ref) < 5e-6
    assert P.count_projector_pairs(PROJECTOR_BACK) == P.count_intersections()
    assert torch.equal(out, P.bp_views(y))


@pytest.mark.parametrize("name", ["partial_tiles", "dense", "two_chunks"])
@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
def test_quarter_not_finite(name, bad):
    """A value that is not finite reaches the voxels that its ray crosses and no others;
    every other voxel keeps its sum."""
    cfg = QUARTER[name]
    P = Plan(cfg, Options(siddon_bp=SIDDON_BP_GATHER))
    y = torch.rand((P.nproj, P.nv, P.nu), device="cuda", generator=torch.Generator("cuda").manual_seed(202))
    clean = P.bp_views(y)
    pixel = (3, P.nv // 2 - 2, P.nu // 2)
    one = torch.zeros_like(y)
    one[pixel] = 1.0
    crossed = P.bp_views(one) > 0
    assert crossed.any() and not crossed.all()
    y[pixel] = bad
    out = P.bp_views(y)
    assert torch.equal(~torch.isfinite(out), crossed)
    assert torch.equal(out[~crossed], clean[~crossed])

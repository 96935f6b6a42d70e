"""The column forward projector's two kernels (few warps: several pieces' loads in flight;
many warps: full occupancy) give the same bits: a call of few views takes one, of many the
other, on a volume large enough for both; and paths whose length is no multiple of a block."""
import pytest

from conftest import small_cfg

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from recon_b200 import FP_COLUMNS, SUM_PLAIN, Options, Plan  # noqa: E402

# 128 rows make a block and 300 columns x 300 views x 4 warps are 360 000 warps (16 rounds
# of 32 an SM are 75 776); five views stay below
BIG = small_cfg(Xdim=61, Ydim=57, Zdim=50, XVoxSize=0.5, YVoxSize=0.5, ZVoxSize=0.5, AxPixels=400, TAxPixels=300,
                AxPixDim=0.15, TAxPixDim=0.15, NumProj=300)


@pytest.mark.parametrize("over", [{}, {"Dz": 0.3}])
def test_few_views_equal_many(over):
    P = Plan({**BIG, **over})
    assert P.forward_projector == FP_COLUMNS and P.mirror_pairs == (not over)
    vol = torch.rand(P.shape_vol, device="cuda", generator=torch.Generator("cuda").manual_seed(501))
    many = P.fp_views(vol)
    assert many.abs().sum() > 0
    for first in (0, 37, 295):
        assert torch.equal(P.fp_views(vol, first, 5).view(torch.int32), many[first:first + 5].view(torch.int32))
    # plain sums always take the same kernel: the lengths and voxels are the same
    plain = Plan({**BIG, **over}, Options(sum=SUM_PLAIN)).fp_views(vol, 37, 5)
    assert ((plain - many[37:42]).norm() / plain.norm()).item() < 1e-6

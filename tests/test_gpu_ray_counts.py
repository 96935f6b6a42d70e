"""The ray design's pair count comes from its own kernel (bp_column_kernel), in the launches
that its back projections take: tiles of rows, paths in stretches (few views), and 32 rows of
every view at a time (an accumulator larger than L2)."""
import pytest

from conftest import small_cfg

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from recon_b200 import PROJECTOR_BACK, PROJECTOR_FORWARD, SIDDON_BP_RAY, Options, Plan  # noqa: E402
from test_gpu_ray_columns import GEOMS  # noqa: E402


def _counted_by(P, kernel):
    other = Plan(small_cfg(ZVoxSize=0.05, NumProj=1), Options(siddon_bp=SIDDON_BP_RAY))
    other.bp_views(other.new_sinogram())
    assert P.last_kernel(PROJECTOR_BACK) == "bp_ray_kernel" != kernel
    pairs = P.count_projector_pairs(PROJECTOR_BACK)
    assert P.last_kernel(PROJECTOR_BACK) == kernel
    return pairs


@pytest.mark.parametrize("name", list(GEOMS))
@pytest.mark.parametrize("views", [0, 1, 2, 12])
def test_counts(name, views):
    P = Plan({**GEOMS[name], "NumProj": views}, Options(siddon_bp=SIDDON_BP_RAY))
    if views == 0:
        assert P.count_projector_pairs(PROJECTOR_BACK) == 0
        return
    pairs = _counted_by(P, "bp_column_kernel")
    assert pairs > 0 or name == "one_voxel"
    assert pairs == P.count_intersections() == P.count_projector_pairs(PROJECTOR_FORWARD)


@pytest.mark.parametrize("dz", [0.0, 0.3])
def test_count_beyond_l2(dz):
    P = Plan(small_cfg(Xdim=250, Ydim=246, Zdim=248, XVoxSize=0.2, YVoxSize=0.2, ZVoxSize=0.2, AxPixels=150,
                       TAxPixels=141, AxPixDim=0.6, TAxPixDim=0.6, NumProj=40, Dz=dz), Options(siddon_bp=SIDDON_BP_RAY))
    assert _counted_by(P, "bp_column_kernel") == P.count_intersections()

"""The gather back projector's kernel for a few views: volumes that do not fill its eight
columns by four rows, one to four voxel pairs per lane and a second chunk of slices, several
candidate rows and detector columns, and values that are not finite; against FP64 and the
kernel for many views.  A voxel sums a few products of lengths whose planes are good to about
4e-6 mm in pieces of the order of a voxel, some of them short: 1e-5 relative L2, as every
back projection is held to; the two kernels sum the same products, 1e-6."""
import numpy as np
import pytest

from conftest import rel_l2, small_cfg

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from oracle import oracle as O  # noqa: E402
from recon_b200 import SIDDON_BP_GATHER, Options, Plan  # noqa: E402
from recon_b200.configs import geom_dict  # noqa: E402

GEOMS = {
    "one_pair": small_cfg(Xdim=9, Ydim=5, Zdim=10),
    "two_pairs": small_cfg(Xdim=30, Ydim=33, Zdim=100, TAxPixels=110),
    "two_chunks": small_cfg(Xdim=17, Ydim=18, Zdim=262, ZVoxSize=0.25, TAxPixels=190, TAxPixDim=0.6),
    "dense": small_cfg(TAxPixDim=0.7, AxPixDim=0.9, TAxPixels=90, AxPixels=100),
    "many_columns": small_cfg(Xdim=131, Ydim=130, XVoxSize=0.25, YVoxSize=0.25),
}


@pytest.mark.parametrize("name", list(GEOMS))
def test_few_views(name):
    cfg = GEOMS[name]
    P = Plan(cfg, Options(siddon_bp=SIDDON_BP_GATHER))
    assert P.mirror_pairs
    g = O.Geom.from_dict(geom_dict(cfg))
    n = P.nproj
    y = torch.rand((n, P.nv, P.nu), device="cuda", generator=torch.Generator("cuda").manual_seed(601)) - 0.2
    zero = torch.zeros_like(y)
    many = P.bp_views(y).double()
    total = torch.zeros_like(many)
    first = 0
    for count in (1, 2, 4, n - 7):
        part = P.bp_views(y[first:first + count].contiguous(), first, count)
        only = zero.clone()
        only[first:first + count] = y[first:first + count]
        ref = O.x_bp_all(g, n, np.float32(cfg["DeltaAng"]), only.cpu().numpy().astype(np.float64).ravel())
        assert rel_l2(part.cpu().numpy(), ref) < 1e-5, count
        total += part.double()
        first += count
    assert rel_l2(total.cpu().numpy(), many.cpu().numpy()) < 1e-6
    assert torch.equal(P.bp_view(y[3].contiguous(), P.angle(3)), P.bp_views(y[3:4].contiguous(), 3, 1))
    # away from the plan's angles: the scratch slot
    Q = Plan({**cfg, "NumProj": 1, "DeltaAng": 0.0}, Options(siddon_bp=SIDDON_BP_GATHER))
    assert torch.equal(Q.bp_view(y[0].contiguous(), 41.5), P.bp_view(y[0].contiguous(), 41.5))
    # a value that is not finite reaches the voxels that its ray crosses
    one = torch.zeros_like(y[:1])
    one[0, P.nv // 2 - 2, P.nu // 2] = 1.0
    crossed = P.bp_views(one, 2, 1) > 0
    assert crossed.any()
    clean = P.bp_views(y[2:3].contiguous(), 2, 1)
    bad = y[2:3].clone()
    bad[0, P.nv // 2 - 2, P.nu // 2] = float("inf")
    out = P.bp_views(bad, 2, 1)
    assert torch.equal(~torch.isfinite(out), crossed)
    assert torch.equal(out[~crossed], clean[~crossed])

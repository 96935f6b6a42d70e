"""Which kernel serves a call: the geometries of the kernels' own tests take the kernels that
they are there for, and the calls outside a kernel's bounds the one that it falls back to."""
import pytest

from conftest import small_cfg

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from recon_b200 import (ARITH_COMPAT, BP_VOXEL, PROJECTOR_BACK, PROJECTOR_FORWARD, SIDDON_BP_GATHER,  # noqa: E402
                        SIDDON_BP_RAY, SUM_PLAIN, Options, Plan)
from test_gpu_fp_wide import BIG  # noqa: E402
from test_gpu_ray_columns import GEOMS as RAY  # noqa: E402
from test_gpu_staged import QUARTER  # noqa: E402
from test_gpu_voxel_staged import GEOMS as VOXEL  # noqa: E402


def back(P, count=None, first=0):
    count = P.nproj - first if count is None else count
    P.bp_views(torch.ones((count, P.nv, P.nu), device="cuda"), first, count)
    return P.last_kernel(PROJECTOR_BACK)


def forward(P, count=None):
    P.fp_views(torch.ones(P.shape_vol, device="cuda"), 0, P.nproj if count is None else count)
    return P.last_kernel(PROJECTOR_FORWARD)


def iteration(P):
    P.mlem_prepare()
    P.mlem_iteration(P.new_sinogram(), P.new_volume(1.0))
    return P.last_kernel(PROJECTOR_FORWARD), P.last_kernel(PROJECTOR_BACK)


@pytest.mark.parametrize("name", list(QUARTER))
def test_quarter_turns(name):
    P = Plan(QUARTER[name], Options(siddon_bp=SIDDON_BP_GATHER))
    assert back(P) == "bp_staged_quarter_kernel"
    assert iteration(P)[1] == "bp_staged_quarter_kernel"
    assert back(P, 3) != "bp_staged_quarter_kernel"
    P.sensitivity()  # (few tiles of a tall volume: the smaller ones of the other kernel)
    tall = QUARTER[name]["Zdim"] > 128
    assert P.last_kernel(PROJECTOR_BACK) == ("bp_gather_quarter_kernel" if tall else "bp_staged_quarter_kernel")
    P.mlem_forward_quarters(P.new_sinogram(), P.new_volume(1.0), 0, 1)
    P.mlem_backward_quarters(P.new_volume(), 0, 1)
    assert P.last_kernel(PROJECTOR_BACK) == "bp_staged_quarter_kernel"


def test_quarter_turns_without_stages():
    """More rows than a box holds; a box of more than 12 KiB."""
    base = dict(Xdim=16, Ydim=16, Zdim=32, NumProj=4, DeltaAng=90.0)
    for over in (dict(TAxPixels=2400, TAxPixDim=0.05), dict(AxPixels=300, TAxPixels=300, AxPixDim=0.2, TAxPixDim=0.2)):
        P = Plan(small_cfg(**{**base, **over}), Options(siddon_bp=SIDDON_BP_GATHER))
        assert P.quarter_turns and P.mirror_pairs
        assert back(P) == "bp_gather_quarter_kernel"


FEW_ROWS = dict(TAxPixels=24, TAxPixDim=3.0)  # rows further apart than voxels: one candidate
FEW_LINES = {  # columns (x, y): views that take the few-view kernel, with one candidate row, with several
    (95, 95): ([], []),
    (96, 96): ([1, 2], []),
    (112, 112): ([1, 2], [1]),
    (128, 128): ([1, 2, 3, 4], [1, 2]),
    (160, 160): ([1, 2, 3, 4], [1]),
    (200, 200): ([1, 2, 3, 4], [1, 2]),
}


@pytest.mark.parametrize("x, y", list(FEW_LINES))
@pytest.mark.parametrize("several", [False, True])
def test_few_views(x, y, several):
    cfg = small_cfg(Xdim=x, Ydim=y, Zdim=24, XVoxSize=0.25, YVoxSize=0.25, **({} if several else FEW_ROWS))
    if several:
        cfg.update(Zdim=130, ZVoxSize=0.25, TAxPixels=150, TAxPixDim=0.3)
    P = Plan(cfg, Options(siddon_bp=SIDDON_BP_GATHER))
    few = FEW_LINES[(x, y)][several]
    for n in range(1, 6):
        assert back(P, n) == ("bp_gather_few_kernel" if n in few else "bp_gather_pairs_kernel"), n
    P.bp_view(torch.ones((P.nv, P.nu), device="cuda"), 41.5)
    assert P.last_kernel(PROJECTOR_BACK) == ("bp_gather_few_kernel" if 1 in few else "bp_gather_pairs_kernel")


def test_large_detectors():
    """Up to 4096 rows and 8192 columns the few-view gather's bounds hold; it drops no ray there."""
    for rows, columns in ((4096, 64), (4098, 64), (48, 8192), (48, 8193)):
        cfg = small_cfg(Xdim=112, Ydim=112, XVoxSize=0.3, YVoxSize=0.3, TAxPixels=rows, TAxPixDim=72.0 / rows,
                        AxPixels=columns, AxPixDim=96.0 / min(columns, 96))
        P = Plan(cfg, Options(siddon_bp=SIDDON_BP_GATHER))
        y = torch.rand((1, P.nv, P.nu), device="cuda", generator=torch.Generator("cuda").manual_seed(341))
        out = P.bp_views(y, 3, 1)
        small = rows <= 4096 and columns <= 8192
        assert P.last_kernel(PROJECTOR_BACK) == ("bp_gather_few_kernel" if small else "bp_gather_pairs_kernel")
        exact = Plan(cfg, Options(siddon_bp=SIDDON_BP_RAY)).bp_views(y, 3, 1)
        # FP32 sums of at most a few hundred products a voxel against exact ones
        assert ((out - exact).norm() / exact.norm()).item() < 2e-6
        assert torch.equal(out != 0, exact != 0)


def test_other_gathers():
    # columns a fifth of a voxel: more than four of them meet a voxel column
    fine = Plan(small_cfg(AxPixels=300, AxPixDim=0.25), Options(siddon_bp=SIDDON_BP_GATHER))
    assert back(fine, 1) == "bp_gather_pairs_kernel"
    assert back(Plan(small_cfg(Dz=0.4), Options(siddon_bp=SIDDON_BP_GATHER)), 1) == "bp_gather_kernel"
    # (pairs of rows come from the column forward projector)
    assert back(Plan(small_cfg(ZVoxSize=0.05), Options(siddon_bp=SIDDON_BP_GATHER)), 1) == "bp_gather_mirror_kernel"


@pytest.mark.parametrize("name", list(RAY))
def test_ray_design(name):
    """Sinograms of few rays and small volumes go ray by ray, the rest along detector columns."""
    P = Plan(RAY[name], Options(siddon_bp=SIDDON_BP_RAY))
    assert back(P) == back(P, 1) == "bp_ray_kernel"
    assert iteration(P)[1] == "bp_column_kernel"
    P.sensitivity()
    assert P.last_kernel(PROJECTOR_BACK) == "bp_column_kernel"


def test_ray_design_sizes():
    many = dict(AxPixels=256, TAxPixels=192, AxPixDim=0.375, TAxPixDim=0.375)
    P = Plan(small_cfg(**many), Options(siddon_bp=SIDDON_BP_RAY))  # 49152 rays a view
    assert [back(P, n) for n in (1, 4, 5)] == ["bp_ray_kernel", "bp_ray_kernel", "bp_column_kernel"]
    P = Plan(small_cfg(AxPixels=160, TAxPixels=100, AxPixDim=0.6, TAxPixDim=0.7), Options(siddon_bp=SIDDON_BP_RAY))
    assert [back(P, n) for n in (10, 11)] == ["bp_ray_kernel", "bp_column_kernel"]  # 16000 rays a view
    for z, kernel in ((64, "bp_ray_kernel"), (65, "bp_column_kernel")):  # 2^20 voxels, and more
        P = Plan(small_cfg(Xdim=128, Ydim=128, Zdim=z, XVoxSize=0.25, YVoxSize=0.25, ZVoxSize=0.25),
                 Options(siddon_bp=SIDDON_BP_RAY))
        assert back(P, 1) == kernel


def test_ray_walk():
    P = Plan(small_cfg(ZVoxSize=0.05), Options(siddon_bp=SIDDON_BP_RAY))
    assert back(P) == "bp_ray_kernel" and forward(P) == "fp_kernel"
    assert iteration(P) == ("fp_kernel", "bp_ray_kernel")


@pytest.mark.parametrize("over", [{}, {"Dz": 0.3}])
def test_forward(over):
    P = Plan({**BIG, **over})
    assert forward(P, 5) == "fp_column_wide_kernel" and forward(P) == "fp_column_kernel"
    assert forward(Plan({**BIG, **over}, Options(sum=SUM_PLAIN)), 5) == "fp_column_kernel"
    assert forward(Plan({**BIG, **over}, Options(fp_block=32)), 5) == "fp_column_block_kernel"


@pytest.mark.parametrize("name", list(VOXEL))
def test_voxel_update(name):
    P = Plan(VOXEL[name], Options(bp=BP_VOXEL))
    staged = name not in ("shorter_image", "dense_rows")
    assert iteration(P)[1] == ("voxel::bp_staged_kernel" if staged else "voxel::bp_gather_kernel")


def test_compat():
    P = Plan(small_cfg(), Options(arith=ARITH_COMPAT))
    assert forward(P) == forward(P, 1) == "compat::fp_kernel"
    assert back(P) == back(P, 1) == "compat::bp_scatter_kernel"
    assert iteration(P) == ("compat::fp_kernel", "compat::bp_scatter_kernel")

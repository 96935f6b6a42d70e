"""COMPAT back projections of several views whose magnitudes differ, and of views that hold
values that are not finite: every view adds what it adds on its own.  Views of like
magnitude share one fixed-point scale; the others must lose nothing by the company."""
import numpy as np
import pytest

from conftest import small_cfg

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from recon_b200 import ARITH_COMPAT, Options, Plan  # noqa: E402

GEOMS = {
    "even": small_cfg(),
    "odd": small_cfg(Xdim=31, Ydim=45, Zdim=27, XVoxSize=0.7, YVoxSize=0.9, ZVoxSize=1.1, AxPixels=61, TAxPixels=75),
    "tilted": small_cfg(xangle=0.02, yangle=-0.01, zangle=0.03),
    "tilted_groups": small_cfg(xangle=0.02, yangle=-0.01, zangle=0.03, NumProj=48),
    "few_pixels": small_cfg(AxPixels=5, TAxPixels=3, AxPixDim=9.0, TAxPixDim=9.0),
    "one_slice": small_cfg(Zdim=1, TAxPixels=3, AxPixels=9, NumProj=7, DeltaAng=51.0),
}


def _plan(name):
    return Plan(GEOMS[name], Options(arith=ARITH_COMPAT))


def _sino(P, seed):
    return torch.rand((P.nproj, P.nv, P.nu), device="cuda", generator=torch.Generator("cuda").manual_seed(seed)) + 0.1


def _quantum(P, cfg, view):
    """A bound on one unit of a view's own fixed-point accumulator: 2^-F, F = 62 - count bits
    - e, with max |value| times the longest ray below 2^e."""
    hu = 0.5 * P.nu * cfg["AxPixDim"] * abs(cfg["M"]) + abs(cfg["Dx"])
    hv = 0.5 * P.nv * cfg["TAxPixDim"] * abs(cfg["M"]) + abs(cfg["Dz"])
    sc = abs(cfg["R"]) / max(1e-6, abs(cfg["Ry"]) - hu - hv)
    longest = 2.0 * (abs(cfg["R"]) + abs(cfg["Rf"]) + sc * (hu + hv)) + 1.0
    bits = int(np.ceil(np.log2(P.nu * P.nv))) + 1
    return 2.0 * float(view.abs().max()) * longest * 2.0 ** (bits - 62)


def _within(P, cfg, got, y, views):
    """got is the sum of the single views: len(views) roundings of partial sums no larger than
    the sum of the magnitudes, each view's own, and the units of each view's own accumulator
    (64 contributions a voxel, either side) in the voxels that it reaches or that touch them."""
    ones = torch.ones_like(y[0])
    total = torch.zeros_like(got, dtype=torch.float64)
    bound = torch.zeros_like(total)
    parts = []
    for n in views:
        p = P.bp_view(y[n], P.angle(n)).double()
        reach = (P.bp_view(ones, P.angle(n)) != 0).float()
        near = torch.nn.functional.max_pool3d(reach[None, None], 3, 1, 1)[0, 0].double()
        total += p
        bound += (len(views) + 1) * 2.0**-24 * p.abs() + 64 * _quantum(P, cfg, y[n]) * near
        parts.append(p)
    assert bool(((got.double() - total).abs() <= bound).all())
    return parts


@pytest.mark.parametrize("name", list(GEOMS))
@pytest.mark.parametrize("scale", [2.0**-4, 1e-3, 1e-9, 1e-16, 1e-30])
def test_dim_views(name, scale):
    P, cfg = _plan(name), GEOMS[name]
    y = _sino(P, 311)
    y[1::2] *= scale
    y[2] *= scale**0.5
    parts = _within(P, cfg, P.bp_views(y), y, range(P.nproj))
    got = P.bp_views(y[:4], 0, 4)
    _within(P, cfg, got, y, range(4))
    # voxels that only the dim views reach
    only = (parts[0] == 0) & (parts[2] == 0) & ((parts[1] != 0) | (parts[3] != 0))
    if bool(only.any()):
        assert bool((got[only] != 0).all())


@pytest.mark.parametrize("name", list(GEOMS))
def test_every_view_a_magnitude_of_its_own(name):
    P, cfg = _plan(name), GEOMS[name]
    y = _sino(P, 312)
    for n in range(P.nproj):
        y[n] *= 10.0 ** (-3.0 * ((5 * n) % P.nproj))
    _within(P, cfg, P.bp_views(y), y, range(P.nproj))


@pytest.mark.parametrize("name", list(GEOMS))
@pytest.mark.parametrize("bad", [float("nan"), float("inf"), float("-inf")])
def test_views_that_are_not_finite_add_nothing(name, bad):
    P = _plan(name)
    y = _sino(P, 313)
    y[3] *= 1e-6
    good = y.clone()
    good[1] = 0.0
    good[4] = 0.0
    y[1, P.nv // 2, P.nu // 2] = bad
    y[4, 0, 0] = bad
    want = P.bp_views(good)
    assert bool((want != 0).any())
    assert torch.equal(P.bp_views(y).view(torch.int32), want.view(torch.int32))
    assert not bool(P.bp_view(y[1], P.angle(1)).any())
    every = y.clone()
    every[:, 0, 0] = bad
    assert not bool(P.bp_views(every).any())
    assert not bool(P.bp_views(torch.zeros_like(y)).any())


def test_like_views_keep_their_bits_in_a_replayed_graph():
    P = _plan("odd")
    y = _sino(P, 314)
    y[5] *= 1e-12
    want = P.bp_views(y)
    out = torch.empty_like(want)
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        P.bp_views(y, out=out)
    for _ in range(3):
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out.view(torch.int32), want.view(torch.int32))
    assert np.isfinite(out.cpu().numpy()).all()

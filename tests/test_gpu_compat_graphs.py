"""COMPAT forward projections and MLEM iterations recorded in graphs: replays on several
streams, beside each other and beside calls outside graphs, project each its own volume."""
import pytest

from conftest import small_cfg

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)

from recon_b200 import ARITH_COMPAT, Options, Plan  # noqa: E402

GEOMS = {
    "pow2": small_cfg(Xdim=96, Ydim=96, Zdim=64, XVoxSize=0.5, YVoxSize=0.5, ZVoxSize=0.5, AxPixels=128, TAxPixels=96),
    "odd": small_cfg(Xdim=71, Ydim=85, Zdim=47, XVoxSize=0.7, YVoxSize=0.9, ZVoxSize=1.1, AxPixels=101, TAxPixels=75),
}


def _record(call):
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=torch.cuda.Stream()):
        call()
    return graph


def _equal(a, b):
    return torch.equal(a.view(torch.int32), b.view(torch.int32))


@pytest.mark.parametrize("name", list(GEOMS))
@pytest.mark.parametrize("views", [5, 6, 12])
def test_replays_on_two_streams(name, views):
    P = Plan(GEOMS[name], Options(arith=ARITH_COMPAT))
    gen = torch.Generator("cuda").manual_seed(321)
    vols = [torch.rand(P.shape_vol, device="cuda", generator=gen) for _ in range(3)]
    want = [P.fp_views(v, 0, views) for v in vols]
    outs = [torch.zeros_like(w) for w in want]
    torch.cuda.synchronize()
    graphs = [_record(lambda k=k: P.fp_views(vols[k], 0, views, out=outs[k])) for k in range(2)]
    streams = [torch.cuda.Stream() for _ in range(3)]
    for _ in range(8):
        for o in outs:
            o.zero_()
        torch.cuda.synchronize()
        for _ in range(4):
            for k in range(2):
                with torch.cuda.stream(streams[k]):
                    graphs[k].replay()
            with torch.cuda.stream(streams[2]):
                P.fp_views(vols[2], 0, views, out=outs[2])
        torch.cuda.synchronize()
        for o, w in zip(outs, want):
            assert _equal(o, w)


def test_forked_branches_of_one_graph():
    P = Plan(GEOMS["odd"], Options(arith=ARITH_COMPAT))
    gen = torch.Generator("cuda").manual_seed(322)
    vols = [torch.rand(P.shape_vol, device="cuda", generator=gen) for _ in range(2)]
    want = [P.fp_views(v) for v in vols]
    outs = [torch.zeros_like(w) for w in want]
    torch.cuda.synchronize()
    side = torch.cuda.Stream()

    def branches():
        here = torch.cuda.current_stream()
        side.wait_stream(here)
        with torch.cuda.stream(side):
            P.fp_views(vols[1], out=outs[1])
        P.fp_views(vols[0], out=outs[0])
        here.wait_stream(side)

    graph = _record(branches)
    for _ in range(16):
        graph.replay()
        torch.cuda.synchronize()
        assert _equal(outs[0], want[0]) and _equal(outs[1], want[1])


@pytest.mark.parametrize("name", list(GEOMS))
def test_iteration_beside_projections(name):
    """An iteration, recorded or not, shares nothing with forward projections on other streams."""
    P = Plan(GEOMS[name], Options(arith=ARITH_COMPAT))
    gen = torch.Generator("cuda").manual_seed(323)
    vol = torch.rand(P.shape_vol, device="cuda", generator=gen)
    g = P.fp_views(vol)
    P.mlem_prepare()
    start = torch.rand(P.shape_vol, device="cuda", generator=gen) + 0.5
    expect = start.clone()
    for _ in range(4):
        P.mlem_iteration(g, expect)
    f, out = start.clone(), torch.empty_like(g)
    torch.cuda.synchronize()
    graph = _record(lambda: P.mlem_iteration(g, f))
    torch.cuda.synchronize()
    one, two = torch.cuda.Stream(), torch.cuda.Stream()
    for recorded in (True, False):
        f.copy_(start)
        torch.cuda.synchronize()
        for _ in range(4):
            with torch.cuda.stream(one):
                graph.replay() if recorded else P.mlem_iteration(g, f)
            with torch.cuda.stream(two):
                P.fp_views(vol, out=out)
        torch.cuda.synchronize()
        assert _equal(f, expect)
        assert _equal(out, g)

"""Action batches under stream capture: a context's first call can be captured, and a captured launch
keeps its own workspace -- calls of any size that follow, on the context's stream or another one,
neither move nor share it."""
import pytest

torch = pytest.importorskip("torch")

import fjmodels_gb300 as F  # noqa: E402
from tests.test_gpu_streams import _inputs, _out  # noqa: E402

pytestmark = pytest.mark.gpu


def test_first_call_captured_then_larger_calls():
    want, other = _out(300), F.Context(0)
    pot, delta, pts = _inputs(other, 300, 1)
    other.uvOrb_actions(pot, delta, pts, want)
    torch.cuda.synchronize()
    other.close()
    ctx = F.Context(0)  # nothing called on it yet
    got, graph = _out(300), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        ctx.uvOrb_actions(pot, delta, pts, got)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(got, want)
    # calls that need ever more workspace, then the graph again, side by side with one of them
    x, w = F.tanh_sinh_rule(8)
    big = _inputs(ctx, 30_000, 2)[2]
    m6 = torch.zeros((6, 300), dtype=torch.float64, device="cuda")
    ctx.uvOrb_actions(pot, delta, big, _out(30_000))
    ctx.moments_points(pot, delta, F.DFParams("Hernquist"), F.Rule(x, w), pts[:, :2].contiguous(), m6)
    big_want, big_got = _out(30_000), _out(30_000)
    ctx.uvOrb_actions(pot, delta, big, big_want)
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    for _ in range(5):
        got.zero_()
        big_got.zero_()
        torch.cuda.synchronize()
        ctx.uvOrb_actions(pot, delta, big, big_got)
        with torch.cuda.stream(side):
            graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(got, want) and torch.equal(big_got, big_want)
    # two captured launches of one context share nothing either
    got2, graph2 = _out(300), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph2):
        ctx.uvOrb_actions(pot, delta, pts, got2)
    got.zero_()
    torch.cuda.synchronize()
    graph2.replay()
    with torch.cuda.stream(side):
        graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(got, want) and torch.equal(got2, want)
    # a workspace whose graph is gone serves the next capture
    del graph2
    for _ in range(3):
        g3 = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g3):
            ctx.uvOrb_actions(pot, delta, pts, got2)
        got2.zero_()
        g3.replay()
        torch.cuda.synchronize()
        assert torch.equal(got2, want)
        del g3
    del graph
    torch.cuda.synchronize()
    ctx.close()

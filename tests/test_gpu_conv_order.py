"""The convolution's passes follow each other without gaps: chains of calls that
read what the call before wrote, on one stream and in a graph, give what the same
calls with a wait after each give, bit for bit."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


# short and long transforms, and one of each
@pytest.mark.parametrize("W,H,k", [(100, 90, 7), (1100, 900, 33), (300, 1200, 9)])
def test_chains(W, H, k):
    import ghostlight_gb300 as gl
    r = np.random.default_rng(W)
    kern = r.random((k, k)).astype(np.float32)
    kern /= kern.sum()
    start = [torch.from_numpy(r.random((H, W)).astype(np.float32)).cuda() for _ in range(3)]
    plans = [gl.ConvPlan(W, H, kern), gl.ConvPlan(W, H, kern[::-1].copy())]
    a, b = [torch.empty_like(i) for i in start], [torch.empty_like(i) for i in start]

    def chain(wait):
        for x, s in zip(a, start):
            x.copy_(s)
        for q in range(6):
            plans[q & 1].execute(a, b)
            if wait:
                torch.cuda.synchronize()
            plans[1 - (q & 1)].execute(b, a)
            if wait:
                torch.cuda.synchronize()
            plans[0].execute(a, a)               # in place
            if wait:
                torch.cuda.synchronize()
        return torch.stack(a)

    want = chain(True).clone()
    for _ in range(20):
        assert torch.equal(chain(False), want)
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        chain(False)
    for _ in range(5):
        for x in a:
            x.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(torch.stack(a), want)
    for p in plans:
        p.close()

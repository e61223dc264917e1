"""Maps that follow one another on a stream read what the one before wrote.

The map kernels start while the previous kernel of the stream still runs and
wait for it before they read a vector.  A chain w = A^T (A (... u)), queued
without a synchronisation between its maps, must give the bits of the same
chain with one after every map: on the default stream, on a side stream and
replayed from a graph."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FORMS = [(5, "DQG", 1), (10, "DQG", 1), (10, "DQG", 7), (10, "DQG", 32), (14, "DQG", 1), (14, "DQG", 6),
         (7, "DQGT2", 1), (7, "DQGT2", 3), (6, "DQGT1", 20)]


@pytest.mark.parametrize("n,positivity,nvec", FORMS)
def test_chain_of_maps(v2g, n, positivity, nvec):
    import torch

    s = v2g.V2RDMSolver([n], n // 2, n // 2, options=dict(POSITIVITY=positivity))
    g = torch.Generator(device="cuda").manual_seed(n + nvec)
    u0 = torch.randn(s.dimx * nvec, dtype=torch.float64, device="cuda", generator=g)
    u, v = u0.clone(), torch.empty(s.nconstraints * nvec, dtype=torch.float64, device="cuda")
    length = 12

    def chain(stream, wait):
        for _ in range(length):
            s.map_batched_device(nvec, u.data_ptr(), v.data_ptr(), stream.cuda_stream)
            if wait:
                stream.synchronize()
            s.map_batched_device(nvec, v.data_ptr(), u.data_ptr(), stream.cuda_stream, transpose=True)
            if wait:
                stream.synchronize()

    def result(stream, wait):
        with torch.cuda.stream(stream):
            u.copy_(u0)
            chain(stream, wait)
        stream.synchronize()
        return u.cpu().numpy(), v.cpu().numpy()

    side = torch.cuda.Stream()
    want = result(side, True)
    assert np.isfinite(want[0]).all() and np.abs(want[0]).max() > 0
    for _ in range(5):
        for stream in (side, torch.cuda.default_stream()):
            assert all(np.array_equal(a, b) for a, b in zip(want, result(stream, False)))
    graph = torch.cuda.CUDAGraph()
    u.copy_(u0)
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=side):
        chain(side, False)
    for _ in range(5):
        u.copy_(u0)
        graph.replay()
        torch.cuda.synchronize()
        assert all(np.array_equal(a, b) for a, b in zip(want, (u.cpu().numpy(), v.cpu().numpy())))

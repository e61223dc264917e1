"""The batched device maps take vectors on any 8-byte boundary.

With an even number of instances a lane's two are adjacent and read by one
16-byte load, which needs a 16-byte boundary; other vectors take two 8-byte
loads.  The sums run in the same order, so the bits are the same."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,positivity,nvec", [(4, "DQG", 2), (6, "DQGT2", 6), (10, "DQG", 32), (14, "DQG", 6),
                                               (10, "DQG", 34), (5, "DQG", 256), (5, "DQG", 3), (10, "DQG", 1)])
@pytest.mark.parametrize("shift_in,shift_out", [(1, 0), (0, 1), (1, 1)])
def test_vectors_on_8_byte_boundaries(v2g, n, positivity, nvec, shift_in, shift_out):
    import torch

    s = v2g.V2RDMSolver([n], n // 2, n // 2, options=dict(POSITIVITY=positivity))
    rng = np.random.default_rng(n + nvec)
    for nin, nout, transpose in ((s.dimx, s.nconstraints, False), (s.nconstraints, s.dimx, True)):
        u = rng.standard_normal(nin * nvec)
        got = []
        for i, o in ((0, 0), (shift_in, shift_out)):
            d_in = torch.empty(u.size + 1, dtype=torch.float64, device="cuda")[i:i + u.size]
            d_in.copy_(torch.from_numpy(u))
            d_out = torch.full((nout * nvec + 1,), float("nan"), dtype=torch.float64, device="cuda")[o:o + nout * nvec]
            assert (d_in.data_ptr() % 16, d_out.data_ptr() % 16) == (8 * i, 8 * o)
            s.map_batched_device(nvec, d_in.data_ptr(), d_out.data_ptr(), transpose=transpose)
            got.append(d_out.cpu().numpy())
        assert np.isfinite(got[0]).all() and np.array_equal(got[0], got[1])

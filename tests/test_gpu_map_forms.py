"""The forms of the map kernels against the exported constraint matrix.

The lane mapping, the rows per thread and the treatment of long rows depend on
the number of interleaved vectors and on the layout's size; every form must
give A u and A^T w.  A row sum has at most a few hundred terms of order one, so
1e-12 of the largest result is far above FP64 rounding.  A non-finite input
entry must reach exactly the rows that hold its column: the padding slots of
the tables read nothing."""
import numpy as np
import pytest

from helpers import csr_of

pytestmark = pytest.mark.gpu

FORMS = [(2, "DQG", 1), (4, "DQG", 2), (4, "DQG", 256), (5, "DQGT2", 3), (7, "DQGT2", 1), (7, "DQGT2", 17),
         (10, "DQG", 1), (10, "DQG", 19), (10, "DQG", 32), (10, "DQG", 33), (9, "DQG", 129), (8, "DQG", 255),
         (14, "DQG", 1), (14, "DQG", 6)]


@pytest.mark.parametrize("n,positivity,nvec", FORMS)
@pytest.mark.parametrize("poison", [False, True])
def test_map_forms_match_the_matrix(v2g, n, positivity, nvec, poison):
    import torch

    s = v2g.V2RDMSolver([n], n // 2, n // 2, options=dict(POSITIVITY=positivity))
    A = csr_of(s)
    rng = np.random.default_rng(100 * n + nvec)
    for M, transpose in ((A, False), (A.T.tocsr(), True)):
        u = rng.standard_normal((M.shape[1], nvec))
        col, vec = int(rng.integers(M.shape[1])), int(rng.integers(nvec))
        if poison:
            u[col, vec] = np.inf
        hit = np.zeros((M.shape[0], nvec), dtype=bool)
        if poison:
            hit[M[:, [col]].nonzero()[0], vec] = True
            u0 = u.copy()
            u0[col, vec] = 0.0
            want = M @ u0
        else:
            want = M @ u
        d_in = torch.from_numpy(u.reshape(-1)).cuda()
        d_out = torch.full((M.shape[0] * nvec,), float("nan"), dtype=torch.float64, device="cuda")
        s.map_batched_device(nvec, d_in.data_ptr(), d_out.data_ptr(), transpose=transpose)
        got = d_out.cpu().numpy().reshape(want.shape)
        assert np.array_equal(~np.isfinite(got), hit)
        assert np.abs(got - want)[~hit].max() <= 1e-12 * max(1.0, np.abs(want).max())

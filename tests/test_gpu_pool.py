"""The solver's memory pools: calls from several threads, and memory given back.

Threads project, solve and multiply at once on handles of their own; every
result must equal the same call alone, bit for bit where the call is
deterministic on its own (projections and products are).  After a call that
needed several GiB, what stays reserved is at most the pool's 1 GiB plus the
context's own use."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_calls_from_several_threads(v2g):
    from v2rdm_casscf_b200.hamiltonian import synthetic

    def project(n, seed):
        s = v2g.V2RDMSolver.from_active_space(synthetic(n, seed))
        rng = np.random.default_rng(seed)
        x, y, z = (rng.uniform(-2, 0, k) for k in (s.dimx, s.nconstraints, s.dimx))
        out = []
        for _ in range(3):
            s.set_state(x, y, z, 1.0)
            s.update_xz(1.0)
            a, _, b, _ = s.get_state()
            out += [a, b, s.ATu(y)]
        return out

    jobs = [(4, 1), (6, 2), (8, 3), (7, 4), (6, 5), (5, 6)]
    alone = [project(*j) for j in jobs]
    got = [None] * len(jobs)
    errors = []

    def work(i):
        try:
            got[i] = project(*jobs[i])
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    for a, b in zip(alone, got):
        assert all(np.array_equal(u, v) for u, v in zip(a, b))


def test_memory_is_given_back(v2g):
    import torch

    dims = [4096] * 16
    n = sum(d * d for d in dims)
    a, b, c = (torch.zeros(n, dtype=torch.float64, device="cuda") for _ in range(3))
    torch.cuda.synchronize()
    v2g.block_gemm_device([64], a.data_ptr(), b.data_ptr(), c.data_ptr())
    before = torch.cuda.mem_get_info()[0]
    v2g.block_gemm_device(dims, a.data_ptr(), b.data_ptr(), c.data_ptr())  # 4 GiB of split operands
    v2g.block_gemm_device([64], a.data_ptr(), b.data_ptr(), c.data_ptr())  # synchronises
    torch.cuda.synchronize()
    assert before - torch.cuda.mem_get_info()[0] <= (1 << 30) + (64 << 20)

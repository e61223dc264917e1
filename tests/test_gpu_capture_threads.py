"""Calls of other threads do not disturb a solve whose CG runs from a graph.

A group above the persistent CG's limits captures one CG iteration into a graph.
Other threads meanwhile allocate, copy and free on the legacy default stream,
which may not become dependent on a capture.  Every thread's results must be
those of the same calls alone: the solves capped at a few outer iterations (a
capture each), the projections, maps and products bit for bit."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_graph_solves_beside_other_calls(v2g):
    import torch
    from v2rdm_casscf_b200.hamiltonian import synthetic

    def group(seed):
        return [v2g.V2RDMSolver.from_active_space(synthetic(4, seed + k), start="feasible", projection="adaptive",
                                                  options=dict(MAXITER=3)) for k in range(9)]

    def solve(solvers):
        for s in solvers:
            s.set_state(*(np.zeros(k) for k in (s.dimx, s.nconstraints, s.dimx)), 1.0)
        return np.array([r["e_primal"] for r in v2g.solve_batch(solvers)])

    def projector(n, seed):
        s = v2g.V2RDMSolver.from_active_space(synthetic(n, seed))
        rng = np.random.default_rng(seed)
        x, y, z = (rng.uniform(-2, 0, k) for k in (s.dimx, s.nconstraints, s.dimx))

        def call():
            s.set_state(x, y, z, 1.0)
            s.update_xz(1.0)
            a, _, b, _ = s.get_state()
            return np.concatenate([a, b, s.ATu(y)])

        return call

    def multiplier(seed):
        g = torch.Generator(device="cuda").manual_seed(seed)
        a, b = (torch.randn(3 * 128 * 128, dtype=torch.float64, device="cuda", generator=g) for _ in range(2))
        c = torch.empty_like(a)
        torch.cuda.synchronize()

        def call():
            v2g.block_gemm_device([128, 100, 128], a.data_ptr(), b.data_ptr(), c.data_ptr(), tensor_cores=False)
            return c.cpu().numpy()

        return call

    solvers, second = group(30), group(60)
    want = solve(solvers)
    calls = [projector(4, 1), projector(6, 2), projector(5, 3), multiplier(4), lambda: solve(second)]
    alone = [c() for c in calls]
    stop, errors = threading.Event(), []

    def other(i):
        try:
            while not stop.is_set():
                assert np.array_equal(calls[i](), alone[i])
        except BaseException as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=other, args=(i,)) for i in range(len(calls))]
    for t in threads:
        t.start()
    try:
        for _ in range(40):
            assert np.array_equal(solve(solvers), want)
    finally:
        stop.set()
        for t in threads:
            t.join()
    assert not errors

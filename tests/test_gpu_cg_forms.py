"""The dual step's CG solves the system it is given, whatever form its kernel takes.

After one outer iteration from the feasible start (z = 0, mu = tau = 1, x with
A x = b to 1e-10 |b|) the dual step has solved A A^T y = A c - (A x - b) to the
first iteration's tolerance |r| < 0.01.  The residual is formed here from the
exported matrix; the allowance of 1e-6 covers the distance of CG's recurred
residual from the true one and of A x from b.  The layouts are such that the
map of A, of A^T, both or neither asks for several rows per thread, alone and
in groups, on the resident, the persistent and the launched route."""
import numpy as np
import pytest

from helpers import csr_of

pytestmark = pytest.mark.gpu

FORMS = [(14, "DG", True, 1), (14, "DG", True, 2), (12, "DQ", True, 7), (13, "DQ", True, 5), (15, "D", True, 5),
         (10, "DQG", False, 8), (14, "DQG", False, 1), (13, "DQG", True, 1), (13, "DQG", True, 6), (13, "DQG", True, 8),
         (6, "DQG", True, 1), (6, "DQG", True, 5), (8, "DQGT2", True, 3), (9, "DQG", True, 12)]


@pytest.mark.parametrize("n,positivity,spin,count", FORMS)
@pytest.mark.parametrize("launched", [False, True])
def test_first_dual_step_solves_its_system(v2g, n, positivity, spin, count, launched):
    from v2rdm_casscf_b200.hamiltonian import synthetic

    # timing every map (profile) takes the launched maps
    solvers = [v2g.V2RDMSolver.from_active_space(synthetic(n, 70 + k), profile=launched, start="feasible",
                                                 projection="adaptive",
                                                 options=dict(POSITIVITY=positivity, CONSTRAIN_SPIN=spin, MAXITER=1))
               for k in range(count)]
    v2g.solve_batch(solvers)
    A = csr_of(solvers[0])
    for s in solvers:
        assert s.result["oiter"] == 1
        y = s.get_state()[1]
        r = A @ (s.c - A.T @ y)
        assert np.linalg.norm(r) <= 0.01 + 1e-6

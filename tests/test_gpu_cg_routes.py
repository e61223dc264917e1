"""The routes of the CG (resident, persistent, launched) give the reference's energies.

The route depends on the rows and the number of instances of a layout group:
n = 4 and 8 take the resident kernel up to the counts whose rows have lanes of
their own, the persistent one up to eight instances, map launches above.  Every
group holds the reference's instance first and neighbours of it after, each of
which stops on its own; the first must land on the reference's energy (1e-6 Eh,
as every solve test), and an instance solved in the group on the energy it has
alone (2e-6: both stop on the same tolerances)."""
import os

import pytest

from tests.helpers import GOLDEN, load

pytestmark = pytest.mark.gpu

PRODUCT = dict(projection="adaptive", start="feasible", anderson_memory=10, cg_extrapolate=True)


@pytest.mark.parametrize("name,count", [("energy_batch_n8_s3", c) for c in (1, 2, 3, 8, 9)]
                         + [("solve_synthetic_n4_s0", c) for c in (1, 2, 3, 8, 9)]
                         + [("energy_batch_n12_s13", 1)])
def test_cg_routes_reach_the_reference_energy(v2g, name, count):
    from v2rdm_casscf_b200.hamiltonian import ActiveSpace, synthetic

    g = load(os.path.join(GOLDEN, name + ".npz"))
    n = int(g["n"]) if "n" in g else 4
    seed = int(g["seed"]) if "seed" in g else 0
    a = synthetic(n, seed)
    opts = dict(R_CONVERGENCE=1e-6, E_CONVERGENCE=1e-7, MU_UPDATE_FREQUENCY=250)

    def solver(k):
        b = synthetic(n, 500 + k)
        space = a if k == 0 else ActiveSpace(a.h + 0.01 * b.h, a.L + 0.01 * b.L, a.na, a.nb)
        return v2g.V2RDMSolver.from_active_space(space, options=opts, **PRODUCT)

    res = v2g.solve_batch([solver(k) for k in range(count)])
    assert all(r["status"] == 0 for r in res)
    assert abs(res[0]["e_total"] - float(g["e_primal"])) <= 1e-6
    if count > 1:
        alone = v2g.solve_batch([solver(count - 1)])[0]
        assert abs(res[-1]["e_total"] - alone["e_total"]) <= 2e-6

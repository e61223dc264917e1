"""The per-iteration diagnostics (V2G_DIAG) of a solve, whatever its projection.

Groups projected by the matrix sign keep no eigenvectors to report on, groups
above its limit do: a solve with diagnostics must take its outer iterations and
write a line per instance and iteration either way."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SCRIPT = """
import sys
import v2rdm_casscf_b200 as V
from v2rdm_casscf_b200.hamiltonian import synthetic
n, count = int(sys.argv[1]), int(sys.argv[2])
solvers = [V.V2RDMSolver.from_active_space(synthetic(n, k), start="feasible", projection="adaptive",
                                           options=dict(MAXITER=3)) for k in range(count)]
for r in V.solve_batch(solvers):
    assert r["oiter"] == 3, r
"""


@pytest.mark.parametrize("n,count", [(4, 2), (10, 1), (14, 20)])
def test_diagnostics_of_a_solve(v2g, tmp_path, n, count):
    out = tmp_path / "diag"
    env = dict(os.environ, V2G_DIAG="1", V2G_DIAG_FILE=str(out), PYTHONPATH=ROOT)
    r = subprocess.run([sys.executable, "-c", SCRIPT, str(n), str(count)], env=env, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    lines = out.read_text().splitlines()
    assert sum(" b " in k and " ep " in k for k in lines) == 3 * count
    assert sum(" group " in k for k in lines) == 3

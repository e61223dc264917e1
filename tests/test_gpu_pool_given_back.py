"""What the pools hold unused stands in nobody's way.

Each check runs in a process of its own, on memory figures of the whole device
with allowances far below the amounts at stake: the pools are empty again once
the last handle has gone, and while they hold something, a call that the device
has room for without them still gets it."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PRELUDE = """
import numpy as np
import torch
import v2rdm_casscf_b200 as V
from v2rdm_casscf_b200.hamiltonian import synthetic
MB = 1 << 20

def free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]

def hold():
    # the split operands of two products leave about 512 MiB in the pool
    dims = [4096] * 2
    n = sum(d * d for d in dims)
    t = [torch.zeros(n, dtype=torch.float64, device="cuda") for _ in range(3)]
    torch.cuda.synchronize()
    V.block_gemm_device(dims, *(x.data_ptr() for x in t))
    del t
    torch.cuda.empty_cache()

def fill(left):
    return torch.empty(free() - left, dtype=torch.uint8, device="cuda")
"""


def run(script):
    r = subprocess.run([sys.executable, "-c", PRELUDE + script], env=dict(os.environ, PYTHONPATH=ROOT),
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return r


def test_pools_are_empty_after_the_last_handle(v2g):
    run("""
def project(n):
    s = V.V2RDMSolver.from_active_space(synthetic(n, 1))
    s.update_xz(1.0)
    return s

s = project(4)
del s
net = V.WarmStart()
before = free()
s = project(18)
held = before - free()
del s
one_owner = before - free()  # the network still lives
assert held > 64 * MB and one_owner > 64 * MB, (held, one_owner)
del net
assert before - free() <= 16 * MB, before - free()
s = project(18)
del s
assert before - free() <= 16 * MB, before - free()
""")


def test_anderson_history_beside_held_memory(v2g):
    # the history of one n = 14 instance takes 0.13 GiB of the 0.5 that the pool holds
    r = run("""
keep = V.V2RDMSolver([2], 1, 1)
hold()
s = V.V2RDMSolver.from_active_space(synthetic(14, 1), start="feasible", projection="adaptive", anderson_memory=10,
                                    options=dict(MAXITER=2))
s.update_xz(1.0)
block = fill(100 * MB)
assert V.solve_batch([s])[0]["oiter"] == 2
""")
    assert "Anderson" not in r.stderr

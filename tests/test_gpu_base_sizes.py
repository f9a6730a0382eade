"""Base levels whose factorisation takes close to 48 KB of shared memory, each
in a process of its own (what a kernel was allowed once stays allowed): the
solve's residual of 1e-10 is checked on the host."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

SCRIPT = """
import numpy as np, scipy.sparse as sp, ugcore_gb300 as ug
from ugcore_gb300 import problems
p = problems.Problem(ug.Context(0), problems.config("c0", mx=%d, my=%d, nref=2))
assert p.solve()["ok"]
rowptr, col, val = p.A.export_csr()
b, x = p.b.numpy(), p.x.numpy()
r = b - sp.csr_matrix((val, col, rowptr)) @ x
assert np.linalg.norm(r) <= 1.1e-10 * np.linalg.norm(b), np.linalg.norm(r)
"""


@pytest.mark.parametrize("mx,my", [(3, 12), (5, 8), (4, 10), (6, 7)])   # 52, 54, 55, 56 unknowns
def test_solves(mx, my):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    done = subprocess.run([sys.executable, "-c", SCRIPT % (mx, my)], cwd=root, capture_output=True, text=True)
    assert done.returncode == 0, done.stderr

"""Large FP64 and FP32 factorisations in turn, in one process that starts with
them: the interchanges of both are composed by one kernel, whose shared memory
passes the default limit from 6145 rows on. The matrices are permuted diagonals,
so the interchanges are known: column j's pivot is the one entry it has."""
import pathlib
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

SCRIPT = """
import numpy as np
import hornsculpt_b200 as hs

def factor(n, fp32):
    rows = np.roll(np.arange(n), 7)
    a = np.zeros((1, n, n), complex)
    a[0, rows, np.arange(n)] = 1.0 + np.arange(n) / n
    factors, piv, info = hs.debug_lu_factor(a, fp32=fp32)
    order = np.arange(n)
    for i, q in enumerate(piv[0]):
        order[i], order[q] = order[q], order[i]
    assert info == 0 and np.array_equal(order, rows)
    assert np.allclose(np.diag(factors[0]), a[0, rows, np.arange(n)], rtol=1e-6)

for n, fp32 in ((6400, False), (6200, True), (6400, False)):
    factor(n, fp32)
print("factored")
"""


def test_both_precisions_in_turn():
    root = pathlib.Path(__file__).resolve().parent.parent
    done = subprocess.run([sys.executable, "-c", SCRIPT], cwd=root, capture_output=True, text=True, timeout=300)
    assert done.returncode == 0 and "factored" in done.stdout, done.stdout + done.stderr

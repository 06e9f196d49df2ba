"""FP32 factorisation of more rows than the cluster's registers hold (16 CTAs of
512 threads with two rows: 16,384): its first two panels, the second a ragged one
of the outer block, come from the shared-memory cluster kernel with rows kept in
global memory, and their row moves from the interchange sequence. LAPACK's
acceptance ratio (xGET01, threshold 30), as in test_gpu_lu.py. The matrix goes
through the C hook as it lies on the device, column-major."""
import ctypes as C

import numpy as np
import pytest
import torch

from hornsculpt_b200 import _lib
from tests.test_gpu_lu import EPS32, XGET01_THRESHOLD, _permutation

pytestmark = pytest.mark.gpu


def test_panels_beyond_the_registers():
    n = 16384 + 33
    generator = torch.Generator(device="cuda").manual_seed(11)
    columns = torch.randn(n, n, 2, generator=generator, device="cuda", dtype=torch.float32).double()
    source = columns.cpu().numpy()
    factors = np.empty_like(source)
    piv = np.empty(n, np.int32)
    info = C.c_int32()
    _lib.check(_lib.load().hs_bem_debug_lu(1, n, 1, source.ctypes.data, factors.ctypes.data, piv.ctypes.data,
                                           C.byref(info)))
    assert info.value == 0
    order = _permutation(piv)
    assert np.array_equal(np.sort(order), np.arange(n))
    del source
    a = torch.view_as_complex(columns)[:, torch.as_tensor(order, device="cuda")].T  # P A
    norm = torch.linalg.matrix_norm(a, ord=1).item()
    lu = torch.view_as_complex(torch.as_tensor(factors, device="cuda")).T
    lower = torch.tril(lu, -1) + torch.eye(n, dtype=lu.dtype, device="cuda")
    residual = a - lower @ torch.triu(lu)
    one = torch.linalg.matrix_norm(residual, ord=1).item() / (n * norm)
    assert one / EPS32 < XGET01_THRESHOLD

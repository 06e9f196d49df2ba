"""LU panels at the edges of their shapes: half panels, one CTA against a
cluster, the wider CTAs of large batches and tall panels, two rows per thread,
and panels beyond the cluster's registers. FP64 pivots equal LAPACK's and the
factors pass its acceptance ratio (xGET01, threshold 30), as in
test_gpu_lu.py; the largest sizes are held to the ratio alone."""
import numpy as np
import pytest

import hornsculpt_b200 as hs
from tests.test_gpu_lu import EPS32, EPS64, XGET01_THRESHOLD, _lapack, _permutation, _random, _residuals

pytestmark = pytest.mark.gpu


def _check(a, fp32, lapack):
    factors, piv, info = hs.debug_lu_factor(a, fp32=fp32)
    assert info == 0
    for b in range(len(a)):
        seen = a[b].astype(np.complex64).astype(np.complex128) if fp32 else a[b]
        one, _ = _residuals(seen, factors[b], piv[b])
        assert one / (EPS32 if fp32 else EPS64) < XGET01_THRESHOLD
        assert np.array_equal(np.sort(_permutation(piv[b])), np.arange(a.shape[1]))
        if lapack:
            assert np.array_equal(piv[b], _lapack(a[b], fp32=False)[1])


@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 31, 32, 33, 48, 63, 65, 255, 256, 257, 288, 511, 513])
def test_small_panels(n):
    a = _random(n, 2, seed=n)
    _check(a, False, True)
    _check(a, True, False)


@pytest.mark.parametrize("n,batch", [(600, 64), (2600, 16)])
def test_panels_of_large_batches(n, batch):
    """More CTAs than the device holds with 256 threads each: the wider shapes."""
    a = _random(n, batch, seed=n)
    _check(a, False, False)
    _check(a, True, False)


@pytest.mark.parametrize("n", [4097, 8225])
def test_tall_panels(n):
    """Beyond 16 x 256 and 16 x 512 rows; FP64 beyond the cluster's registers."""
    a = _random(n, 1, seed=n)
    _check(a, False, False)
    _check(a, True, False)


def test_ties_take_the_lowest_row():
    """Equal magnitudes everywhere in the first column, over several CTAs: row 0 is chosen, as zgetrf does."""
    a = _random(1200, 1, seed=5)
    a[0, :, 0] = 1.0
    factors, piv, info = hs.debug_lu_factor(a)
    assert info == 0 and piv[0, 0] == 0
    assert np.array_equal(piv[0], _lapack(a[0], fp32=False)[1])

"""Tridiagonals that hold NaN (a recurrence that broke down) beside sound ones: every output is written, and the sound
ones' are their own."""
import numpy as np
import pytest

import qsi_subspace_ed_gb300 as q

pytestmark = pytest.mark.gpu


# 118: the largest with its vectors in shared memory; odd sizes carry a padding row
@pytest.mark.parametrize("m", [3, 4, 31, 118, 127])
def test_every_output_is_written(m):
    rng = np.random.default_rng(m)
    a, b = rng.standard_normal((3, m)), np.zeros((3, m))
    b[::2] = 0.1 + np.abs(rng.standard_normal((2, m)))
    a[1, 1 % m] = a[1, m // 2] = np.nan
    before = [q.tridiag_ritz(np.full((3, m), 7e77), np.full((3, m), 1e77)) for _ in range(3)]  # what memory held
    ev, first = q.tridiag_ritz(a, b)
    assert np.isfinite(before[0][0]).all()
    for k in (0, 2):
        w = np.linalg.eigvalsh(np.diag(a[k]) + np.diag(b[k, :m - 1], 1) + np.diag(b[k, :m - 1], -1))
        np.testing.assert_allclose(ev[k], w, rtol=0, atol=1e-12)
        assert abs(np.sum(first[k] ** 2) - 1) < 1e-12
    # nothing couples: the diagonal in order, NaN before the numbers, unit vectors
    n_nan = np.isnan(a[1]).sum()
    assert np.isnan(ev[1, :n_nan]).all()
    np.testing.assert_array_equal(ev[1, n_nan:], np.sort(a[1][~np.isnan(a[1])]))
    assert np.count_nonzero(first[1]) == 1 and first[1].sum() == 1

"""Bins of large buckets, whose slots have room for few bits of a tag: no state of the basis is taken for absent, also
where a state that found its bin full meets a last slot that is marked and carries the all-ones tag.  And bases whose
states share their top bits, which the buckets leave out."""
import numpy as np
import pytest

import qsi_subspace_ed_gb300 as q

pytestmark = pytest.mark.gpu


def patterns(n, up=None, far=None):
    """The patterns 0 .. n-1 of the low spins, with spin `up` up in all of them, or with one more state far above, beside
    which they are all in one bucket."""
    lohi = np.zeros((n + (far is not None), 2), dtype=np.uint64)
    lohi[:n, 0] = np.arange(n, dtype=np.uint64)
    for bit, rows in ((up, slice(n)), (far, slice(n, n + 1))):
        if bit is not None:
            lohi[rows, bit // 64] |= np.uint64(1) << np.uint64(bit % 64)
    return lohi


def check(lohi):
    H = q.SymbolicOpSum()
    for c, s in [(0.3, "0x"), (0.5, "11x"), (0.9, "20x")]:  # every flip of 2^k patterns stays in the basis
        H.add_term(c, q.SymbolicPMROperator(s))
    H.add_term(0.7, q.SymbolicPMROperator("64x"))  # leaves it, from a shared bit as from the others
    b = q.ZBasis(lohi)
    op = q.LazyOpSum(b, H)
    n = len(lohi)
    x = np.random.default_rng(n).standard_normal(n)
    row, y = np.zeros(n), np.zeros(n)
    op.set_kernel(0)  # bisects the bucket
    op.evaluate(x, row)
    op.set_kernel(1)
    op.evaluate(x, y)
    assert np.array_equal(y, row), np.count_nonzero(y != row)
    op.materialise(True)
    y[:] = 0.0
    op.evaluate(x, y)
    assert np.array_equal(y, row), np.count_nonzero(y != row)
    return b, row, x


# nine, eight and seven bits of tag; 2^23 - 1 states need as many bits of offset as 2^23: two offsets are no state's
@pytest.mark.parametrize("n,far", [(1 << 23, 68), ((1 << 23) - 1, 40), (1 << 24, 64), (1 << 25, 64)])
def test_no_state_of_a_large_bucket_is_lost(n, far):
    check(patterns(n, far=far))


# the shared bit next to the others, in either word, at the ends of the words, above 96 bits (no bins)
@pytest.mark.parametrize("n", [1, 2, 1000, 1 << 21])
@pytest.mark.parametrize("up", [21, 40, 62, 63, 64, 65, 95, 96, 127])
def test_states_that_share_their_top_bits(n, up):
    lohi = patterns(n, up=up)
    b, row, x = check(lohi)
    assert b.index_info()["bucket_bits"] <= max(1, (n - 1).bit_length())
    i = np.arange(n)
    want = np.zeros(n)
    for c, k in [(0.3, 0), (0.5, 11), (0.9, 20)]:
        j = i ^ (1 << k)
        want += np.where(j < n, c * x[np.minimum(j, n - 1)], 0.0)
    np.testing.assert_allclose(row, want, rtol=0, atol=1e-14 * np.abs(x).max())
    ask = lohi[::7].copy()
    assert np.array_equal(b.search(ask), np.arange(n)[::7])
    ask[:, up // 64] ^= np.uint64(1) << np.uint64(up % 64)  # without the shared bit; below, with another one
    assert np.all(b.search(ask) < 0)
    ask[:, 1] |= np.uint64(1) << np.uint64(50)
    assert np.all(b.search(ask) < 0)

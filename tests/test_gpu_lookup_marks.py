"""Bins of large buckets, whose slots have room for few bits of a tag: no state of the basis is taken for absent, also
where a state that found its bin full meets a last slot that is marked and carries the all-ones tag."""
import numpy as np
import pytest

import qsi_subspace_ed_gb300 as q

pytestmark = pytest.mark.gpu


def pinned(n, up):
    """All n patterns of the low spins with spin `up` up: one bucket, since all states share their top bits."""
    lohi = np.zeros((n, 2), dtype=np.uint64)
    lohi[:, 0] = np.arange(n, dtype=np.uint64)
    lohi[:, up // 64] |= np.uint64(1) << np.uint64(up % 64)
    return lohi


# nine, eight and seven bits of tag; 2^23 - 1 states need as many bits of offset as 2^23: two offsets are no state's
@pytest.mark.parametrize("n,up", [(1 << 23, 68), ((1 << 23) - 1, 40), (1 << 24, 64), (1 << 25, 64)])
def test_no_state_of_a_large_bucket_is_lost(n, up):
    H = q.SymbolicOpSum()
    for c, s in [(0.3, "0x"), (0.5, "11x"), (0.9, "20x")]:  # every flip stays in the basis (2^k states)
        H.add_term(c, q.SymbolicPMROperator(s))
    op = q.LazyOpSum(q.ZBasis(pinned(n, up)), H)
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

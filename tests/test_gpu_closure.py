"""Operators whose terms leave the basis at few or many, early or late rows: the closure pass at creation stops at the
first miss any warp meets, while the others are at every point of theirs.  Created many times; the applies bitwise those
of the row-per-thread kernel, which takes nothing from that pass."""
import numpy as np
import pytest

import qsi_subspace_ed_gb300 as q

pytestmark = pytest.mark.gpu

N = 300_000
PAIRS = [(0.7, "0+ 1-"), (0.7, "0- 1+"), (0.2, "2+ 3-"), (0.2, "2- 3+"), (0.5, "4+ 5- 6+ 7- 8+ 9-"), (0.5, "4- 5+ 6- 7+ 8- 9+")]
FLIPS = [(0.3, "0x"), (0.4, "7x"), (-0.2, "3x 9z")]


@pytest.mark.parametrize("terms", [PAIRS, FLIPS], ids=["pairs", "flips"])
@pytest.mark.parametrize("missing", ["first", "last", "middle", "every 5,000th", "every third"])
def test_terms_that_leave_the_basis(terms, missing):
    keep = np.ones(N, dtype=bool)
    keep[{"first": slice(1, 2), "last": slice(N - 2, N - 1), "middle": slice(N // 2, N // 2 + 5),
          "every 5,000th": slice(77, None, 5000), "every third": slice(1, None, 3)}[missing]] = False
    lohi = np.zeros((keep.sum(), 2), dtype=np.uint64)
    lohi[:, 0] = np.arange(N, dtype=np.uint64)[keep]
    basis = q.ZBasis(lohi)
    H = q.SymbolicOpSum()
    for c, s in terms:
        H.add_term(c, q.SymbolicPMROperator(s))
    x = np.random.default_rng(1).standard_normal(len(lohi))
    row, y = np.zeros_like(x), np.zeros_like(x)
    for k in range(20):
        op = q.LazyOpSum(basis, H)
        if k == 0:
            op.set_kernel(0)
            op.evaluate(x, row)
            op.set_kernel(1)
        y[:] = 7.0
        op.evaluate(x, y)
        assert np.array_equal(y, row), k
        op.close()

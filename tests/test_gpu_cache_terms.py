"""Materialised operators around 256 terms, where a term's number stops fitting a byte."""
import numpy as np
import pytest

import qsi_subspace_ed_gb300 as q

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("terms", [255, 256, 257])
def test_terms_around_a_byte(terms):
    n = 1000  # some flips leave the basis
    lohi = np.zeros((n, 2), dtype=np.uint64)
    lohi[:, 0] = np.arange(n, dtype=np.uint64)
    H = q.SymbolicOpSum()
    for m in range(1, terms + 1):  # each flips another set of spins, with its own coefficient
        H.add_term(0.01 * m, q.SymbolicPMROperator(" ".join(f"{k}x" for k in range(10) if (m >> k) & 1)))
    op = q.LazyOpSum(q.ZBasis(lohi), H)
    rng = np.random.default_rng(terms)
    x, X = rng.standard_normal(n), rng.standard_normal((n, 16)).astype(np.float32)
    row, y, ref, Y = np.zeros(n), np.zeros(n), np.zeros_like(X), np.zeros_like(X)
    op.apply_batched(X, ref)
    op.set_kernel(0)
    op.evaluate(x, row)
    op.set_kernel(1)
    op.materialise(True)
    op.evaluate(x, y)
    op.apply_batched(X, Y)
    assert np.array_equal(y, row) and np.array_equal(Y, ref)

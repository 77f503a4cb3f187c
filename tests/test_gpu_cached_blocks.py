"""Blocks of FP32 and FP64 vectors on a materialised operator against the look-ups, bitwise: rows of every number of
entries up to more than two groups of eight, misses among them, and tile counts about the one (152 SMs of 32 warps) up
to which a tile's row sets go to warps of their own."""
import numpy as np
import pytest

import qsi_subspace_ed_gb300 as q

pytestmark = pytest.mark.gpu


def operator(n, terms):
    lohi = np.zeros((n, 2), dtype=np.uint64)
    lohi[:, 0] = np.arange(n, dtype=np.uint64)
    H = q.SymbolicOpSum()
    for k in range(terms):  # flips of spin k from up: rows with as many entries as spins up; those of k + 1 may leave
        H.add_term(0.1 * (k + 1), q.SymbolicPMROperator(f"{k}-"))
        H.add_term(-0.03 * (k + 1), q.SymbolicPMROperator(f"{k}+ {k + 1}z"))
    H.add_term(0.7, q.SymbolicPMROperator("3z"))
    return q.LazyOpSum(q.ZBasis(lohi), H)


@pytest.mark.parametrize("n,terms", [(1, 1), (31, 3), (33, 6), (5000, 12), (152 * 32 * 32, 17), (152 * 32 * 32 + 1, 18)])
def test_materialised_blocks_are_those_of_the_look_ups(n, terms):
    op = operator(n, terms)
    rng = np.random.default_rng(n)
    counts = [4, 8, 16, 17, 31, 32, 33, 64, 65, 100, 128, 130] if n < 10000 else [4, 8, 16, 32, 65]
    cases = [(R, t, acc) for R in counts for t in (np.float32, np.float64) for acc in (False, True)]
    X = {t: rng.standard_normal((n, max(counts))).astype(t) for t in (np.float32, np.float64)}
    got = []
    for cached in (False, True):
        op.materialise(cached)
        for i, (R, t, acc) in enumerate(cases):
            x = np.ascontiguousarray(X[t][:, :R])
            y = 0.5 * x if acc else np.full_like(x, 7.0)
            op.apply_batched(x, y, accumulate=acc)
            if not cached:
                got.append(y)
            else:
                assert np.array_equal(y, got[i]), (R, t, acc)

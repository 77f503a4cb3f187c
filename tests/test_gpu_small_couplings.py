"""Solves whose Krylov space all but closes inside a cycle: a coupling (beta) between rounding and 1e-6 of the norm,
where the basis stays orthogonal only if each step removes what the vanishing norm brings up, and past exact closures."""
import numpy as np
import pytest

import qsi_subspace_ed_gb300 as q

pytestmark = pytest.mark.gpu

SPINS = 12


def operator(eps, scale=1.0):
    """Sum of X over the spins (13 levels -12, -10 .. 12) plus eps times an irregular field: the thirteenth coupling is
    of the order of eps."""
    lohi = np.zeros((1 << SPINS, 2), dtype=np.uint64)
    lohi[:, 0] = np.arange(1 << SPINS, dtype=np.uint64)
    H = q.SymbolicOpSum()
    for k in range(SPINS):
        H.add_term(scale, q.SymbolicPMROperator(f"{k}x"))
    if eps:
        for k in range(SPINS):
            H.add_term(scale * eps * np.cos(1.7 * k + 0.3), q.SymbolicPMROperator(f"{k}z"))
            H.add_term(scale * eps * 0.3 * np.sin(2.3 * k), q.SymbolicPMROperator(f"{k}x {(k + 5) % SPINS}x"))
    return q.LazyOpSum(q.ZBasis(lohi), H)


def residuals(op, e, v):
    out = []
    for k in range(len(e)):
        y = np.zeros(op.rows())
        op.evaluate(np.ascontiguousarray(v[:, k]), y)
        out.append(np.linalg.norm(y - e[k] * v[:, k]))
    return np.array(out)


# 24 steps: 13, then the eleven levels that have more copies, a second closure at the end
@pytest.mark.parametrize("eps", [1e-6, 1e-8, 1e-9, 1e-10, 1e-11, 1e-12, 1e-13, 3e-14, 1e-14, 1e-15, 0.0])
@pytest.mark.parametrize("scale", [1.0, 1e5, 1e-4])
def test_vectors_stay_orthonormal(eps, scale):
    op = operator(eps, scale)
    e, v, rep = q.diagonalise(op, nev=8, ncv=24, tol=max(100 * eps, 1e-11), seed=5, max_iter=300)
    # a few hundred roundings per product and sum, of vectors of norm one
    np.testing.assert_allclose(v.T @ v, np.eye(8), rtol=0, atol=1e-12)
    assert np.all(np.diff(e) >= -1e-12 * scale)
    assert residuals(op, e, v).max() < scale * SPINS * max(200 * eps, 1e-9)
    # levels near -12, -10, .. and none more often than the space has it (1, 12, ...)
    assert np.abs(e / scale + SPINS - 2 * np.rint((e / scale + SPINS) / 2)).max() < 1e-9 + 10 * eps
    assert np.count_nonzero(e < (1 - SPINS) * scale) == 1


@pytest.mark.parametrize("ncv", [14, 16, 20])
def test_levels_past_exact_closures(ncv):
    """No perturbation: after the 13 levels the solve goes on from a direction orthogonal to all vectors before, and
    what it returns are eigenpairs, no level more often than its multiplicity."""
    op = operator(0.0)
    e, v, _ = q.diagonalise(op, nev=4, ncv=ncv, tol=1e-11, seed=2, max_iter=300)
    np.testing.assert_allclose(v.T @ v, np.eye(4), rtol=0, atol=1e-12)
    assert residuals(op, e, v).max() < 1e-9
    assert abs(e[0] + 12) < 1e-10 and np.all(np.diff(e) >= -1e-12)
    levels = np.rint(e)
    assert np.abs(e - levels).max() < 1e-9 and np.count_nonzero(levels == -12) == 1

"""Signs of the eigenvectors: those that cyclic Jacobi in the circle method's pair order, from the identity, gives the
projected eigenproblem's columns, and so the same for a seed whatever the kernels' shape."""
import numpy as np
import pytest

import qsi_subspace_ed_gb300 as q
from qsi_subspace_ed_gb300 import workloads

pytestmark = pytest.mark.gpu


def pairs(M):
    """Rounds of the circle method: player 0 stays, the others move up one position, positions t and M - 1 - t meet."""
    at = list(range(M))
    for _ in range(M - 1):
        yield np.sort([[at[t], at[M - 1 - t]] for t in range(M // 2)], axis=1).T
        at = [at[0], at[-1]] + at[1:-1]


def jacobi(T):
    """Eigenvalues ascending and eigenvectors of T; odd sizes carry a decoupled last row above the spectrum."""
    m = len(T)
    M = m + (m & 1)
    A, V = np.zeros((M, M)), np.eye(M)
    A[:m, :m] = T
    if M != m:
        A[-1, -1] = 2 * np.abs(T).sum(axis=1).max() + 1
    tiny = 1e-17 * np.linalg.norm(A)
    for _ in range(20):
        before = V.copy()
        for p, r in pairs(M):
            apq, d = A[p, r], A[r, r] - A[p, p]
            turn = np.abs(apq) > tiny
            theta = d / np.where(turn, 2 * apq, 1)
            t = np.where(turn, np.where(theta >= 0, 1, -1) / (np.abs(theta) + np.hypot(theta, 1)), 0)
            c = 1 / np.hypot(t, 1)
            s = t * c
            A[p], A[r] = c[:, None] * A[p] - s[:, None] * A[r], s[:, None] * A[p] + c[:, None] * A[r]
            A[:, p], A[:, r] = c * A[:, p] - s * A[:, r], s * A[:, p] + c * A[:, r]
            V[:, p], V[:, r] = c * V[:, p] - s * V[:, r], s * V[:, p] + c * V[:, r]
        if np.array_equal(V, before):
            break
    order = np.argsort(np.diag(A), kind="stable")[:m]
    return np.diag(A)[order], V[:m, order]


# one and two pairs per round, odd sizes, the vectors in shared (up to 118) and in global memory, the largest
@pytest.mark.parametrize("m", [2, 3, 4, 15, 16, 25, 64, 118, 120, 127, 128])
def test_first_components_have_the_signs_of_the_rotations(m):
    rng = np.random.default_rng(m)
    a, b = rng.standard_normal((2, m)), 0.1 + np.abs(rng.standard_normal((2, m)))
    ev, first = q.tridiag_ritz(a, b)
    for k in range(2):
        w, V = jacobi(np.diag(a[k]) + np.diag(b[k, :m - 1], 1) + np.diag(b[k, :m - 1], -1))
        np.testing.assert_allclose(ev[k], w, rtol=0, atol=1e-12)
        seen = np.abs(V[0]) > 1e-9  # smaller components may come out with either sign
        assert seen.any() and np.array_equal(np.sign(first[k][seen]), np.sign(V[0][seen]))


# 32-spin Q = 0 basis, seeds 0 .. 15: the sign of each vector's product with default_rng(0).standard_normal
@pytest.mark.parametrize("options,signs", [
    (dict(nev=1, ncv=15), "- - - + + + - + - + - - - - + +"),
    (dict(nev=3, ncv=20), "-++ +-+ -+- -+- ++- ++- --+ -+- +-- --- --- +++ -++ +-- +-- ---"),
    (dict(nev=2, ncv=24, precision="mixed"), "++ -+ -+ -+ +- -- ++ +- ++ +- +- ++ +- +- -+ -+"),
    (dict(nev=3, ncv=30, precision="mixed", block=16), "--+ +-+ ++- +-+ +-+ +-+ +-+ --- +-- +-- -++ +-+ ++- +-- +++ ++-"),
])
def test_solves_return_the_same_vectors_for_a_seed(options, signs):
    lat = workloads.lattice("pyro_1x2x1")
    lohi = q.enumerate_basis(lat)
    basis = q.ZBasis(lohi)
    probe = np.random.default_rng(0).standard_normal(len(lohi))
    got = []
    for seed in range(16):
        g, B = workloads.ring_zeeman_params(seed)
        op = q.LazyOpSum(basis, q.build_ring_zeeman(lat, g, B))
        _, vec, _ = q.diagonalise(op, tol=1e-10, seed=seed, **options)
        got.append("".join("+" if d > 0 else "-" for d in probe @ vec))
    assert " ".join(got) == signs

"""The Krylov drivers' device kernels at the edges of their tiles and batches: the Jacobi eigensolver with its
eigenvectors in shared and in global memory, Krylov bases around groups of eight vectors, invariant subspaces inside a
cycle, eigval0 around its batches of iterations, and solves that materialise the operator for themselves."""
import numpy as np
import pytest

import qsi_subspace_ed_gb300 as q
from oracle import oracle as O
from qsi_subspace_ed_gb300 import workloads

pytestmark = pytest.mark.gpu

EPS = 2.220446049250313e-16


@pytest.mark.parametrize("m", [1, 2, 3, 24, 25, 100, 118, 119, 120, 127, 128])
@pytest.mark.parametrize("kind", ["random", "clustered", "diagonal", "graded"])
def test_tridiagonal_eigensolver(m, kind):
    rng = np.random.default_rng(m)
    a, b = rng.standard_normal((3, m)), np.abs(rng.standard_normal((3, m)))
    if kind == "clustered":
        a[:], b[:] = 1.0, 1e-9 * b
    elif kind == "diagonal":
        b[:] = 0.0
    elif kind == "graded":
        a *= 10.0 ** -np.linspace(0, 12, m)
        b *= 10.0 ** -np.linspace(0, 12, m)
    ev, first = q.tridiag_ritz(a, b)
    for k in range(3):
        T = np.diag(a[k]) + np.diag(b[k, :m - 1], 1) + np.diag(b[k, :m - 1], -1)
        norm = max(np.linalg.norm(T), 1e-300)
        tol = 10 * m * EPS * norm  # backward error of a sweep's m rotations per element, ten sweeps
        np.testing.assert_allclose(ev[k], np.linalg.eigvalsh(T), rtol=0, atol=tol)
        w = first[k] ** 2
        assert abs(w.sum() - 1) <= 10 * m * EPS
        for p, ref in ((1, T[0, 0]), (2, (T @ T)[0, 0]), (3, (T @ T @ T)[0, 0])):
            assert abs((w * ev[k] ** p).sum() - ref) <= p * tol * norm ** (p - 1)


def flip_operator(n_bits, n, fields=True):
    """sum_k c_k X_k (+ fields h_k Z_k) on the states 0 .. n-1, and its dense matrix."""
    H = q.SymbolicOpSum()
    D = np.zeros((n, n))
    i = np.arange(n)
    for k in range(n_bits):
        H.add_term(-0.3 - 0.1 * k, q.SymbolicPMROperator(f"{k}x"))
        j = i ^ (1 << k)
        ok = j < n
        D[j[ok], i[ok]] += -0.3 - 0.1 * k
        if fields:
            H.add_term(0.05 * (k + 1) ** 2, q.SymbolicPMROperator(f"{k}z"))
            D[i, i] += 0.05 * (k + 1) ** 2 * (2 * ((i >> k) & 1) - 1)
    lohi = np.zeros((n, 2), dtype=np.uint64)
    lohi[:, 0] = i
    return q.LazyOpSum(q.ZBasis(lohi), H), D


# dimensions around one row per thread and block (512, 1024), ncv around groups of eight Krylov vectors
@pytest.mark.parametrize("n,ncv", [(31, 8), (500, 9), (513, 16), (1023, 17), (1025, 24), (2048, 25), (3000, 40)])
@pytest.mark.parametrize("precision", ["f64", "mixed"])
def test_lowest_levels(n, ncv, precision):
    op, D = flip_operator(max(1, (n - 1).bit_length()), n)
    ref = np.linalg.eigvalsh(D)
    ev, vec, rep = q.diagonalise(op, nev=2, ncv=ncv, tol=1e-11, max_iter=500, seed=3, precision=precision)
    np.testing.assert_allclose(ev, ref[:2], rtol=0, atol=1e-9)
    r = D @ vec - vec * ev
    assert np.abs(r).max() < 1e-4 and np.abs(vec.T @ vec - np.eye(2)).max() < 1e-6


@pytest.mark.parametrize("precision", ["f64", "mixed"])
def test_invariant_subspace_inside_a_cycle(precision):
    """Without fields the spectrum of 6 commuting flips has few distinct levels, so the Krylov space closes before ncv:
    the solve continues from new directions and finds the lowest level's value and its neighbours."""
    n = 64
    H = q.SymbolicOpSum()
    for k in range(6):
        H.add_term(-1.0, q.SymbolicPMROperator(f"{k}x"))
    lohi = np.zeros((n, 2), dtype=np.uint64)
    lohi[:, 0] = np.arange(n)
    op = q.LazyOpSum(q.ZBasis(lohi), H)  # levels -6, -4 (x6), -2 (x15), ...
    ev, vec, _ = q.diagonalise(op, nev=4, ncv=20, tol=1e-10, max_iter=200, seed=1, precision=precision)
    assert abs(ev[0] + 6) < 1e-9
    assert np.all(np.isfinite(vec)) and np.abs(vec.T @ vec - np.eye(4)).max() < 1e-6
    assert np.all(np.abs(ev[1:] + 4) < 1e-6) or np.all(np.isin(np.round(ev, 6), [-6, -4, -2, 0, 2, 4, 6]))


@pytest.mark.parametrize("its", [1, 2, 127, 128, 129, 300])
def test_eigval0_around_its_batches(its):
    op, D = flip_operator(9, 400)
    kw = dict(seed=4, abs_tol=1e-10, rel_tol=1e-12, min_iterations=5, max_iterations=its)
    e, vec, n_it = q.eigval0(op, **kw)
    e1, none, n1 = q.eigval0(op, calc_eigenvector=False, **kw)
    assert none is None and e1 == e and n1 == n_it == its
    al, be = plain_lanczos(D, O.set_random_unit(400, 4), its)
    T = np.diag(al) + np.diag(be[:-1], 1) + np.diag(be[:-1], -1)
    np.testing.assert_allclose(e, np.linalg.eigvalsh(T)[0], rtol=0, atol=1e-10)
    assert np.all(np.isfinite(vec)) and np.linalg.norm(vec) > 0


def plain_lanczos(D, v, its):
    u, beta = np.zeros(len(v)), 0.0
    al, be = [], []
    for _ in range(its):
        w = D @ v - beta * u
        a = v @ w
        w -= a * v
        beta = np.linalg.norm(w)
        u, v = v, w / beta
        al.append(a)
        be.append(beta)
    return np.array(al), np.array(be)


def test_eigval0_stops_on_a_vanishing_beta():
    n = 64
    H = q.SymbolicOpSum()
    for k in range(6):
        H.add_term(-1.0, q.SymbolicPMROperator(f"{k}x"))
    lohi = np.zeros((n, 2), dtype=np.uint64)
    lohi[:, 0] = np.arange(n)
    op = q.LazyOpSum(q.ZBasis(lohi), H)  # seven distinct levels: the recurrence closes at the seventh step, whose
    # coefficients the reference leaves out
    kw = dict(abs_tol=1e-8, rel_tol=1e-16, min_iterations=10, max_iterations=400)
    e, vec, its = q.eigval0(op, seed=2, **kw)
    e_o, vec_o, its_o = O.eigval0_oracle(*op.triplets(), n, 2, **kw)
    assert its == its_o == 6 and abs(e - e_o) < 1e-10
    assert np.abs(vec - vec_o).max() < 1e-9 or np.abs(vec + vec_o).max() < 1e-9


# Gram tiles of 64 vectors: 8 operators x nvec images, nvec vectors
@pytest.mark.parametrize("nvec", [1, 3, 8, 9, 17])
@pytest.mark.parametrize("n", [15, 256, 700])
def test_expectations_tiles(nvec, n):
    """Off-diagonal, many-term, Z-carrying, diagonal and mixed operators against dense matrices."""
    lohi = np.zeros((n, 2), dtype=np.uint64)
    lohi[:, 0] = np.arange(n)
    specs = [["0+ 1-"], ["0x", "1x", "2+ 3-"], ["0+ 1- 2z"], ["2z"], ["1z", "0x"], ["3-"], ["0+ 1+ 2- 3-"], ["9x"]]
    ops, mats = [], []
    i = np.arange(n)
    for k, terms in enumerate(specs):
        H, M = q.SymbolicOpSum(), np.zeros((n, n))
        for t, s in enumerate(terms):
            op, c = q.SymbolicPMROperator(s), 0.5 + 0.25 * t + 0.1 * k
            H.add_term(c, op)
            for j in i:
                new, sign = op.applyState(int(j))
                if sign and new < n:
                    M[new, j] += c * sign
        ops.append(H)
        mats.append(M)
    psi = np.random.default_rng(5).standard_normal((n, nvec))
    expect, cross = q.expectations(q.ZBasis(lohi), ops, psi, cross=True)
    only, none = q.expectations(q.ZBasis(lohi), ops, psi)
    W = np.stack([M @ psi for M in mats])  # (ops, n, nvec)
    scale = n * np.abs(W).max() * max(np.abs(W).max(), np.abs(psi).max())
    np.testing.assert_allclose(expect, np.einsum("lni,nj->lij", W, psi), rtol=0, atol=8 * EPS * scale)
    np.testing.assert_allclose(cross, np.einsum("lni,mnj->lmij", W, W), rtol=0, atol=8 * EPS * scale)
    assert none is None and np.array_equal(only, expect)


# 8,191 / 8,192 rows: without and with a solve's own lookup cache; cut-off bases: some cached entries are empty
@pytest.mark.parametrize("pairs,n", [(0, 3618), (2, 8191), (2, 8192), (2, 20_011)])
def test_solves_with_their_own_cache(pairs, n):
    """Bitwise those of the row-per-thread kernel, which has no cache: the materialised sums are the same."""
    lat = workloads.lattice("pyro_1x2x1")
    g, B = workloads.ring_zeeman_params(5)
    lohi = q.enumerate_basis(lat, n_spinon_pairs=pairs)[:n]
    assert len(lohi) == n
    op = q.LazyOpSum(q.ZBasis(lohi), q.build_ring_zeeman(lat, g, B, Jpm=0.05 if pairs else 0.0))
    got = []
    for kernel in (1, 0):
        op.set_kernel(kernel)
        out = []
        for precision in ("f64", "mixed"):
            ev, vec, rep = q.diagonalise(op, nev=2, ncv=12, tol=1e-10, seed=4, precision=precision)
            assert rep.applies >= 50
            out += [ev, vec]
        out += list(q.eigval0(op, seed=3, max_iterations=60)[:2])
        out += list(q.ftlm([op, op], [2, 4], M=44, seed=6, precision="f64")[1])
        got.append(out)
    for a, b in zip(*got):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("scale", [1e-120, 1.0, 1e120])
@pytest.mark.parametrize("n", [300, 1025, 4097])
def test_eigval0_levels_and_scales(n, scale):
    """One to five blocks of rows, tridiagonals of one to several chunks, and spectra of any width: the lowest level of the
    dense matrix, scaled, and its vector."""
    bits = max(1, (n - 1).bit_length())
    H = q.SymbolicOpSum()
    for k in range(bits):
        H.add_term(-scale * (1 + 0.01 * k), q.SymbolicPMROperator(f"{k}x"))
        H.add_term(scale * 0.3 * (k + 1), q.SymbolicPMROperator(f"{k}z"))
    lohi = np.zeros((n, 2), dtype=np.uint64)
    lohi[:, 0] = np.arange(n)
    op = q.LazyOpSum(q.ZBasis(lohi), H)
    D = np.zeros((n, n))
    r, c, v = op.triplets(tol=0.0)
    np.add.at(D, (r, c), v / scale)
    w, V = np.linalg.eigh(D)
    its = min(n - 50, 700)
    e, vec, got = q.eigval0(op, seed=4, abs_tol=scale * 1e-13, rel_tol=1e-16, min_iterations=10, max_iterations=its)
    # 700 steps reach the lowest level to rounding (width below 150, multisection and recurrence of 1e-15 of it)
    assert abs(e / scale - w[0]) < 1e-11
    if scale < 1:
        return  # the stop rule divides by at least 1e-10, so the second pass ends at min_iterations
    # the second pass stops when the level moves by less than 1e-13: residual^2 <= about ten times that, times the width
    assert np.linalg.norm(D @ vec - w[0] * vec) < 1e-4 * np.linalg.norm(vec)

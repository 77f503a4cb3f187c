"""The bin index and the tile kernels' term tables where they can go wrong: full bins and shared tags (settled by
bisection), lookups that leave the basis, conjugate pairs stored as one entry, terms without literals, with more than
eight, and with Z factors.  Every apply against the oracle's push loop and, bitwise, the row-per-thread kernel, which
shares neither the index nor the tables."""
import numpy as np
import pytest

import qsi_subspace_ed_gb300 as q
from oracle import oracle as O
from qsi_subspace_ed_gb300 import workloads

pytestmark = pytest.mark.gpu


def opsum(specs):
    H = q.SymbolicOpSum()
    for c, s in specs:
        H.add_term(c, q.SymbolicPMROperator(s))
    return H


def integers(n, lo_shift=0, hi_shift=None):
    """States 0 .. n-1 with their low ten bits at lo_shift and the others higher (in the high word when given)."""
    i = np.arange(n, dtype=np.uint64)
    low, high = (i & np.uint64(1023)) << np.uint64(lo_shift), i >> np.uint64(10)
    out = np.zeros((n, 2), dtype=np.uint64)
    out[:, 0] = low if hi_shift is not None else low | (high << np.uint64(lo_shift + 10))
    if hi_shift is not None:
        out[:, 1] = high << np.uint64(hi_shift)
    return out


FLIPS = [(0.3 * (k + 1), f"{k}x") for k in range(10)]  # no literals: every row admits them
MIXED = [(0.7, "0+ 1-"), (0.7, "0- 1+"), (-0.4, "2+ 3- 4z"), (-0.4, "2- 3+ 4z"), (0.2, "5+ 6-"), (0.9, "5- 6+"),
         (0.1, "0+ 1- 2+ 3- 4+ 5- 6+ 7- 8+ 9-"), (0.1, "0- 1+ 2- 3+ 4- 5+ 6- 7+ 8- 9+"), (0.05, "1z"), (0.6, "7+")]
PAIRS = [(0.7, "0+ 1-"), (0.7, "0- 1+"), (0.7, "0+ 1-"), (0.2, "2+ 3-"), (0.2, "2- 3+"), (0.5, "4+ 5- 6+ 7- 8+ 9-"),
         (0.5, "4- 5+ 6- 7+ 8- 9+"), (0.3, "4+ 5- 6+ 7- 8+ 9-")]


def check(lohi, H, bits, terms=18):
    n = len(lohi)
    x = np.random.default_rng(3).standard_normal(n)
    x[::7] = 0.0
    x[3::11] = 1e-15  # not above the apply tolerance
    ref = O.apply_port(lohi, H.specs(), x, threads=1)
    b = q.ZBasis(lohi)
    op = q.LazyOpSum(b, H)
    op.set_kernel(0)
    row = np.zeros(n)
    op.evaluate(x, row)
    # two roundings per term and row (product, sum), in another order
    np.testing.assert_allclose(row, ref, rtol=0, atol=2 * terms * 2.3e-16 * max(np.abs(ref).max(), 1.0))
    X = np.stack([x] * 3, axis=1)
    for use in (1, 0):
        for w in bits:
            b.set_index(use_hash=True, bucket_bits=w)
            assert b.index_info()["hash"]
            op.set_kernel(1, use)
            y = np.full(n, 7.0)
            op.evaluate(x, y)
            assert np.array_equal(y, row), (use, w)
            Y = np.full_like(X, 7.0)
            op.apply_batched(X, Y)
            assert all(np.array_equal(Y[:, k], row) for k in range(3)), (use, w)
            op.materialise(True)
            y = np.full(n, 7.0)
            op.evaluate(x, y)
            assert np.array_equal(y, row), (use, w)
            op.materialise(False)


# 1023, 1024: the last states' flips leave the basis or not; 200,000 states in two buckets: 15-bit tags, shared ones
# in the thousands of bins, and bins that overflow
@pytest.mark.parametrize("n,bits", [(1, (1,)), (31, (1, 5)), (1023, (1, 8, 10)), (1024, (1, 8, 10)), (200_000, (1, 9, 18))])
@pytest.mark.parametrize("terms", ["flips", "mixed", "pairs"])
@pytest.mark.parametrize("place", [(0, None), (3, None), (0, 0), (0, 21)])
def test_applies_on_integer_bases(n, bits, terms, place):
    lo_shift, hi_shift = place
    if hi_shift == 21 and n < 1024:
        hi_shift = 0
    specs = {"flips": FLIPS, "mixed": MIXED, "pairs": PAIRS}[terms]
    if lo_shift:
        specs = [(c, " ".join(f"{int(t[:-1]) + lo_shift}{t[-1]}" for t in s.split())) for c, s in specs]
    check(integers(n, lo_shift, hi_shift), opsum(specs), bits)


@pytest.mark.parametrize("pairs", [0, 1, 2])
def test_applies_on_spinon_bases(pairs):
    """Closed (no pairs), and hopping whose images leave the basis (one and two pairs)."""
    lat = workloads.lattice("pyro_1x2x1")
    g, B = workloads.ring_zeeman_params(5)
    lohi = q.enumerate_basis(lat, n_spinon_pairs=pairs)
    check(lohi, q.build_ring_zeeman(lat, g, B, Jpm=0.05 if pairs else 0.0), (4, 14))


def test_one_sided_terms():
    """Rings without their conjugates: a non-symmetric operator, nothing to pair."""
    lat = workloads.lattice("pyro_1x2x1")
    H = q.SymbolicOpSum()
    for k, op in enumerate(q.get_ring_ops(lat)[0]):
        H.add_term(0.1 * (k + 1), op)
    check(q.enumerate_basis(lat), H, (6, 14))


def xor_terms(n_bits, most):
    """A term flipping each non-empty set of bits, up to `most` of them, every one with its own coefficient."""
    return [(0.01 * (m + 1), " ".join(f"{k}x" for k in range(n_bits) if (m >> k) & 1)) for m in range(1, min(most + 1, 1 << n_bits))]


# 30, 31, 32 distinct coefficients: 16- and 32-bit cache slots; 64, 65 terms on every row: lists of 2,048 and 2,080
# hits, around a slot's 11 bits of position; 1,023 terms: a list that no block's shared memory holds
@pytest.mark.parametrize("n", [40, 1000, 1024])
@pytest.mark.parametrize("most", [30, 31, 32, 64, 65, 1023])
def test_long_lists_and_many_coefficients(n, most):
    bits = max(6, (n - 1).bit_length())
    if most >= 1 << bits:
        pytest.skip("more terms than sets of bits")
    check(integers(n), opsum(xor_terms(bits, most)), (1, 8), terms=most)


@pytest.mark.parametrize("R", [1, 2, 3, 4, 5, 7, 8, 9, 15, 16, 17, 20, 32, 33])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("pairs", [0, 2])
def test_few_vectors(R, dtype, pairs):
    """Rows summed several at a time (R <= 16), with 16-byte gathers (FP32, 4 and 8) and one at a time: every column
    bitwise the one of a 33-column apply, plain and accumulating, for short lists, and materialised."""
    if R == 1 and dtype == np.float32:
        pytest.skip("one FP32 vector is summed in FP64, not double-float")
    lat = workloads.lattice("pyro_1x2x1")
    g, B = workloads.ring_zeeman_params(5)
    lohi = q.enumerate_basis(lat, n_spinon_pairs=pairs)[:20_011]  # cut off: some lookups leave the basis
    op = q.LazyOpSum(q.ZBasis(lohi), q.build_ring_zeeman(lat, g, B, Jpm=0.05))
    rng = np.random.default_rng(R)
    n = len(lohi)
    wide = rng.standard_normal((n, 33)).astype(dtype)
    wide[::5, ::3] = 0
    wide0 = rng.standard_normal((n, 33)).astype(dtype)
    for acc in (False, True):
        ref = wide0.copy()
        op.apply_batched(wide, ref, accumulate=acc)
        for cap in (8, 256):
            op.set_kernel(1, 1, list_cap=cap)
            for cached in (False, True):
                op.materialise(cached)
                X, Y = wide[:, :R].copy(), wide0[:, :R].copy()
                op.apply_batched(X, Y, accumulate=acc)
                assert np.array_equal(Y, ref[:, :R]), (acc, cap, cached)
            op.materialise(False)


@pytest.mark.parametrize("kept", [1, 2])
def test_pairs_that_leave_one_way(kept):
    """A third of the states that admit one operator of the pair on spins 0 and 1 are missing, so that only the other's
    images leave the basis, first or second in the pair; shared tags, so a lookup that takes a match for the state errs."""
    lohi = integers(200_000)
    i = np.arange(200_000)
    lohi = lohi[~(((i & 3) == 3 - kept) & ((i >> 10) % 3 == 0))]
    check(lohi, opsum(PAIRS[:2] + PAIRS[3:7]), (1, 9))


@pytest.mark.parametrize("R", [1, 3, 20])
@pytest.mark.parametrize("special", [False, True])
@pytest.mark.parametrize("add", [False, True])
def test_fp32_vectors_of_every_magnitude(R, special, add):
    """FP32 vectors summed in FP64, widened by integer instructions: zeros of both signs, subnormals, the tolerance's
    neighbours, the largest floats, infinities and NaN, bitwise as the row kernels' conversions."""
    lat = workloads.lattice("pyro_1x2x1")
    lohi = q.enumerate_basis(lat)
    g, B = workloads.ring_zeeman_params(5)
    op = q.LazyOpSum(q.ZBasis(lohi), q.build_ring_zeeman(lat, g, B))
    rng = np.random.default_rng(R)
    n = len(lohi)
    x = np.ldexp(rng.standard_normal((n, R)), rng.integers(-160, 120, (n, R))).astype(np.float32)
    pick = rng.integers(0, 12, (n, R))
    for k, v in enumerate([0.0, -0.0, 1e-15, np.nextafter(np.float32(1e-15), np.float32(1)), 1e-45, -1e-39]):
        x[pick == k] = v
    y0 = np.ldexp(rng.standard_normal((n, R)), rng.integers(-160, 60, (n, R))).astype(np.float32)
    if special:
        x[5::97], x[7::89], x[9::83] = np.inf, -np.inf, np.nan
    got = []
    for kernel, cached in ((0, False), (1, False), (1, True)):
        op.set_kernel(kernel, 3)  # batched sums in FP64 too
        if cached:
            op.materialise(True)
        y = y0.copy()
        op.apply_batched(x, y, accumulate=add)
        got.append(y)
    assert np.array_equal(got[0], got[1], equal_nan=True) and np.array_equal(got[0], got[2], equal_nan=True)


@pytest.mark.parametrize("R,chunk,width", [(32, 16, 0), (64, 0, 16), (128, 128, 8), (256, 256, 0), (256, 256, 8), (512, 512, 0), (512, 512, 16)])
def test_vectors_per_lane_and_pass(R, chunk, width):
    """Built-in and asked-for vectors per lane with passes of up to all vectors, wider than a warp of four-vector lanes
    too: bitwise the same, with the look-ups and materialised."""
    lat = workloads.lattice("pyro_1x2x1")
    g, B = workloads.ring_zeeman_params(5)
    op = q.LazyOpSum(q.ZBasis(q.enumerate_basis(lat)), q.build_ring_zeeman(lat, g, B))
    X = np.random.default_rng(R).standard_normal((op.rows(), R)).astype(np.float32)
    ref = np.zeros((op.rows(), R), dtype=np.float32)
    op.set_tuning(0, 0, which=1, vec_width=4)
    op.apply_batched(X, ref)
    op.set_tuning(0, chunk, which=1, vec_width=width)
    for cached in (False, True):
        op.materialise(cached)
        Y = np.zeros_like(ref)
        op.apply_batched(X, Y)
        assert np.array_equal(Y, ref), cached

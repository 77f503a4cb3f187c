// Device-side data structures shared by the CUDA translation units.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "qsi_internal.h"

namespace qsi {

// A 128-bit basis state as stored in HBM: x = low word, y = high word.
using state2 = ulonglong2;

// Pull-form off-diagonal term: applicability masks are those of the
// transposed operator, so a row state s is admitted when
// (s & down) == 0 && (s & up) == up, and its column is s ^ X.
// The matrix element is cs * (-1)^popcount(~s & Z).
struct PullTerm {
    uint64_t x0, x1, z0, z1, up0, up1, dn0, dn1;
    double cs;       // coefficient times construction sign
    int32_t has_z;
    float cs_hi;     // cs as a double-float pair (cs_hi + cs_lo), for FP32 accumulation
    float cs_lo;
    int32_t pad;
};

// Push-form term (the reference's own orientation; used for connectivity
// export and for generic diagonal terms).
struct PushTerm {
    uint64_t x0, x1, z0, z1, up0, up1, dn0, dn1;
    double c;
    int32_t sign;
    int32_t pad;
};

// The off-diagonal terms as the tile kernels stage them in shared memory.  Two consecutive terms with the same flip, Z
// mask and coefficient and opposite requirements (an operator and its conjugate) are one entry with its pair bit set:
// a row admits at most one of the two, so its hits and their order are those of the separate terms, at half the
// admission tests.  Literals are spin + 128 when the spin must be down.
struct TileTerms {
    const uint4* x;           // flipped bits, four words
    const double* cs;         // coefficient, and as a (hi, lo) float pair
    const float2* ff;
    const ulonglong2* z;      // Z masks (nullptr: no term has one)
    const uint2* lit8;        // up to eight literals, the last repeated, max_lits of them used (nullptr: lits)
    const uint32_t* pair;     // pair bits, 32 terms per word
    const uint16_t* lit_off;  // literal lists of any length, when some term has none or more than eight
    const uint8_t* lits;
    int n, n_lits, max_lits;
};

// Diagonal part: single-site pure-z terms grouped by weight w into masks,
// contributing w * (2 * popcount(s & M) - popcount(M)); remaining diagonal
// terms are evaluated one by one.
constexpr int kMaxZClasses = 32;
struct DiagSpec {
    int n_cls;
    int n_generic;
    double w2[kMaxZClasses];  // 2*w
    uint64_t m0[kMaxZClasses], m1[kMaxZClasses];
    double constant;  // -sum_k w_k * popcount(M_k)
};

// Sorted basis with a direct bucket table over the top `bits` bits below
// `shift`: bucket(s) = s >> shift; tab[v] = [first, end) is the index range of
// the states in bucket v ({0, 0} for an empty bucket), so one 8-byte load
// gives a lookup both bounds.
struct BasisView {
    const state2* states;
    const uint2* tab;
    int64_t n;
    int shift;
    uint32_t n_buckets;
};

constexpr uint32_t kEmpty = 0xFFFFFFFFu;

__device__ __forceinline__ bool less128(uint64_t alo, uint64_t ahi, uint64_t blo, uint64_t bhi) {
    return ahi < bhi || (ahi == bhi && alo < blo);
}

__device__ __forceinline__ uint64_t bucket_of(const BasisView& B, uint64_t lo, uint64_t hi, bool& in_range) {
    uint64_t v;
    if (B.shift >= 64) {
        v = hi >> (B.shift - 64);
    } else if (B.shift == 0) {
        v = lo;
        if (hi) v = ~0ULL;
    } else {
        if (hi >> B.shift) v = ~0ULL;
        else v = (hi << (64 - B.shift)) | (lo >> B.shift);
    }
    in_range = v < B.n_buckets;
    return v;
}

// Exact index of state (lo, hi) in [a, b), or -1: lower-bound bisection.  The state at the final position was loaded
// by the bisection itself whenever that position lies inside the range (the last probe that moved the upper end
// there), and a search that never moved the upper end ends past the range, where the state cannot be: no reload
// either way.
__device__ __forceinline__ int64_t range_find(const state2* __restrict__ states, uint32_t a, uint32_t b, uint64_t lo,
                                              uint64_t hi) {
    state2 e = make_ulonglong2(0, 0);
    bool seen = false;  // e holds states[b]
    while (a < b) {
        const uint32_t m = a + ((b - a) >> 1);
        const state2 t = __ldg(states + m);
        if (less128(t.x, t.y, lo, hi)) {
            a = m + 1;
        } else {
            b = m;
            e = t;
            seen = true;
        }
    }
    return (seen && e.x == lo && e.y == hi) ? (int64_t)a : -1;
}

// Exact index of state (lo, hi) in the basis, or -1: bisection over the state's bucket.
__device__ __forceinline__ int64_t basis_find(const BasisView& B, uint64_t lo, uint64_t hi) {
    bool ok;
    const uint64_t v = bucket_of(B, lo, hi, ok);
    if (!ok) return -1;
    const uint2 ab = __ldg(B.tab + v);
    return range_find(B.states, ab.x, ab.y, lo, hi);
}

// Hash index of the basis: a direct-mapped cache of bucket searches in bins of eight 4-byte slots (one 32-byte
// sector, one load instruction).  The states of a bucket [a, b) share the bins bin_of(a) .. bin_of(b - 1), one bin per
// 3.2 states of the basis, so neighbouring states' bins are neighbours too; a hash of the state picks its bin and a
// tag, and its slot holds the tag in the upper bits and the state's offset from a in the lower off_bits.  A lookup is
// three dependent loads and no loop: the bucket's bounds, its bin, and what it was looked up for.
//
// The bins decide nothing alone.  A state that finds its bin full is left out (0.1-0.3% of the states measured), and
// a state whose tag another state of its bin carries too has both slots marked with offset off_mask (k_bins_check),
// so for a state of the basis its first match is itself, marked, or absent with a full bin; the last two are settled
// by bisecting the bucket.  A state outside the basis may match a tag by chance: callers that can meet one compare
// the state found (kClosed = false).
//
// Why bins: a table of 16-byte {state, index} slots with linear probing (load 1/2, 1.5 probes on average) made a
// warp wait for its unluckiest lane, four to six dependent loads per lookup, and spent 340 warp instructions per 32
// lookups in hash arithmetic and probe loops; it also took 32 bytes per state where the bins take 10.  FP64 apply of
// the 64-spin Q=0 basis (2.9 M states): 615 us with that table, 321 with the bins; 96-spin 12.12.12.12 sector (196 M):
// 69.4 -> 37.1 ms.
struct BinView {
    BasisView B;
    const uint32_t* bins;
    uint32_t off_mask;
};
constexpr int kBinSlots = 8;

__host__ __device__ __forceinline__ uint32_t bin_of(uint32_t i) { return (i >> 2) + (i >> 4); }

// Bin selector (a 32-bit fraction) and tag bits of a state of at most 96 bits: a multilinear hash of its words, its
// 64-bit sum folded once for the bin and once more for the tag.
__device__ __forceinline__ void bin_hash(uint32_t w0, uint32_t w1, uint32_t w2, uint32_t& frac, uint32_t& tag) {
    const uint64_t h = (uint64_t)w0 * 0x9E3779B1u + (uint64_t)w1 * 0x85EBCA6Bu + (uint64_t)w2 * 0xC2B2AE35u;
    frac = (uint32_t)(h >> 32) * 0x9E3779B1u + (uint32_t)h;
    tag = (frac ^ (frac >> 15)) * 0x85EBCA6Bu + (uint32_t)h;
}
// The tag in a slot's upper bits; the all-ones tag belongs to free slots (kEmpty).
__device__ __forceinline__ uint32_t slot_tag(uint32_t tag, uint32_t off_mask) {
    const uint32_t t = tag & ~off_mask;
    return t == ~off_mask ? 0u : t;
}
__device__ __forceinline__ uint32_t pick_bin(uint2 ab, uint32_t frac) {
    const uint32_t f0 = bin_of(ab.x);
    return f0 + __umulhi(frac, bin_of(ab.y - 1) - f0 + 1);
}
__device__ __forceinline__ void load_bin(const uint32_t* p, uint32_t (&w)[kBinSlots]) {
    asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]), "=r"(w[4]), "=r"(w[5]), "=r"(w[6]), "=r"(w[7])
        : "l"(p));
}
// Smallest slot ^ tag of a bin: below off_mask it is the offset of the slot that carries the tag (an offset beyond the
// bucket's size belongs to a neighbouring bucket that shares the bin), off_mask a marked slot, above it no slot
// carries the tag.
__device__ __forceinline__ uint32_t bin_match(const uint32_t (&w)[kBinSlots], uint32_t tag) {
    uint32_t m = w[0] ^ tag;
#pragma unroll
    for (int k = 1; k < kBinSlots; ++k) m = min(m, w[k] ^ tag);
    return m;
}

// Column lookups.  Every class takes the admitted rows' states as 32-bit words with the bucket number (see
// term_words) and returns a candidate index per state, kEmpty when the state is not in the basis; a candidate of a
// class with kCheck set has to be compared with the state at that index (matches()).  For the materialised
// operator's cache, cursor(tile, lane) is where the row's entries start, once per tile, and k0 the admission ordinal
// of the batch's first term.
struct Word4 {
    uint32_t w0, w1, w2, w3;  // w3: the bucket number for BinView lookups, bits 96..127 otherwise
};
__device__ __forceinline__ Word4 split_state(uint64_t lo, uint64_t hi) {
    return Word4{(uint32_t)lo, (uint32_t)(lo >> 32), (uint32_t)hi, (uint32_t)(hi >> 32)};
}

struct LookupTable {
    BasisView B;
    static constexpr int kNB = 4, kMinBlocks = 3;  // lookups per batch per lane, resident 256-thread blocks
    static constexpr bool kCheck = false;
    __device__ __forceinline__ int64_t find(uint64_t lo, uint64_t hi) const { return basis_find(B, lo, hi); }
    __device__ __forceinline__ Word4 words(uint64_t lo, uint64_t hi) const { return split_state(lo, hi); }
    __device__ __forceinline__ uint64_t cursor(int64_t, int) const { return 0; }
    __device__ __forceinline__ bool matches(const Word4&, uint32_t) const { return true; }
    template <int NB>
    __device__ __forceinline__ void find_batch(const Word4 (&s)[NB], int n, uint32_t (&J)[NB], uint64_t = 0, int = 0) const {
#pragma unroll
        for (int u = 0; u < NB; ++u) {
            J[u] = kEmpty;
            if (u < n)
                J[u] = (uint32_t)basis_find(B, (uint64_t)s[u].w1 << 32 | s[u].w0, (uint64_t)s[u].w3 << 32 | s[u].w2);
        }
    }
};

// kClosed: every state looked up is in the basis (qsi_op::closed), so a match needs no comparison.  Bucket numbers
// are linear over XOR, so a row's number XOR a term's is the flipped state's; terms that flip a bit above the basis's
// highest never land in it and are pruned before they get here.
template <bool kClosed>
struct LookupBins {
    BinView H;
    // two lookups in flight per lane at 64 registers: 318 us on the 64-spin Q=0 basis, against 397 / 390 / 506 with
    // one, three or four (the last two spill), and 412 at three resident blocks
    static constexpr int kNB = 2, kMinBlocks = 4;
    static constexpr bool kCheck = !kClosed;
    __device__ __forceinline__ Word4 words(uint64_t lo, uint64_t hi) const {
        bool ok;
        Word4 s = split_state(lo, hi);
        s.w3 = (uint32_t)bucket_of(H.B, lo, hi, ok);
        return s;
    }
    __device__ __forceinline__ uint64_t cursor(int64_t, int) const { return 0; }
    __device__ __forceinline__ bool matches(const Word4& s, uint32_t J) const {
        if (kClosed) return true;
        const uint4 e = __ldg(reinterpret_cast<const uint4*>(H.B.states + J));
        return e.x == s.w0 && e.y == s.w1 && e.z == s.w2 && e.w == 0;
    }
    template <int NB>
    __device__ __forceinline__ void find_batch(const Word4 (&s)[NB], int n, uint32_t (&J)[NB], uint64_t = 0, int = 0) const {
        uint2 ab[NB];
#pragma unroll
        for (int u = 0; u < NB; ++u) ab[u] = (u < n) ? __ldg(H.B.tab + s[u].w3) : make_uint2(0, 0);
        uint32_t w[NB][kBinSlots], tag[NB];
#pragma unroll
        for (int u = 0; u < NB; ++u) {
            uint32_t frac;
            bin_hash(s[u].w0, s[u].w1, s[u].w2, frac, tag[u]);
            tag[u] = slot_tag(tag[u], H.off_mask);
            if (ab[u].x != ab[u].y) load_bin(H.bins + (size_t)pick_bin(ab[u], frac) * kBinSlots, w[u]);
        }
#pragma unroll
        for (int u = 0; u < NB; ++u) {
            J[u] = kEmpty;
            if (ab[u].x == ab[u].y) continue;
            const uint32_t m = bin_match(w[u], tag[u]);
            if (m < ab[u].y - ab[u].x) J[u] = ab[u].x + m;
            else if (kClosed || m == H.off_mask || w[u][kBinSlots - 1] != kEmpty)
                J[u] = (uint32_t)range_find(H.B.states, ab[u].x, ab[u].y, (uint64_t)s[u].w1 << 32 | s[u].w0, s[u].w2);
        }
    }
    // One state of any width.
    __device__ __forceinline__ int64_t find(uint64_t lo, uint64_t hi) const {
        bool ok;
        bucket_of(H.B, lo, hi, ok);
        if (!ok || (hi >> 32)) return -1;
        const Word4 s[1] = {words(lo, hi)};
        uint32_t J[1];
        find_batch<1>(s, 1, J);
        return (J[0] != kEmpty && matches(s[0], J[0])) ? (int64_t)J[0] : -1;
    }
};

// The materialised operator's lookup cache (qsi_op_materialise): the column of every admitted term of every row,
// kEmpty for a column outside the basis, in the order the tile kernels visit them (with the term's index and the
// sign of its matrix element on the row beside it, for the single-vector kernel that reads only the cache).  Tile t's entries start at
// 32 * off[t]; the row in lane l has its k-th admitted term at 32 * (off[t] + k) + l, so a warp reads one
// coalesced 128-byte line per admission ordinal.  Results are those of the lookups it replaces, bit for bit.
// Bit 31 of a cached column holds the sign of the term's matrix element on that row (columns are below 2^31).
constexpr uint32_t kCacheNeg = 0x80000000u;
struct CacheView {
    const uint32_t* cols;
    const uint64_t* off;
};
struct LookupCache {
    CacheView C;
    static constexpr int kNB = 8, kMinBlocks = 3;
    static constexpr bool kCheck = false;
    __device__ __forceinline__ Word4 words(uint64_t, uint64_t) const { return Word4{0, 0, 0, 0}; }
    __device__ __forceinline__ uint64_t cursor(int64_t tile, int lane) const { return C.off[tile] * 32 + lane; }
    __device__ __forceinline__ bool matches(const Word4&, uint32_t) const { return true; }
    template <int NB>
    __device__ __forceinline__ void find_batch(const Word4 (&)[NB], int n, uint32_t (&J)[NB], uint64_t cur, int k0) const {
#pragma unroll
        for (int u = 0; u < NB; ++u) {
            J[u] = kEmpty;
            if (u < n) {
                const uint32_t c = __ldg(C.cols + cur + (uint64_t)(k0 + u) * 32);
                J[u] = (c == kEmpty) ? kEmpty : (c & ~kCacheNeg);
            }
        }
    }
};

// 32x32 bit-matrix transpose across a warp: lane r holds row r (bit c = [r][c]);
// on return lane r holds column r (bit c = [c][r]).  Five shuffle stages,
// each swapping the off-diagonal j x j blocks.
__device__ __forceinline__ uint32_t warp_transpose32(uint32_t w, int lane) {
    const uint32_t m0[5] = {0x0000FFFFu, 0x00FF00FFu, 0x0F0F0F0Fu, 0x33333333u, 0x55555555u};
#pragma unroll
    for (int k = 0; k < 5; ++k) {
        const int j = 16 >> k;
        const uint32_t m = m0[k];
        const uint32_t x = __shfl_xor_sync(0xffffffffu, w, j);
        w = (lane & j) ? ((w & ~m) | ((x & ~m) >> j)) : ((w & m) | ((x & m) << j));
    }
    return w;
}

__device__ __forceinline__ double diag_value(const DiagSpec& D, const PushTerm* gen, uint64_t s0, uint64_t s1) {
    double d = D.constant;
    for (int k = 0; k < D.n_cls; ++k) d += D.w2[k] * (double)(__popcll(s0 & D.m0[k]) + __popcll(s1 & D.m1[k]));
    for (int k = 0; k < D.n_generic; ++k) {
        const PushTerm& T = gen[k];
        bool ok = ((s0 & T.dn0) | (s1 & T.dn1)) == 0 && (s0 & T.up0) == T.up0 && (s1 & T.up1) == T.up1;
        if (!ok) continue;
        int par = (__popcll(~s0 & T.z0) + __popcll(~s1 & T.z1)) & 1;
        d += T.c * (double)(T.sign * (1 - 2 * par));
    }
    return d;
}

}  // namespace qsi

#define QSI_CUDA(call)                                                                            \
    do {                                                                                          \
        cudaError_t e_ = (call);                                                                  \
        if (e_ != cudaSuccess) {                                                                  \
            return ::qsi::fail(e_ == cudaErrorMemoryAllocation ? QSI_OOM : QSI_CUDA_ERROR,        \
                               "%s: %s (%s:%d)", #call, cudaGetErrorString(e_), __FILE__, __LINE__); \
        }                                                                                         \
    } while (0)

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
    int reversible;           // every pair's requirements are on spins it flips: each operator undoes the other
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

// Conversions between FP32 and FP64 with integer instructions: the conversion instructions run on GB300's FP64 pipe, 17-20
// cycles per warp each, where a materialised apply of an FP32 vector has one multiply-add per hit (64-spin Q=0 basis:
// 178 us with them, 90 without).
// (double)x exactly; kNormal: x is known to be neither zero nor subnormal.
template <bool kNormal = false>
__device__ __forceinline__ double widen(float x) {
    const uint32_t b = __float_as_uint(x), m = b & 0x7FFFFFFFu;
    uint32_t hi = (m >> 3) + 0x38000000u, lo = b << 29;  // exponent bias 127 -> 1023
    if (m >= 0x7F800000u) {
        hi += 0x38000000u;  // infinity, NaN
    } else if (!kNormal && m < 0x00800000u) {  // m * 2^-149, m exact as a float
        const uint32_t c = __float_as_uint((float)m);
        hi = m ? (c >> 3) + 0x38000000u - (149u << 20) : 0u;
        lo = c << 29;
    }
    return __hiloint2double((int)(hi | (b & 0x80000000u)), (int)lo);
}
__device__ __forceinline__ double widen(double x) { return x; }
template <bool kNormal>
__device__ __forceinline__ double widen(double x) {
    return x;
}

// v as a (hi, lo) float pair: hi the nearest float, lo the nearest float to the rest.
__device__ __forceinline__ float2 split_f64(double v) {
    const uint64_t u = (uint64_t)__double_as_longlong(v);
    const int e = (int)(u >> 52) & 0x7FF;
    if ((uint32_t)(e - 960) > 180u) {  // zero; outside 2^-63 .. 2^118, where hi or lo may not be normal floats
        if ((u << 1) == 0) return make_float2(__uint_as_float((uint32_t)(u >> 32)), 0.f);
        const float h = (float)v;
        return make_float2(h, (float)(v - (double)h));
    }
    const uint64_t m = (u & 0xFFFFFFFFFFFFFull) | 0x10000000000000ull;
    const uint32_t q = (uint32_t)((m + 0x0FFFFFFF + ((m >> 29) & 1)) >> 29);  // to nearest, ties to even
    const int rest = (int)((uint32_t)m - (q << 29));                         // m - q 2^29, at most 2^28
    const uint32_t sign = (uint32_t)(u >> 32) & 0x80000000u;
    const float h = __uint_as_float((((uint32_t)(e - 896) << 23) + (q - 0x800000u)) | sign);
    const float l = (float)rest * __uint_as_float((uint32_t)(e - 948) << 23 | sign);  // 2^(e - 1075)
    return make_float2(h, l);
}

// Sorted basis with a direct bucket table over the `bits` highest bits in which
// its states differ: bucket(s) = (s ^ top) >> shift, top the bits above them that
// all states share (spins that are up everywhere; with those in the bucket
// number all states of such a basis were in one bucket: 16 flips on 2^24
// patterns with spin 64 up took 7.1 ms, 1.2 without); tab[v] = {first, size} is the
// index range of the states in bucket v ({0, 0} for an empty bucket), so one
// 8-byte load gives a lookup both bounds.
struct BasisView {
    const state2* states;
    const uint2* tab;
    int64_t n;
    int shift;
    uint32_t n_buckets;
    uint64_t top0, top1;
};

constexpr uint32_t kEmpty = 0xFFFFFFFFu;

__device__ __forceinline__ bool less128(uint64_t alo, uint64_t ahi, uint64_t blo, uint64_t bhi) {
    return ahi < bhi || (ahi == bhi && alo < blo);
}

__device__ __forceinline__ uint64_t bucket_of(const BasisView& B, uint64_t lo, uint64_t hi, bool& in_range) {
    lo ^= B.top0;
    hi ^= B.top1;
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

// The 32 bits from `shift` on, linear over XOR: that of a state of the basis XOR that of the shared bits is its bucket.
__device__ __forceinline__ uint32_t bucket_word(const BasisView& B, uint64_t lo, uint64_t hi) {
    if (B.shift >= 64) return (uint32_t)(hi >> (B.shift - 64));
    return (uint32_t)(B.shift == 0 ? lo : (hi << (64 - B.shift)) | (lo >> B.shift));
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
    const uint2 t = __ldg(B.tab + v);
    return range_find(B.states, t.x, t.x + t.y, lo, hi);
}

// Hash index of the basis: a direct-mapped cache of bucket searches in bins of eight 4-byte slots (one 32-byte
// sector, one load instruction).  The states of a bucket {a, m} share the bins first_bin(a) .. first_bin(a) +
// first_bin(m), one bin per two states of the basis, so neighbouring states' bins are neighbours too.  (One per 3.2
// or 2.7 states leaves more states out, and one lookup in the slow path holds its warp: 5.37 and 5.02 ms against
// 4.93 for the apply of the 96-spin 8.8.16.16 sector.)  A state's
// key, a 64-bit hash, picks its bin with the upper word and gives a tag with the lower; its slot holds the tag in the
// upper bits and the state's offset from a in the lower off_bits.  A lookup is three dependent loads and no loop: the
// bucket's bounds, its bin, and what it was looked up for.
//
// Keys are linear over XOR (each spin has a 64-bit word, a state's key is the XOR of its up spins'), and so are bucket
// numbers: the key and the bucket of a flipped state are those of the row XOR those of the term's flips, three XORs per
// lookup, with the rows' keys stored (8 bytes per state) and the terms' computed when they are staged.
//
// The bins decide nothing alone.  A state that finds its bin full is left out (few in a thousand), and
// a state whose tag another state of its bin carries too has both slots marked with offset off_mask - 1 (k_bins_check),
// so for a state of the basis its first match is itself, marked, or absent with a full bin; the last two are settled
// by bisecting the bucket.  Offset off_mask stays unused: with it a slot of the all-ones tag would be a free slot
// (kEmpty), and its full bin one with room, whose left-out states no lookup would find.  The shorter the tags, the
// likelier: a bucket of 2^24 states leaves eight bits, and so many are in one bucket where a few others lie far above
// them.  A state outside the basis may match a tag by chance: callers that can meet one compare the state found
// (kClosed = false).
//
// Why bins: a table of 16-byte {state, index} slots with linear probing (load 1/2, 1.5 probes on average) made a
// warp wait for its unluckiest lane, four to six dependent loads per lookup, and spent 340 warp instructions per 32
// lookups in hash arithmetic and probe loops.  FP64 apply of the 64-spin Q=0 basis (2.9 M states): 615 us with that
// table, 321 with bins of a multilinear hash per lookup, 280 with linear keys.
struct BinView {
    BasisView B;
    const uint32_t* bins;
    const uint2* keys;  // per state: {bin fraction, tag bits}
    uint32_t off_mask;
};
constexpr int kBinSlots = 8;

__host__ __device__ __forceinline__ uint32_t first_bin(uint32_t i) { return i >> 1; }

__device__ __forceinline__ uint2 state_key(uint64_t lo, uint64_t hi) {
    uint64_t k = 0;
    for (int w = 0; w < 2; ++w)
        for (uint64_t rest = w ? hi : lo; rest; rest &= rest - 1) {
            uint64_t z = (uint64_t)(64 * w + __ffsll((long long)rest)) * 0x9E3779B97F4A7C15ULL;  // splitmix64
            z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
            z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
            k ^= z ^ (z >> 31);
        }
    return make_uint2((uint32_t)(k >> 32), (uint32_t)k);
}
// The bin of a key: a multiplication breaks the linearity, which would send whole families of states that differ by a
// few independent flips to one bin (at one bin per 3.2 states, bins of up to 34 states and 1.0% of the 96-spin
// 8.8.16.16 basis left out instead of 0.4%).
__device__ __forceinline__ uint32_t pick_bin(uint2 bucket, uint32_t k0, uint32_t k1) {
    return first_bin(bucket.x) + __umulhi(__umulhi(k0, 0x9E3779B1u) ^ k1, first_bin(bucket.y) + 1);
}
__device__ __forceinline__ void load_bin(const uint32_t* p, uint32_t (&w)[kBinSlots]) {
    asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]), "=r"(w[4]), "=r"(w[5]), "=r"(w[6]), "=r"(w[7])
        : "l"(p));
}
// Smallest slot ^ tag of a bin: below off_mask - 1 it is the offset of the slot that carries the tag (an offset beyond the
// bucket's size belongs to a neighbouring bucket that shares the bin), off_mask - 1 a marked slot; from off_mask on
// no slot carries the tag (off_mask itself: a free slot met by the all-ones tag).
__device__ __forceinline__ uint32_t bin_match(const uint32_t (&w)[kBinSlots], uint32_t tag) {
    uint32_t m = w[0] ^ tag;
#pragma unroll
    for (int k = 1; k < kBinSlots; ++k) m = min(m, w[k] ^ tag);
    return m;
}

// Column lookups.  Every class describes rows and terms by four words whose XOR describes the flipped state, and
// returns for flipped states an index, kEmpty when the state is not in the basis.  state(u) gives the whole flipped
// state u where the words do not settle a lookup.
struct Word4 {
    uint32_t w0, w1, w2, w3;
};
__device__ __forceinline__ Word4 flip_words(const Word4& a, const uint4& x) {
    return Word4{a.w0 ^ x.x, a.w1 ^ x.y, a.w2 ^ x.z, a.w3 ^ x.w};
}

struct LookupTable {
    BasisView B;
    static constexpr int kNB = 4, kMinBlocks = 3;  // lookups per batch per lane, resident 256-thread blocks
    __device__ __forceinline__ Word4 row_words(int64_t, const state2 s) const {
        return Word4{(uint32_t)s.x, (uint32_t)(s.x >> 32), (uint32_t)s.y, (uint32_t)(s.y >> 32)};
    }
    __device__ __forceinline__ uint4 term_words(const uint4 x) const { return x; }
    template <int NB, class F>
    __device__ __forceinline__ void find_batch(const Word4 (&s)[NB], int n, uint32_t (&J)[NB], F&&) const {
#pragma unroll
        for (int u = 0; u < NB; ++u) {
            J[u] = kEmpty;
            if (u < n)
                J[u] = (uint32_t)basis_find(B, (uint64_t)s[u].w1 << 32 | s[u].w0, (uint64_t)s[u].w3 << 32 | s[u].w2);
        }
    }
};

// kClosed: every state looked up is in the basis (qsi_op::closed), so a match needs no comparison.  Terms that flip a
// bit which all states share never land in the basis and are pruned before they get here.
template <bool kClosed>
struct LookupBins {
    BinView H;
    // two lookups in flight per lane at 64 registers: 282 us on the 64-spin Q=0 basis, against 373 with one (at 48
    // registers), 317 with three and 342 with four at three resident blocks
    static constexpr int kNB = 2, kMinBlocks = 4;
    __device__ __forceinline__ Word4 row_words(int64_t row, const state2 s) const {
        const uint2 k = row < H.B.n ? __ldg(H.keys + row) : make_uint2(0, 0);
        return Word4{bucket_word(H.B, s.x, s.y), k.x, k.y, 0};
    }
    __device__ __forceinline__ uint4 term_words(const uint4 x) const {
        const uint64_t lo = (uint64_t)x.y << 32 | x.x, hi = (uint64_t)x.w << 32 | x.z;
        const uint2 k = state_key(lo, hi);
        return make_uint4(bucket_word(H.B, lo ^ H.B.top0, hi ^ H.B.top1), k.x, k.y, 0);  // the shared bits taken out here
    }
    template <int NB, class F>
    __device__ __forceinline__ void find_batch(const Word4 (&s)[NB], int n, uint32_t (&J)[NB], F&& state) const {
        uint2 bucket[NB];
#pragma unroll
        for (int u = 0; u < NB; ++u) bucket[u] = (u < n) ? __ldg(H.B.tab + s[u].w0) : make_uint2(0, 0);
        uint32_t w[NB][kBinSlots];
#pragma unroll
        for (int u = 0; u < NB; ++u)
            if (kClosed ? u < n : bucket[u].y != 0) load_bin(H.bins + (size_t)pick_bin(bucket[u], s[u].w1, s[u].w2) * kBinSlots, w[u]);
#pragma unroll
        for (int u = 0; u < NB; ++u) {
            J[u] = kEmpty;
            if (kClosed ? u >= n : bucket[u].y == 0) continue;
            const uint32_t m = bin_match(w[u], s[u].w2 & ~H.off_mask);
            if (m < bucket[u].y) {
                J[u] = bucket[u].x + m;
                if (!kClosed) {
                    const state2 t = state(u), e = __ldg(H.B.states + J[u]);
                    if (e.x != t.x || e.y != t.y) J[u] = kEmpty;
                }
            } else if (kClosed || m == H.off_mask - 1 || w[u][kBinSlots - 1] != kEmpty) {
                const state2 t = state(u);
                J[u] = (uint32_t)range_find(H.B.states, bucket[u].x, bucket[u].x + bucket[u].y, t.x, t.y);
            }
        }
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
    const void* tids;  // term of every entry: uint8, or uint16 beyond 256 terms
    int tid_bytes;
};
struct LookupCache {
    CacheView C;
    __device__ __forceinline__ uint4 term_words(const uint4 x) const { return x; }
    __device__ __forceinline__ uint64_t cursor(int64_t tile, int lane) const { return C.off[tile] * 32 + lane; }
    __device__ __forceinline__ uint32_t term(uint64_t at) const {
        return C.tid_bytes == 1 ? __ldg((const uint8_t*)C.tids + at) : __ldg((const uint16_t*)C.tids + at);
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

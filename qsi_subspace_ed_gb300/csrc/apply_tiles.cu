// Bit-sliced tile kernels of the pull-gather apply, the materialised operator's kernels, and the hash index.
//
// A warp owns a tile of 32 consecutive basis rows.  The tile's 32 states are
// transposed with warp shuffles into one 32-bit word per spin (bit l = spin
// of row l), so one lane evaluates one off-diagonal term for all 32 rows with
// a few AND/XOR operations over that term's literals (the spins its
// transposed up/down masks constrain).  A second transpose hands each row its
// admitted terms as a bit set, visited in term order, so every row is summed
// in the same fixed order as the one-row-per-thread kernel (deterministic,
// bit-identical results).
//
// Single vector: each lane finds its own row's columns and gathers x.
// Batched (R vectors, [row][R] layout): lanes first look up all columns of
// the tile, term by term, into a shared-memory hit list; then the warp walks
// the list row by row and gathers each column's R values with coalesced loads.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <condition_variable>
#include <cstring>
#include <map>
#include <mutex>
#include <vector>
#include <type_traits>

#include <cub/device/device_scan.cuh>

#include "qsi_device.cuh"
#include "qsi_handles.h"

namespace qsi {

struct TileParams {
    BasisView B;
    TileTerms T;
    DiagSpec D;
    const double* diag;  // per-row diagonal, precomputed with diag_value
    const float2* diag_ff;  // the same as (hi, lo) float pairs
    int nwords;
    int vchunk;             // vectors per pass of the 16-byte batched kernel (0: as many as 32 lanes hold)
    // operator families (family mode kernels only): the terms' coefficients encode their class as +-(class + 1)
    // and fcoef[class * fR + column] is the coefficient of that class in each column's operator
    const double* fcoef = nullptr;
    int fR = 1;
};

static TileParams tile_params(const qsi_op* op, int vchunk) {
    return TileParams{op->basis->view(), op->tile, op->diag, op->d_diag, op->d_diag_ff, op->nwords, vchunk};
}

// Family mode: the coefficient of a hit whose term's coefficient encodes +-(class + 1), for column col.
__device__ __forceinline__ double fam_coef(const TileParams& P, double enc, int col) {
    const double c = P.fcoef[((int)(fabs(enc) + 0.5) - 1) * P.fR + col];
    return enc < 0 ? -c : c;
}
// Family mode: the diagonal of state s for column col, sum over the single-site z groups of the template's
// diagonal (weight +-(class + 1) each) of coefficient(class) * sign * (2 popcount(s & M) - |M|), in group order.
__device__ __forceinline__ double fam_diag(const TileParams& P, uint64_t s0, uint64_t s1, int col) {
    double d = 0.0;
    for (int k = 0; k < P.D.n_cls; ++k) {
        const double w = 0.5 * P.D.w2[k];
        const int cls = (int)(fabs(w) + 0.5) - 1;
        const int cnt = __popcll(P.D.m0[k]) + __popcll(P.D.m1[k]);
        const int v = 2 * (__popcll(s0 & P.D.m0[k]) + __popcll(s1 & P.D.m1[k])) - cnt;
        const double c = P.fcoef[cls * P.fR + col];
        d += (w < 0 ? -c : c) * (double)v;
    }
    return d;
}

// |x| > 1e-15 (APPLY_TOL, operator_matrix.hpp:113) as integer compares on the
// bit pattern: magnitude above the threshold and not a NaN.  For FP32 x the
// threshold is the largest float whose value is <= 1e-15, so the test equals
// fabs((double)x) > 1e-15 exactly.
constexpr uint64_t kTolBitsF64 = 0x3CD203AF9EE75616ULL;  // 1e-15
constexpr uint32_t kTolBitsF32 = 0x26901D7CU;            // largest float <= 1e-15
// The FP64 word is split by an opaque move: written as a mask of the 64-bit pattern, the sign clear compiles to an
// FP64 |v| (a DADD, which takes GB300's FP64 pipe 20 cycles per warp where the multiply-add the test guards takes
// 17), and the materialised apply, bound by that pipe, issued one for every entry slot (96-spin 8.8.16.16 sector,
// 30.8 M states: 3.63 -> 2.45 ms; five FP64 vectors on a 64-spin sector of 443,256 states: 838 -> 517 us).
__device__ __forceinline__ bool above_tol(double v) {
    uint32_t lo, hi;
    asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "d"(v));
    const uint64_t m = ((uint64_t)(hi & 0x7FFFFFFFu) << 32) | lo;
    return m - (kTolBitsF64 + 1) <= 0x7FF0000000000000ULL - (kTolBitsF64 + 1);  // tolerance < m <= inf, one compare
}
__device__ __forceinline__ bool above_tol(float v) {
    const uint32_t m = __float_as_uint(v) & 0x7FFFFFFFu;
    return m - (kTolBitsF32 + 1) <= 0x7F800000u - (kTolBitsF32 + 1);  // kTolBitsF32 < m <= inf, one compare
}
// v where the tolerance test admits it (or keep is set), else 0: selected, not branched, so the
// double-float update that follows runs unconditionally (adding 0 leaves the sum unchanged).  The float
// compare |v| > largest-float-below-1e-15 is the same test as above_tol (false for NaN, true for inf).
__device__ __forceinline__ float tol_select(float v, bool keep) {
    return (keep || fabsf(v) > __uint_as_float(kTolBitsF32)) ? v : 0.0f;
}

// Double-float accumulator (hi + lo, two FP32 words, ~2^-48 relative):
// error-free product c*x with c = ch + cl and error-free sum into hi.
struct FF {
    float hi, lo;
};
__device__ __forceinline__ void ff_fma(FF& a, float ch, float cl, float x) {
    const float p = ch * x;
    const float e = fmaf(ch, x, -p) + cl * x;
    const float s = a.hi + p;
    const float bb = s - a.hi;
    const float err = (a.hi - (s - bb)) + (p - bb);
    a.hi = s;
    a.lo += err + e;
}
// Two double-float accumulators held as packed FP32 pairs and updated with the f32x2 instructions of
// sm_100-family GPUs (one instruction per operation for both): the same operations, in the same order,
// as ff_fma on each lane of the pair.
struct FF2 {
    uint64_t hi, lo;
};
__device__ __forceinline__ uint64_t pk2(float a, float b) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 unpk2(uint64_t v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ uint64_t sub2(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
// a += (ch + cl) * x on both lanes; cn = -ch.  q = cn*x = -(ch*x) exactly, so hi - q is hi + p and
// fma(ch, x, q) is the exact error of the product p = ch*x, as in ff_fma.
__device__ __forceinline__ void ff2_fma(FF2& a, uint64_t ch, uint64_t cn, uint64_t cl, uint64_t x) {
    const uint64_t q = mul2(cn, x);
    const uint64_t e = fma2(cl, x, fma2(ch, x, q));
    const uint64_t s = sub2(a.hi, q);
    const uint64_t bb = sub2(s, a.hi);
    const uint64_t err = sub2(sub2(a.hi, sub2(s, bb)), add2(q, bb));
    a.hi = s;
    a.lo = add2(a.lo, add2(err, e));
}

// Shared-memory layout common to the tile kernels.
struct TileSmem {
    uint4* x;           // the terms' flips as the lookup class describes them
    ulonglong2* z;
    double* cs;         // or (hi, lo) float pairs
    uint2* lit8;
    uint32_t* pair;
    uint16_t* off;
    uint8_t* lit;
    unsigned char* tail;  // per-warp scratch follows
};

static size_t tile_smem(const TileTerms& T) {
    size_t used = (size_t)T.n * (16 + (T.z ? 16 : 0) + 8);
    if (T.lit8) used += (size_t)T.n * 8 + (size_t)(T.n + 31) / 32 * 4;
    else used += (size_t)(T.n + 1) * 2 + (size_t)T.n_lits;
    return (used + 15) & ~(size_t)15;
}

template <class LK>
__device__ __forceinline__ TileSmem stage_terms(const TileParams& P, const LK& lk, bool ff, unsigned char* smem) {
    const TileTerms& T = P.T;
    TileSmem S;
    S.x = reinterpret_cast<uint4*>(smem);
    S.z = reinterpret_cast<ulonglong2*>(S.x + T.n);
    S.cs = reinterpret_cast<double*>(S.z + (T.z ? T.n : 0));
    S.lit8 = reinterpret_cast<uint2*>(S.cs + T.n);
    S.pair = reinterpret_cast<uint32_t*>(S.lit8 + T.n);
    S.off = reinterpret_cast<uint16_t*>(S.cs + T.n);
    S.lit = reinterpret_cast<uint8_t*>(S.off + T.n + 1);
    const size_t used = (size_t)T.n * (16 + (T.z ? 16 : 0) + 8) +
                        (T.lit8 ? (size_t)T.n * 8 + (size_t)(T.n + 31) / 32 * 4 : (size_t)(T.n + 1) * 2 + (size_t)T.n_lits);
    S.tail = smem + ((used + 15) & ~(size_t)15);
    for (int k = threadIdx.x; k < T.n; k += blockDim.x) {
        S.x[k] = lk.term_words(T.x[k]);
        if (T.z) S.z[k] = T.z[k];
        S.cs[k] = ff ? reinterpret_cast<const double*>(T.ff)[k] : T.cs[k];
    }
    if (T.lit8) {
        for (int k = threadIdx.x; k < T.n; k += blockDim.x) S.lit8[k] = T.lit8[k];
        for (int k = threadIdx.x; k < (T.n + 31) / 32; k += blockDim.x) S.pair[k] = T.pair[k];
    } else {
        for (int k = threadIdx.x; k <= T.n; k += blockDim.x) S.off[k] = T.lit_off[k];
        for (int k = threadIdx.x; k < T.n_lits; k += blockDim.x) S.lit[k] = T.lits[k];
    }
    __syncthreads();
    return S;
}

// Transposes the tile's states into per-spin words: spinw[i] bit l = spin i of row l, spinw[128 + i] its complement.
constexpr int kSpinWords = 256;
__device__ __forceinline__ void tile_spin_words(const state2 s, int nwords, int lane, uint32_t* spinw) {
    const uint32_t w[4] = {(uint32_t)s.x, (uint32_t)(s.x >> 32), (uint32_t)s.y, (uint32_t)(s.y >> 32)};
#pragma unroll
    for (int k = 0; k < 4; ++k)
        if (k < nwords) {
            const uint32_t t = warp_transpose32(w[k], lane);
            spinw[32 * k + lane] = t;
            spinw[128 + 32 * k + lane] = ~t;
        }
    __syncwarp();
}

// Rows that admit term t0 + lane (bit l = row l).  kForward: of a pair only the rows that admit its first operator, with
// *skew the number of rows that admit the first less those that admit the second.
template <bool kForward = false>
__device__ __forceinline__ uint32_t tile_admitted(const TileSmem& S, const TileTerms& T, int t0, int lane,
                                                  uint32_t vmask, const uint32_t* spinw, int* skew = nullptr) {
    const int t = t0 + lane;
    uint32_t A = 0;
    if (t < T.n) {
        if (T.lit8) {
            const uint2 L = S.lit8[t];
            uint32_t all = spinw[L.x & 0xff], any = all;
#pragma unroll
            for (int k = 1; k < 8; ++k) {
                if (k >= T.max_lits) break;
                const uint32_t w = spinw[((k < 4 ? L.x : L.y) >> (8 * (k & 3))) & 0xff];
                all &= w;
                any |= w;
            }
            if ((S.pair[t0 >> 5] >> lane) & 1) {
                if constexpr (kForward) *skew += __popc(all & vmask) - __popc(~any & vmask);
                else all |= ~any;
            }
            A = all & vmask;
        } else {
            A = vmask;
            const int e = S.off[t + 1];
            for (int k = S.off[t]; k < e; ++k) A &= spinw[S.lit[k]];
        }
    }
    return A;
}

// Whether term t's matrix element on state s carries a minus sign from its Z mask.
__device__ __forceinline__ bool term_negative(const TileSmem& S, bool has_z, uint32_t t, const state2 s) {
    if (!has_z) return false;
    const ulonglong2 z = S.z[t];
    return (__popcll(~s.x & z.x) + __popcll(~s.y & z.y)) & 1;
}
__device__ __forceinline__ double term_coeff(const TileSmem& S, bool has_z, uint32_t t, const state2 s) {
    const double cs = S.cs[t];
    return term_negative(S, has_z, t, s) ? -cs : cs;
}

// Per-warp scratch in shared memory of the matrix-free kernels, rounds = 32-term rounds:
//   spin words, then (they are done with once the tile's admission is known) the rows' flippable words and list bases;
//   adm[rounds * 32]: admission word of row l in round r at r * 32 + l;
//   ts[rounds * 32]: {rows that admit term t, t's first position in the hit list};
//   list: the hits of the tile (or of as many of its rows as fit), term by term.
struct WarpScratch {
    uint32_t* spinw;
    Word4* rows;
    uint32_t* base;
    uint32_t* adm;
    uint2* ts;
    unsigned char* list;
};
__host__ __device__ constexpr size_t scratch_bytes(int rounds) { return 4 * kSpinWords + (size_t)rounds * (128 + 256); }
__device__ __forceinline__ WarpScratch warp_scratch(unsigned char* p, int rounds) {
    WarpScratch W;
    W.spinw = reinterpret_cast<uint32_t*>(p);
    W.rows = reinterpret_cast<Word4*>(p);
    W.base = reinterpret_cast<uint32_t*>(p + 32 * sizeof(Word4));
    W.ts = reinterpret_cast<uint2*>(p + 4 * kSpinWords);
    W.adm = reinterpret_cast<uint32_t*>(W.ts + rounds * 32);
    W.list = reinterpret_cast<unsigned char*>(W.adm + rounds * 32);
    return W;
}

// A hit in the list: its term (an operator's term table holds at most 2,327), its row in the tile and its ordinal
// among the row's hits.
__device__ __forceinline__ uint32_t pack_hit(uint32_t t, uint32_t l, uint32_t k) { return t << 19 | l << 14 | k; }
__device__ __forceinline__ uint32_t hit_term(uint32_t e) { return e >> 19; }
__device__ __forceinline__ uint32_t hit_row(uint32_t e) { return (e >> 14) & 31; }
__device__ __forceinline__ uint32_t hit_ordinal(uint32_t e) { return e & 0x3fff; }

// Admission of the tile's rows: fills adm, the rows of ts and rows; returns this lane's number of hits.
template <bool kForward = false, class LK>
__device__ __forceinline__ int tile_admit(const TileSmem& S, const TileParams& P, const LK& lk, const WarpScratch& W,
                                          const state2 s, int64_t row, int n_rounds, int lane, int* skew = nullptr) {
    const uint32_t vmask = __ballot_sync(0xffffffffu, row < P.B.n);
    const Word4 words = lk.row_words(row, s);
    tile_spin_words(s, P.nwords, lane, W.spinw);
    int cnt = 0;
    for (int r = 0; r < n_rounds; ++r) {
        const uint32_t A = tile_admitted<kForward>(S, P.T, r * 32, lane, vmask, W.spinw, skew);
        const uint32_t a = warp_transpose32(A, lane);
        W.ts[r * 32 + lane].x = A;
        W.adm[r * 32 + lane] = a;
        cnt += __popc(a);
    }
    __syncwarp();
    W.rows[lane] = words;
    return cnt;
}

// Rows [row_start, row_end) whose list slots (per_row each) fit cap, at least one row; *base: this lane's first slot.
__device__ __forceinline__ int chunk_rows(int row_start, int per_row, int cap, int lane, int& base) {
    const int c = (lane >= row_start) ? per_row : 0;
    int incl = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    base = incl - c;
    return 32 - __clz(__ballot_sync(0xffffffffu, lane >= row_start && (incl <= cap || lane == row_start)));
}
__device__ __forceinline__ uint32_t row_mask(int row_start, int row_end) {
    return (0xffffffffu >> (32 - row_end)) & (0xffffffffu << row_start);
}

// Lists the hits of the rows in mask, term by term and by row inside a term (slot i at list + i * stride), and returns
// their number.  Neighbouring rows flipped by one term land on neighbouring states, so a warp that takes 32
// consecutive hits of this order touches 0.49 sectors per load and lane where one hit of each row takes 0.75 (64-spin
// Q=0 basis), and all its lanes have work, where rows of 10.5 hits on average wait for the tile's longest of 14.3 and
// the rows outside a chunk for the chunk.  FP32 batched apply, 30.8 M states: R = 64 45.4 -> 38.7 ms, R = 16 23.0 ->
// 18.1 ms against lookups row by row.
__device__ __forceinline__ int list_hits(const WarpScratch& W, uint32_t mask, int n_rounds, int lane, int stride) {
    int total = 0;
    for (int r = 0; r < n_rounds; ++r) {
        const int c = __popc(W.ts[r * 32 + lane].x & mask);
        int incl = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        W.ts[r * 32 + lane].y = (uint32_t)(total + incl - c);
        total += __shfl_sync(0xffffffffu, incl, 31);
    }
    __syncwarp();
    if ((mask >> lane) & 1) {
        const uint32_t below = mask & ((1u << lane) - 1);
        uint32_t k = 0;
        for (int r = 0; r < n_rounds; ++r)
            for (uint32_t a = W.adm[r * 32 + lane]; a; a &= a - 1) {
                const uint32_t t = r * 32 + __ffs(a) - 1;
                const uint2 p = W.ts[t];
                *reinterpret_cast<uint32_t*>(W.list + (size_t)(p.y + __popc(p.x & below)) * stride) = pack_hit(t, lane, k++);
            }
    }
    __syncwarp();
    return total;
}

// State of row `row` flipped by term t.
__device__ __forceinline__ state2 flipped_state(const TileParams& P, int64_t row, uint32_t t) {
    const state2 s = __ldg(P.B.states + row);
    const uint4 x = __ldg(P.T.x + t);
    return make_ulonglong2(s.x ^ ((uint64_t)x.y << 32 | x.x), s.y ^ ((uint64_t)x.w << 32 | x.z));
}

// Looks the list's hits up, NB per lane at a time: f(i, n, hits, indices) with the lane's first slot i and number of
// hits n <= NB; index kEmpty for a state outside the basis.
template <int NB, class LK, class F>
__device__ __forceinline__ void look_up_hits(const TileSmem& S, const TileParams& P, const WarpScratch& W, const LK& lk,
                                             int64_t tile, int total, int lane, int stride, F&& f) {
    for (int i0 = lane; i0 < total; i0 += 32 * NB) {
        uint32_t e[NB], J[NB];
        Word4 w[NB];
        int n = 0;
#pragma unroll
        for (int u = 0; u < NB; ++u) {
            e[u] = 0;
            w[u] = Word4{0, 0, 0, 0};
            if (i0 + 32 * u < total) {
                e[u] = *reinterpret_cast<const uint32_t*>(W.list + (size_t)(i0 + 32 * u) * stride);
                w[u] = flip_words(W.rows[hit_row(e[u])], S.x[hit_term(e[u])]);
                ++n;
            }
        }
        lk.find_batch(w, n, J, [&](int u) { return flipped_state(P, tile * 32 + hit_row(e[u]), hit_term(e[u])); });
        f(i0, n, e, J);
    }
}

// Calls f(term, slot) for this lane's hits in term order; slot: the hit's position in the list.
template <class F>
__device__ __forceinline__ void for_row_hits(const WarpScratch& W, uint32_t mask, int n_rounds, int lane, F&& f) {
    const uint32_t below = mask & ((1u << lane) - 1);
    for (int r = 0; r < n_rounds; ++r)
        for (uint32_t a = W.adm[r * 32 + lane]; a; a &= a - 1) {
            const uint32_t t = r * 32 + __ffs(a) - 1;
            const uint2 p = W.ts[t];
            f(t, p.y + __popc(p.x & below));
        }
}

// Single vector: every lane looks its own row's hits up, gathers x and adds, kNB hits at a time in step with the other
// lanes.  Bound by the L1's data pipe (76% busy), which serves one sector per cycle of the scattered loads, 2.26 per
// hit, then by latency.  The hit list of the batched kernel below needs a third fewer sectors, but the list's own
// shared-memory traffic and instructions cost more than that saves where a hit brings one value: 351 us against 282
// on the 64-spin Q=0 basis.
template <typename XT, typename YT, class LK, bool kFam = false>
__global__ void __launch_bounds__(256, LK::kMinBlocks) k_apply_tile(TileParams P, LK lk, const XT* __restrict__ x,
                                                                 YT* __restrict__ y, int accumulate) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const TileSmem S = stage_terms(P, lk, false, smem_raw);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int n_rounds = (P.T.n + 31) >> 5;
    const bool has_z = P.T.z != nullptr;
    uint32_t* spinw = reinterpret_cast<uint32_t*>(S.tail) + wid * (kSpinWords + 32 * n_rounds);
    uint32_t* adm = spinw + kSpinWords;
    const int64_t ntiles = (P.B.n + 31) >> 5;
    for (int64_t tile = (int64_t)blockIdx.x * nw + wid; tile < ntiles; tile += (int64_t)gridDim.x * nw) {
        const int64_t row = tile * 32 + lane;
        const bool valid = row < P.B.n;
        const state2 s = valid ? P.B.states[row] : make_ulonglong2(0, 0);
        const Word4 rw = lk.row_words(row, s);
        double acc = valid ? (kFam ? fam_diag(P, s.x, s.y, 0) : P.diag[row]) * widen(x[row]) : 0.0;
        const uint32_t vmask = __ballot_sync(0xffffffffu, valid);
        tile_spin_words(s, P.nwords, lane, spinw);
        int cnt = 0;
        for (int r = 0; r < n_rounds; ++r) {
            const uint32_t a = warp_transpose32(tile_admitted(S, P.T, r * 32, lane, vmask, spinw), lane);
            adm[r * 32 + lane] = a;
            cnt += __popc(a);
        }
        const int width = __reduce_max_sync(0xffffffffu, cnt);
        int r = 0;
        uint32_t a = n_rounds ? adm[lane] : 0;
        for (int k0 = 0; k0 < width; k0 += LK::kNB) {  // up to kNB hits of every row, summed in term order
            constexpr int kNB = LK::kNB;
            uint32_t tt[kNB], J[kNB];
            Word4 w[kNB];
#pragma unroll
            for (int u = 0; u < kNB; ++u) {
                while (!a && r + 1 < n_rounds) a = adm[++r * 32 + lane];
                tt[u] = 0;
                w[u] = rw;
                if (a) {
                    tt[u] = r * 32 + 31 - __clz(a & -a);
                    a &= a - 1;
                    w[u] = flip_words(rw, S.x[tt[u]]);
                }
            }
            lk.find_batch(w, min(max(cnt - k0, 0), kNB), J, [&](int u) { return flipped_state(P, row, tt[u]); });
            XT xv[kNB];
#pragma unroll
            for (int u = 0; u < kNB; ++u) xv[u] = (J[u] != kEmpty) ? x[J[u]] : (XT)0;
#pragma unroll
            for (int u = 0; u < kNB; ++u)
                if (above_tol(xv[u])) {
                    const double cs = term_coeff(S, has_z, tt[u], s);
                    acc += (kFam ? fam_coef(P, cs, 0) : cs) * widen<true>(xv[u]);
                }
        }
        if (valid) {
            if (accumulate) acc += widen(y[row]);
            y[row] = (YT)acc;
        }
        __syncwarp();
    }
}

// Family mode with a few columns (FP64 [row][R], 2 <= R <= RC): as the single-vector tile kernel, with the hits'
// columns left in the list and each lane summing all R columns of its row, the R values of a hit gathered from one
// place.  Each column's sum is the one k_apply_tile forms for that column alone (same terms in the same order, same
// coefficients and tests), so a member's result does not depend on the batch it ran in.
template <class LK, int RC>
__global__ void __launch_bounds__(256, RC <= 4 ? 4 : 2) k_apply_tile_cols(TileParams P, LK lk, const double* __restrict__ x,
                                                            double* __restrict__ y, int accumulate, int cap) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const TileSmem S = stage_terms(P, lk, false, smem_raw);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int n_rounds = (P.T.n + 31) >> 5;
    const bool has_z = P.T.z != nullptr;
    const int R = P.fR;
    const WarpScratch W = warp_scratch(S.tail + wid * (scratch_bytes(n_rounds) + (size_t)cap * 4), n_rounds);
    uint32_t* js = reinterpret_cast<uint32_t*>(W.list);
    const int64_t ntiles = (P.B.n + 31) >> 5;
    for (int64_t tile = (int64_t)blockIdx.x * nw + wid; tile < ntiles; tile += (int64_t)gridDim.x * nw) {
        const int64_t row = tile * 32 + lane;
        const bool valid = row < P.B.n;
        const state2 s = valid ? P.B.states[row] : make_ulonglong2(0, 0);
        double acc[RC];
#pragma unroll
        for (int c = 0; c < RC; ++c) acc[c] = (valid && c < R) ? fam_diag(P, s.x, s.y, c) * x[row * R + c] : 0.0;
        const int cnt = tile_admit(S, P, lk, W, s, row, n_rounds, lane);
        for (int row_start = 0; row_start < 32;) {
            int base;
            const int row_end = chunk_rows(row_start, cnt, cap, lane, base);
            const uint32_t mask = row_mask(row_start, row_end);
            const int total = list_hits(W, mask, n_rounds, lane, 4);
            constexpr int kNB = 2;
            look_up_hits<kNB>(S, P, W, lk, tile, total, lane, 4,
                              [&](int i0, int n, const uint32_t (&)[kNB], const uint32_t (&J)[kNB]) {
#pragma unroll
                for (int u = 0; u < kNB; ++u)
                    if (u < n) js[i0 + 32 * u] = J[u];
            });
            __syncwarp();
            if ((mask >> lane) & 1)
                for_row_hits(W, mask, n_rounds, lane, [&](uint32_t t, uint32_t slot) {
                    const uint32_t J = js[slot];
                    if (J == kEmpty) return;
                    const double cs = term_coeff(S, has_z, t, s);
                    const double* xj = x + (int64_t)J * R;
                    double xv[RC];
#pragma unroll
                    for (int c = 0; c < RC; ++c) xv[c] = (c < R) ? xj[c] : 0.0;
#pragma unroll
                    for (int c = 0; c < RC; ++c)
                        if (c < R && above_tol(xv[c])) acc[c] += fam_coef(P, cs, c) * xv[c];
                });
            __syncwarp();
            row_start = row_end;
        }
        if (valid) {
#pragma unroll
            for (int c = 0; c < RC; ++c) {
                if (c >= R) break;
                double v = acc[c];
                if (accumulate) v += y[row * R + c];
                y[row * R + c] = v;
            }
        }
    }
}

// KM values selecting 16-byte FP32 gathers of 4 (kVec4) or 8 (kVec8) vectors per lane (see k_apply_tile_batched), and
// the bases, vector counts and pointers each takes.  Their hit lists mark the diagonal slot with the top bit of
// the row index.
constexpr int kVec4 = 0;
constexpr int kVec8 = -1;
constexpr int kVec16 = -2;
// A few vectors (R <= kGroupMax) without 16-byte gathers: the warp sums 32 / lpc rows at once, lpc = R rounded up to a
// power of two lanes each.  (With one row per warp the lanes beyond R idle, and GB300's FP64 pipe takes 17 cycles per
// instruction however few of its lanes work.)
constexpr int kGroup = -3;
constexpr int kGroupMax = 16;
constexpr uint32_t kDiagSlot = 0x80000000u;
constexpr int kWideFrom = 32;
inline bool vec4_ok(int64_t n, int R, const void* x, const void* y) {
    return n < (int64_t)kDiagSlot - 1 && R >= 4 && (R & 3) == 0 &&
           (R <= 128 ? (R & (R - 1)) == 0 : (R & 127) == 0) &&
           ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y)) & 15) == 0;
}
inline bool vec8_ok(int64_t n, int R, const void* x, const void* y) {
    return vec4_ok(n, R, x, y) && R >= 32 && (R <= 256 ? (R & (R - 1)) == 0 : (R & 255) == 0);
}
inline bool vec16_ok(int64_t n, int R, const void* x, const void* y) {
    return vec4_ok(n, R, x, y) && R >= 64 && (R <= 512 ? (R & (R - 1)) == 0 : (R & 511) == 0);
}

// Blocks per SM: two where a lane sums four FP32 vectors without 16-byte gathers (KM = 4), which spill at three (100 vectors on
// the 64-spin Q=0 basis 6,100 -> 4,620 us, 388 to 36,056 rows 59-125 -> 44-92); FP64 sums stay at three (8,260 us there, 8,480
// at two).
template <typename XT, class LK, bool kFF, int KM, bool kFam = false>
__global__ void __launch_bounds__(256, KM == kVec8 || KM == kVec16 || (KM == 4 && kFF) ? 2 : 3) k_apply_tile_batched(TileParams P, LK lk, const XT* __restrict__ x,
                                                            XT* __restrict__ y, int R, int accumulate, int cap,
                                                            const float2* __restrict__ ycoef) {
    // accumulate: y <- H x + c y per column, c = 1, or the (hi, lo) float pair ycoef[column] (double-float paths)
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const TileSmem S = stage_terms(P, lk, kFF, smem_raw);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int n_rounds = (P.T.n + 31) >> 5;
    const bool has_z = P.T.z != nullptr;
    // per-warp scratch, then the rows' slots in row order (coefficients, columns)
    constexpr bool kCached = std::is_same<LK, LookupCache>::value;
    unsigned char* mine = S.tail + (size_t)wid * (scratch_bytes(n_rounds) + (size_t)cap * 16);
    const WarpScratch W = warp_scratch(mine, n_rounds);
    double* hc = reinterpret_cast<double*>(W.list);  // coefficients (8-byte aligned)
    float2* hcf = reinterpret_cast<float2*>(hc);     // the same slots as (hi, lo) floats
    uint32_t* hJ = reinterpret_cast<uint32_t*>(hc + cap);
    WarpScratch WL = W;  // with the hits in list order behind them
    WL.list = reinterpret_cast<unsigned char*>(hJ + cap);
    // KM == kVec4 / kVec8 (FP32, R accepted by vec4_ok / vec8_ok): 16-byte gathers.  A lane owns VPL = 4 or 8
    // consecutive vectors, lpc lanes cover one column's vectors (up to 32*VPL per pass), and the warp's
    // cpw = 32/lpc lane groups sum cpw rows at once.  Otherwise a lane owns KM vectors and the warp sums one
    // row at a time.
    constexpr bool v4 = (KM == kVec4 || KM == kVec8 || KM == kVec16);
    constexpr int VPL = (KM == kVec16) ? 16 : (KM == kVec8) ? 8 : 4;
    static_assert(!v4 || kFF, "16-byte gathers are for FP32 vectors with double-float accumulation");
    int lpc = 32, cpw = 1;
    if constexpr (v4) {
        const int vc = P.vchunk > 0 ? min(P.vchunk, 32 * VPL) : 32 * VPL;  // the warp's lanes at most
        lpc = (R >= vc ? vc : R) / VPL;
        cpw = 32 / lpc;
    }
    const int64_t ntiles = (P.B.n + 31) >> 5;
    for (int64_t tile = (int64_t)blockIdx.x * nw + wid; tile < ntiles; tile += (int64_t)gridDim.x * nw) {
        const int64_t row = tile * 32 + lane;
        const bool valid = row < P.B.n;
        state2 s = make_ulonglong2(0, 0);
        int cnt = 0, width = 0;
        uint64_t cur = 0;
        if constexpr (kCached) {  // the row's entries are read from the cache, misses left out
            cur = lk.cursor(tile, lane);
            width = (int)((lk.cursor(tile + 1, lane) - cur) >> 5);
#pragma unroll 8
            for (int k = 0; k < width; ++k) cnt += __ldg(lk.C.cols + cur + (uint64_t)k * 32) != kEmpty;
            if constexpr (kFam) s = valid ? P.B.states[row] : s;
        } else {
            if (valid) s = P.B.states[row];
            cnt = tile_admit(S, P, lk, W, s, row, n_rounds, lane);
        }
        const int pc = v4 ? cnt + 1 : cnt;  // list slots of this row: (the diagonal,) the hits
        const double d = valid ? P.diag[row] : 0.0;
        for (int row_start = 0; row_start < 32;) {
            // rows [row_start, row_end) whose slots fit the list (at least one row; cap >= a row's slots)
            int base;
            const int row_end = chunk_rows(row_start, pc, cap, lane, base);
            const bool in_chunk = lane >= row_start && lane < row_end;
            if constexpr (v4) {  // the diagonal leads the row's list (gathered like a hit, no tolerance test)
                if (in_chunk) {
                    hJ[base] = valid ? (uint32_t)row | kDiagSlot : kEmpty;
                    hcf[base] = valid ? P.diag_ff[row] : make_float2(0.f, 0.f);
                }
            }
            auto put = [&](uint32_t slot, uint32_t J, uint32_t t, bool neg) {
                hJ[slot] = J;
                if constexpr (kFF) {
                    const float2 f = reinterpret_cast<const float2*>(S.cs)[t];
                    hcf[slot] = neg ? make_float2(-f.x, -f.y) : f;
                } else {
                    const double c = S.cs[t];
                    hc[slot] = neg ? -c : c;
                }
            };
            if constexpr (kCached) {
                if (in_chunk) {
                    int k = base + (v4 ? 1 : 0);
                    constexpr int kE = KM == kGroup ? 4 : 8;  // entries read at once (the group's kernel has registers for four)
                    for (int e0 = 0; e0 < width; e0 += kE) {
                        uint32_t c[kE], t[kE];
#pragma unroll
                        for (int u = 0; u < kE; ++u) {
                            const uint64_t at = cur + (uint64_t)(e0 + u) * 32;
                            const bool in = e0 + u < width;
                            c[u] = in ? __ldg(lk.C.cols + at) : kEmpty;
                            t[u] = in ? lk.term(at) : 0;
                        }
#pragma unroll
                        for (int u = 0; u < kE; ++u)
                            if (c[u] != kEmpty) put(k++, c[u] & ~kCacheNeg, t[u], c[u] & kCacheNeg);
                    }
                }
            } else {
                W.base[lane] = base + (v4 ? 1 : 0);
                const int total = list_hits(WL, row_mask(row_start, row_end), n_rounds, lane, 4);
                constexpr int kNB = 2;
                look_up_hits<kNB>(S, P, WL, lk, tile, total, lane, 4,
                                  [&](int, int n, const uint32_t (&e)[kNB], const uint32_t (&J)[kNB]) {
#pragma unroll
                    for (int u = 0; u < kNB; ++u) {
                        if (u >= n) continue;
                        const uint32_t t = hit_term(e[u]), l = hit_row(e[u]);
                        bool neg = false;
                        if (has_z) neg = term_negative(S, true, t, P.B.states[tile * 32 + l]);
                        put(W.base[l] + hit_ordinal(e[u]), J[u], t, neg);
                    }
                });
            }
            __syncwarp();
            if constexpr (KM == kGroup) {
                int lpc = 1;
                while (lpc < R) lpc *= 2;
                const int g = lane / lpc, c = lane % lpc;
                constexpr int kU = 8;  // column gathers in flight per lane
                for (int l0 = row_start; l0 < row_end; l0 += 32 / lpc) {
                    const int l = l0 + g;
                    const int64_t rl = tile * 32 + l;
                    const bool mine = l < row_end && rl < P.B.n;
                    const int kb = __shfl_sync(0xffffffffu, base, l & 31);
                    int nl = __shfl_sync(0xffffffffu, cnt, l & 31);
                    if (!mine) nl = 0;
                    const int steps = __reduce_max_sync(0xffffffffu, nl);
                    const bool on = mine && c < R;
                    std::conditional_t<kFF, FF, double> acc{};
                    if (on) {
                        const XT xd = x[rl * R + c];
                        if constexpr (kFF) {
                            const float2 dd = P.diag_ff[rl];
                            ff_fma(acc, dd.x, dd.y, (float)xd);
                        } else {
                            double dl;
                            if constexpr (kFam) {
                                const state2 t = P.B.states[rl];
                                dl = fam_diag(P, t.x, t.y, c);
                            } else {
                                dl = P.diag[rl];
                            }
                            acc = dl * widen(xd);
                        }
                    }
                    for (int s0 = 0; s0 < steps; s0 += kU) {
                        XT xv[kU];
#pragma unroll
                        for (int u = 0; u < kU; ++u) {
                            const uint32_t J = (s0 + u < nl) ? hJ[kb + s0 + u] : kEmpty;
                            xv[u] = (on && J != kEmpty) ? x[(int64_t)J * R + c] : (XT)0;
                        }
#pragma unroll
                        for (int u = 0; u < kU; ++u) {
                            if (!above_tol(xv[u])) continue;
                            if constexpr (kFF) {
                                const float2 ck = hcf[kb + s0 + u];
                                ff_fma(acc, ck.x, ck.y, (float)xv[u]);
                            } else {
                                const double ck = hc[kb + s0 + u];
                                acc += (kFam ? fam_coef(P, ck, c) : ck) * widen<true>(xv[u]);
                            }
                        }
                    }
                    if (on) {
                        if constexpr (kFF) {
                            if (accumulate) {
                                const float2 yc = ycoef ? ycoef[c] : make_float2(1.0f, 0.0f);
                                ff_fma(acc, yc.x, yc.y, (float)y[rl * R + c]);
                            }
                            y[rl * R + c] = (XT)(acc.hi + acc.lo);
                        } else {
                            if (accumulate) acc += widen(y[rl * R + c]);
                            y[rl * R + c] = (XT)acc;
                        }
                    }
                }
            } else if constexpr (kFF) {
                // FP32 storage, double-float accumulation, no FP64 instruction.  The chunk's hit list
                // is walked in order across row boundaries with kU column gathers in flight.
                static_assert(std::is_same<XT, float>::value, "double-float accumulation is for FP32 vectors");
                // Column gathers in flight per lane, bound by their latency.  64 vectors, with the look-ups / materialised,
                // four vectors per lane and a list of 256:
                //   floats, blocks          32, 2        32, 3        24, 3        20, 3        16, 3
                //   96-spin 8.8.16.16 ms  40.1 / 38.9  40.4 / 30.2  37.7 / 28.5  38.5 / 29.8  45.9 / 31.4
                //   64-spin Q=0 ms        2.48 / 2.30  2.62 / 1.87  2.38 / 1.78  2.38 / 1.84  2.73 / 1.91
                // eight vectors per lane and a list of 512, whose shared memory holds it to two blocks:
                //   96-spin 8.8.16.16 ms  32.1 / 33.1               44.5 / 39.7
                //   64-spin Q=0 ms        1.88 / 1.82               2.55 / 2.18
                constexpr int kU = !v4 ? 8 : VPL == 4 ? 6 : 32 / VPL;
                const int kbeg = __shfl_sync(0xffffffffu, base, row_start);
                const int last = row_end - 1;
                const int kend = __shfl_sync(0xffffffffu, base + pc, last);
                if constexpr (v4) {
                    // Lane group g (lpc lanes, VPL vectors each) sums rows row_start + g, + g + cpw, ...: each
                    // group walks its own row's slots, kU column gathers in flight per lane, and the warp
                    // steps as long as its longest row of the set.
                    constexpr int NQ = VPL / 4;  // float4 loads per lane and column
                    const int g = lane / lpc, rr = VPL * (lane % lpc);
                    for (int r0 = 0; r0 < R; r0 += VPL * lpc) {
                        for (int l0 = row_start; l0 < row_end; l0 += cpw) {
                            const int l = l0 + g;
                            const bool mine = l < row_end;
                            const int lsrc = mine ? l : row_end - 1;
                            const int kb = __shfl_sync(0xffffffffu, base, lsrc);
                            int nl = __shfl_sync(0xffffffffu, pc, lsrc);
                            if (!mine) nl = 0;
                            int steps = nl;
#pragma unroll
                            for (int o = 16; o; o >>= 1) steps = max(steps, __shfl_xor_sync(0xffffffffu, steps, o));
                            FF2 acc[2 * NQ];  // vector pairs (0, 1), (2, 3), ... of this lane
#pragma unroll
                            for (int i = 0; i < 2 * NQ; ++i) acc[i] = FF2{0, 0};
                            auto run_batch = [&](int s0, auto width) {
                                constexpr int W = decltype(width)::value;
                                float4 xv[W][NQ];
                                float2 ck[W];
                                uint32_t dg = 0;  // bit u: slot u holds the diagonal
#pragma unroll
                                for (int u = 0; u < W; ++u) {
                                    const int k = kb + s0 + u;
                                    const uint32_t J = (s0 + u < nl) ? hJ[k] : kEmpty;
                                    if (J != kEmpty && (J & kDiagSlot)) dg |= 1u << u;
                                    ck[u] = (J == kEmpty) ? make_float2(0.f, 0.f) : hcf[k];
                                    const float4* src =
                                        reinterpret_cast<const float4*>(x + (int64_t)(J & ~kDiagSlot) * R + r0 + rr);
#pragma unroll
                                    for (int q = 0; q < NQ; ++q)
                                        xv[u][q] = (J == kEmpty) ? make_float4(0.f, 0.f, 0.f, 0.f) : src[q];
                                }
#pragma unroll
                                for (int u = 0; u < W; ++u) {
                                    const bool all = (dg >> u) & 1;
                                    const uint64_t ch = pk2(ck[u].x, ck[u].x), cn = pk2(-ck[u].x, -ck[u].x),
                                                   cl = pk2(ck[u].y, ck[u].y);
#pragma unroll
                                    for (int q = 0; q < NQ; ++q) {
                                        ff2_fma(acc[2 * q], ch, cn, cl,
                                                pk2(tol_select(xv[u][q].x, all), tol_select(xv[u][q].y, all)));
                                        ff2_fma(acc[2 * q + 1], ch, cn, cl,
                                                pk2(tol_select(xv[u][q].z, all), tol_select(xv[u][q].w, all)));
                                    }
                                }
                            };
                            for (int s0 = 0; s0 < steps;) {  // full batches, and a half batch for a short tail
                                if (steps - s0 > kU / 2) {
                                    run_batch(s0, std::integral_constant<int, kU>{});
                                    s0 += kU;
                                } else {
                                    constexpr int kH = kU / 2 > 0 ? kU / 2 : 1;
                                    run_batch(s0, std::integral_constant<int, kH>{});
                                    s0 += kH;
                                }
                            }
                            const int64_t rl = tile * 32 + l;
                            if (mine && rl < P.B.n) {
                                float4* yp = reinterpret_cast<float4*>(y + rl * R + r0 + rr);
#pragma unroll
                                for (int q = 0; q < NQ; ++q) {
                                    if (accumulate) {
                                        const float4 yv = yp[q];
                                        if (ycoef) {
                                            const float4 ca = *reinterpret_cast<const float4*>(ycoef + r0 + rr + 4 * q);
                                            const float4 cb =
                                                *reinterpret_cast<const float4*>(ycoef + r0 + rr + 4 * q + 2);
                                            ff2_fma(acc[2 * q], pk2(ca.x, ca.z), pk2(-ca.x, -ca.z), pk2(ca.y, ca.w),
                                                    pk2(yv.x, yv.y));
                                            ff2_fma(acc[2 * q + 1], pk2(cb.x, cb.z), pk2(-cb.x, -cb.z),
                                                    pk2(cb.y, cb.w), pk2(yv.z, yv.w));
                                        } else {
                                            const uint64_t one = pk2(1.0f, 1.0f), mone = pk2(-1.0f, -1.0f),
                                                           zero = pk2(0.f, 0.f);
                                            ff2_fma(acc[2 * q], one, mone, zero, pk2(yv.x, yv.y));
                                            ff2_fma(acc[2 * q + 1], one, mone, zero, pk2(yv.z, yv.w));
                                        }
                                    }
                                    const float2 a = unpk2(add2(acc[2 * q].hi, acc[2 * q].lo)),
                                                 b = unpk2(add2(acc[2 * q + 1].hi, acc[2 * q + 1].lo));
                                    yp[q] = make_float4(a.x, a.y, b.x, b.y);
                                }
                            }
                        }
                    }
                } else {
                for (int r0 = 0; r0 < R; r0 += 32 * KM) {
                    int l = row_start;
                    int lend = __shfl_sync(0xffffffffu, base + pc, l);
                    FF acc[KM];
                    auto start_row = [&](int rr_l) {
                        const int64_t rl = tile * 32 + rr_l;
                        const float2 dd = (rl < P.B.n) ? P.diag_ff[rl] : make_float2(0.f, 0.f);
#pragma unroll
                        for (int m = 0; m < KM; ++m) {
                            const int rr = r0 + lane + 32 * m;
                            acc[m] = FF{0.f, 0.f};
                            if (rr < R && rl < P.B.n) ff_fma(acc[m], dd.x, dd.y, (float)x[rl * R + rr]);
                        }
                    };
                    auto finish_row = [&](int rr_l) {
                        const int64_t rl = tile * 32 + rr_l;
                        if (rl >= P.B.n) return;
#pragma unroll
                        for (int m = 0; m < KM; ++m) {
                            const int rr = r0 + lane + 32 * m;
                            if (rr < R) {
                                if (accumulate) {
                                    const float2 c = ycoef ? ycoef[rr] : make_float2(1.0f, 0.0f);
                                    ff_fma(acc[m], c.x, c.y, (float)y[rl * R + rr]);
                                }
                                y[rl * R + rr] = (XT)(acc[m].hi + acc[m].lo);
                            }
                        }
                    };
                    start_row(l);
                    for (int k0 = kbeg; k0 < kend; k0 += kU) {
                        float xv[kU][KM];
                        float2 ck[kU];
#pragma unroll
                        for (int u = 0; u < kU; ++u) {
                            const uint32_t J = (k0 + u < kend) ? hJ[k0 + u] : kEmpty;
                            ck[u] = (J == kEmpty) ? make_float2(0.f, 0.f) : hcf[k0 + u];
#pragma unroll
                            for (int m = 0; m < KM; ++m) {
                                const int rr = r0 + lane + 32 * m;
                                xv[u][m] = (J != kEmpty && rr < R) ? (float)x[(int64_t)J * R + rr] : 0.f;
                            }
                        }
#pragma unroll
                        for (int u = 0; u < kU; ++u) {
                            const int k = k0 + u;
                            if (k >= kend) break;
                            while (k >= lend) {  // rows whose hits are complete
                                finish_row(l);
                                ++l;
                                lend = __shfl_sync(0xffffffffu, base + pc, l);
                                start_row(l);
                            }
#pragma unroll
                            for (int m = 0; m < KM; ++m) ff_fma(acc[m], ck[u].x, ck[u].y, tol_select(xv[u][m], false));
                        }
                    }
                    finish_row(l);
                    for (++l; l <= last; ++l) {  // trailing rows without hits
                        start_row(l);
                        finish_row(l);
                    }
                }
                }
            } else {
            for (int l = row_start; l < row_end; ++l) {
                const int b0 = __shfl_sync(0xffffffffu, base, l);
                const int nl = __shfl_sync(0xffffffffu, cnt, l);
                const double dl = __shfl_sync(0xffffffffu, d, l);
                const uint64_t sl0 = __shfl_sync(0xffffffffu, s.x, l), sl1 = __shfl_sync(0xffffffffu, s.y, l);
                const int64_t rl = tile * 32 + l;
                if (rl >= P.B.n) break;
                for (int r0 = 0; r0 < R; r0 += 32 * KM) {
                    {
                        double acc[KM];
#pragma unroll
                        for (int m = 0; m < KM; ++m) {
                            const int rr = r0 + lane + 32 * m;
                            acc[m] = (rr < R) ? (kFam ? fam_diag(P, sl0, sl1, rr) : dl) * widen(x[rl * R + rr]) : 0.0;
                        }
                        for (int k = b0; k < b0 + nl; k += 4) {
                            XT xv[4][KM];
                            double ck[4];
#pragma unroll
                            for (int u = 0; u < 4; ++u) {
                                const uint32_t J = (k + u < b0 + nl) ? hJ[k + u] : kEmpty;
                                ck[u] = (J == kEmpty) ? 0.0 : hc[k + u];
#pragma unroll
                                for (int m = 0; m < KM; ++m) {
                                    const int rr = r0 + lane + 32 * m;
                                    xv[u][m] = (J != kEmpty && rr < R) ? x[(int64_t)J * R + rr] : (XT)0;
                                }
                            }
#pragma unroll
                            for (int u = 0; u < 4; ++u)
#pragma unroll
                                for (int m = 0; m < KM; ++m)
                                    if (above_tol(xv[u][m]))
                                        acc[m] += (kFam ? fam_coef(P, ck[u], r0 + lane + 32 * m) : ck[u]) * widen<true>(xv[u][m]);
                        }
#pragma unroll
                        for (int m = 0; m < KM; ++m) {
                            const int rr = r0 + lane + 32 * m;
                            if (rr < R) {
                                double v = acc[m];
                                if (accumulate) v += widen(y[rl * R + rr]);
                                y[rl * R + rr] = (XT)v;
                            }
                        }
                    }
                }
            }
            }
            __syncwarp();
            row_start = row_end;
        }
    }
}

// Per-row diagonal, evaluated once per operator with the same arithmetic as
// diag_value in the row kernels.
__global__ void k_diag_precompute(BasisView B, DiagSpec D, const PushTerm* __restrict__ dgen, double* __restrict__ out,
                                  float2* __restrict__ out_ff) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < B.n; i += (int64_t)gridDim.x * blockDim.x) {
        const state2 s = B.states[i];
        const double d = diag_value(D, dgen, s.x, s.y);
        out[i] = d;
        const float h = (float)d;
        out_ff[i] = make_float2(h, (float)(d - (double)h));
    }
}

qsi_status build_diag(qsi_op* op) {
    cudaStream_t st = op->stream;
    QSI_CUDA(cudaMallocAsync(&op->d_diag, (size_t)op->basis->n * sizeof(double), st));
    QSI_CUDA(cudaMallocAsync(&op->d_diag_ff, (size_t)op->basis->n * sizeof(float2), st));
    k_diag_precompute<<<grid_for(op->basis->n, 256), 256, 0, st>>>(op->basis->view(), op->diag, op->d_diag_generic,
                                                                    op->d_diag, op->d_diag_ff);
    QSI_CUDA(cudaGetLastError());
    QSI_CUDA(cudaStreamSynchronize(st));
    return QSI_OK;
}

// ------------------------------------------------------------------ hash index build
// The keys of the states (of at most 96 bits), by tables of the twelve bytes' keys.
__global__ void __launch_bounds__(256) k_state_keys(BasisView B, uint2* __restrict__ keys) {
    __shared__ uint2 part[12][256];
    for (int e = threadIdx.x; e < 12 * 256; e += blockDim.x) {
        const int byte = e >> 8;
        const uint64_t v = (uint64_t)(e & 255) << (8 * (byte & 7));
        part[byte][e & 255] = byte < 8 ? state_key(v, 0) : state_key(0, v);
    }
    __syncthreads();
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < B.n; i += (int64_t)gridDim.x * blockDim.x) {
        const state2 s = B.states[i];
        uint2 k = make_uint2(0, 0);
#pragma unroll
        for (int byte = 0; byte < 12; ++byte) {
            const uint2 p = part[byte][((byte < 8 ? s.x : s.y) >> (8 * (byte & 7))) & 255];
            k.x ^= p.x;
            k.y ^= p.y;
        }
        keys[i] = k;
    }
}

__device__ __forceinline__ uint32_t* state_bin(const BinView& H, uint32_t* bins, int64_t i, uint32_t& offset, uint32_t& tag) {
    bool ok;
    const uint2 bucket = H.B.tab[bucket_of(H.B, H.B.states[i].x, H.B.states[i].y, ok)], key = H.keys[i];
    offset = (uint32_t)i - bucket.x;
    tag = key.y & ~H.off_mask;
    return bins + (size_t)pick_bin(bucket, key.x, key.y) * kBinSlots;
}

// Every state takes the first free slot of its bin; a state that finds it full is left out.
__global__ void k_bins_insert(BinView H, uint32_t* bins) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < H.B.n; i += (int64_t)gridDim.x * blockDim.x) {
        uint32_t offset, tag;
        uint32_t* p = state_bin(H, bins, i, offset, tag);
        for (int k = 0; k < kBinSlots; ++k)
            if (atomicCAS(p + k, kEmpty, tag | offset) == kEmpty) break;
    }
}

// Marks the slots that a state of the basis would take for its own though they are not: afterwards a state's first
// match is itself or a marked slot, or its bin is full and has no match.
__global__ void k_bins_check(BinView H, uint32_t* bins) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < H.B.n; i += (int64_t)gridDim.x * blockDim.x) {
        uint32_t offset, tag, w[kBinSlots];
        uint32_t* p = state_bin(H, bins, i, offset, tag);
        for (int k = 0; k < kBinSlots; ++k) w[k] = *(volatile uint32_t*)(p + k);
        const uint32_t m = bin_match(w, tag), mark = H.off_mask - 1;
        if (m >= mark || m == offset) continue;
        for (int k = 0; k < kBinSlots; ++k)
            if ((w[k] ^ tag) < mark) *(volatile uint32_t*)(p + k) = tag | mark;
    }
}

void drop_hash(qsi_basis* b) {
    if (b->d_bins) cudaFree(b->d_bins);
    if (b->d_keys) cudaFree(b->d_keys);
    b->d_bins = nullptr;
    b->d_keys = nullptr;
    b->n_bins = 0;
}

// The bins over the basis's current bucket table (built again whenever the table is).
qsi_status build_hash(qsi_basis* b) {
    if (b->hb >= 96) return fail(QSI_INVALID_ARG, "hash index needs states of at most 96 bits");
    if (b->n >= ((int64_t)1 << 31)) return fail(QSI_INVALID_ARG, "hash index needs fewer than 2^31 states");
    auto build = [&]() -> qsi_status {
        if (!b->d_keys) {
            QSI_CUDA(cudaMalloc(&b->d_keys, (size_t)b->n * sizeof(uint2)));
            k_state_keys<<<std::min(grid_for(b->n, 256), 608), 256>>>(b->view(), b->d_keys);
        }
        if (!b->d_bins) {
            // a bucket's last bin: first_bin(a) + first_bin(m) <= first_bin(n)
            b->n_bins = (uint64_t)first_bin((uint32_t)b->n) + 1;
            QSI_CUDA(cudaMalloc(&b->d_bins, b->n_bins * kBinSlots * sizeof(uint32_t)));
        }
        b->off_mask = 15;
        while (b->off_mask <= b->largest_bucket) b->off_mask = 2 * b->off_mask + 1;  // offsets below the mark, off_mask - 1
        QSI_CUDA(cudaMemset(b->d_bins, 0xFF, b->n_bins * kBinSlots * sizeof(uint32_t)));
        k_bins_insert<<<grid_for(b->n, 256), 256>>>(b->bview(), b->d_bins);
        k_bins_check<<<grid_for(b->n, 256), 256>>>(b->bview(), b->d_bins);
        QSI_CUDA(cudaGetLastError());
        QSI_CUDA(cudaStreamSynchronize(nullptr));
        return QSI_OK;
    };
    const qsi_status s = build();
    if (s != QSI_OK) drop_hash(b);
    return s;
}

// ------------------------------------------------------------------ term tables
qsi_status upload_tile_terms(qsi_op* op, const std::vector<PullTerm>& pull) {
    std::vector<const PullTerm*> kept;
    std::vector<uint32_t> pair((pull.size() + 31) / 32 + 1, 0);
    std::vector<std::vector<uint8_t>> lits(pull.size());
    bool short_lists = true, any_z = false, reversible = true;
    for (size_t k = 0; k < pull.size(); ++k) {
        const PullTerm& t = pull[k];
        const uint64_t um[2] = {t.up0, t.up1}, dm[2] = {t.dn0, t.dn1};
        for (int bit = 0; bit < 128; ++bit) {
            if ((um[bit >> 6] >> (bit & 63)) & 1) lits[k].push_back((uint8_t)bit);
            if ((dm[bit >> 6] >> (bit & 63)) & 1) lits[k].push_back((uint8_t)(0x80 | bit));
        }
        short_lists = short_lists && !lits[k].empty() && lits[k].size() <= 8;
        any_z = any_z || t.has_z;
    }
    std::vector<std::vector<uint8_t>*> klits;
    for (size_t k = 0; k < pull.size(); ++k) {
        const PullTerm& t = pull[k];
        klits.push_back(&lits[k]);
        kept.push_back(&t);
        if (short_lists && k + 1 < pull.size()) {
            const PullTerm& c = pull[k + 1];
            if (c.x0 == t.x0 && c.x1 == t.x1 && c.z0 == t.z0 && c.z1 == t.z1 && c.cs == t.cs && c.up0 == t.dn0 &&
                c.up1 == t.dn1 && c.dn0 == t.up0 && c.dn1 == t.up1) {
                pair[(kept.size() - 1) >> 5] |= 1u << ((kept.size() - 1) & 31);
                reversible = reversible && !((t.up0 | t.dn0) & ~t.x0) && !((t.up1 | t.dn1) & ~t.x1);
                ++k;
            }
        }
    }
    TileTerms& T = op->tile;
    T = TileTerms{};
    T.n = (int)kept.size();
    std::vector<uint4> x;
    std::vector<double> cs;
    std::vector<float2> ff;
    std::vector<ulonglong2> z;
    std::vector<uint2> lit8;
    std::vector<uint16_t> off{0};
    std::vector<uint8_t> flat;
    for (int k = 0; k < T.n; ++k) {
        const PullTerm& t = *kept[k];
        const std::vector<uint8_t>& l = *klits[k];
        x.push_back(make_uint4((uint32_t)t.x0, (uint32_t)(t.x0 >> 32), (uint32_t)t.x1, (uint32_t)(t.x1 >> 32)));
        cs.push_back(t.cs);
        ff.push_back(make_float2(t.cs_hi, t.cs_lo));
        if (any_z) z.push_back(make_ulonglong2(t.z0, t.z1));
        if (short_lists) {
            uint32_t w[2] = {0, 0};
            for (int j = 0; j < 8; ++j) w[j >> 2] |= (uint32_t)l[std::min<size_t>(j, l.size() - 1)] << (8 * (j & 3));
            lit8.push_back(make_uint2(w[0], w[1]));
            T.max_lits = std::max(T.max_lits, (int)l.size());
        } else {
            flat.insert(flat.end(), l.begin(), l.end());
            if (flat.size() > 65535) return fail(QSI_INVALID_ARG, "qsi_op_create: more than 65535 literals in the term list");
            off.push_back((uint16_t)flat.size());
        }
    }
    T.n_lits = (int)flat.size();
    T.reversible = reversible;
    size_t total = 0;
    auto place = [&](size_t bytes) {
        const size_t at = total;
        total += (bytes + 15) & ~(size_t)15;
        return at;
    };
    const size_t n = (size_t)T.n, o_x = place(n * 16), o_cs = place(n * 8), o_ff = place(n * 8), o_z = place(z.size() * 16),
                 o_l8 = place(lit8.size() * 8), o_p = place(pair.size() * 4), o_off = place(off.size() * 2),
                 o_lit = place(flat.size());
    std::vector<unsigned char> host(total + 16, 0);
    auto put = [&](size_t at, const void* src, size_t bytes) {
        if (bytes) std::memcpy(host.data() + at, src, bytes);
    };
    put(o_x, x.data(), n * 16);
    put(o_cs, cs.data(), n * 8);
    put(o_ff, ff.data(), n * 8);
    put(o_z, z.data(), z.size() * 16);
    put(o_l8, lit8.data(), lit8.size() * 8);
    put(o_p, pair.data(), pair.size() * 4);
    put(o_off, off.data(), off.size() * 2);
    put(o_lit, flat.data(), flat.size());
    QSI_CUDA(cudaMalloc(&op->d_tile_terms, host.size()));
    QSI_CUDA(cudaMemcpy(op->d_tile_terms, host.data(), host.size(), cudaMemcpyHostToDevice));
    unsigned char* d = op->d_tile_terms;
    T.x = reinterpret_cast<const uint4*>(d + o_x);
    T.cs = reinterpret_cast<const double*>(d + o_cs);
    T.ff = reinterpret_cast<const float2*>(d + o_ff);
    T.z = any_z ? reinterpret_cast<const ulonglong2*>(d + o_z) : nullptr;
    T.lit8 = (short_lists && n) ? reinterpret_cast<const uint2*>(d + o_l8) : nullptr;
    T.pair = reinterpret_cast<const uint32_t*>(d + o_p);
    T.lit_off = reinterpret_cast<const uint16_t*>(d + o_off);
    T.lits = reinterpret_cast<const uint8_t*>(d + o_lit);
    return QSI_OK;
}

// What find_closed reads: missed != 0 when an admitted term of some row leaves the basis; with kForward also the sum over
// all rows and pairs of tile_admitted's skew.
struct Closure {
    unsigned long long skew;
    int missed;
};

// kForward (every pair is reversible): only the first operator of a pair is looked up.  It maps the rows that admit it one
// to one onto states that admit the second, so when none of them leaves the basis, at least as many rows admit the
// second; when the sum over all pairs says that no more do, each row that admits a second operator is the image of
// one that admits the first and is mapped back onto it, inside the basis.
template <bool kForward, class LK>
__global__ void __launch_bounds__(256) k_find_miss(TileParams P, LK lk, Closure* __restrict__ out, int cap) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const TileSmem S = stage_terms(P, lk, false, smem_raw);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int n_rounds = (P.T.n + 31) >> 5;
    const WarpScratch W = warp_scratch(S.tail + wid * (scratch_bytes(n_rounds) + (size_t)cap * 4), n_rounds);
    const int64_t ntiles = (P.B.n + 31) >> 5;
    long long skew = 0;
    for (int64_t tile = (int64_t)blockIdx.x * nw + wid; tile < ntiles; tile += (int64_t)gridDim.x * nw) {
        // any block may set the flag at any time: one lane reads it for the warp, which then leaves or stays as a whole
        if (__shfl_sync(0xffffffffu, lane == 0 ? *(volatile int*)&out->missed : 0, 0)) break;
        const int64_t row = tile * 32 + lane;
        const bool valid = row < P.B.n;
        const state2 s = valid ? P.B.states[row] : make_ulonglong2(0, 0);
        int here = 0;
        const int cnt = tile_admit<kForward>(S, P, lk, W, s, row, n_rounds, lane, &here);
        skew += here;
        bool miss = false;
        for (int row_start = 0; row_start < 32;) {
            int base;
            const int row_end = chunk_rows(row_start, cnt, cap, lane, base);
            const int total = list_hits(W, row_mask(row_start, row_end), n_rounds, lane, 4);
            constexpr int kNB = 2;
            look_up_hits<kNB>(S, P, W, lk, tile, total, lane, 4,
                              [&](int, int n, const uint32_t (&)[kNB], const uint32_t (&J)[kNB]) {
#pragma unroll
                for (int u = 0; u < kNB; ++u) miss = miss || (u < n && J[u] == kEmpty);
            });
            __syncwarp();
            row_start = row_end;
        }
        if (__any_sync(0xffffffffu, miss) && lane == 0) *(volatile int*)&out->missed = 1;
    }
    if constexpr (kForward) {
#pragma unroll
        for (int o = 16; o; o >>= 1) skew += __shfl_down_sync(0xffffffffu, skew, o);
        if (lane == 0 && skew) atomicAdd(&out->skew, (unsigned long long)skew);
    }
}

// Block, shared memory and list capacity of a matrix-free tile kernel whose list slots take slot_bytes (0: no list): a
// list holds want hits or a row of all terms; blocks have eight warps, fewer where a long term list leaves no room.
struct TileLaunch {
    int block, cap;
    size_t smem;
};
constexpr int kListCap = 512;
static TileLaunch tile_launch(const qsi_op* op, size_t slot_bytes, int want) {
    TileLaunch L;
    L.cap = (std::max(want, op->tile.n + 1) + 7) & ~7;  // a batched row: the diagonal and every term
    const int rounds = (op->tile.n + 31) / 32;
    const size_t per_warp = slot_bytes ? scratch_bytes(rounds) + (size_t)L.cap * slot_bytes : 4 * kSpinWords + (size_t)rounds * 128;
    for (L.block = 256; L.block > 32; L.block /= 2)
        if (tile_smem(op->tile) + L.block / 32 * per_warp <= 227 * 1024) break;
    L.smem = tile_smem(op->tile) + L.block / 32 * per_warp;
    return L;
}

// Determines op->closed: with a hash index, one pass of compared lookups; a first miss ends it.  With one operator of
// each pair it takes 209 us on the 64-spin Q=0 basis and 3.2 ms on the 96-spin 8.8.16.16 sector, 305 us and 5.8 ms with
// both.  Applies of a closed operator take a tag match for the state itself, which saves each of their lookups the 16-byte
// load of the state at the index found.
qsi_status find_closed(qsi_op* op) {
    op->closed = 0;
    if (!op->basis->d_bins) return QSI_OK;
    const TileParams P = tile_params(op, 0);
    cudaStream_t st = op->stream;
    Closure* d_out = nullptr;
    QSI_CUDA(cudaMallocAsync(&d_out, sizeof(Closure), st));
    cudaError_t e = cudaMemsetAsync(d_out, 0, sizeof(Closure), st);
    const int64_t ntiles = (P.B.n + 31) / 32;
    const LookupBins<false> lk{op->basis->bview()};
    auto k = op->tile.reversible ? k_find_miss<true, LookupBins<false>> : k_find_miss<false, LookupBins<false>>;
    const TileLaunch L = tile_launch(op, 4, kListCap);
    if (L.smem > 48 * 1024) cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L.smem);
    k<<<grid_for(ntiles, L.block / 32), L.block, L.smem, st>>>(P, lk, d_out, L.cap);
    Closure c{0, 1};
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(&c, d_out, sizeof(c), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    cudaFreeAsync(d_out, st);
    if (e != cudaSuccess) return fail(QSI_CUDA_ERROR, "qsi_op_create (closure): %s", cudaGetErrorString(e));
    op->closed = !c.missed && !c.skew;
    return QSI_OK;
}

// ------------------------------------------------------------------ lookup cache (materialised operator)
// Single-vector apply of a materialised operator: a sliced-ELL product over the cache alone (no states, no
// admission test): lane l of tile t sums row 32 t + l as the diagonal, then its entries in cache order (the
// admission order of the tile kernels) with coefficient +-cs of the entry's term and the entry's sign, the same
// sums in the same order as k_apply_tile, so the result is bitwise the matrix-free one.
//
// Latency-bound: six entries in flight per lane at 40 registers and six resident blocks.  With eight (64 registers, four
// blocks, and 11.5 entries per tile padded to 16) the 64-spin Q=0 basis takes 166 us against 93, the 96-spin 8.8.16.16
// sector 2.34 ms against 1.29; four entries at eight blocks 95 us and 1.38 ms.
constexpr int kCachedBlocks = 6;
template <typename XT, typename YT, typename TT>
__global__ void __launch_bounds__(256, kCachedBlocks) k_apply_cached(const double* __restrict__ coef, int n_off,
                                                      const double* __restrict__ diag, CacheView C,
                                                      const TT* __restrict__ tids, int64_t n, const XT* __restrict__ x,
                                                      YT* __restrict__ y, int accumulate) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double* cs = reinterpret_cast<double*>(smem_raw);
    for (int k = threadIdx.x; k < n_off; k += blockDim.x) cs[k] = coef[k];
    __syncthreads();
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int64_t ntiles = (n + 31) >> 5;
    for (int64_t tile = (int64_t)blockIdx.x * nw + wid; tile < ntiles; tile += (int64_t)gridDim.x * nw) {
        const int64_t row = tile * 32 + lane;
        const bool valid = row < n;
        const uint64_t o0 = C.off[tile];
        const int width = (int)(C.off[tile + 1] - o0);
        double acc = valid ? diag[row] * widen(x[row]) : 0.0;
        const uint32_t* cp = C.cols + o0 * 32 + lane;
        const TT* tp = tids + o0 * 32 + lane;
        constexpr int kU = 6;  // entries in flight per lane
        for (int k0 = 0; k0 < width; k0 += kU) {
            uint32_t c[kU];
            TT t[kU];
            XT xv[kU];
#pragma unroll
            for (int u = 0; u < kU; ++u) {
                const bool in = k0 + u < width;
                c[u] = in ? __ldg(cp + (uint64_t)(k0 + u) * 32) : kEmpty;
                t[u] = in ? __ldg(tp + (uint64_t)(k0 + u) * 32) : (TT)0;
            }
#pragma unroll
            for (int u = 0; u < kU; ++u) xv[u] = (c[u] != kEmpty) ? x[c[u] & ~kCacheNeg] : (XT)0;
#pragma unroll
            for (int u = 0; u < kU; ++u)
                if (c[u] != kEmpty && above_tol(xv[u])) {
                    // -cs for a negative entry as a flip of the sign bit (integer work, exactly the negation), so
                    // the FP64 pipe, GB300's bottleneck here, sees one multiply-add per hit
                    const double v = __longlong_as_double(__double_as_longlong(cs[t[u]]) ^
                                                          ((unsigned long long)(c[u] & kCacheNeg) << 32));
                    acc += v * widen<true>(xv[u]);
                }
        }
        if (valid) {
            if (accumulate) acc += widen(y[row]);
            y[row] = (YT)acc;
        }
    }
}

static CacheView cache_view(const qsi_op* op) {
    return CacheView{op->d_cache_cols, op->d_cache_off, op->d_cache_tid, op->cache_tid_bytes};
}

static qsi_status launch_cached(qsi_op* op, const void* x, void* y, int xdtype, int ydtype, int accumulate,
                                cudaStream_t st) {
    const int64_t n = op->basis->n;
    const int block = 256, nw = block / 32;
    const int64_t ntiles = (n + 31) / 32;
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    // four waves of the resident blocks: 8 blocks per SM, one wave and a third, took 114 us on the 64-spin Q=0 basis
    const int bps = op->tune[0].grid_bps > 0 ? op->tune[0].grid_bps : 4 * kCachedBlocks;
    const int grid = (int)std::max<int64_t>(1, std::min<int64_t>((ntiles + nw - 1) / nw, (int64_t)sms * bps));
    const size_t smem = (size_t)std::max(op->tile.n, 1) * 8;
    const CacheView C = cache_view(op);
    auto go = [&](auto xt, auto yt, auto tt) {
        using XT = decltype(xt);
        using YT = decltype(yt);
        using TT = decltype(tt);
        auto k = k_apply_cached<XT, YT, TT>;
        if (smem > 48 * 1024) cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        k<<<grid, block, smem, st>>>(op->tile.cs, op->tile.n, op->d_diag, C, (const TT*)op->d_cache_tid, n,
                                     (const XT*)x, (YT*)y, accumulate);
    };
    auto by_tid = [&](auto xt, auto yt) {
        if (op->cache_tid_bytes == 1) go(xt, yt, uint8_t{});
        else go(xt, yt, uint16_t{});
    };
    if (xdtype == QSI_F64) by_tid(double{}, double{});
    else if (ydtype == QSI_F64) by_tid(float{}, double{});
    else by_tid(float{}, float{});
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return fail(QSI_CUDA_ERROR, "cached apply launch: %s", cudaGetErrorString(e));
    return QSI_OK;
}


// 4 .. 32 FP32 vectors of a materialised operator (vec4_ok): R / 4 lanes of four vectors each sum a row, 128 / R rows per
// warp at once, reading the cache where it lies.  The diagonal, then the entries in cache order in double-float, as in
// k_apply_tile_batched, so the results are bitwise its.
//
// k_apply_tile_batched reads the cache twice and passes every entry through its list in shared memory, whose size and
// whose registers leave three blocks per SM; here it is four, waiting for gathers.  Against it, in us:
//   vectors                  4             16             32             64
//   64-spin Q=0              441 -> 187    716 -> 571     1086 -> 1074   1781 -> 2072
//   96-spin 8.8.16.16        8545 -> 2993  12269 -> 9342  18289 -> 16578 28492 -> 31712
// Each row's columns and terms are read by all its lanes, from 64 vectors on by too many.  Other depths: six entries in
// flight and three blocks 186, 612, 1171 us at 4, 16, 32 vectors (64-spin), more blocks spill.
constexpr int kCachedVecMax = 32;
constexpr int kCachedVecBlocks = 4;
template <typename TT, bool kSplit>
__global__ void __launch_bounds__(256, kCachedVecBlocks) k_apply_cached_vec4(const float2* __restrict__ coef, int n_off,
                                                      const float2* __restrict__ diag_ff, CacheView C,
                                                      const TT* __restrict__ tids, int64_t n, const float* __restrict__ x,
                                                      float* __restrict__ y, int R, int accumulate,
                                                      const float2* __restrict__ ycoef) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float2* cs = reinterpret_cast<float2*>(smem_raw);
    for (int k = threadIdx.x; k < n_off; k += blockDim.x) cs[k] = coef[k];
    __syncthreads();
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int lpc = R / 4, cpw = 32 / lpc, g = lane / lpc, rr = 4 * (lane % lpc);
    const int64_t ntiles = (n + 31) >> 5;
    // a warp's share: a tile, or (kSplit) the cpw rows of a tile that it sums at once
    const int split = kSplit ? lpc : 1, rows = kSplit ? cpw : 32;
    for (int64_t part = (int64_t)blockIdx.x * nw + wid; part < ntiles * split; part += (int64_t)gridDim.x * nw) {
        const int64_t tile = part / split;
        const int first = kSplit ? (int)(part % split) * rows : 0;
        const uint64_t o0 = C.off[tile];
        const int width = (int)(C.off[tile + 1] - o0);
        const float* xr = x + rr;
        for (int l0 = first; l0 < first + rows; l0 += cpw) {
            const int64_t row = tile * 32 + l0 + g;
            const bool valid = row < n;
            const uint32_t* cp = C.cols + o0 * 32 + l0 + g;
            const TT* tp = tids + o0 * 32 + l0 + g;
            FF2 a0{0, 0}, a1{0, 0};
            auto add = [&](float2 f, const float4 v, bool all) {
                const uint64_t ch = pk2(f.x, f.x), cn = pk2(-f.x, -f.x), cl = pk2(f.y, f.y);
                ff2_fma(a0, ch, cn, cl, pk2(tol_select(v.x, all), tol_select(v.y, all)));
                ff2_fma(a1, ch, cn, cl, pk2(tol_select(v.z, all), tol_select(v.w, all)));
            };
            constexpr int kU = 4;  // entries in flight per lane, and as many columns read ahead
            uint32_t c[kU];
            TT t[kU];
            auto fetch = [&](int k0) {
#pragma unroll
                for (int u = 0; u < kU; ++u) {
                    const bool in = k0 + u < width;
                    c[u] = in ? __ldg(cp + (uint64_t)(k0 + u) * 32) : kEmpty;
                    t[u] = in ? __ldg(tp + (uint64_t)(k0 + u) * 32) : (TT)0;
                }
            };
            fetch(0);
            if (valid) add(diag_ff[row], *reinterpret_cast<const float4*>(xr + row * R), true);
            for (int k0 = 0; k0 < width; k0 += kU) {
                float4 v[kU];
                float2 f[kU];
#pragma unroll
                for (int u = 0; u < kU; ++u) {
                    v[u] = make_float4(0.f, 0.f, 0.f, 0.f);
                    f[u] = make_float2(0.f, 0.f);
                    if (c[u] == kEmpty) continue;
                    v[u] = *reinterpret_cast<const float4*>(xr + (int64_t)(c[u] & ~kCacheNeg) * R);
                    f[u] = cs[t[u]];
                    if (c[u] & kCacheNeg) f[u] = make_float2(-f[u].x, -f[u].y);
                }
                fetch(k0 + kU);
#pragma unroll
                for (int u = 0; u < kU; ++u) add(f[u], v[u], false);
            }
            if (!valid) continue;
            float4* yp = reinterpret_cast<float4*>(y + row * R + rr);
            if (accumulate) {
                const float4 yv = *yp;
                if (ycoef) {
                    const float4 ca = *reinterpret_cast<const float4*>(ycoef + rr);
                    const float4 cb = *reinterpret_cast<const float4*>(ycoef + rr + 2);
                    ff2_fma(a0, pk2(ca.x, ca.z), pk2(-ca.x, -ca.z), pk2(ca.y, ca.w), pk2(yv.x, yv.y));
                    ff2_fma(a1, pk2(cb.x, cb.z), pk2(-cb.x, -cb.z), pk2(cb.y, cb.w), pk2(yv.z, yv.w));
                } else {
                    const uint64_t one = pk2(1.0f, 1.0f), mone = pk2(-1.0f, -1.0f), zero = pk2(0.f, 0.f);
                    ff2_fma(a0, one, mone, zero, pk2(yv.x, yv.y));
                    ff2_fma(a1, one, mone, zero, pk2(yv.z, yv.w));
                }
            }
            const float2 a = unpk2(add2(a0.hi, a0.lo)), b = unpk2(add2(a1.hi, a1.lo));
            *yp = make_float4(a.x, a.y, b.x, b.y);
        }
    }
}

static qsi_status launch_cached_vec4(qsi_op* op, const float* x, float* y, int R, int accumulate, const float2* ycoef,
                                     cudaStream_t st) {
    const int64_t n = op->basis->n, ntiles = (n + 31) / 32;
    const qsi_tuning& T = op->tune[1];
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int bps = T.grid_bps > 0 ? T.grid_bps : 4 * kCachedVecBlocks;
    // Fewer tiles than resident warps: a tile's row sets go to warps of their own instead of one after another (32 vectors:
    // 7,236 rows 20.5 -> 8 us, 18.5 for the batched kernel before this one; 36,056 rows 29 -> 19 us).  With more tiles every
    // warp has work anyway, and the shared loop costs 1-3% (2.9 M rows, 32 vectors: 1048 -> 1077 us).
    const bool split = R > 4 && ntiles <= (int64_t)sms * kCachedVecBlocks * 8;
    const int64_t parts = ntiles * (split ? R / 4 : 1);
    const int grid = (int)std::max<int64_t>(1, std::min<int64_t>((parts + 7) / 8, (int64_t)sms * bps));
    const size_t smem = (size_t)std::max(op->tile.n, 1) * 8;
    auto go = [&](auto tt) {
        using TT = decltype(tt);
        auto k = split ? k_apply_cached_vec4<TT, true> : k_apply_cached_vec4<TT, false>;
        k<<<grid, 256, smem, st>>>(op->tile.ff, op->tile.n, op->d_diag_ff, cache_view(op), (const TT*)op->d_cache_tid, n, x, y,
                                   R, accumulate, ycoef);
    };
    if (op->cache_tid_bytes == 1) go(uint8_t{});
    else go(uint16_t{});
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return fail(QSI_CUDA_ERROR, "cached apply launch: %s", cudaGetErrorString(e));
    return QSI_OK;
}

// Admitted terms of the tile's widest row: the tile's number of cache lines.
__global__ void __launch_bounds__(256) k_cache_widths(TileParams P, uint64_t* __restrict__ width) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const TileSmem S = stage_terms(P, LookupTable{P.B}, false, smem_raw);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int n_rounds = (P.T.n + 31) >> 5;
    const WarpScratch W = warp_scratch(S.tail + wid * scratch_bytes(n_rounds), n_rounds);
    const int64_t ntiles = (P.B.n + 31) >> 5;
    for (int64_t tile = (int64_t)blockIdx.x * nw + wid; tile < ntiles; tile += (int64_t)gridDim.x * nw) {
        const int64_t row = tile * 32 + lane;
        const bool valid = row < P.B.n;
        const state2 s = valid ? P.B.states[row] : make_ulonglong2(0, 0);
        int cnt = tile_admit(S, P, LookupTable{P.B}, W, s, row, n_rounds, lane);
#pragma unroll
        for (int o = 16; o; o >>= 1) cnt = max(cnt, __shfl_xor_sync(0xffffffffu, cnt, o));
        if (lane == 0) width[tile] = (uint64_t)cnt;
        __syncwarp();
    }
}

// The column of every admitted term of every row (kEmpty outside the basis), looked up with lk, at the positions
// LookupCache reads them from.
template <class LK, typename TT>
__global__ void __launch_bounds__(256) k_cache_fill(TileParams P, LK lk, const uint64_t* __restrict__ off,
                                                    uint32_t* __restrict__ cols, TT* __restrict__ tids, int cap) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const TileSmem S = stage_terms(P, lk, false, smem_raw);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int n_rounds = (P.T.n + 31) >> 5;
    const bool has_z = P.T.z != nullptr;
    const WarpScratch W = warp_scratch(S.tail + wid * (scratch_bytes(n_rounds) + (size_t)cap * 4), n_rounds);
    const int64_t ntiles = (P.B.n + 31) >> 5;
    for (int64_t tile = (int64_t)blockIdx.x * nw + wid; tile < ntiles; tile += (int64_t)gridDim.x * nw) {
        const int64_t row = tile * 32 + lane;
        const bool valid = row < P.B.n;
        const state2 s = valid ? P.B.states[row] : make_ulonglong2(0, 0);
        const int cnt = tile_admit(S, P, lk, W, s, row, n_rounds, lane);
        const uint64_t o0 = off[tile] * 32;
        for (int row_start = 0; row_start < 32;) {
            int base;
            const int row_end = chunk_rows(row_start, cnt, cap, lane, base);
            const int total = list_hits(W, row_mask(row_start, row_end), n_rounds, lane, 4);
            constexpr int kNB = 2;
            look_up_hits<kNB>(S, P, W, lk, tile, total, lane, 4,
                              [&](int, int n, const uint32_t (&e)[kNB], const uint32_t (&J)[kNB]) {
#pragma unroll
                for (int u = 0; u < kNB; ++u) {
                    if (u >= n) continue;
                    // the column, with the sign of the term's matrix element on this row in the top bit
                    const uint32_t t = hit_term(e[u]), l = hit_row(e[u]);
                    const bool neg = has_z && term_negative(S, true, t, P.B.states[tile * 32 + l]);
                    const uint64_t at = o0 + (uint64_t)hit_ordinal(e[u]) * 32 + l;
                    cols[at] = J[u] != kEmpty ? (J[u] | (neg ? kCacheNeg : 0u)) : kEmpty;
                    tids[at] = (TT)t;
                }
            });
            __syncwarp();
            row_start = row_end;
        }
    }
}

// ------------------------------------------------------------------ launchers
template <class K>
static void set_smem(K kernel, size_t smem) {
    if (smem > 48 * 1024) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
}

// Grid of one wave (the blocks that fit on the GPU at once, each working through tiles with a grid
// stride) or of bps blocks per SM when bps > 0; at most one block per 8 tiles.
template <class K>
static int one_wave(K kernel, int block, size_t smem, int64_t ntiles, int bps = 0) {
    int dev = 0, sms = 148, per_sm = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (bps > 0) per_sm = bps;
    else if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, block, smem) != cudaSuccess || per_sm < 1)
        per_sm = 1;
    return (int)std::max<int64_t>(1, std::min<int64_t>((ntiles + block / 32 - 1) / (block / 32), (int64_t)sms * per_sm));
}

// Grid of the single-vector tile kernels: several waves of blocks measured faster than one.
static int tile_grid(int64_t ntiles, int block, int bps) {
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int nw = block / 32;
    return (int)std::max<int64_t>(1, std::min<int64_t>((ntiles + nw - 1) / nw, (int64_t)sms * (bps > 0 ? bps : 8)));
}

// From kWideFrom vectors on eight per lane and a list of 512, since a row's look-ups then cost less beside its gathers; a
// cache has no look-ups and does best with four and at most 256, or sixteen where they are asked for (figures at the kernel).
BatchedChoice batched_choice(const qsi_op* op, int R, int dtype, const void* x, const void* y) {
    const qsi_tuning& T = op->tune[1];
    const int64_t n = op->basis->n;
    const bool gathers = dtype == QSI_F32 && op->ff_accumulate, cached = op->d_cache_cols != nullptr;
    int width = 4;
    if (gathers && T.vec_width == 16 && vec16_ok(n, R, x, y)) width = 16;
    else if (gathers && !cached && (T.vec_width == 8 || (T.vec_width == 0 && R >= kWideFrom)) && vec8_ok(n, R, x, y)) width = 8;
    int list = T.list_cap > 0 ? T.list_cap : width == 8 ? 512 : 256;
    if (gathers && cached && width == 4) list = std::min(list, 256);
    return {width, list};
}

template <class LK>
static qsi_status launch_tiles_lk(qsi_op* op, LK lk, const void* x, void* y, int R, int xdtype, int ydtype,
                                  int accumulate, cudaStream_t st, bool batched, const float2* ycoef) {
    const qsi_tuning& T = op->tune[batched];
    TileParams P = tile_params(op, T.vec_chunk);
    const int64_t ntiles = (P.B.n + 31) / 32;
    if (!batched) {
        if constexpr (std::is_same<LK, LookupCache>::value) return fail(QSI_INVALID_ARG, "tile apply: no cached form");
        else {
            auto go = [&](auto xt, auto yt) {
                using XT = decltype(xt);
                using YT = decltype(yt);
                auto k = k_apply_tile<XT, YT, LK>;
                const TileLaunch L = tile_launch(op, 0, 0);
                set_smem(k, L.smem);
                k<<<tile_grid(ntiles, L.block, T.grid_bps), L.block, L.smem, st>>>(P, lk, (const XT*)x, (YT*)y, accumulate);
            };
            if (xdtype == QSI_F64) go(double{}, double{});
            else if (ydtype == QSI_F64) go(float{}, double{});
            else go(float{}, float{});
        }
    } else {
        const BatchedChoice C = batched_choice(op, R, xdtype, x, y);
        const TileLaunch L = tile_launch(op, 16, C.list);
        const int block = L.block, cap = L.cap;
        const size_t smem = L.smem;
        if (smem > 227 * 1024) return fail(QSI_INVALID_ARG, "batched apply: %zu bytes of shared memory needed", smem);
        auto go = [&](auto km) -> void {
            constexpr int KM = decltype(km)::value;
            if (xdtype == QSI_F64) {
                auto k = k_apply_tile_batched<double, LK, false, KM>;
                set_smem(k, smem);
                k<<<one_wave(k, block, smem, ntiles, T.grid_bps), block, smem, st>>>(P, lk, (const double*)x, (double*)y, R,
                                                                         accumulate, cap, ycoef);
            } else if (op->ff_accumulate) {
                auto k = C.width == 16             ? k_apply_tile_batched<float, LK, true, kVec16>
                         : vec4_ok(P.B.n, R, x, y) ? k_apply_tile_batched<float, LK, true, kVec4>
                                                   : k_apply_tile_batched<float, LK, true, KM>;
                if constexpr (!std::is_same<LK, LookupCache>::value)
                    if (C.width == 8) k = k_apply_tile_batched<float, LK, true, kVec8>;
                set_smem(k, smem);
                k<<<one_wave(k, block, smem, ntiles, T.grid_bps), block, smem, st>>>(P, lk, (const float*)x, (float*)y, R,
                                                                         accumulate, cap, ycoef);
            } else {
                auto k = k_apply_tile_batched<float, LK, false, KM>;
                set_smem(k, smem);
                k<<<one_wave(k, block, smem, ntiles, T.grid_bps), block, smem, st>>>(P, lk, (const float*)x, (float*)y, R,
                                                                         accumulate, cap, ycoef);
            }
        };
        if (R <= kGroupMax) go(std::integral_constant<int, kGroup>{});
        else if (R <= 32) go(std::integral_constant<int, 1>{});
        else if (R <= 64) go(std::integral_constant<int, 2>{});
        else go(std::integral_constant<int, 4>{});
    }
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return fail(QSI_CUDA_ERROR, "tile apply launch: %s", cudaGetErrorString(e));
    return QSI_OK;
}

qsi_status preload_apply_f64_rows();  // operator.cu: the row-per-thread kernel

qsi_status preload_apply_f64() {
    cudaFuncAttributes a;
    QSI_CUDA(cudaFuncGetAttributes(&a, k_apply_tile<double, double, LookupBins<true>>));
    QSI_CUDA(cudaFuncGetAttributes(&a, k_apply_tile<double, double, LookupBins<false>>));
    QSI_CUDA(cudaFuncGetAttributes(&a, k_apply_tile<double, double, LookupTable>));
    return preload_apply_f64_rows();
}

// Family mode applies of the template operator tmpl: y = H(p_c) x per column c (FP64, [row][R]), fcoef
// [classes][R] on the device.  One column runs the single-vector tile kernel, several the batched one; both sum a
// row in the same order, so a column's result does not depend on R.
template <class LK>
static qsi_status launch_family_lk(qsi_op* tmpl, LK lk, const double* x, double* y, int R, const double* fcoef,
                                   int accumulate, cudaStream_t st) {
    const qsi_tuning& T = tmpl->tune[0];
    TileParams P = tile_params(tmpl, 0);
    P.fcoef = fcoef;
    P.fR = R;
    const int64_t ntiles = (P.B.n + 31) / 32;
    if (R == 1) {
        const TileLaunch L = tile_launch(tmpl, 0, 0);
        auto k = k_apply_tile<double, double, LK, true>;
        set_smem(k, L.smem);
        k<<<tile_grid(ntiles, L.block, T.grid_bps), L.block, L.smem, st>>>(P, lk, x, y, accumulate);
    } else if (R <= 8) {  // a few columns: every lane sums all columns of its row
        const TileLaunch L = tile_launch(tmpl, 4, kListCap);
        auto k = (R <= 2) ? k_apply_tile_cols<LK, 2> : (R <= 4) ? k_apply_tile_cols<LK, 4> : k_apply_tile_cols<LK, 8>;
        set_smem(k, L.smem);
        k<<<tile_grid(ntiles, L.block, 0), L.block, L.smem, st>>>(P, lk, x, y, accumulate, L.cap);
    } else {
        const TileLaunch L = tile_launch(tmpl, 16, batched_choice(tmpl, R, QSI_F64, x, y).list);
        const int block = L.block, cap = L.cap;
        const size_t smem = L.smem;
        if (smem > 227 * 1024) return fail(QSI_INVALID_ARG, "family apply: %zu bytes of shared memory needed", smem);
        auto go = [&](auto km) {
            constexpr int KM = decltype(km)::value;
            auto k = k_apply_tile_batched<double, LK, false, KM, true>;
            set_smem(k, smem);
            k<<<one_wave(k, block, smem, ntiles, tmpl->tune[1].grid_bps), block, smem, st>>>(P, lk, x, y, R, accumulate,
                                                                                             cap, nullptr);
        };
        if (R <= kGroupMax) go(std::integral_constant<int, kGroup>{});
        else if (R <= 32) go(std::integral_constant<int, 1>{});
        else if (R <= 64) go(std::integral_constant<int, 2>{});
        else go(std::integral_constant<int, 4>{});
    }
    QSI_CUDA(cudaGetLastError());
    return QSI_OK;
}

qsi_status launch_family(qsi_op* tmpl, const double* x, double* y, int R, const double* fcoef, int accumulate,
                         cudaStream_t st) {
    if (R < 1 || R > 128) return fail(QSI_INVALID_ARG, "family apply: %d columns (1..128)", R);
    if (tmpl->basis->d_bins && tmpl->tune[R > 1].use_hash) {
        if (tmpl->closed)
            return launch_family_lk(tmpl, LookupBins<true>{tmpl->basis->bview()}, x, y, R, fcoef, accumulate, st);
        return launch_family_lk(tmpl, LookupBins<false>{tmpl->basis->bview()}, x, y, R, fcoef, accumulate, st);
    }
    return launch_family_lk(tmpl, LookupTable{tmpl->basis->view()}, x, y, R, fcoef, accumulate, st);
}

static qsi_status launch_tiles(qsi_op* op, const void* x, void* y, int R, int xdtype, int ydtype, int accumulate,
                               cudaStream_t st, bool batched, const float2* ycoef) {
    auto go = [&](auto lk) { return launch_tiles_lk(op, lk, x, y, R, xdtype, ydtype, accumulate, st, batched, ycoef); };
    if (op->d_cache_cols) {
        if (batched && xdtype == QSI_F32 && op->ff_accumulate && R <= kCachedVecMax &&
            vec4_ok(op->basis->n, R, x, y))
            return launch_cached_vec4(op, (const float*)x, (float*)y, R, accumulate, ycoef, st);
        return go(LookupCache{cache_view(op)});
    }
    if (op->basis->d_bins && op->tune[batched].use_hash) {
        if (op->closed) return go(LookupBins<true>{op->basis->bview()});
        return go(LookupBins<false>{op->basis->bview()});
    }
    return go(LookupTable{op->basis->view()});
}

qsi_status launch_apply_tiles(qsi_op* op, const void* x, void* y, int R, int xdtype, int ydtype, int accumulate,
                              cudaStream_t st) {
    if (R == 1 && op->d_cache_cols) return launch_cached(op, x, y, xdtype, ydtype, accumulate, st);
    return launch_tiles(op, x, y, R, xdtype, ydtype, accumulate, st, R > 1, nullptr);
}

qsi_status launch_apply_ff(qsi_op* op, const float* x, float* y, int R, int accumulate, const float2* ycoef,
                           cudaStream_t st) {
    return launch_tiles(op, x, y, R, QSI_F32, QSI_F32, accumulate, st, true, ycoef);
}

// Allocates and frees the operator's lookup cache: a solve's own (cache_pooled) in the order of the operator's stream, so
// that solves overlap, a handle's behind the applies of every stream (cudaFree waits for them).
static cudaError_t cache_alloc(qsi_op* op, void** p, size_t bytes) {
    return op->cache_pooled ? cudaMallocAsync(p, bytes, op->stream) : cudaMalloc(p, bytes);
}
static void drop_cache(qsi_op* op) {
    for (void* p : {(void*)op->d_cache_cols, (void*)op->d_cache_off, op->d_cache_tid}) {
        if (op->cache_pooled) cudaFreeAsync(p, op->stream);
        else cudaFree(p);
    }
    op->d_cache_cols = nullptr;
    op->d_cache_off = nullptr;
    op->d_cache_tid = nullptr;
    op->cache_entries = 0;
}

// Builds (enable) or frees the operator's lookup cache; *bytes: its size.  A cache of more than `most` bytes is not
// built (QSI_OK, 0 bytes).
qsi_status materialise(qsi_op* op, bool enable, int64_t* bytes, size_t most) {
    drop_cache(op);
    if (enable) {
        if (op->kernel != 1) return fail(QSI_INVALID_ARG, "qsi_op_materialise: the cache serves the tile kernels (kernel 1)");
        cudaStream_t st = op->stream;
        const int64_t ntiles = (op->basis->n + 31) / 32;
        TileParams P = tile_params(op, 0);
        const TileLaunch L = tile_launch(op, 4, kListCap);
        const int grid = tile_grid(ntiles, L.block, 8);
        // widths, their exclusive scan (tile offsets in cache lines), then the columns
        // the scratch arrays are freed, and a failure leaves no partial cache behind, on every path out
        uint64_t* width = nullptr;
        void* tmp = nullptr;
        auto scratch_free = [&]() {
            cudaFreeAsync(tmp, st);
            cudaFreeAsync(width, st);
            tmp = nullptr;
            width = nullptr;
        };
        auto fail_partial = [&](cudaError_t e, const char* what) {
            scratch_free();
            drop_cache(op);
            return fail(e == cudaErrorMemoryAllocation ? QSI_OOM : QSI_CUDA_ERROR, "qsi_op_materialise: %s: %s", what,
                        cudaGetErrorString(e));
        };
        cudaError_t e = cudaMallocAsync(&width, (size_t)(ntiles + 1) * 8, st);
        if (e == cudaSuccess) e = cache_alloc(op, (void**)&op->d_cache_off, (size_t)(ntiles + 1) * 8);
        if (e == cudaSuccess) e = cudaMemsetAsync(width + ntiles, 0, 8, st);
        if (e != cudaSuccess) return fail_partial(e, "tile offsets");
        set_smem(k_cache_widths, L.smem);
        k_cache_widths<<<grid, L.block, L.smem, st>>>(P, width);
        size_t tmp_bytes = 0;
        e = cub::DeviceScan::ExclusiveSum(nullptr, tmp_bytes, width, op->d_cache_off, ntiles + 1, st);
        if (e == cudaSuccess) e = cudaMallocAsync(&tmp, tmp_bytes, st);
        if (e == cudaSuccess) e = cub::DeviceScan::ExclusiveSum(tmp, tmp_bytes, width, op->d_cache_off, ntiles + 1, st);
        uint64_t lines = 0;
        if (e == cudaSuccess) e = cudaMemcpyAsync(&lines, op->d_cache_off + ntiles, 8, cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        if (e != cudaSuccess) return fail_partial(e, "tile widths");
        scratch_free();
        const size_t n_entries = (size_t)lines * 32;
        op->cache_tid_bytes = op->tile.n <= 256 ? 1 : 2;
        if (n_entries * (4 + op->cache_tid_bytes) > most) {
            drop_cache(op);
            if (bytes) *bytes = 0;
            return QSI_OK;
        }
        e = cache_alloc(op, (void**)&op->d_cache_cols, std::max<size_t>(n_entries, 1) * 4);
        if (e == cudaSuccess) e = cache_alloc(op, &op->d_cache_tid, std::max<size_t>(n_entries, 1) * op->cache_tid_bytes);
        if (e != cudaSuccess) {
            drop_cache(op);
            return fail(e == cudaErrorMemoryAllocation ? QSI_OOM : QSI_CUDA_ERROR,
                        "qsi_op_materialise: %zu bytes for the cache: %s", n_entries * (4 + op->cache_tid_bytes),
                        cudaGetErrorString(e));
        }
        auto unfilled = [&](cudaError_t err) {  // a cache that was not filled completely is never used
            drop_cache(op);
            return fail(QSI_CUDA_ERROR, "qsi_op_materialise: %s", cudaGetErrorString(err));
        };
        e = cudaMemsetAsync(op->d_cache_cols, 0xFF, n_entries * 4, st);  // the lanes below their tile's width
        if (e == cudaSuccess) e = cudaMemsetAsync(op->d_cache_tid, 0, n_entries * op->cache_tid_bytes, st);
        if (e != cudaSuccess) return unfilled(e);
        auto fill = [&](auto lk, auto* tids) {
            auto k = k_cache_fill<decltype(lk), std::remove_pointer_t<decltype(tids)>>;
            set_smem(k, L.smem);
            k<<<grid, L.block, L.smem, st>>>(P, lk, op->d_cache_off, op->d_cache_cols, tids, L.cap);
        };
        auto by_tid = [&](auto lk) {
            if (op->cache_tid_bytes == 1) fill(lk, (uint8_t*)op->d_cache_tid);
            else fill(lk, (uint16_t*)op->d_cache_tid);
        };
        if (!op->basis->d_bins) by_tid(LookupTable{op->basis->view()});
        else if (op->closed) by_tid(LookupBins<true>{op->basis->bview()});
        else by_tid(LookupBins<false>{op->basis->bview()});
        e = cudaGetLastError();
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        if (e != cudaSuccess) return unfilled(e);
        op->cache_entries = n_entries;
    }
    if (bytes)
        *bytes = op->d_cache_cols ? (int64_t)(op->cache_entries * (4 + op->cache_tid_bytes) +
                                              ((op->basis->n + 31) / 32 + 1) * 8)
                                  : 0;
    return QSI_OK;
}

// Rows from which a solve builds its own cache, and applies after which it does: those that pay for the building and the
// release.  2.9 M rows (64-spin Q=0 basis): 276 -> 93 us per apply against 0.78 ms; 31 M (96-spin 8.8.16.16 sector): 4.8 ->
// 1.3 ms against 8.5 ms; 221,628: 36 -> 12.5 us against 0.37 ms; 15,528: 14.7 -> 8.0 us against 0.08 ms; 3,618 rows
// (10.4 -> 7.9 us) are launch-bound, and a solve of 115 applies takes 5.25 ms instead of 5.18.
constexpr int64_t kCacheMinRows = 8192;
static int64_t applies_for_cache(int64_t n) { return n >= (1 << 20) ? 6 : 16; }

// The solves that hold a cache, and how often memory was asked of them.
struct SolveCaches {
    struct Holder {
        int device;
        uint64_t asked;  // when the cache was built
    };
    std::mutex m;
    std::condition_variable gone;
    std::map<const SolveOp*, Holder> live;
    std::atomic<uint64_t> asked{0};
};
static SolveCaches& solve_caches() {
    static SolveCaches c;
    return c;
}

void SolveOp::plan(int64_t applies) {
    const int64_t n = op_->basis->n;
    if (tried_ || op_->kernel != 1 || op_->family || op_->d_cache_cols || n < kCacheMinRows ||
        n >= ((int64_t)1 << 31) - 1 || applies < applies_for_cache(n) || op_->solve_cache == 0)
        return;
    tried_ = true;
    size_t free_b = 0, total_b = 0;
    if (cudaMemGetInfo(&free_b, &total_b) == cudaSuccess) {
        view_ = *op_;
        view_.cache_pooled = true;
        const size_t most = free_b / 4;
        materialise(&view_, true, nullptr, op_->solve_cache < 0 ? most : std::min(most, (size_t)op_->solve_cache));
    }
    cudaGetLastError();  // without a cache the solve applies the operator as it is
    if (view_.d_cache_cols) {
        SolveCaches& c = solve_caches();
        std::lock_guard<std::mutex> l(c.m);
        asked_ = c.asked;
        c.live[this] = {op_->device, asked_};
    }
}

qsi_op* SolveOp::get() {
    if (view_.d_cache_cols && solve_caches().asked.load(std::memory_order_relaxed) != asked_) drop();
    return hold();
}

bool SolveOp::drop() {
    if (!view_.d_cache_cols) return false;
    drop_cache(&view_);
    SolveCaches& c = solve_caches();
    if (c.asked != asked_) {  // another thread waits for the memory: out of the pool, too
        cudaMemPool_t pool;
        cudaStreamSynchronize(op_->stream);
        if (cudaDeviceGetDefaultMemPool(&pool, op_->device) == cudaSuccess) cudaMemPoolTrimTo(pool, 0);
    }
    std::lock_guard<std::mutex> l(c.m);
    c.live.erase(this);
    c.gone.notify_all();
    return true;
}

bool reclaim_solve_caches() {
    int dev = 0;
    cudaGetLastError();
    if (cudaGetDevice(&dev) != cudaSuccess) return false;
    SolveCaches& c = solve_caches();
    std::unique_lock<std::mutex> l(c.m);
    const uint64_t mine = c.asked + 1;
    auto none = [&] {
        for (const auto& e : c.live)
            if (e.second.device == dev && e.second.asked < mine) return false;
        return true;
    };
    if (none()) return false;
    c.asked = mine;
    c.gone.wait(l, none);
    return true;
}

}  // namespace qsi

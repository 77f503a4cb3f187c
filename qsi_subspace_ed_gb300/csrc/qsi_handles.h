// Handle layouts behind the opaque qsi_basis / qsi_op pointers of the C-ABI.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <vector>

#include "qsi_device.cuh"

struct qsi_basis {
    int64_t n = 0;
    int bits = 0, shift = 0;
    uint32_t n_buckets = 0;
    qsi::state2* d_states = nullptr;
    uint2* d_tab = nullptr;
    int hb = 0;                      // highest bit used by any state
    int vb = 0;                      // highest bit in which two states differ
    uint64_t top0 = 0, top1 = 0;     // the bits above vb, which all states share
    uint32_t* d_bins = nullptr;      // optional hash index over the bucket table (states <= 96 bits)
    uint64_t n_bins = 0;
    uint2* d_keys = nullptr;         // ... and the states' keys
    uint32_t largest_bucket = 0;
    uint32_t off_mask = 0;           // offset field of a slot: wide enough for the largest bucket and two marks
    qsi::BasisView view() const { return qsi::BasisView{d_states, d_tab, n, shift, n_buckets, top0, top1}; }
    qsi::BinView bview() const { return qsi::BinView{view(), d_bins, d_keys, off_mask}; }
};

// Launch settings of one class of applies (single vector, batched).  None of them changes results.
struct qsi_tuning {
    int use_hash = 1;    // look columns up through the basis hash index when it exists (else bucket table)
    int list_cap = 0;    // hit-list entries per warp in the batched tile kernel (0: built-in choice)
    int grid_bps = 0;    // tile-kernel blocks per SM (0: built-in choice)
    int vec_chunk = 0;   // vectors per pass of the 16-byte batched kernel (0: up to 32 lanes' worth)
    int vec_width = 0;   // FP32 vectors per lane of the 16-byte batched kernel: 4, 8 or 16 (0: built-in choice)
};

struct qsi_family;

struct qsi_op {
    qsi_basis* basis = nullptr;
    qsi_family* family = nullptr;  // member of an operator family: FP64 single-vector applies join its batches
    double* d_fcoef = nullptr;     // the member's class coefficients on the device (family mode, one column)
    std::vector<double> fcoef;     // ... and on the host
    qsi::PullTerm* d_pull = nullptr;        // transposed off-diagonal terms (apply)
    qsi::PushTerm* d_push_off = nullptr;    // off-diagonal terms as given (export)
    qsi::PushTerm* d_push_diag = nullptr;   // diagonal terms as given (export)
    qsi::PushTerm* d_diag_generic = nullptr;
    int n_pull = 0, n_push_off = 0, n_push_diag = 0, n_diag_generic = 0;
    int n_pull_pruned = 0;                  // transposed terms removed because they map no row into the basis
    qsi::DiagSpec diag{};
    size_t smem_bytes = 0;
    unsigned char* d_tile_terms = nullptr;  // the tile kernels' term tables, one block (see TileTerms)
    qsi::TileTerms tile{};                  // views into it
    int closed = 0;                 // every admitted term of every row lands in the basis (find_closed)
    int nwords = 4;                 // 32-bit words that hold any basis or term bit
    int kernel = 1;                 // 0 = row-per-thread / warp-per-row, 1 = bit-sliced tiles
    int ff_accumulate = 1;          // FP32 batched applies accumulate rows in double-float (else FP64)
    qsi_tuning tune[2];             // [0] single-vector applies, [1] batched applies (R > 1)
    double* d_diag = nullptr;       // per-row diagonal (tile kernels)
    float2* d_diag_ff = nullptr;    // the same as double-float pairs (FP32 batched kernel)
    uint32_t* d_cache_cols = nullptr;  // lookup cache of the materialised operator (qsi_op_materialise), or null
    uint64_t* d_cache_off = nullptr;   // its tile offsets in 32-entry lines
    void* d_cache_tid = nullptr;       // the term index of every entry (uint8, or uint16 beyond 256 terms)
    int cache_tid_bytes = 1;
    size_t cache_entries = 0;
    bool cache_pooled = false;         // from the stream-ordered allocator (SolveOp)
    int64_t solve_cache = -1;          // most bytes for a solve's own cache (negative: SolveOp's quarter)
    cudaStream_t stream = nullptr;
    int device = 0;        // the device current at qsi_op_create (owner of every buffer and of the stream)
    void* d_x = nullptr;   // staging for host-pointer applies
    void* d_y = nullptr;
    size_t staging_bytes = 0;
};

namespace qsi {
int grid_for(int64_t n, int block);
qsi_status launch_apply(qsi_op* op, const void* x, void* y, int R, int dtype, int accumulate, cudaStream_t st);
// y = H x with x stored as xdtype and y always FP64 (single vector).
qsi_status launch_apply_to_f64(qsi_op* op, const void* x, double* y, int xdtype, cudaStream_t st);
qsi_status launch_apply_tiles(qsi_op* op, const void* x, void* y, int R, int xdtype, int ydtype, int accumulate,
                              cudaStream_t st);
// Family mode apply of a family's template operator: y = H(p_c) x per column c of [row][R] FP64 blocks.
qsi_status launch_family(qsi_op* tmpl, const double* x, double* y, int R, const double* fcoef, int accumulate,
                         cudaStream_t st);
// A member's single-vector FP64 apply, run in a batch with the family's other waiting members.
qsi_status family_apply(qsi_op* op, const double* x, double* y, int accumulate, cudaStream_t st);
// Called by qsi_op_destroy for a family member.
void family_release_member(qsi_op* op);
qsi_status build_hash(qsi_basis* b);
void drop_hash(qsi_basis* b);
// qsi_op_create; check_closed: determine op->closed (one pass of lookups over the basis), else it stays 0.
qsi_status create_op(qsi_basis* b, const qsi_term* terms, int32_t n_terms, bool check_closed, qsi_op** out);
// An off-diagonal term in the pull form of the applies.
PullTerm transposed_term(const qsi_term& t);
// Builds op->tile from the transposed terms.
qsi_status upload_tile_terms(qsi_op* op, const std::vector<PullTerm>& pull);
qsi_status find_closed(qsi_op* op);
// Builds (enable) or frees an operator's lookup cache (qsi_op_materialise); *bytes: its size in device memory.  A cache of
// more than `most` bytes is not built (QSI_OK, 0 bytes).
qsi_status materialise(qsi_op* op, bool enable, int64_t* bytes, size_t most = SIZE_MAX);

// An operator as one solve applies it: with a lookup cache of the solve's own, in a copy of the handle, once enough
// applies are known to use it and if it takes no more than a quarter of the free device memory, or less if the handle
// says so; the results are bitwise those of the operator without it.  A family's members apply in their family's
// batches and get none.
// The cache is memory to spare: the solve gives it up for its own later allocations (alloc) and, at its next apply or its
// end, for any call of another thread that ran out of memory (reclaim_solve_caches).
class SolveOp {
   public:
    explicit SolveOp(qsi_op* op) : op_(op) {}
    ~SolveOp() { drop(); }
    SolveOp(const SolveOp&) = delete;
    SolveOp& operator=(const SolveOp&) = delete;
    // applies: those done so far and those sure to follow.
    void plan(int64_t applies);
    // The operator for the next apply; for all applies of a graph: hold().
    qsi_op* get();
    qsi_op* hold() { return view_.d_cache_cols ? &view_ : op_; }
    // Frees the cache behind the applies enqueued on the operator's stream; whether there was one.
    bool drop();
    // An allocation on the operator's stream that comes before the cache when both don't fit.
    template <class Buf>
    cudaError_t alloc(Buf& b, size_t count) {
        cudaError_t e = b.alloc(count, op_->stream);
        if (e == cudaErrorMemoryAllocation && drop()) {
            cudaGetLastError();
            cudaStreamSynchronize(op_->stream);
            e = b.alloc(count, op_->stream);
        }
        return e;
    }

   private:
    qsi_op* op_;
    qsi_op view_;
    bool tried_ = false;
    uint64_t asked_ = 0;  // requests for memory when the cache was built
};
// Fills the bucket table of a basis at its current width (b->bits, b->shift, b->n_buckets).
qsi_status build_buckets(qsi_basis* b);
// Loads the single-vector FP64 apply kernels on the current device (CUDA loads device code lazily, on first use).
qsi_status preload_apply_f64();
// Looks the static staging arrays of qsi_op_apply_static up on the current device (once per device).
qsi_status static_stage_prepare();
qsi_status build_diag(qsi_op* op);
// What a batched apply of R vectors runs with: FP32 vectors per lane of its 16-byte gathers (4, 8 or 16) and hit-list entries
// per warp, as op->tune[1] asks for and R, the vectors' addresses and the operator's form allow.
struct BatchedChoice {
    int width, list;
};
BatchedChoice batched_choice(const qsi_op* op, int R, int dtype, const void* x, const void* y);
// Y <- H X + c Y for R FP32 vectors [row][R] summed in double-float (the tile kernels, also for R = 1): c = 0
// (accumulate = 0), 1, or per column the (hi, lo) float pair ycoef[column].
qsi_status launch_apply_ff(qsi_op* op, const float* x, float* y, int R, int accumulate, const float2* ycoef,
                           cudaStream_t st);
qsi_status jacobi_eigh(const std::vector<double>& A, int m, int n_mat, std::vector<double>& w, std::vector<double>& V, cudaStream_t st);
}  // namespace qsi

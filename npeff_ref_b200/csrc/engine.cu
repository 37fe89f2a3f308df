// Host side of the D-NPEFF engine and its C ABI (see include/dnpeff.h).
//
// One engine = one column shard of the pruned PEF matrix A on one device:
//   A  as CSR (rows = examples) and CSC (rows = features), fp32 + int32 + int64 offsets
//   W  [n_rows, ld] row-major, replicated on every engine of a job
//   H  [n_cols_shard, ld] row-major: the reference's column-major r x m_s matrix
//      (multi_mu_dense_factors_device_contexts1.h:413-429), rows ld floats apart
//   ld = r, or r rounded up to a rank of the tensor-core kernels (padded_rank) with columns
//   r .. ld zero in W, H, both products and both Gram matrices
// Iteration (multi_mu_dense_factors_nmf1.h:175-182): W first, then H.
#include <algorithm>
#include <atomic>
#include <chrono>
#include <functional>
#include <mutex>
#include <vector>

#include "common.cuh"
#include "kernels_dense.cuh"
#include "kernels_hoyer.cuh"
#include "kernels_prep.cuh"
#include "kernels_small.cuh"
#include "kernels_spmm.cuh"
#include "kernels_tc.cuh"
#include "kernels_block.cuh"
#include "memory.cuh"
#include "nccl_dyn.h"
#include "transfer.cuh"

using namespace dnpeff;

namespace {

// Exclusive scan of N items into out[0..N) (int64).  Callers that want the
// total pass N+1 items whose last one is zero.
template <typename TIn>
int scan_exclusive(const TIn* in, int64_t* out, int64_t N, cudaStream_t st) {
    if (N <= 0) return DNPEFF_OK;
    int64_t nb = ceil_div(N, 4096);
    if (nb == 1) {
        k_scan_block<TIn><<<1, 1024, 0, st>>>(in, out, nullptr, N);
        DN_LAUNCH_CHECK();
        DN_COUNT_LAUNCH(1);
        return DNPEFF_OK;
    }
    DevBuf<int64_t> bs, bsp;
    DN_TRY(bs.alloc((size_t)nb));
    DN_TRY(bsp.alloc((size_t)nb));
    k_scan_block<TIn><<<(unsigned)nb, 1024, 0, st>>>(in, out, bs.p, N);
    DN_LAUNCH_CHECK();
    DN_TRY(scan_exclusive<int64_t>(bs.p, bsp.p, nb, st));
    k_scan_add<<<(unsigned)nb, 1024, 0, st>>>(out, bsp.p, N);
    DN_LAUNCH_CHECK();
    DN_COUNT_LAUNCH(2);
    if (!current_arena()) DN_CUDA(cudaStreamSynchronize(st));  // bs/bsp are released on return
    return DNPEFF_OK;
}

struct TimedRegion {
    int id;
    cudaEvent_t a, b;
};

}  // namespace

struct dnpeff_engine {
    dnpeff_params p;
    int device = 0;
    cudaStream_t st = nullptr;
    bool own_stream = false;
    cudaStream_t up = nullptr;  // uploads that overlap the loader; made by the first of them
    DeviceArena arena;          // all device memory of the engine

    int64_t n = 0, m_full = 0, m_kept = 0, c0 = 0, ms = 0, nnz = 0;
    int ld = 0;  // row stride of W, H and everything of their shape (padded_rank)
    ShardMap map = {0, 0, 1, 0, 0};
    bool loaded = false, have_factors = false, csc_ready = false, csc_hot_ready = false;

    float* a_vals = nullptr;
    int32_t* a_col = nullptr;
    int64_t* a_rowptr = nullptr;
    // CSC arrays.  With the popular block kept dense only the other columns are ever
    // read from the CSC: the arrays then hold entries [c_base, nnz) of the full CSC
    // (c_base = c_colptr[n_hot]) and are addressed through csc_vals()/csc_rows(),
    // which shift the pointers so that the offsets in c_colptr apply unchanged.
    float* c_vals = nullptr;
    int32_t* c_row = nullptr;
    int64_t* c_colptr = nullptr;
    int64_t c_base = 0;
    float* w_spare = nullptr;  // n x r, wide ranks only: a W update is written here, then W and w_spare change places
    int32_t* new_to_og = nullptr;

    // Internal column order: [n_hot popular columns][the rest], each in local-id
    // order.  H, WA and the CSC use it; perm[jp] = local id, inv_perm[local] = jp.
    int32_t* perm = nullptr;
    int32_t* inv_perm = nullptr;
    int64_t n_hot = 0;
    BucketMap bm = {0, 1, 1, 0, 0};
    int n_tail_blocks = 0;
    float* b_vals = nullptr;      // rows of A with entries grouped by bucket, internal ids
    int32_t* b_col = nullptr;
    uint32_t* tail_off = nullptr;  // [n][n_tail_blocks + 1]
    std::vector<int64_t> tail_nnz;  // stored entries per tail block
    int* work_counter = nullptr;
    int* d_err = nullptr;
    // Popular block of A kept dense for the tensor-core product (null: the popular
    // part goes through the tiled sparse kernel): x1 = rows x popular columns,
    // x2 = its transpose, both in the blocked layout of k_block_tc.
    __half* x1 = nullptr;
    __half* x2 = nullptr;
    BlockTcPlan plan_x1 = {}, plan_x2 = {};
    uint32_t* x1_max = nullptr;  // bits of the largest magnitude per row of x1; then
    uint32_t* x2_max = nullptr;  // per row of x2, and
    uint32_t* y_max[2] = {nullptr, nullptr};  // per column of the factor, of products in turn (ld words each), then
    unsigned long long* x1_sum = nullptr;     // sums that say where the halves do not do (blk_faint), per row of x1; then
    unsigned long long* x2_sum = nullptr;     // per row of x2, and
    unsigned char* blk_again = nullptr;       // a byte per row of a product
    __half* blk_ysplit = nullptr;
    float* blk_partial = nullptr;

    float* W = nullptr;
    float* H = nullptr;
    float* AHG = nullptr;  // [n*r | r*r]: A*H^T partial and H*H^T partial, one allreduce
    float* WA = nullptr;   // [ms*r], made on the first H update
    float* WW = nullptr;   // [r*r]
    float* gram_scratch = nullptr;
    size_t gram_scratch_floats = 0;
    float* tc_scratch = nullptr;  // 2*r*r: the update's small matrix split for the tensor cores
    double* words = nullptr;        // device: what the next pointers, d_err and work_counter point into
    double* red_partial = nullptr;  // device, 2*kRedBlocks doubles
    double* red_out = nullptr;      // device, 4 doubles
    void* h_pinned = nullptr;       // kPinnedBytes of page-locked host memory for scalar read-backs
    int64_t hot_nnz = 0;            // stored entries in popular columns
    SpmmPlan plan_csr, plan_csc;
    // small problems (kernels_small.cuh): cuts of the two sides, carries, partials
    SmallCut* small_cuts = nullptr;
    float* small_carry = nullptr;
    float* small_partial = nullptr;
    unsigned int* small_barrier = nullptr;
    bool small_ready = false;     // all of them, with the cuts made

    double a_sq = 0.0, a_sum = 0.0;
    double a_sq_global = -1.0;
    int64_t w_row_offset = 0;  // global index of this engine's first row (generated W only)

    ncclComm_t comm = nullptr;
    int comm_rank = 0, comm_size = 1;

    bool timing = false;
    std::vector<TimedRegion> regions;
    std::vector<cudaEvent_t> ev_pool;
    double t_ms[DNPEFF_N_TIMERS] = {0};
    int64_t t_n[DNPEFF_N_TIMERS] = {0};
    int64_t launches0 = 0;

    // dnpeff_set_option values; 0 = the built-in default
    int opt_loader_slabs = 0;
    int64_t opt_tail_block_bytes = 0;
    int opt_popular_divisor = 0;
    uint32_t opt_wait_limit = kTiledSpinLimit;
    bool opt_keep_csr = false;
    bool opt_refuse_cooperative = false;
    bool opt_keep_memory = false;
};

namespace {

int check_kernel_status(dnpeff_engine* e);

// A pointer `base` elements before p (never dereferenced below p + base).
template <typename T>
T* shifted(T* p, int64_t base) {
    return reinterpret_cast<T*>(reinterpret_cast<uintptr_t>(p) - (uintptr_t)base * sizeof(T));
}
float* csc_vals(const dnpeff_engine* e) { return shifted(e->c_vals, e->c_base); }
int32_t* csc_rows(const dnpeff_engine* e) { return shifted(e->c_row, e->c_base); }

constexpr int kRedBlocks = 4 * kNumSMs;
constexpr int kMaxHotTiles = 1024;            // tiles of popular columns per row walk
// Slice of H gathered per tail launch.  It has to stay L2-resident (126 MB, shared
// with the A*H^T accumulator and the streamed entries) while all rows sweep it, and
// every further launch costs about 11 us: 48 MB is the measured optimum on B200.
constexpr int64_t kTailBlockBytes = 48 << 20;
constexpr int kMaxTailBlocks = 512;
// Most that padding the rank may add to an engine of a sharded job: an eighth of the GPU's 180 GB.  The
// allreduce of A*H^T grows with the stride too, and is not bounded: by arithmetic 1.4 ns a row at rank 130 as 256 (504
// more bytes at 725 GB/s, twice), about what the CUDA cores take for the contractions of a row of W.
constexpr double kShardedPadBytes = 22.5e9;
constexpr int kSmallIters = 256;              // iterations per launch of the small-problem kernel
constexpr int kFitSteps = 256;                // W-only steps per launch (a tile's step takes 5 to 40 us)

struct DeviceGuard {
    int prev = -1;
    explicit DeviceGuard(int dev) {
        cudaGetDevice(&prev);
        if (prev != dev) cudaSetDevice(dev);
        else prev = -1;
    }
    ~DeviceGuard() {
        if (prev >= 0) cudaSetDevice(prev);
    }
};

struct ScopedTimer {
    dnpeff_engine* e;
    int id;
    cudaEvent_t a = nullptr, b = nullptr;
    ScopedTimer(dnpeff_engine* e_, int id_) : e(e_), id(id_) {
        if (!e->timing) return;
        a = get();
        b = get();
        cudaEventRecord(a, e->st);
    }
    ~ScopedTimer() {
        if (!e->timing) return;
        cudaEventRecord(b, e->st);
        e->regions.push_back({id, a, b});
    }
    cudaEvent_t get() {
        if (!e->ev_pool.empty()) {
            cudaEvent_t x = e->ev_pool.back();
            e->ev_pool.pop_back();
            return x;
        }
        cudaEvent_t x;
        cudaEventCreate(&x);
        return x;
    }
};

// DNPEFF_NO_TC=1 keeps the dense contractions on the CUDA-core kernels (A/B runs).
bool tensor_cores_enabled() {
    static int v = -1;
    if (v < 0) {
        const char* s = getenv("DNPEFF_NO_TC");
        v = (s && s[0] == '1') ? 0 : 1;
    }
    return v == 1;
}

// DNPEFF_TRACE=1 prints the wall time of the loader's phases to stderr (each
// phase is closed with a stream synchronisation, so the trace slows the load).
struct PhaseTrace {
    cudaStream_t st;
    bool on;
    std::chrono::high_resolution_clock::time_point t;
    explicit PhaseTrace(cudaStream_t s) : st(s) {
        const char* v = getenv("DNPEFF_TRACE");
        on = v && v[0] == '1';
        if (on) t = std::chrono::high_resolution_clock::now();
    }
    void mark(const char* what) {
        if (!on) return;
        cudaStreamSynchronize(st);
        auto n = std::chrono::high_resolution_clock::now();
        fprintf(stderr, "[dnpeff] %-28s %8.2f ms\n", what, std::chrono::duration<double, std::milli>(n - t).count());
        t = n;
    }
};

// Ranks that the tensor-core contractions do not take as they are get the next one they do take
// as row stride, with zero columns behind the real ones: they stay zero under the update (their
// numerators and Gram entries are zero, x = 0 * (0 / (0 + eps))), and the sparse products gather
// the real columns only.  That needs eps > 0: with eps = 0 the padding would divide 0 by 0.
// Above 512 only the gathers gain: a multiple of 4 keeps them on 16-byte loads.
int padded_rank(int r, float eps) {
    if (!tensor_cores_enabled() || !(eps > 0.f)) return r;
    if (r <= 128) return (r + 31) / 32 * 32;
    if (r <= 512) return (r + 127) / 128 * 128;
    return r <= 1024 ? (r + 3) / 4 * 4 : r;
}

// Popular columns hold at least ceil(n / div) entries.  In the dense tensor-core block a column of 20000
// rows costs 16 ns a product whatever it holds (rank 128), its entries 31 ps each in the sparse one: even at
// a 37th stored, and flat around it (ms per iteration at 16, 32, 48 and 64, configuration 2: 24.3, 22.7, 22.7, 23.4;
// a sixteenth of configuration 3, rank 256: -, 13.1, 13.1, 13.6; of 5, rank 512: -, 17.0, 17.0, 17.5; 5003 x 300007 at
// rank 100: -, 0.97, 0.98, 1.00).
// With few rows much of the block is the padding of its last tile.  The sparse tiled kernel needs longer columns.
int hot_divisor(const dnpeff_engine* e, bool dense, int64_t n) {
    if (e->opt_popular_divisor >= 2) return e->opt_popular_divisor;
    return dense ? (n >= 1024 ? 32 : 16) : 8;
}

// G = X^T X: tcgen05 kernel where the rank allows, CUDA-core kernel otherwise.  Gsplit (or NULL):
// where the update runs on the tensor cores, the same matrix in that kernel's layout.
int gram_any(const float* X, int64_t rows, int r, float* G, float* Gsplit, float* scratch, int* err, cudaStream_t st,
             uint32_t wait_limit = kTiledSpinLimit) {
    if (tensor_cores_enabled() && gram_tc_ok(r)) return gram_blk_launch(X, rows, r, G, Gsplit, scratch, err, st, wait_limit);
    if (tensor_cores_enabled() && gram_wide_ok(r) && rows > 0)
        return gram_wide_launch(X, rows, r, G, Gsplit, scratch, err, st, wait_limit);
    DN_TRY(gram_launch(X, rows, r, G, scratch, st));
    if (Gsplit && tensor_cores_enabled() && (mu_update_ws_ok(r) || mu_update_ws_wide_ok(r)))
        DN_TRY(tc_split_g_launch(G, r, Gsplit, st));
    return DNPEFF_OK;
}

size_t gram_any_scratch(int64_t rows, int r) {
    size_t a = gram_plan(rows, r).scratch_floats;
    size_t b = gram_tc_ok(r) ? gram_blk_plan(rows).scratch_floats : 0;
    if (gram_wide_ok(r)) b = gram_wide_plan(rows, r).scratch_floats;
    return a > b ? a : b;
}

// Several steps on the CUDA cores, whose time grows with the rows, or on the tensor cores, whose time grows by
// waves of 148 tiles of 128 rows.  us per step at 2000, 10000 and 18944 rows | a full wave: rank 32 0.33, 1.1, 1.4 | 6.0;
// 64 0.76, 3.7, 6.0 | 8.1; 96 1.9, 8.3, 14.8 | 10.1; 128 2.6, 11.6, - | 10.7.  So 32 and 64 stay on the CUDA cores; the
// lines cross at 9000 rows at 128, and at 96 at 12000 rows a wave (12000: 10.1 either way; 18945: 15.6 against 18.1;
// 25000: 20.2 against 20.0; 37888: 29.6 against 20.1; 37889: 30.2 against 27.8; 50000: 39.4 against 30.1).
bool fit_on_cuda_cores(int64_t rows, int r) {
    const int64_t waves = ceil_div(rows, (int64_t)kNumSMs * 128);
    return r < 96 || rows <= (r == 96 ? 12000 * waves : 9000);
}

// `steps` updates of X.  gsplit: 2*r*r floats that hold the split G already (have_split) or are
// scratch for it.
// The wide-rank kernels cannot update X in place: a result goes to Num when the caller is done with
// it (num_is_scratch, a single step), else to the caller's spare buffer of rows * r floats
// (out_buf), else to a temporary; several steps go back and forth.  With `moved` given, the
// result stays where it is and *moved tells the caller to exchange its two buffers; without it, a
// device copy brings the result back to X.
int mu_update_any(float* X, const float* Num, const float* G, int64_t rows, int r, float eps, float* gsplit,
                  bool have_split, int* err, cudaStream_t st, bool num_is_scratch = false, float* out_buf = nullptr,
                  uint32_t wait_limit = kTiledSpinLimit, bool* moved = nullptr, int steps = 1) {
    if (moved) *moved = false;
    const bool narrow = tensor_cores_enabled() && mu_update_ws_ok(r);
    const bool wide = tensor_cores_enabled() && mu_update_ws_wide_ok(r);
    if (narrow && rows > 0 && steps > 1 && fit_on_cuda_cores(rows, r))
        return fit_steps_launch(X, Num, G, rows, r, steps, eps, st);
    if ((narrow || wide) && rows > 0) {
        if (!have_split) DN_TRY(tc_split_g_launch(G, r, gsplit, st));
        if (narrow) return mu_update_ws_launch(X, Num, X, gsplit, rows, r, steps, eps, err, st, wait_limit);
        DevBuf<float> tmp;
        float* out = num_is_scratch && steps == 1 ? const_cast<float*>(Num) : out_buf;
        if (!out) {
            DN_TRY(tmp.alloc((size_t)(rows * r)));
            out = tmp.p;
        }
        DN_TRY(mu_update_ws_launch(X, Num, out, gsplit, rows, r, steps, eps, err, st, wait_limit));
        if (steps % 2 == 0) return DNPEFF_OK;
        if (moved && !tmp.p) {
            *moved = true;
            return DNPEFF_OK;
        }
        DN_CUDA(cudaMemcpyAsync(X, out, sizeof(float) * (size_t)(rows * r), cudaMemcpyDeviceToDevice, st));
        if (tmp.p && !tmp.arena) DN_CUDA(cudaStreamSynchronize(st));  // tmp is released on return
        return DNPEFF_OK;
    }
    for (int i = 0; i < steps; i++) DN_TRY(mu_update_launch(X, Num, G, rows, r, eps, st));
    return DNPEFF_OK;
}

template <typename T>
int dev_alloc(dnpeff_engine* e, T** p, size_t count) {
    return e->arena.alloc(sizeof(T) * std::max<size_t>(count, 1), (void**)p);
}
template <typename T>
void dev_free(dnpeff_engine* e, T*& p) {
    if (p) e->arena.release(p);
    p = nullptr;
}

void free_small(dnpeff_engine* e) {
    dev_free(e, e->small_cuts); dev_free(e, e->small_carry);
    dev_free(e, e->small_partial); dev_free(e, e->small_barrier);
    e->small_ready = false;
}

void free_matrix(dnpeff_engine* e) {
    dev_free(e, e->a_vals); dev_free(e, e->a_col); dev_free(e, e->a_rowptr);
    dev_free(e, e->c_vals); dev_free(e, e->c_row); dev_free(e, e->c_colptr);
    e->c_base = 0;
    dev_free(e, e->w_spare);
    dev_free(e, e->new_to_og);
    dev_free(e, e->perm); dev_free(e, e->inv_perm);
    dev_free(e, e->b_vals); dev_free(e, e->b_col); dev_free(e, e->tail_off);
    dev_free(e, e->x1); dev_free(e, e->x2); dev_free(e, e->x1_max); dev_free(e, e->blk_ysplit); dev_free(e, e->blk_partial);
    e->tail_nnz.clear();
    e->n_hot = 0; e->n_tail_blocks = 0; e->hot_nnz = 0;
    dev_free(e, e->W); dev_free(e, e->H); dev_free(e, e->AHG); dev_free(e, e->WA); dev_free(e, e->WW);
    dev_free(e, e->gram_scratch);
    dev_free(e, e->tc_scratch);
    e->gram_scratch_floats = 0;
    free_small(e);
    dev_free(e, e->plan_csr.long_list);
    dev_free(e, e->plan_csc.long_list);
    e->plan_csr = SpmmPlan();
    e->plan_csc = SpmmPlan();
    e->loaded = e->have_factors = e->csc_ready = e->csc_hot_ready = false;
    e->a_sq_global = -1.0;
}

// Small device -> host reads through the engine's page-locked scratch (a copy into pageable
// memory would queue behind a large upload that is still in flight), several per wait: add()
// what is needed, then finish() once.
struct SmallReads {
    dnpeff_engine* e;
    size_t used = 0;
    struct Item {
        void* out;
        size_t off, bytes;
    };
    std::vector<Item> items;
    explicit SmallReads(dnpeff_engine* e_) : e(e_) {}
    int add(const void* dptr, size_t bytes, void* out) {
        const size_t off = (used + 15) / 16 * 16;
        if (!e->h_pinned || off + bytes > kPinnedBytes) {
            DN_CUDA(cudaMemcpyAsync(out, dptr, bytes, cudaMemcpyDeviceToHost, e->st));
            return DNPEFF_OK;
        }
        DN_CUDA(cudaMemcpyAsync((char*)e->h_pinned + off, dptr, bytes, cudaMemcpyDeviceToHost, e->st));
        items.push_back({out, off, bytes});
        used = off + bytes;
        return DNPEFF_OK;
    }
    int finish() {
        DN_CUDA(cudaStreamSynchronize(e->st));
        for (const Item& i : items) memcpy(i.out, (const char*)e->h_pinned + i.off, i.bytes);
        items.clear();
        used = 0;
        return DNPEFF_OK;
    }
};

int read_small(dnpeff_engine* e, const void* dptr, size_t bytes, void* out) {
    SmallReads r(e);
    DN_TRY(r.add(dptr, bytes, out));
    return r.finish();
}

int data_error(int flags) {
    if (flags & kErrColRange) return fail(DNPEFF_ERR_DATA, "column index outside [0, n_cols_full)");
    if (flags & kErrRowPtr) return fail(DNPEFF_ERR_DATA, "row offsets are not non-decreasing");
    if (flags & kErrDuplicate) return fail(DNPEFF_ERR_DATA, "a row holds the same column twice");
    return DNPEFF_OK;
}

// getSizeOfSplit (src/util/matrix_util.h:10-20): equal widths, remainder to the last.
void shard_range(int64_t total, int n_shards, int idx, int64_t* start, int64_t* size) {
    int64_t base = total / n_shards;
    *start = base * idx;
    *size = (idx == n_shards - 1) ? base + total % n_shards : base;
}

// The values may arrive in slabs of rows (a host upload still in flight): rows
// [row_end[s-1], row_end[s]) are part first_part + s of the upload (none: valid already).
// Everything that needs the column ids only runs before the first wait.
struct LoadSlabs {
    std::vector<int64_t> row_end;
    Upload* upload = nullptr;
    size_t first_part = 0;
    int count() const { return (int)row_end.size(); }
    int wait(int s, cudaStream_t st) const { return upload ? upload->wait(first_part + (size_t)s, st) : DNPEFF_OK; }
};

// d_retained != nullptr: the kept columns are that list of original ids (device
// pointer, n_retained of them) instead of the columns with >= min_count entries.
// The rows every engine of a job holds when the matrix arrives in row slices
// (dnpeff_set_csr_rows): equal-size contiguous ranges, the remainder spread over
// the leading engines.
void row_slice(int64_t n_total, int n_parts, int idx, int64_t* begin, int64_t* count) {
    *begin = n_total * idx / n_parts;
    *count = n_total * (idx + 1) / n_parts - *begin;
}

// Row slice of the input (dnpeff_set_csr_rows): the arrays hold rows
// [row_begin, row_begin + n_in) of the matrix and every engine of the job is making
// the same call on its own slice.  Column counts are summed over the engines, and
// every entry travels to the engine that owns its column.
struct RowSlice {
    int64_t n_in;
    int64_t row_begin;
};

int load_device(dnpeff_engine* e, int64_t n, int64_t m_full, int64_t k, const int64_t* d_rowptr,
                const float* d_vals, const int32_t* d_col, const float* d_norms, int32_t min_count,
                const int32_t* d_retained = nullptr, int64_t n_retained = 0, const LoadSlabs* slabs = nullptr,
                const RowSlice* slice = nullptr) {
    if (n < 0 || m_full < 0 || (d_rowptr == nullptr && k < 0))
        return fail(DNPEFF_ERR_INVALID, "negative shape");
    if (n >= INT32_MAX || m_full >= INT32_MAX)
        return fail(DNPEFF_ERR_UNSUPPORTED, "n_rows and n_cols_full must fit int32");
    cudaStream_t st = e->st;
    free_matrix(e);
    ArenaScope arena_scope(&e->arena);
    SmallReads reads(e);
    const int r = e->p.rank;
    const int64_t n_in = slice ? slice->n_in : n;  // rows the input arrays hold

    int64_t nnz_in = n_in * k;
    if (d_rowptr) {
        if (n_in > 0) {
            DN_TRY(read_small(e, d_rowptr + n_in, sizeof(int64_t), &nnz_in));
        } else {
            nnz_in = 0;
        }
    }
    if (nnz_in < 0) return fail(DNPEFF_ERR_DATA, "negative nnz");

    DevBuf<int> err;
    DN_TRY(err.alloc_zero(1, st));
    int herr = 0;
    PhaseTrace trace(st);
    trace.mark("upload / inputs ready");

    // 1. explicit entries per original column
    DevBuf<int32_t> counts, flags, og_to_new;
    DevBuf<int64_t> pos;
    DN_TRY(counts.alloc_zero((size_t)m_full + 1, st));
    if (nnz_in > 0) {
        int64_t blocks = std::min<int64_t>(ceil_div(nnz_in, 256), (int64_t)kNumSMs * 16);
        k_count_columns<<<(unsigned)blocks, 256, 0, st>>>(d_col, nnz_in, m_full, counts.p, err.p);
        DN_LAUNCH_CHECK();
        DN_COUNT_LAUNCH(1);
    }
    if (slice) {
        // the pruning decision needs the counts over all rows: one integer sum over the
        // engines; a bad index seen by any of them fails the load on all of them
        DN_NCCL(nccl_api().AllReduce(counts.p, counts.p, (size_t)m_full + 1, ncclInt32, ncclSum, e->comm, st));
        DN_NCCL(nccl_api().AllReduce(err.p, err.p, 1, ncclInt32, ncclMax, e->comm, st));
    }
    trace.mark("count columns");
    // 2. keep mask -> ascending renumbering, or the caller's list of kept columns
    DN_TRY(og_to_new.alloc((size_t)m_full + 1));
    int64_t m_kept = 0;
    // (the maps are made before the id check below is read: they index by column only)
    if (d_retained) {
        if (n_retained < 0 || n_retained >= INT32_MAX) return fail(DNPEFF_ERR_INVALID, "bad retained-column count");
        m_kept = n_retained;
        DevBuf<int> bad;
        DN_TRY(bad.alloc_zero(1, st));
        DN_TRY(dev_alloc(e, &e->new_to_og, (size_t)m_kept));
        DN_CUDA(cudaMemsetAsync(og_to_new.p, 0xFF, sizeof(int32_t) * ((size_t)m_full + 1), st));
        if (m_kept > 0) {
            k_retain_maps<<<(unsigned)ceil_div(m_kept, 256), 256, 0, st>>>(d_retained, m_kept, m_full, og_to_new.p,
                                                                          e->new_to_og, bad.p);
            DN_LAUNCH_CHECK();
            DN_COUNT_LAUNCH(1);
        }
        int hbad = 0;
        DN_TRY(reads.add(err.p, sizeof(int), &herr));
        DN_TRY(reads.add(bad.p, sizeof(int), &hbad));
        DN_TRY(reads.finish());
        if (herr) return data_error(herr);
        if (hbad) return fail(DNPEFF_ERR_DATA, "retained column id outside [0, n_cols_full)");
    } else {
        DN_TRY(flags.alloc_zero((size_t)m_full + 1, st));
        DN_TRY(pos.alloc((size_t)m_full + 1));
        if (m_full > 0) {
            k_keep_flags<<<(unsigned)ceil_div(m_full, 256), 256, 0, st>>>(counts.p, m_full, min_count, flags.p);
            DN_LAUNCH_CHECK();
            DN_COUNT_LAUNCH(1);
        }
        DN_TRY(scan_exclusive<int32_t>(flags.p, pos.p, m_full + 1, st));
        DN_TRY(reads.add(err.p, sizeof(int), &herr));
        DN_TRY(reads.add(pos.p + m_full, sizeof(int64_t), &m_kept));
        DN_TRY(reads.finish());
        if (herr) return data_error(herr);
        DN_TRY(dev_alloc(e, &e->new_to_og, (size_t)m_kept));
        if (m_full > 0) {
            k_build_maps<<<(unsigned)ceil_div(m_full, 256), 256, 0, st>>>(flags.p, pos.p, m_full,
                                                                         og_to_new.p, e->new_to_og);
            DN_LAUNCH_CHECK();
            DN_COUNT_LAUNCH(1);
        }
    }

    trace.mark("pruning maps");
    // 3. this engine's range of kept columns
    int64_t c0 = 0, ms = 0;
    ShardMap map;
    if (e->p.shard_mode == DNPEFF_SHARD_CYCLIC) {
        int64_t G = e->p.n_shards, d = e->p.shard_index;
        ms = m_kept > d ? (m_kept - d + G - 1) / G : 0;
        c0 = d;
        map = {c0, ms, (int32_t)G, (int32_t)d, 1};
    } else {
        shard_range(m_kept, e->p.n_shards, e->p.shard_index, &c0, &ms);
        map = {c0, ms, 1, 0, 0};
    }

    // 4. shard row lengths -> row offsets
    DevBuf<int32_t> row_count;
    DN_TRY(row_count.alloc_zero((size_t)n + 1, st));
    DN_TRY(dev_alloc(e, &e->a_rowptr, (size_t)(n + 1)));
    // Row slices: for every engine d of the job, the lengths of this slice's rows
    // inside d's columns (rc_to[d], with offsets off_to[d] for the extraction); the
    // lengths travel to d, which puts the slices of all engines one after the other.
    const int G = slice ? e->comm_size : 1;
    std::vector<ShardMap> map_of((size_t)G);
    // (one allocation each for all destinations: device allocations are driver calls
    // that the processes of a box serialise on)
    DevBuf<int32_t> rc_all;
    DevBuf<int64_t> off_all;
    std::vector<int32_t*> rc_to((size_t)G, nullptr);
    std::vector<int64_t*> off_to((size_t)G, nullptr);
    if (slice) {
        DN_TRY(rc_all.alloc_zero((size_t)G * ((size_t)n_in + 1), st));
        DN_TRY(off_all.alloc((size_t)G * ((size_t)n_in + 1)));
        for (int d = 0; d < G; d++) {
            rc_to[(size_t)d] = rc_all.p + (size_t)d * ((size_t)n_in + 1);
            off_to[(size_t)d] = off_all.p + (size_t)d * ((size_t)n_in + 1);
        }
    }
    std::vector<int64_t> send_count((size_t)G, 0), slice_begin((size_t)G + 1, 0);
    if (slice) {
        for (int d = 0; d < G; d++) {
            if (e->p.shard_mode == DNPEFF_SHARD_CYCLIC) {
                int64_t w = m_kept > d ? (m_kept - d + G - 1) / G : 0;
                map_of[(size_t)d] = {d, w, (int32_t)G, (int32_t)d, 1};
            } else {
                int64_t b = 0, w = 0;
                shard_range(m_kept, G, d, &b, &w);
                map_of[(size_t)d] = {b, w, 1, 0, 0};
            }
            int64_t sb = 0, sc = 0;
            row_slice(n, G, d, &sb, &sc);
            slice_begin[(size_t)d] = sb;
            if (n_in > 0) {
                int64_t blocks = std::min<int64_t>(n_in, (int64_t)kNumSMs * 32);
                k_row_counts<<<(unsigned)blocks, 256, 0, st>>>(d_col, d_rowptr, k, n_in, og_to_new.p, map_of[(size_t)d],
                                                              rc_to[(size_t)d], err.p);
                DN_LAUNCH_CHECK();
                DN_COUNT_LAUNCH(1);
            }
            DN_TRY(scan_exclusive<int32_t>(rc_to[(size_t)d], off_to[(size_t)d], n_in + 1, st));
        }
        // entries bound for each engine: the last offset of every destination, one read-back
        for (int d = 0; d < G; d++)
            DN_TRY(reads.add(off_to[(size_t)d] + n_in, sizeof(int64_t), &send_count[(size_t)d]));
        DN_TRY(reads.finish());
        slice_begin[(size_t)G] = n;
        if (slice->row_begin != slice_begin[(size_t)e->comm_rank] ||
            n_in != slice_begin[(size_t)e->comm_rank + 1] - slice_begin[(size_t)e->comm_rank])
            return fail(DNPEFF_ERR_INVALID, "row slice of engine %d must be rows [%lld, %lld)", e->comm_rank,
                        (long long)slice_begin[(size_t)e->comm_rank], (long long)slice_begin[(size_t)e->comm_rank + 1]);
        int gs = DNPEFF_OK;
        DN_NCCL(nccl_api().GroupStart());
        for (int d = 0; d < G; d++) {
            const int64_t cnt_d = slice_begin[(size_t)d + 1] - slice_begin[(size_t)d];
            if (d == e->comm_rank) continue;
            if (n_in > 0) DN_NCCL_IN_GROUP(gs, nccl_api().Send(rc_to[(size_t)d], (size_t)n_in, ncclInt32, d, e->comm, st));
            if (cnt_d > 0)
                DN_NCCL_IN_GROUP(gs, nccl_api().Recv(row_count.p + slice_begin[(size_t)d], (size_t)cnt_d, ncclInt32, d,
                                                     e->comm, st));
        }
        DN_NCCL(nccl_api().GroupEnd());
        DN_TRY(gs);
        if (n_in > 0)
            DN_CUDA(cudaMemcpyAsync(row_count.p + slice->row_begin, rc_to[(size_t)e->comm_rank], sizeof(int32_t) * (size_t)n_in,
                                    cudaMemcpyDeviceToDevice, st));
    } else if (n > 0) {
        int64_t blocks = std::min<int64_t>(n, (int64_t)kNumSMs * 32);
        k_row_counts<<<(unsigned)blocks, 256, 0, st>>>(d_col, d_rowptr, k, n, og_to_new.p, map,
                                                      row_count.p, err.p);
        DN_LAUNCH_CHECK();
        DN_COUNT_LAUNCH(1);
    }
    DN_TRY(scan_exclusive<int32_t>(row_count.p, e->a_rowptr, n + 1, st));
    trace.mark("row counts + scan");
    // 5. (the order-preserving extraction needs the values and comes further down,
    //    slab by slab; everything up to there needs the column ids only)
    // 6. internal column order: popular columns first (they get the tiled,
    //    shared-memory kernels), then the rest; both parts in local-id order
    DevBuf<int32_t> cnt_s, hot_flags, cnt_p;
    DevBuf<int64_t> hot_pos;
    DN_TRY(cnt_s.alloc((size_t)ms + 1));
    k_gather_counts<<<(unsigned)ceil_div(ms + 1, 256), 256, 0, st>>>(counts.p, e->new_to_og, map, cnt_s.p);
    DN_LAUNCH_CHECK();
    DN_COUNT_LAUNCH(1);
    int ld = padded_rank(r, e->p.eps);
    // Asking the device for its free memory takes 0.1 ms or more: not for small matrices.
    constexpr double kSmallBytes = 256 << 20;
    // Three arrays of either side's shape: the factors and the products of theirs.
    const int64_t ms_most = m_kept / e->p.n_shards + e->p.n_shards;  // of any shard
    const double pad_bytes = (double)(ld - r) * 12.0 * (double)(n + (e->p.n_shards > 1 ? ms_most : ms));
    if (e->p.n_shards > 1) {
        // The engines of a job must agree on the stride without asking one another: by sizes that
        // all of them know.
        if (pad_bytes > kShardedPadBytes) ld = r;
    } else if (pad_bytes > kSmallBytes) {
        // not a quarter of the free memory more than without the padding
        size_t free_b = 0;
        DN_TRY(e->arena.at_hand(&free_b));
        if (pad_bytes > 0.25 * (double)free_b) ld = r;
    }
    e->ld = ld;
    const bool fast = spmm_fast_rank(ld);
    bool dense = fast && tensor_cores_enabled() && block_tc_ok(ld);
    int tile = fast ? spmm_tile_rows(ld) : 128;
    int32_t hot_thr = (int32_t)std::max<int64_t>(2, ceil_div(n, hot_divisor(e, dense, n)));
    if (!fast || n < 32) hot_thr = INT32_MAX;  // no hot part
    DN_TRY(hot_flags.alloc((size_t)ms + 1));
    DN_TRY(hot_pos.alloc((size_t)ms + 1));
    k_hot_flags<<<(unsigned)ceil_div(ms + 1, 256), 256, 0, st>>>(cnt_s.p, ms, hot_thr, hot_flags.p);
    DN_LAUNCH_CHECK();
    DN_COUNT_LAUNCH(1);
    DN_TRY(scan_exclusive<int32_t>(hot_flags.p, hot_pos.p, ms + 1, st));
    // Row slabs: the caller's (an upload in flight), or cuts of about 256 Mi input entries,
    // which bound the temporary that holds a slab in input order.  a_rowptr at the slab
    // boundaries comes back together with the other counts.
    LoadSlabs own;
    std::vector<int64_t> slab_off(1, 0);
    auto ask_slab_offsets = [&]() -> int {
        if (!slabs) {
            const int64_t S = std::min<int64_t>(std::max<int64_t>(ceil_div(nnz_in, (int64_t)256 << 20), 1), 64);
            for (int64_t sl = 0; sl < S; sl++) own.row_end.push_back(sl + 1 == S ? n : n * (sl + 1) / S);
            slabs = &own;
        }
        slab_off.assign((size_t)slabs->count() + 1, 0);
        for (int sl = 0; sl < slabs->count() && n > 0; sl++)
            DN_TRY(reads.add(e->a_rowptr + slabs->row_end[(size_t)sl], sizeof(int64_t), &slab_off[(size_t)sl + 1]));
        return DNPEFF_OK;
    };
    int64_t n_hot = 0, nnz = 0;
    DN_TRY(reads.add(e->a_rowptr + n, sizeof(int64_t), &nnz));
    DN_TRY(reads.add(err.p, sizeof(int), &herr));
    DN_TRY(reads.add(hot_pos.p + ms, sizeof(int64_t), &n_hot));
    if (!slice) DN_TRY(ask_slab_offsets());
    DN_TRY(reads.finish());
    if (herr) return data_error(herr);
    // The shard's CSR in input order is an intermediate: it is kept only on request
    // (option keep_canonical_csr, for dnpeff_export_shard_csr); otherwise one slab
    // of it at a time lives in a temporary on its way into the bucketed layout.
    if (e->opt_keep_csr) {
        DN_TRY(dev_alloc(e, &e->a_vals, (size_t)nnz));
        DN_TRY(dev_alloc(e, &e->a_col, (size_t)nnz));
    }
    int64_t max_hot = (int64_t)kMaxHotTiles * tile;
    if (dense && 8.0 * (double)n * (double)n_hot > kSmallBytes) {
        // both dense copies (8 bytes per element of the block) within a third of
        // the memory that is free now
        size_t free_b = 0;
        DN_TRY(e->arena.at_hand(&free_b));
        max_hot = (int64_t)(free_b / 3 / (8 * (size_t)std::max<int64_t>(n, 1)));
        max_hot = std::min<int64_t>(max_hot / 128 * 128, (int64_t)1 << 21);
        if (max_hot < 128) {
            dense = false;
            max_hot = (int64_t)kMaxHotTiles * tile;
        }
    }
    if (n_hot > max_hot || n_hot < 8) {
        // too many (cap the tile loop) or too few to be worth a launch: raise the
        // bar until the count fits, or drop the hot part
        if (n_hot > max_hot) {
            // keep the max_hot most popular: find the count threshold by bisection on the host
            std::vector<int32_t> hc((size_t)ms);
            DN_CUDA(cudaMemcpyAsync(hc.data(), cnt_s.p, sizeof(int32_t) * (size_t)ms, cudaMemcpyDeviceToHost, st));
            DN_CUDA(cudaStreamSynchronize(st));
            std::vector<int32_t> sorted(hc);
            std::nth_element(sorted.begin(), sorted.begin() + (size_t)max_hot, sorted.end(), std::greater<int32_t>());
            hot_thr = sorted[(size_t)max_hot] + 1;
        } else {
            hot_thr = INT32_MAX;
        }
        k_hot_flags<<<(unsigned)ceil_div(ms + 1, 256), 256, 0, st>>>(cnt_s.p, ms, hot_thr, hot_flags.p);
        DN_LAUNCH_CHECK();
        DN_COUNT_LAUNCH(1);
        DN_TRY(scan_exclusive<int32_t>(hot_flags.p, hot_pos.p, ms + 1, st));
        DN_TRY(read_small(e, hot_pos.p + ms, sizeof(int64_t), &n_hot));
    }
    DN_TRY(dev_alloc(e, &e->perm, (size_t)(ms)));
    DN_TRY(dev_alloc(e, &e->inv_perm, (size_t)(ms)));
    if (ms > 0) {
        k_build_perm<<<(unsigned)ceil_div(ms, 256), 256, 0, st>>>(hot_flags.p, hot_pos.p, ms, n_hot, e->perm, e->inv_perm);
        DN_LAUNCH_CHECK();
        DN_COUNT_LAUNCH(1);
    }
    // column offsets of the CSC in internal order (the arrays are filled on first use)
    DN_TRY(cnt_p.alloc((size_t)ms + 1));
    DN_TRY(dev_alloc(e, &e->c_colptr, (size_t)(ms + 1)));
    k_permute_counts<<<(unsigned)ceil_div(ms + 1, 256), 256, 0, st>>>(cnt_s.p, e->perm, ms, cnt_p.p);
    DN_LAUNCH_CHECK();
    DN_COUNT_LAUNCH(1);
    DN_TRY(scan_exclusive<int32_t>(cnt_p.p, e->c_colptr, ms + 1, st));

    trace.mark("popular columns, permutation");
    // 6b. rows of A partitioned into buckets: hot tiles, then tail column blocks
    //     narrow enough for their slice of H to stay in L2 while it is gathered
    DevBuf<int64_t> edges;
    std::vector<int64_t> tail_edge;
    {
        int64_t tail_cols = ms - n_hot;
        const int64_t tail_bytes = e->opt_tail_block_bytes > 0 ? e->opt_tail_block_bytes : kTailBlockBytes;
        const int64_t min_block = e->opt_tail_block_bytes > 0 ? 32 : 4096;
        int64_t block = std::max<int64_t>(min_block, (tail_bytes / (4 * (int64_t)ld)) / 32 * 32);
        int64_t nb = ceil_div(std::max<int64_t>(tail_cols, 1), block);
        if (nb > kMaxTailBlocks) {
            block = ceil_div(ceil_div(tail_cols, kMaxTailBlocks), 32) * 32;
            nb = ceil_div(tail_cols, block);
        }
        if (tail_cols <= 0) nb = 0;
        if (n_hot <= 0) dense = false;
        if (dense) tile = (int)std::max<int64_t>(n_hot, 1);  // the dense block needs no tiles: one hot bucket
        BucketMap bm;
        bm.n_hot = n_hot;
        bm.tile = tile;
        bm.block = (int32_t)block;
        bm.n_hot_tiles = (int32_t)ceil_div(n_hot, tile);
        bm.n_buckets = bm.n_hot_tiles + (int32_t)nb;
        e->bm = bm;
        e->n_hot = n_hot;
        e->n_tail_blocks = (int)nb;
        DN_TRY(dev_alloc(e, &e->b_vals, (size_t)(nnz)));
        DN_TRY(dev_alloc(e, &e->b_col, (size_t)(nnz)));
        DN_TRY(dev_alloc(e, &e->tail_off, (size_t)(n * (nb + 1))));
        if (dense) {
            e->plan_x1 = block_tc_plan(n, n_hot, ld);
            e->plan_x2 = block_tc_plan(n_hot, n, ld);
            DN_TRY(dev_alloc(e, &e->x1, e->plan_x1.x_halves));
            DN_TRY(dev_alloc(e, &e->x2, e->plan_x2.x_halves));
            const size_t maxima = e->plan_x1.xmax_words + e->plan_x2.xmax_words + 2 * (size_t)ld;
            const size_t sums = e->plan_x1.xmax_words + e->plan_x2.xmax_words, flags4 = (size_t)(std::max(n, n_hot) + 3) / 4;
            DN_TRY(dev_alloc(e, &e->x1_max, maxima + 2 * sums + flags4));
            e->x2_max = e->x1_max + e->plan_x1.xmax_words;
            e->y_max[0] = e->x2_max + e->plan_x2.xmax_words;
            e->y_max[1] = e->y_max[0] + ld;
            e->x1_sum = (unsigned long long*)(e->x1_max + maxima);
            e->x2_sum = e->x1_sum + e->plan_x1.xmax_words;
            e->blk_again = (unsigned char*)(e->x1_sum + sums);
            DN_CUDA(cudaMemsetAsync(e->x1_max, 0, sizeof(uint32_t) * (maxima + 2 * sums + flags4), st));
            DN_TRY(dev_alloc(e, &e->blk_ysplit, std::max(e->plan_x1.ysplit_halves, e->plan_x2.ysplit_halves)));
            DN_TRY(dev_alloc(e, &e->blk_partial, std::max(e->plan_x1.partial_floats, e->plan_x2.partial_floats)));
            DN_CUDA(cudaMemsetAsync(e->x1, 0, sizeof(__half) * e->plan_x1.x_halves, st));
        }
        trace.mark("index-only phases done");
        // slab by slab, as the values arrive: extraction with the row normalisation
        // applied, bucketing of the rows, the dense copy of the popular part
        // Row slices: every engine extracts, for each engine d, its slice's entries in
        // d's columns (normalised, column ids local to d, input order) and sends them;
        // what arrives from engine s lands at rows [slice_begin[s], slice_begin[s+1]) of
        // this shard's CSR in input order, which is then complete and bucketed below.
        DevBuf<float> canon_v;
        DevBuf<int32_t> canon_c;
        if (slice) {
            if (slabs)
                for (int sl = 0; sl < slabs->count(); sl++) DN_TRY(slabs->wait(sl, st));
            slabs = nullptr;
            nnz_in = nnz;  // (the slabs below are of the complete shard)
            if (!e->opt_keep_csr) {
                DN_TRY(canon_v.alloc((size_t)std::max<int64_t>(nnz, 1)));
                DN_TRY(canon_c.alloc((size_t)std::max<int64_t>(nnz, 1)));
            }
            float* const cv = e->opt_keep_csr ? e->a_vals : canon_v.p;
            int32_t* const cc = e->opt_keep_csr ? e->a_col : canon_c.p;
            // one pair of send buffers, the destinations' parts one after the other
            DevBuf<float> sv_all;
            DevBuf<int32_t> sc_all;
            std::vector<int64_t> send_off((size_t)G + 1, 0);
            for (int d = 0; d < G; d++)
                send_off[(size_t)d + 1] = send_off[(size_t)d] + (d == e->comm_rank ? 0 : send_count[(size_t)d]);
            DN_TRY(sv_all.alloc((size_t)std::max<int64_t>(send_off[(size_t)G], 1)));
            DN_TRY(sc_all.alloc((size_t)std::max<int64_t>(send_off[(size_t)G], 1)));
            std::vector<int64_t> recv_off((size_t)G + 1, 0);
            for (int d = 0; d <= G; d++)
                DN_TRY(reads.add(e->a_rowptr + slice_begin[(size_t)d], sizeof(int64_t), &recv_off[(size_t)d]));
            DN_TRY(ask_slab_offsets());
            DN_TRY(reads.finish());
            for (int d = 0; d < G; d++) {
                const bool self = d == e->comm_rank;
                // this engine's own part goes straight to its place
                float* ov = self ? cv + recv_off[(size_t)d] : nullptr;
                int32_t* oc = self ? cc + recv_off[(size_t)d] : nullptr;
                if (!self) {
                    ov = sv_all.p + send_off[(size_t)d];
                    oc = sc_all.p + send_off[(size_t)d];
                } else if (send_count[(size_t)d] != recv_off[(size_t)d + 1] - recv_off[(size_t)d]) {
                    return fail(DNPEFF_ERR_INVALID, "internal: row-slice bookkeeping out of step");
                }
                if (n_in > 0) {
                    k_extract_shard<<<(unsigned)std::min<int64_t>(n_in, (int64_t)kNumSMs * 32), 256, 0, st>>>(
                        d_vals, d_col, d_rowptr, k, 0, n_in, d_norms, og_to_new.p, map_of[(size_t)d], off_to[(size_t)d],
                        ov, oc);
                    DN_LAUNCH_CHECK();
                    DN_COUNT_LAUNCH(1);
                }
            }
            int gs = DNPEFF_OK;
            DN_NCCL(nccl_api().GroupStart());
            for (int d = 0; d < G; d++) {
                if (d == e->comm_rank) continue;
                if (send_count[(size_t)d] > 0) {
                    DN_NCCL_IN_GROUP(gs, nccl_api().Send(sv_all.p + send_off[(size_t)d], (size_t)send_count[(size_t)d],
                                                         ncclFloat, d, e->comm, st));
                    DN_NCCL_IN_GROUP(gs, nccl_api().Send(sc_all.p + send_off[(size_t)d], (size_t)send_count[(size_t)d],
                                                         ncclInt32, d, e->comm, st));
                }
                const int64_t cnt = recv_off[(size_t)d + 1] - recv_off[(size_t)d];
                if (cnt > 0) {
                    DN_NCCL_IN_GROUP(gs, nccl_api().Recv(cv + recv_off[(size_t)d], (size_t)cnt, ncclFloat, d, e->comm, st));
                    DN_NCCL_IN_GROUP(gs, nccl_api().Recv(cc + recv_off[(size_t)d], (size_t)cnt, ncclInt32, d, e->comm, st));
                }
            }
            DN_NCCL(nccl_api().GroupEnd());
            DN_TRY(gs);
            DN_CUDA(cudaStreamSynchronize(st));  // the send buffers are released here
            trace.mark("row slices exchanged");
        }
        const int n_slabs = slabs->count();
        DevBuf<float> t_vals;
        DevBuf<int32_t> t_col;
        if (!e->opt_keep_csr && !slice && n > 0) {
            int64_t longest = 1;
            for (int sl = 0; sl < n_slabs; sl++) longest = std::max(longest, slab_off[(size_t)sl + 1] - slab_off[(size_t)sl]);
            DN_TRY(t_vals.alloc((size_t)longest));
            DN_TRY(t_col.alloc((size_t)longest));
        }
        int64_t row0 = 0;
        for (int sl = 0; sl < n_slabs && n > 0; sl++) {
            const int64_t row1 = slabs->row_end[sl];
            DN_TRY(slabs->wait(sl, st));
            if (row1 <= row0) continue;
            const int64_t rows = row1 - row0;
            // the slab in input order: at its place in the kept CSR, or in the temporary
            // (addressed through a_rowptr all the same: the pointers are shifted)
            float* cv = e->opt_keep_csr ? e->a_vals : (slice ? canon_v.p : shifted(t_vals.p, slab_off[(size_t)sl]));
            int32_t* cc = e->opt_keep_csr ? e->a_col : (slice ? canon_c.p : shifted(t_col.p, slab_off[(size_t)sl]));
            if (!slice) {
                k_extract_shard<<<(unsigned)std::min<int64_t>(rows, (int64_t)kNumSMs * 32), 256, 0, st>>>(
                    d_vals, d_col, d_rowptr, k, row0, row1, d_norms, og_to_new.p, map, e->a_rowptr, cv, cc);
                DN_LAUNCH_CHECK();
                DN_COUNT_LAUNCH(1);
            }
            size_t smem = sizeof(int) * 8 * (size_t)std::max(bm.n_buckets, 1);
            k_bucket_rows<<<(unsigned)std::min<int64_t>(rows, (int64_t)kNumSMs * 16), 256, smem, st>>>(
                cv, cc, e->a_rowptr, row0, row1, e->inv_perm, bm, e->b_vals, e->b_col, e->tail_off);
            DN_LAUNCH_CHECK();
            DN_COUNT_LAUNCH(1);
            if (dense) {
                k_fill_blocks<<<(unsigned)std::min<int64_t>(ceil_div(rows, 8), (int64_t)kNumSMs * 16), 256, 0, st>>>(
                    e->b_vals, e->b_col, e->a_rowptr, e->tail_off, (int)(nb + 1), row0, row1, e->plan_x1.k_chunks,
                    (float*)e->x1, e->x1_max, e->x2_max);
                DN_LAUNCH_CHECK();
                DN_COUNT_LAUNCH(1);
            }
            row0 = row1;
        }
        trace.mark("extract, bucket, dense fill");
        if (dense) {
            dim3 sgrid((unsigned)e->plan_x1.m_tiles, (unsigned)(2 * e->plan_x2.m_tiles));
            k_block_split<<<sgrid, 256, 0, st>>>(e->x1, e->x1_max, e->x1_sum, e->plan_x1.k_chunks, e->x2, e->x2_max, e->x2_sum,
                                                 e->plan_x2.k_chunks);
            DN_LAUNCH_CHECK();
            DN_COUNT_LAUNCH(1);
        }
        trace.mark("dense block split, transposed");
        // stored entries per tail block (decides warp-per-row or block-per-row launches)
        e->tail_nnz.assign((size_t)nb, 0);
        tail_edge.assign((size_t)nb + 1, 0);
        DN_TRY(edges.alloc((size_t)nb + 1));
        k_tail_edges<<<(unsigned)ceil_div(nb + 1, 256), 256, 0, st>>>(e->c_colptr, n_hot, block, ms, (int)(nb + 1), edges.p);
        DN_LAUNCH_CHECK();
        DN_COUNT_LAUNCH(1);
        DN_TRY(reads.add(edges.p, sizeof(int64_t) * (size_t)(nb + 1), tail_edge.data()));
    }

    trace.mark("tail block sizes");
    // 7. |A|^2 and sum(A) of the shard
    k_sum_sumsq<<<kRedBlocks, 256, 0, st>>>(e->b_vals, nnz, e->red_partial);
    DN_LAUNCH_CHECK();
    k_fold<<<1, 256, 0, st>>>(e->red_partial, kRedBlocks, 2, e->red_out);
    DN_LAUNCH_CHECK();
    DN_COUNT_LAUNCH(2);
    double hs[2] = {0, 0};
    DN_TRY(reads.add(e->red_out, sizeof(double) * 2, hs));

    e->n = n; e->m_full = m_full; e->m_kept = m_kept; e->c0 = c0; e->ms = ms; e->nnz = nnz;
    e->map = map;

    // 8. factor and work buffers, long-row lists
    DN_TRY(dev_alloc(e, &e->W, (size_t)(n * ld)));
    DN_TRY(dev_alloc(e, &e->H, (size_t)(ms * ld)));
    DN_TRY(dev_alloc(e, &e->AHG, (size_t)(n * ld + (int64_t)ld * ld)));
    DN_TRY(dev_alloc(e, &e->WW, (size_t)((int64_t)ld * ld)));
    e->gram_scratch_floats = std::max(gram_any_scratch(n, ld), gram_any_scratch(ms, ld));
    DN_TRY(dev_alloc(e, &e->gram_scratch, e->gram_scratch_floats));
    DN_TRY(dev_alloc(e, &e->tc_scratch, 2 * (size_t)ld * ld));
    DevBuf<int> n_long;  // columns for the block kernel (the generic product takes whole columns)
    DN_TRY(n_long.alloc_zero(1, st));
    int h_long = 0;
    if (spmm_fast_rank(ld)) {
        const int64_t cols = ms - e->n_hot;
        DN_TRY(dev_alloc(e, &e->plan_csc.long_list, (size_t)cols));
        DN_TRY(spmm_list_long(e->c_colptr, e->n_hot, cols, e->plan_csc.long_list, n_long.p, st));
    }
    DN_TRY(reads.add(n_long.p, sizeof(int), &h_long));
    DN_TRY(reads.finish());
    e->a_sum = hs[0];
    e->a_sq = hs[1];
    for (int b = 0; b < e->n_tail_blocks; b++) e->tail_nnz[(size_t)b] = tail_edge[(size_t)b + 1] - tail_edge[(size_t)b];
    e->hot_nnz = tail_edge[0];
    e->plan_csc.n_long = h_long;
    e->plan_csc.n_short = ms - e->n_hot - h_long;
    e->plan_csr.n_short = n;
    e->arena.trim(DeviceArena::kKeep);
    e->loaded = true;
    trace.mark("norms, factor buffers, plans");
    return DNPEFF_OK;
}

// CSC fill (see kernels_prep.cuh): every entry takes the next slot of its column in a
// temporary copy, then every column is put in row order.  `mode`: 0 every entry, 1
// only the entries outside the popular columns, 2 only those inside.  The column
// offsets cover all entries in every mode.
int fill_csc(dnpeff_engine* e, int mode) {
    cudaStream_t st = e->st;
    if (e->nnz <= 0 || e->n <= 0 || e->ms <= 0) return DNPEFF_OK;
    const int n_seg_all = e->n_tail_blocks + 1;  // segment 0 = popular part, s >= 1 = tail block s-1
    const int seg_first = mode == 1 ? 1 : 0, seg_last = mode == 2 ? 1 : n_seg_all;
    const int64_t col_first = mode == 1 ? e->n_hot : 0, col_last = mode == 2 ? e->n_hot : e->ms;
    if (seg_first >= seg_last || col_first >= col_last) return DNPEFF_OK;
    RowSegments segs = {e->tail_off, e->n_tail_blocks + 1};
    const size_t bitmap_bytes = 2 * (size_t)ceil_div(e->n, 32) * sizeof(uint32_t);
    ArenaScope arena_scope(&e->arena);
    PhaseTrace trace(st);
    // the temporary copy covers the CSC entries of the columns being filled:
    // offsets [t_base, t_end) of c_colptr
    int64_t t_base = 0, t_end = e->nnz;
    if (mode != 0) {
        if (mode == 1) t_base = e->hot_nnz; else t_end = e->hot_nnz;
    }
    if (t_base < e->c_base) return fail(DNPEFF_ERR_INVALID, "internal: CSC arrays do not cover the requested columns");
    DevBuf<float> tvals_buf;
    DevBuf<int32_t> trow_buf, cursor, long_cols;
    DevBuf<int> err, n_long;
    DN_TRY(tvals_buf.alloc((size_t)std::max<int64_t>(t_end - t_base, 1)));
    DN_TRY(trow_buf.alloc((size_t)std::max<int64_t>(t_end - t_base, 1)));
    float* const tvals = shifted(tvals_buf.p, t_base);
    int32_t* const trow = shifted(trow_buf.p, t_base);
    float* const cvals = csc_vals(e);
    int32_t* const crows = csc_rows(e);
    DN_TRY(cursor.alloc_zero((size_t)e->ms, st));
    DN_TRY(long_cols.alloc((size_t)(col_last - col_first)));
    DN_TRY(err.alloc_zero(1, st));
    DN_TRY(n_long.alloc_zero(1, st));
    trace.mark("  csc: scratch");
    for (int seg = seg_first; seg < seg_last; seg++) {
        k_csc_scatter<<<(unsigned)ceil_div(e->n, 8), 256, 0, st>>>(e->a_rowptr, e->b_col, e->b_vals, e->n, segs, seg,
                                                                  e->c_colptr, cursor.p, tvals, trow);
        DN_COUNT_LAUNCH(1);
    }
    DN_LAUNCH_CHECK();
    trace.mark("  csc: slots");
    k_csc_list_long<<<(unsigned)ceil_div(col_last - col_first, 256), 256, 0, st>>>(e->c_colptr, col_first, col_last,
                                                                                  long_cols.p, n_long.p);
    DN_LAUNCH_CHECK();
    {
        int64_t blocks = std::min<int64_t>(ceil_div(col_last - col_first, 8), (int64_t)kNumSMs * 32);
        k_csc_order_short<<<(unsigned)blocks, 256, 0, st>>>(e->c_colptr, col_first, col_last, tvals, trow,
                                                           cvals, crows, e->n, err.p);
        DN_LAUNCH_CHECK();
        DN_COUNT_LAUNCH(2);
    }
    // a column longer than kCscShortMax needs that many rows; how many there are stays on the device
    if (e->n > kCscShortMax) {
        if (e->n > kCscLongRows) {
            int h_long = 0;
            DN_TRY(read_small(e, n_long.p, sizeof(int), &h_long));
            if (h_long > 0)
                return fail(DNPEFF_ERR_UNSUPPORTED, "columns longer than %d entries need n_rows <= %lld", kCscShortMax,
                            (long long)kCscLongRows);
        } else {
            DN_CUDA(cudaFuncSetAttribute(k_csc_order_long, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bitmap_bytes));
            const int64_t blocks = std::min<int64_t>(col_last - col_first, (int64_t)kNumSMs * 8);
            k_csc_order_long<<<(unsigned)blocks, 256, bitmap_bytes, st>>>(e->c_colptr, long_cols.p, n_long.p, e->n, tvals,
                                                                         trow, cvals, crows, err.p);
            DN_LAUNCH_CHECK();
            DN_COUNT_LAUNCH(1);
        }
    }
    trace.mark("  csc: row order");
    int herr = 0;
    DN_TRY(read_small(e, err.p, sizeof(int), &herr));
    if (herr) return data_error(herr);
    return DNPEFF_OK;
}

// The CSC the H update needs.  With the popular block kept dense the popular
// columns are never read from the CSC, so they are filled only on demand
// (`full`: the export call).
int build_csc(dnpeff_engine* e, bool full = false) {
    PhaseTrace trace(e->st);
    if (full && e->csc_ready && e->c_base > 0) {
        // the arrays were sized for the unpopular columns only: start over at full size
        dev_free(e, e->c_vals);
        dev_free(e, e->c_row);
        e->c_base = 0;
        e->csc_ready = e->csc_hot_ready = false;
    }
    if (!e->csc_ready) {
        trace.mark("(before CSC build)");
        const bool tail_only = e->x2 != nullptr && !full;
        const int64_t base = tail_only ? e->hot_nnz : 0;
        dev_free(e, e->c_vals);  // of a build that failed
        dev_free(e, e->c_row);
        DN_TRY(dev_alloc(e, &e->c_vals, (size_t)(e->nnz - base)));
        DN_TRY(dev_alloc(e, &e->c_row, (size_t)(e->nnz - base)));
        e->c_base = base;
        trace.mark("  csc: arrays allocated");
        DN_TRY(fill_csc(e, tail_only ? 1 : 0));
        e->csc_ready = true;
        e->csc_hot_ready = !tail_only;
        e->arena.trim(DeviceArena::kKeep);
        trace.mark("CSC build");
    }
    if (full && !e->csc_hot_ready) {
        DN_TRY(fill_csc(e, 2));
        e->csc_hot_ready = true;
    }
    return DNPEFF_OK;
}

int allreduce_f32(dnpeff_engine* e, float* buf, size_t count) {
    if (e->comm_size <= 1) return DNPEFF_OK;
    ScopedTimer t(e, 4);
    DN_NCCL(nccl_api().AllReduce(buf, buf, count, ncclFloat, ncclSum, e->comm, e->st));
    return DNPEFF_OK;
}

int device_dot(dnpeff_engine* e, const float* a, const float* b, int64_t count, double* d_out) {
    k_dot<<<kRedBlocks, 256, 0, e->st>>>(a, b, count, e->red_partial);
    DN_LAUNCH_CHECK();
    k_fold<<<1, 256, 0, e->st>>>(e->red_partial, kRedBlocks, 1, d_out);
    DN_LAUNCH_CHECK();
    DN_COUNT_LAUNCH(2);
    return DNPEFF_OK;
}

// The stored entries behind x1 (`columns`: behind x2, whose rows are the popular columns).
BlkValues popular_values(const dnpeff_engine* e, bool columns) {
    return {nullptr, e->b_vals, e->b_col, e->a_rowptr, e->tail_off, e->n_tail_blocks + 1, columns};
}

// A*H^T: the popular columns through the tiled kernel (H tiles staged in shared
// memory), then one launch per tail column block, each adding to AH, so that the
// slice of H being gathered stays L2-resident.
int spmm_ah(dnpeff_engine* e, float* AH) {
    // ld: row stride; r: the columns gathered (a multiple of 4; those past the rank are zero)
    const int ld = e->ld, r = std::min(ld, (e->p.rank + 3) / 4 * 4);
    if (!spmm_fast_rank(ld))
        return spmm_dispatch(e->b_vals, e->b_col, e->a_rowptr, e->n, e->H, ld, AH, e->plan_csr, e->st);
    if (e->n <= 0) return DNPEFF_OK;
    int accumulate = 0;
    const int stride = e->n_tail_blocks + 1;
    if (e->x1) {
        // popular block on the tensor cores: AH = A_pop * H_pop (H's first n_hot rows)
        const BlkOperand x = {e->x1, e->x1_max, e->x1_sum, popular_values(e, false)};
        DN_TRY(block_tc_launch(x, e->plan_x1, e->H, e->n, e->n_hot, ld, AH, e->W, e->blk_again, e->blk_ysplit, e->y_max[0],
                               e->y_max[1], e->blk_partial, e->d_err, e->st, e->opt_wait_limit));
        std::swap(e->y_max[0], e->y_max[1]);
        accumulate = 1;
    } else if (e->n_hot > 0) {
        SpmmCall c;
        c.kind = kSpmmTiled;
        c.vals = e->b_vals; c.ind = e->b_col;
        c.seg = {e->a_rowptr, nullptr, 0, 0};
        c.rows = e->n; c.D = e->H; c.r = ld; c.out = AH;
        c.row_len = e->tail_off; c.row_len_stride = stride;
        c.d_rows = e->n_hot;
        c.work_counter = e->work_counter; c.err = e->d_err;
        DN_TRY(spmm_call(c, e->st));
        accumulate = 1;
    }
    for (int b = 0; b < e->n_tail_blocks; b++) {
        SpmmCall c;
        c.kind = (e->tail_nnz[(size_t)b] / e->n > 512) ? kSpmmBucketBlock : kSpmmBucketWarp;
        c.vals = e->b_vals; c.ind = e->b_col;
        c.seg = {e->a_rowptr, e->tail_off, stride, b};
        c.rows = e->n; c.D = e->H; c.r = r; c.ld = ld; c.out = AH;
        c.accumulate = accumulate;
        c.overlap = b > 0;  // (what the first one follows may be the update of H)
        DN_TRY(spmm_call(c, e->st));
        accumulate = 1;
    }
    if (!accumulate) DN_CUDA(cudaMemsetAsync(AH, 0, sizeof(float) * (size_t)(e->n * ld), e->st));
    return DNPEFF_OK;
}

// A^T*W: the popular columns (long CSC rows) through the tiled kernel with W
// staged tile by tile, the rest by warp/block gathers from the L2-resident W.
int spmm_wa(dnpeff_engine* e) {
    const int ld = e->ld, r = std::min(ld, (e->p.rank + 3) / 4 * 4);  // as in spmm_ah
    if (!spmm_fast_rank(ld))
        return spmm_dispatch(csc_vals(e), csc_rows(e), e->c_colptr, e->ms, e->W, ld, e->WA, e->plan_csc, e->st);
    if (e->x2) {
        // popular columns on the tensor cores: WA[0, n_hot) = A_pop^T * W
        const BlkOperand x = {e->x2, e->x2_max, e->x2_sum, popular_values(e, true)};
        DN_TRY(block_tc_launch(x, e->plan_x2, e->W, e->n_hot, e->n, ld, e->WA, e->H, e->blk_again, e->blk_ysplit, e->y_max[0],
                               e->y_max[1], e->blk_partial, e->d_err, e->st, e->opt_wait_limit));
        std::swap(e->y_max[0], e->y_max[1]);
    } else if (e->n_hot > 0) {
        SpmmCall c;
        c.kind = kSpmmTiled;
        c.vals = csc_vals(e); c.ind = csc_rows(e);
        c.seg = {e->c_colptr, nullptr, 0, 0};
        c.rows = e->n_hot; c.D = e->W; c.r = ld; c.out = e->WA;
        c.d_rows = e->n;
        c.work_counter = e->work_counter; c.err = e->d_err;
        DN_TRY(spmm_call(c, e->st));
    }
    if (e->ms > e->n_hot) {
        SpmmCall c;
        c.kind = kSpmmRows;
        c.vals = csc_vals(e); c.ind = csc_rows(e);
        c.seg = {e->c_colptr, nullptr, 0, 0};
        c.row_first = e->n_hot; c.rows = e->ms - e->n_hot;
        c.D = e->W; c.r = r; c.ld = ld; c.out = e->WA; c.plan = &e->plan_csc;
        DN_TRY(spmm_call(c, e->st));
    }
    return DNPEFF_OK;
}

// The split form of a Gram matrix comes with it, except where the matrix is summed over the
// engines of a job first (*split: whether tc_scratch holds it now).
int compute_ah_hh(dnpeff_engine* e, bool* split) {
    const int r = e->ld;
    float* AH = e->AHG;
    float* HH = e->AHG + e->n * r;
    *split = e->comm_size <= 1;
    {
        ScopedTimer t(e, 0);
        DN_TRY(spmm_ah(e, AH));
    }
    {
        ScopedTimer t(e, 2);
        DN_TRY(gram_any(e->H, e->ms, r, HH, *split ? e->tc_scratch : nullptr, e->gram_scratch, e->d_err, e->st,
                        e->opt_wait_limit));
    }
    DN_TRY(allreduce_f32(e, e->AHG, (size_t)(e->n * r + (int64_t)r * r)));
    return DNPEFF_OK;
}

// `steps` W updates with the products at hand.
int update_w(dnpeff_engine* e, bool split, int steps) {
    const int r = e->ld;
    // Wide ranks write the updated W beside the old one, into the engine's spare n x r
    // buffer (allocated once), and the two buffers change places.
    if (tensor_cores_enabled() && mu_update_ws_wide_ok(r) && e->n > 0 && !e->w_spare)
        DN_TRY(dev_alloc(e, &e->w_spare, (size_t)(e->n * r)));
    ScopedTimer t(e, 3);
    bool moved = false;
    DN_TRY(mu_update_any(e->W, e->AHG, e->AHG + e->n * r, e->n, r, e->p.eps, e->tc_scratch, split, e->d_err, e->st, false,
                         e->w_spare, e->opt_wait_limit, &moved, steps));
    if (moved) std::swap(e->W, e->w_spare);
    return DNPEFF_OK;
}

int step_w(dnpeff_engine* e) {
    bool split = false;
    DN_TRY(compute_ah_hh(e, &split));
    return update_w(e, split, 1);
}

int step_h(dnpeff_engine* e) {
    const int r = e->ld;
    DN_TRY(build_csc(e));
    if (!e->WA) DN_TRY(dev_alloc(e, &e->WA, (size_t)(e->ms * r)));
    {
        ScopedTimer t(e, 1);
        DN_TRY(spmm_wa(e));
    }
    {
        ScopedTimer t(e, 2);
        DN_TRY(gram_any(e->W, e->n, r, e->WW, e->tc_scratch, e->gram_scratch, e->d_err, e->st, e->opt_wait_limit));
    }
    ScopedTimer t(e, 3);
    // wide ranks: the new H is written over W^T*A (not used again), and the buffers change places
    bool moved = false;
    DN_TRY(mu_update_any(e->H, e->WA, e->WW, e->ms, r, e->p.eps, e->tc_scratch, e->n > 0, e->d_err, e->st, true, nullptr,
                         e->opt_wait_limit, &moved));
    if (moved) std::swap(e->H, e->WA);
    return DNPEFF_OK;
}

// Iterations of a problem small enough for the one-launch kernel.
bool small_problem(const dnpeff_engine* e) {
    if (!tensor_cores_enabled() || e->timing || e->p.n_shards > 1 || !small_rank_ok(e->ld)) return false;
    if (e->n <= 0 || e->ms <= 0 || e->nnz <= 0 || e->nnz > ((int64_t)1 << 30)) return false;
    // the large path leaves the popular columns out of its CSC, where they could not be put in order
    if (e->n > kCscLongRows && e->n_hot > 0) return false;
    return small_pays(e->nnz, e->n + e->ms, e->ld, e->hot_nnz, e->n * e->n_hot);
}

// *made: iterations that were made; fewer than asked for where the launch was refused.
int run_small(dnpeff_engine* e, int iters, int* made) {
    ArenaScope arena_scope(&e->arena);
    const int ld = e->ld;
    DN_TRY(build_csc(e, true));
    const size_t partial = (size_t)kNumSMs * ld * ld;
    // words that a launch counts in: barrier, abort flag, chunks of either Gram matrix, then a flag per worker of either side
    const size_t most = (size_t)kNumSMs * small_workers_per_block(ld), sync_words = 4 + 2 * most;
    const int w_workers = small_workers(e->n, e->nnz, ld), h_workers = small_workers(e->ms, e->nnz, ld);
    if (!e->small_ready) {
        free_small(e);  // what an earlier call got before memory ran out
        DN_TRY(dev_alloc(e, &e->small_cuts, 2 * (most + 1)));
        DN_TRY(dev_alloc(e, &e->small_carry, 2 * most * ld));
        DN_TRY(dev_alloc(e, &e->small_partial, 2 * partial));
        DN_TRY(dev_alloc(e, &e->small_barrier, sync_words));
        const uint32_t cost = small_row_cost(ld);
        k_small_cuts<<<(unsigned)(w_workers / 256 + 1), 256, 0, e->st>>>(e->a_rowptr, (uint32_t)e->n, cost, (uint32_t)w_workers,
                                                                       e->small_cuts);
        k_small_cuts<<<(unsigned)(h_workers / 256 + 1), 256, 0, e->st>>>(e->c_colptr, (uint32_t)e->ms, cost, (uint32_t)h_workers,
                                                                       e->small_cuts + most + 1);
        DN_LAUNCH_CHECK();
        DN_COUNT_LAUNCH(2);
        e->small_ready = true;
    }
    unsigned int* const words = e->small_barrier;
    SmallArgs a;
    a.side[0] = {e->b_vals, e->b_col, e->a_rowptr, e->small_cuts, (uint32_t)w_workers, e->W, e->H, e->small_carry, words + 4,
           e->AHG + e->n * ld, words + 2, e->small_partial, 0, e->small_partial + partial};
    a.side[1] = {e->c_vals, e->c_row, e->c_colptr, e->small_cuts + most + 1, (uint32_t)h_workers, e->H, e->W, e->small_carry + most * ld,
           words + 4 + most, e->WW, words + 3, e->small_partial + partial, 0, e->small_partial};
    a.r4 = (e->p.rank + 3) / 4;
    a.eps = e->p.eps;
    a.barrier = e->small_barrier;
    a.wait_limit = e->opt_wait_limit;
    a.err = e->d_err;
    for (*made = 0; *made < iters; *made += a.iters) {
        a.iters = std::min(kSmallIters, iters - *made);
        bool launched = false;
        DN_TRY(small_launch(a, ld, sync_words, e->st, e->opt_refuse_cooperative, &launched));
        if (!launched) break;
    }
    return DNPEFF_OK;
}

int global_a_sq(dnpeff_engine* e, double* out) {
    if (e->a_sq_global < 0.0) {
        if (e->comm_size > 1) {
            DN_CUDA(cudaMemcpyAsync(e->red_out + 3, &e->a_sq, sizeof(double), cudaMemcpyHostToDevice, e->st));
            DN_NCCL(nccl_api().AllReduce(e->red_out + 3, e->red_out + 3, 1, ncclDouble, ncclSum, e->comm, e->st));
            double v = 0;
            DN_CUDA(cudaMemcpyAsync(&v, e->red_out + 3, sizeof(double), cudaMemcpyDeviceToHost, e->st));
            DN_CUDA(cudaStreamSynchronize(e->st));
            e->a_sq_global = v;
        } else {
            e->a_sq_global = e->a_sq;
        }
    }
    *out = e->a_sq_global;
    return DNPEFF_OK;
}

// sqrt(|A|^2 + <W^T W, H H^T> - 2 <A H^T, W>).  <H,(W^T W)H> = <W^T W, H H^T> and
// <W^T A, H> = <A H^T, W> are the reference's two Frobenius products
// (…device_contexts1.h:337-354) written on the small side; after the allreduce
// both are global, so every engine returns the same number.  The three terms
// are accumulated in double.
int loss_from_current(dnpeff_engine* e, bool recompute_ah, double* out) {
    const int r = e->ld;
    ScopedTimer t(e, 5);
    bool split = false;
    if (recompute_ah) DN_TRY(compute_ah_hh(e, &split));
    DN_TRY(gram_any(e->W, e->n, r, e->WW, nullptr, e->gram_scratch, e->d_err, e->st, e->opt_wait_limit));
    DN_TRY(device_dot(e, e->AHG, e->W, e->n * r, e->red_out + 0));
    DN_TRY(device_dot(e, e->WW, e->AHG + e->n * r, (int64_t)r * r, e->red_out + 1));
    double h[2];
    DN_CUDA(cudaMemcpyAsync(h, e->red_out, sizeof(double) * 2, cudaMemcpyDeviceToHost, e->st));
    DN_CUDA(cudaStreamSynchronize(e->st));
    DN_TRY(check_kernel_status(e));
    double a2 = 0;
    DN_TRY(global_a_sq(e, &a2));
    double sq = a2 + h[1] - 2.0 * h[0];
    *out = sq > 0.0 ? sqrt(sq) : 0.0;
    return DNPEFF_OK;
}

// Host arrays to the device, in the engine's stream order; the arrays are free again on return.
int upload_now(dnpeff_engine* e, std::vector<Upload::Part> parts) {
    const size_t n = parts.size();
    Upload u;
    DN_TRY(u.start(std::move(parts), e->device, e->st));
    for (size_t p = 0; p < n; p++) DN_TRY(u.wait(p, e->st));
    return DNPEFF_OK;
}

int init_generated(dnpeff_engine* e, bool do_w, bool do_h) {
    const int r = e->p.rank;
    float scale = e->p.init_scale > 0.f ? e->p.init_scale : 1.0f;
    if (do_w && e->n > 0) {
        k_init_uniform<<<kNumSMs * 8, 256, 0, e->st>>>(e->W, e->w_row_offset * r, e->n, r, e->ld,
                                                       stream_key(e->p.seed, 0), scale);
        DN_LAUNCH_CHECK();
        DN_COUNT_LAUNCH(1);
    }
    if (do_h && e->ms > 0) {
        k_init_uniform_cols<<<kNumSMs * 8, 256, 0, e->st>>>(e->H, e->ms, r, e->ld, e->map, e->perm,
                                                          stream_key(e->p.seed, 1), scale);
        DN_LAUNCH_CHECK();
        DN_COUNT_LAUNCH(1);
    }
    return DNPEFF_OK;
}

// Reads the device error word the bounded waits write (synchronises the stream).
int check_kernel_status(dnpeff_engine* e) {
    int h = 0;
    DN_CUDA(cudaMemcpyAsync(&h, e->d_err, sizeof(int), cudaMemcpyDeviceToHost, e->st));
    DN_CUDA(cudaStreamSynchronize(e->st));
    if (h) {
        // reported once: the word is cleared so that the engine can be used again
        // (after new factors are set; what the interrupted kernels wrote is invalid)
        cudaMemsetAsync(e->d_err, 0, sizeof(int), e->st);
        cudaStreamSynchronize(e->st);
    }
    if (h & kErrTiledTimeout)
        return fail(DNPEFF_ERR_CUDA, "a bulk-copy wait in the tiled SpMM kernel ran out; results are invalid");
    if (h & kErrGridTimeout)
        return fail(DNPEFF_ERR_CUDA, "a grid-wide barrier of the small-problem kernel ran out; results are invalid");
    if (h & kErrTcTimeout)
        return fail(DNPEFF_ERR_CUDA, "a wait in a tensor-core kernel ran out; results are invalid");
    return DNPEFF_OK;
}

int check_ready(dnpeff_engine* e, bool need_factors) {
    if (!e) return fail(DNPEFF_ERR_INVALID, "null engine");
    if (!e->loaded) return fail(DNPEFF_ERR_INVALID, "no matrix loaded: call dnpeff_set_csr first");
    if (need_factors && !e->have_factors)
        return fail(DNPEFF_ERR_INVALID, "factors not initialised: call dnpeff_init_factors first");
    return DNPEFF_OK;
}

// Scratch for the single-kernel entry points, one grow-only buffer per device.
struct OpWorkspace {
    std::mutex mu;
    float* scratch[64] = {nullptr};
    size_t floats[64] = {0};
    int* err[64] = {nullptr};
};
OpWorkspace& op_ws() {
    static OpWorkspace w;
    return w;
}

int op_scratch(size_t floats, float** out) {
    int dev = 0;
    DN_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return fail(DNPEFF_ERR_UNSUPPORTED, "device ordinal %d", dev);
    OpWorkspace& w = op_ws();
    std::lock_guard<std::mutex> lk(w.mu);
    if (w.floats[dev] < floats) {
        if (w.scratch[dev]) {
            DN_CUDA(cudaDeviceSynchronize());
            cudaFree(w.scratch[dev]);
            w.scratch[dev] = nullptr;
            w.floats[dev] = 0;
        }
        DN_CUDA(cudaMalloc((void**)&w.scratch[dev], sizeof(float) * floats));
        w.floats[dev] = floats;
    }
    *out = w.scratch[dev];
    return DNPEFF_OK;
}

// Error word of the single-kernel entry points (one per device), read after the call.
int op_err_word(int** out) {
    int dev = 0;
    DN_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return fail(DNPEFF_ERR_UNSUPPORTED, "device ordinal %d", dev);
    OpWorkspace& w = op_ws();
    std::lock_guard<std::mutex> lk(w.mu);
    if (!w.err[dev]) {
        DN_CUDA(cudaMalloc((void**)&w.err[dev], sizeof(int)));
        DN_CUDA(cudaMemset(w.err[dev], 0, sizeof(int)));
    }
    *out = w.err[dev];
    return DNPEFF_OK;
}

int op_check_err(int* d_err, cudaStream_t st) {
    int h = 0;
    DN_CUDA(cudaMemcpyAsync(&h, d_err, sizeof(int), cudaMemcpyDeviceToHost, st));
    DN_CUDA(cudaStreamSynchronize(st));
    if (h) {
        cudaMemsetAsync(d_err, 0, sizeof(int), st);
        return fail(DNPEFF_ERR_CUDA, "a bounded wait inside a kernel ran out (status %d); results are invalid", h);
    }
    return DNPEFF_OK;
}

}  // namespace

// ===========================================================================
extern "C" {

const char* dnpeff_last_error(void) { return err_buf(); }
int dnpeff_abi_version(void) { return DNPEFF_ABI_VERSION; }

int dnpeff_device_count(int* count) {
    if (!count) return fail(DNPEFF_ERR_INVALID, "null argument");
    *count = 0;
    DN_CUDA(cudaGetDeviceCount(count));
    return DNPEFF_OK;
}

int dnpeff_create(const dnpeff_params* params, int device, void* stream, dnpeff_engine** out) {
    if (!params || !out) return fail(DNPEFF_ERR_INVALID, "null argument");
    if (params->rank <= 0) return fail(DNPEFF_ERR_INVALID, "rank must be positive");
    if (params->n_shards <= 0 || params->shard_index < 0 || params->shard_index >= params->n_shards)
        return fail(DNPEFF_ERR_INVALID, "shard_index/n_shards out of range");
    if (params->shard_mode != DNPEFF_SHARD_CONTIGUOUS && params->shard_mode != DNPEFF_SHARD_CYCLIC)
        return fail(DNPEFF_ERR_INVALID, "unknown shard_mode %d", (int)params->shard_mode);
    int ndev = 0;
    DN_CUDA(cudaGetDeviceCount(&ndev));
    if (device < 0 || device >= ndev)
        return fail(DNPEFF_ERR_CUDA, "device %d not available (%d visible)", device, ndev);
    DN_CUDA(cudaSetDevice(device));
    dnpeff_engine* e = new dnpeff_engine();
    e->p = *params;
    e->device = device;
    if (stream) {
        e->st = (cudaStream_t)stream;
    } else {
        cudaError_t ce = StreamCache::get().take(device, &e->st);
        if (ce != cudaSuccess) {
            delete e;
            return fail(DNPEFF_ERR_CUDA, "cudaStreamCreate: %s", cudaGetErrorString(ce));
        }
        e->own_stream = true;
    }
    e->arena.open(device, e->st);
    // 4 doubles of red_out, the error word and the work counter, then the partials of the reductions
    if (dev_alloc(e, &e->words, 8 + 2 * kRedBlocks) != DNPEFF_OK ||
        cudaMemsetAsync(e->words, 0, 8 * sizeof(double), e->st) != cudaSuccess) {
        dnpeff_destroy(e);
        return fail(DNPEFF_ERR_CUDA, "no device memory for the status words");
    }
    e->red_out = e->words;
    e->d_err = (int*)(e->words + 4);
    e->work_counter = (int*)(e->words + 5);
    e->red_partial = e->words + 8;
    e->h_pinned = PinnedSlots::get().take();  // null: SmallReads falls back to pageable copies
    e->launches0 = launch_counter();
    *out = e;
    return DNPEFF_OK;
}

int dnpeff_destroy(dnpeff_engine* e) {
    if (!e) return DNPEFF_OK;
    DeviceGuard g(e->device);
    cudaStreamSynchronize(e->st);
    if (e->comm) nccl_api().CommDestroy(e->comm);
    if (e->up) StreamCache::get().give(e->device, e->up);
    e->arena.close(e->opt_keep_memory);
    PinnedSlots::get().give(e->h_pinned);
    for (auto& r : e->regions) { cudaEventDestroy(r.a); cudaEventDestroy(r.b); }
    for (auto ev : e->ev_pool) cudaEventDestroy(ev);
    if (e->own_stream) StreamCache::get().give(e->device, e->st);
    delete e;
    return DNPEFF_OK;
}

int dnpeff_release_memory(int device) {
    int ndev = 0;
    DN_CUDA(cudaGetDeviceCount(&ndev));
    if (device < -1 || device >= ndev) return fail(DNPEFF_ERR_INVALID, "device %d of %d", device, ndev);
    SlabCache::get().flush(device);
    StreamCache::get().flush(device);
    StagingRing::get().release();
    return DNPEFF_OK;
}

int dnpeff_set_option(dnpeff_engine* e, const char* name, int64_t value) {
    if (!e || !name) return fail(DNPEFF_ERR_INVALID, "null argument");
    if (value < 0) return fail(DNPEFF_ERR_INVALID, "option values are non-negative");
    if (!strcmp(name, "loader_slabs")) {
        if (value > 8) return fail(DNPEFF_ERR_INVALID, "loader_slabs: at most 8");
        e->opt_loader_slabs = (int)value;
    } else if (!strcmp(name, "tail_block_bytes")) {
        e->opt_tail_block_bytes = value;
    } else if (!strcmp(name, "popular_divisor")) {
        if (value == 1 || value > INT32_MAX) return fail(DNPEFF_ERR_INVALID, "popular_divisor: 0 or >= 2");
        e->opt_popular_divisor = (int)value;
    } else if (!strcmp(name, "keep_canonical_csr")) {
        e->opt_keep_csr = value != 0;
    } else if (!strcmp(name, "keep_memory")) {
        e->opt_keep_memory = value != 0;
    } else if (!strcmp(name, "refuse_cooperative")) {
        e->opt_refuse_cooperative = value != 0;
    } else if (!strcmp(name, "wait_limit")) {
        e->opt_wait_limit = value == 0 || value > kTiledSpinLimit ? kTiledSpinLimit : (uint32_t)value;
    } else {
        return fail(DNPEFF_ERR_INVALID, "unknown option '%s'", name);
    }
    return DNPEFF_OK;
}

int dnpeff_set_csr_device(dnpeff_engine* e, int64_t n_rows, int64_t n_cols_full, int64_t k_per_row,
                          const int64_t* d_rowptr, const float* d_vals, const int32_t* d_colind,
                          const float* d_norms, int32_t min_values_per_parameter) {
    if (!e) return fail(DNPEFF_ERR_INVALID, "null engine");
    DeviceGuard g(e->device);
    int s = load_device(e, n_rows, n_cols_full, k_per_row, d_rowptr, d_vals, d_colind, d_norms,
                        min_values_per_parameter);
    if (s != DNPEFF_OK) free_matrix(e);
    return s;
}

namespace {
int set_csr_host(dnpeff_engine* e, int64_t n_rows, int64_t n_cols_full, int64_t k_per_row,
                 const int64_t* rowptr, const float* vals, const int32_t* colind, const float* norms,
                 int32_t min_values_per_parameter, const int32_t* retained, int64_t n_retained,
                 int64_t n_rows_total = -1, int64_t row_begin = 0);
}

int dnpeff_set_csr(dnpeff_engine* e, int64_t n_rows, int64_t n_cols_full, int64_t k_per_row,
                   const int64_t* rowptr, const float* vals, const int32_t* colind,
                   const float* norms, int32_t min_values_per_parameter) {
    return set_csr_host(e, n_rows, n_cols_full, k_per_row, rowptr, vals, colind, norms,
                        min_values_per_parameter, nullptr, 0);
}

int dnpeff_row_slice(int64_t n_rows_total, int32_t n_engines, int32_t index, int64_t* row_begin, int64_t* n_rows) {
    if (n_rows_total < 0 || n_engines <= 0 || index < 0 || index >= n_engines || !row_begin || !n_rows)
        return fail(DNPEFF_ERR_INVALID, "bad argument");
    row_slice(n_rows_total, n_engines, index, row_begin, n_rows);
    return DNPEFF_OK;
}

int dnpeff_set_csr_rows(dnpeff_engine* e, int64_t n_rows_total, int64_t n_cols_full, int64_t k_per_row,
                        int64_t row_begin, int64_t n_rows, const int64_t* rowptr, const float* vals,
                        const int32_t* colind, const float* norms, int32_t min_values_per_parameter) {
    if (!e) return fail(DNPEFF_ERR_INVALID, "null engine");
    if (n_rows_total < 0 || n_rows < 0 || row_begin < 0 || row_begin + n_rows > n_rows_total)
        return fail(DNPEFF_ERR_INVALID, "row slice outside the matrix");
    if (e->p.n_shards == 1) {
        if (row_begin != 0 || n_rows != n_rows_total)
            return fail(DNPEFF_ERR_INVALID, "a single engine takes the whole matrix");
        return set_csr_host(e, n_rows, n_cols_full, k_per_row, rowptr, vals, colind, norms, min_values_per_parameter,
                            nullptr, 0);
    }
    if (e->comm_size != e->p.n_shards)
        return fail(DNPEFF_ERR_INVALID, "sharded engine without a communicator: call dnpeff_comm_init first");
    return set_csr_host(e, n_rows, n_cols_full, k_per_row, rowptr, vals, colind, norms, min_values_per_parameter,
                        nullptr, 0, n_rows_total, row_begin);
}

int dnpeff_set_csr_rows_device(dnpeff_engine* e, int64_t n_rows_total, int64_t n_cols_full, int64_t k_per_row,
                               int64_t row_begin, int64_t n_rows, const int64_t* d_rowptr, const float* d_vals,
                               const int32_t* d_colind, const float* d_norms, int32_t min_values_per_parameter) {
    if (!e) return fail(DNPEFF_ERR_INVALID, "null engine");
    if (n_rows_total < 0 || n_rows < 0 || row_begin < 0 || row_begin + n_rows > n_rows_total)
        return fail(DNPEFF_ERR_INVALID, "row slice outside the matrix");
    DeviceGuard g(e->device);
    int s;
    if (e->p.n_shards == 1) {
        if (row_begin != 0 || n_rows != n_rows_total)
            return fail(DNPEFF_ERR_INVALID, "a single engine takes the whole matrix");
        s = load_device(e, n_rows, n_cols_full, k_per_row, d_rowptr, d_vals, d_colind, d_norms, min_values_per_parameter);
    } else {
        if (e->comm_size != e->p.n_shards)
            return fail(DNPEFF_ERR_INVALID, "sharded engine without a communicator: call dnpeff_comm_init first");
        RowSlice slice = {n_rows, row_begin};
        s = load_device(e, n_rows_total, n_cols_full, k_per_row, d_rowptr, d_vals, d_colind, d_norms,
                        min_values_per_parameter, nullptr, 0, nullptr, &slice);
    }
    if (s != DNPEFF_OK) free_matrix(e);
    return s;
}

int dnpeff_get_shard(dnpeff_engine* e, int32_t* shard_index, int32_t* n_shards, int32_t* device) {
    if (!e) return fail(DNPEFF_ERR_INVALID, "null engine");
    if (shard_index) *shard_index = e->p.shard_index;
    if (n_shards) *n_shards = e->p.n_shards;
    if (device) *device = e->device;
    return DNPEFF_OK;
}

int dnpeff_comm_agree(dnpeff_engine* e, int32_t ok, int32_t* all_ok) {
    if (!e || !all_ok) return fail(DNPEFF_ERR_INVALID, "null argument");
    *all_ok = ok ? 1 : 0;
    if (e->p.n_shards == 1) return DNPEFF_OK;
    if (e->comm_size != e->p.n_shards)
        return fail(DNPEFF_ERR_INVALID, "sharded engine without a communicator: call dnpeff_comm_init first");
    DeviceGuard g(e->device);
    ArenaScope arena_scope(&e->arena);
    DevBuf<int32_t> flag;
    DN_TRY(flag.alloc(1));
    int32_t h = ok ? 1 : 0;
    DN_CUDA(cudaMemcpyAsync(flag.p, &h, sizeof(int32_t), cudaMemcpyHostToDevice, e->st));
    DN_NCCL(nccl_api().AllReduce(flag.p, flag.p, 1, ncclInt32, ncclMin, e->comm, e->st));
    DN_CUDA(cudaMemcpyAsync(&h, flag.p, sizeof(int32_t), cudaMemcpyDeviceToHost, e->st));
    DN_CUDA(cudaStreamSynchronize(e->st));
    *all_ok = h;
    return DNPEFF_OK;
}

int dnpeff_set_csr_retain(dnpeff_engine* e, int64_t n_rows, int64_t n_cols_full, int64_t k_per_row,
                          const int64_t* rowptr, const float* vals, const int32_t* colind,
                          const float* norms, const int32_t* retained_cols, int64_t n_retained) {
    if (!retained_cols && n_retained > 0) return fail(DNPEFF_ERR_INVALID, "null retained_cols");
    static const int32_t none = 0;
    return set_csr_host(e, n_rows, n_cols_full, k_per_row, rowptr, vals, colind, norms, 1,
                        retained_cols ? retained_cols : &none, n_retained);
}

namespace {
// n_rows_total >= 0: the arrays hold rows [row_begin, row_begin + n_rows) of a matrix of
// n_rows_total rows and every engine of the job makes this call on its own slice.
int set_csr_host(dnpeff_engine* e, int64_t n_rows, int64_t n_cols_full, int64_t k_per_row,
                 const int64_t* rowptr, const float* vals, const int32_t* colind, const float* norms,
                 int32_t min_values_per_parameter, const int32_t* retained, int64_t n_retained,
                 int64_t n_rows_total, int64_t row_begin) {
    if (!e) return fail(DNPEFF_ERR_INVALID, "null engine");
    if (n_rows < 0) return fail(DNPEFF_ERR_INVALID, "negative shape");
    DeviceGuard g(e->device);
    int64_t nnz = rowptr ? (n_rows > 0 ? rowptr[n_rows] : 0) : n_rows * k_per_row;
    if (nnz < 0) return fail(DNPEFF_ERR_DATA, "negative nnz");
    if (nnz > 0 && (!vals || !colind)) return fail(DNPEFF_ERR_INVALID, "null vals/colind");
    free_matrix(e);
    ArenaScope arena_scope(&e->arena);
    DevBuf<float> dv, dn;
    DevBuf<int32_t> dc, dret;
    DevBuf<int64_t> dr;
    DN_TRY(dv.alloc((size_t)nnz));
    DN_TRY(dc.alloc((size_t)nnz));
    if (rowptr) DN_TRY(dr.alloc((size_t)n_rows + 1));
    if (norms) DN_TRY(dn.alloc((size_t)n_rows));
    if (retained) DN_TRY(dret.alloc((size_t)std::max<int64_t>(n_retained, 1)));
    // The index arrays go first; the values follow in slabs of rows, so that counting, pruning,
    // row offsets and the column permutation overlap their upload and every slab is processed
    // as it lands.
    std::vector<Upload::Part> parts;
    if (rowptr) parts.push_back({dr.p, rowptr, sizeof(int64_t) * (size_t)(n_rows + 1)});
    if (norms) parts.push_back({dn.p, norms, sizeof(float) * (size_t)n_rows});
    if (retained) parts.push_back({dret.p, retained, sizeof(int32_t) * (size_t)n_retained});
    parts.push_back({dc.p, colind, sizeof(int32_t) * (size_t)nnz});
    LoadSlabs slabs;
    slabs.first_part = parts.size();
    if (nnz > 0) {
        int n_slabs = nnz >= ((int64_t)64 << 20) ? 4 : 1;
        if (e->opt_loader_slabs > 0) n_slabs = std::min(e->opt_loader_slabs, 8);
        int64_t off0 = 0;
        for (int i = 0; i < n_slabs; i++) {
            const int64_t row1 = i + 1 == n_slabs ? n_rows : n_rows * (i + 1) / n_slabs;
            const int64_t off1 = std::max(off0, rowptr ? rowptr[row1] : row1 * k_per_row);
            parts.push_back({dv.p + off0, vals + off0, sizeof(float) * (size_t)(off1 - off0)});
            slabs.row_end.push_back(row1);
            off0 = off1;
        }
    }
    if (!e->up) DN_CUDA(StreamCache::get().take(e->device, &e->up));
    // the arena may have handed out memory that work queued on the engine's stream still uses
    cudaEvent_t free_before = nullptr;
    DN_CUDA(cudaEventCreateWithFlags(&free_before, cudaEventDisableTiming));
    cudaError_t ce = cudaEventRecord(free_before, e->st);
    if (ce == cudaSuccess) ce = cudaStreamWaitEvent(e->up, free_before, 0);
    cudaEventDestroy(free_before);
    if (ce != cudaSuccess) return fail(DNPEFF_ERR_CUDA, "ordering the upload: %s", cudaGetErrorString(ce));
    int s;
    {
        Upload upload;
        const size_t index_parts = slabs.first_part;
        s = upload.start(std::move(parts), e->device, e->up);
        for (size_t p = 0; p < index_parts && s == DNPEFF_OK; p++) s = upload.wait(p, e->st);
        slabs.upload = &upload;
        RowSlice slice = {n_rows, row_begin};
        const bool sliced = n_rows_total >= 0;
        if (s == DNPEFF_OK)
            s = load_device(e, sliced ? n_rows_total : n_rows, n_cols_full, k_per_row, rowptr ? dr.p : nullptr, dv.p, dc.p,
                            norms ? dn.p : nullptr, min_values_per_parameter, retained ? dret.p : nullptr, n_retained,
                            slabs.count() > 0 ? &slabs : nullptr, sliced ? &slice : nullptr);
    }  // (the upload is over before the buffers it fills are released)
    if (s != DNPEFF_OK) free_matrix(e);
    cudaStreamSynchronize(e->st);
    return s;
}
}  // namespace

int dnpeff_get_shape(dnpeff_engine* e, int64_t* n_rows, int64_t* n_cols_kept, int64_t* col_start,
                     int64_t* n_cols_shard, int64_t* nnz_shard) {
    DN_TRY(check_ready(e, false));
    if (n_rows) *n_rows = e->n;
    if (n_cols_kept) *n_cols_kept = e->m_kept;
    if (col_start) *col_start = e->c0;
    if (n_cols_shard) *n_cols_shard = e->ms;
    if (nnz_shard) *nnz_shard = e->nnz;
    return DNPEFF_OK;
}

int dnpeff_get_layout(dnpeff_engine* e, int64_t* n_hot_cols, int64_t* hot_nnz, int32_t* n_tail_blocks,
                      int32_t* tile_rows) {
    DN_TRY(check_ready(e, false));
    DeviceGuard g(e->device);
    int64_t v = 0;
    DN_CUDA(cudaMemcpyAsync(&v, e->c_colptr + e->n_hot, sizeof(int64_t), cudaMemcpyDeviceToHost, e->st));
    DN_CUDA(cudaStreamSynchronize(e->st));
    if (n_hot_cols) *n_hot_cols = e->n_hot;
    if (hot_nnz) *hot_nnz = v;
    if (n_tail_blocks) *n_tail_blocks = e->n_tail_blocks;
    // the dense block is consumed kBlkKC rows of the factor at a time
    if (tile_rows) *tile_rows = !e->x1 ? e->bm.tile : (e->ld == e->p.rank ? 0 : kBlkKC);
    return DNPEFF_OK;
}

int dnpeff_get_new_to_og(dnpeff_engine* e, int32_t* out) {
    DN_TRY(check_ready(e, false));
    DeviceGuard g(e->device);
    DN_TRY(download(out, e->new_to_og, sizeof(int32_t) * (size_t)e->m_kept, e->device, e->st));
    return DNPEFF_OK;
}

int dnpeff_get_shard_columns(dnpeff_engine* e, int32_t* kept_ids, int32_t* original_ids) {
    DN_TRY(check_ready(e, false));
    DeviceGuard g(e->device);
    ArenaScope arena_scope(&e->arena);
    if (e->ms <= 0) return DNPEFF_OK;
    DevBuf<int32_t> a, b;
    DN_TRY(a.alloc((size_t)e->ms));
    DN_TRY(b.alloc((size_t)e->ms));
    k_shard_columns<<<(unsigned)ceil_div(e->ms, 256), 256, 0, e->st>>>(e->new_to_og, e->map, a.p, b.p);
    DN_LAUNCH_CHECK();
    DN_COUNT_LAUNCH(1);
    if (kept_ids) DN_TRY(download(kept_ids, a.p, sizeof(int32_t) * (size_t)e->ms, e->device, e->st));
    if (original_ids) DN_TRY(download(original_ids, b.p, sizeof(int32_t) * (size_t)e->ms, e->device, e->st));
    return DNPEFF_OK;
}

int dnpeff_export_shard_csr(dnpeff_engine* e, int64_t* rowptr, int32_t* colind, float* vals) {
    DN_TRY(check_ready(e, false));
    DeviceGuard g(e->device);
    if ((colind || vals) && e->nnz > 0 && !e->a_vals)
        return fail(DNPEFF_ERR_INVALID,
                    "the CSR in input order was not kept: set option keep_canonical_csr to 1 before loading");
    if (rowptr) DN_CUDA(cudaMemcpyAsync(rowptr, e->a_rowptr, sizeof(int64_t) * (size_t)(e->n + 1), cudaMemcpyDeviceToHost, e->st));
    if (colind && e->nnz > 0) DN_CUDA(cudaMemcpyAsync(colind, e->a_col, sizeof(int32_t) * (size_t)e->nnz, cudaMemcpyDeviceToHost, e->st));
    if (vals && e->nnz > 0) DN_CUDA(cudaMemcpyAsync(vals, e->a_vals, sizeof(float) * (size_t)e->nnz, cudaMemcpyDeviceToHost, e->st));
    DN_CUDA(cudaStreamSynchronize(e->st));
    return DNPEFF_OK;
}

int dnpeff_export_shard_csc(dnpeff_engine* e, int64_t* colptr, int32_t* rowind, float* vals) {
    DN_TRY(check_ready(e, false));
    DeviceGuard g(e->device);
    DN_TRY(build_csc(e, true));
    // The device CSC is in the engine's internal column order; hand it out in
    // local column order (a test/debug path: reordered on the host).
    std::vector<int64_t> cp((size_t)e->ms + 1);
    std::vector<int32_t> perm((size_t)e->ms), ri((size_t)e->nnz);
    std::vector<float> va((size_t)e->nnz);
    DN_CUDA(cudaMemcpyAsync(cp.data(), e->c_colptr, sizeof(int64_t) * (size_t)(e->ms + 1), cudaMemcpyDeviceToHost, e->st));
    if (e->ms > 0) DN_CUDA(cudaMemcpyAsync(perm.data(), e->inv_perm, sizeof(int32_t) * (size_t)e->ms, cudaMemcpyDeviceToHost, e->st));
    if (e->nnz > 0) {
        DN_CUDA(cudaMemcpyAsync(ri.data(), csc_rows(e), sizeof(int32_t) * (size_t)e->nnz, cudaMemcpyDeviceToHost, e->st));
        DN_CUDA(cudaMemcpyAsync(va.data(), csc_vals(e), sizeof(float) * (size_t)e->nnz, cudaMemcpyDeviceToHost, e->st));
    }
    DN_CUDA(cudaStreamSynchronize(e->st));
    int64_t q = 0;
    for (int64_t j = 0; j < e->ms; j++) {
        int64_t jp = perm[(size_t)j];
        if (colptr) colptr[j] = q;
        for (int64_t p = cp[(size_t)jp]; p < cp[(size_t)jp + 1]; p++, q++) {
            if (rowind) rowind[q] = ri[(size_t)p];
            if (vals) vals[q] = va[(size_t)p];
        }
    }
    if (colptr) colptr[e->ms] = q;
    return DNPEFF_OK;
}

int dnpeff_a_sq_norm(dnpeff_engine* e, double* out) {
    DN_TRY(check_ready(e, false));
    *out = e->a_sq;
    return DNPEFF_OK;
}

int dnpeff_a_sum(dnpeff_engine* e, double* out) {
    DN_TRY(check_ready(e, false));
    *out = e->a_sum;
    return DNPEFF_OK;
}

int dnpeff_set_init_scale(dnpeff_engine* e, float init_scale) {
    if (!e) return fail(DNPEFF_ERR_INVALID, "null engine");
    e->p.init_scale = init_scale;
    return DNPEFF_OK;
}

int dnpeff_init_factors(dnpeff_engine* e, const float* W, const float* H) {
    DN_TRY(check_ready(e, false));
    DeviceGuard g(e->device);
    ArenaScope arena_scope(&e->arena);
    const int r = e->p.rank;
    const int ld = e->ld;
    DN_TRY(init_generated(e, W == nullptr, H == nullptr));
    if (W && e->n > 0) {
        DevBuf<float> tmp;
        if (ld > r) DN_TRY(tmp.alloc((size_t)(e->n * r)));
        DN_TRY((upload_now(e, {{ld > r ? tmp.p : e->W, W, sizeof(float) * (size_t)(e->n * r)}})));
        if (ld > r) {
            k_gather_rows<<<kNumSMs * 8, 256, 0, e->st>>>(tmp.p, nullptr, e->n, r, r, ld, e->W);
            DN_LAUNCH_CHECK();
            DN_COUNT_LAUNCH(1);
        }
    }
    if (H && e->ms > 0) {
        DevBuf<float> tmp;
        DN_TRY(tmp.alloc((size_t)(e->ms * r)));
        DevBuf<float> tmp2;
        DN_TRY(tmp2.alloc((size_t)(e->ms * r)));
        DN_TRY((upload_now(e, {{tmp.p, H, sizeof(float) * (size_t)(e->ms * r)}})));
        k_transpose<<<kNumSMs * 8, dim3(32, 8), 0, e->st>>>(tmp.p, tmp2.p, r, e->ms);
        DN_LAUNCH_CHECK();
        // internal row jp holds local column perm[jp]
        k_gather_rows<<<kNumSMs * 8, 256, 0, e->st>>>(tmp2.p, e->perm, e->ms, r, r, ld, e->H);
        DN_LAUNCH_CHECK();
        DN_COUNT_LAUNCH(2);
    }
    DN_CUDA(cudaStreamSynchronize(e->st));
    e->have_factors = true;
    return DNPEFF_OK;
}

int dnpeff_set_w_row_offset(dnpeff_engine* e, int64_t first_row) {
    if (!e) return fail(DNPEFF_ERR_INVALID, "null engine");
    if (first_row < 0) return fail(DNPEFF_ERR_INVALID, "negative row offset");
    e->w_row_offset = first_row;
    return DNPEFF_OK;
}

int dnpeff_set_h_csr(dnpeff_engine* e, const int64_t* h_rowptr, const int32_t* h_colind, const float* h_vals) {
    DN_TRY(check_ready(e, false));
    if (!h_rowptr) return fail(DNPEFF_ERR_INVALID, "null h_rowptr");
    DeviceGuard g(e->device);
    ArenaScope arena_scope(&e->arena);
    const int r = e->p.rank;
    const int64_t nnz = h_rowptr[r];
    if (h_rowptr[0] != 0 || nnz < 0) return fail(DNPEFF_ERR_DATA, "row offsets of H must start at 0");
    for (int t = 0; t < r; t++)
        if (h_rowptr[t + 1] < h_rowptr[t]) return fail(DNPEFF_ERR_DATA, "row offsets of H are not non-decreasing");
    if (nnz > 0 && (!h_colind || !h_vals)) return fail(DNPEFF_ERR_INVALID, "null column ids / values of H");
    if (!e->have_factors) DN_TRY(init_generated(e, true, false));  // W as dnpeff_init_factors(NULL, .) makes it
    DN_CUDA(cudaMemsetAsync(e->H, 0, sizeof(float) * (size_t)std::max<int64_t>(e->ms * e->ld, 1), e->st));
    if (nnz > 0 && e->ms > 0) {
        DevBuf<int64_t> drp;
        DevBuf<int32_t> dc;
        DevBuf<float> dv;
        DevBuf<int> err;
        DN_TRY(drp.alloc((size_t)r + 1));
        DN_TRY(dc.alloc((size_t)nnz));
        DN_TRY(dv.alloc((size_t)nnz));
        DN_TRY(err.alloc_zero(1, e->st));
        DN_TRY((upload_now(e, {{drp.p, h_rowptr, sizeof(int64_t) * (size_t)(r + 1)},
                              {dc.p, h_colind, sizeof(int32_t) * (size_t)nnz},
                              {dv.p, h_vals, sizeof(float) * (size_t)nnz}})));
        k_scatter_h_csr<<<(unsigned)ceil_div(nnz, 256), 256, 0, e->st>>>(drp.p, dc.p, dv.p, r, nnz, e->m_kept, e->map,
                                                                         e->inv_perm, e->H, e->ld, err.p);
        DN_LAUNCH_CHECK();
        DN_COUNT_LAUNCH(1);
        int herr = 0;
        DN_TRY(read_small(e, err.p, sizeof(int), &herr));
        if (herr) return fail(DNPEFF_ERR_DATA, "a column id of H is outside [0, n_cols_kept)");
    }
    DN_CUDA(cudaStreamSynchronize(e->st));
    e->have_factors = true;
    return DNPEFF_OK;
}

int dnpeff_get_w(dnpeff_engine* e, float* out) {
    DN_TRY(check_ready(e, true));
    DeviceGuard g(e->device);
    ArenaScope arena_scope(&e->arena);
    const int r = e->p.rank;
    DevBuf<float> tmp;
    const float* src = e->W;
    if (e->n > 0 && e->ld > r) {
        DN_TRY(tmp.alloc((size_t)(e->n * r)));
        k_gather_rows<<<kNumSMs * 8, 256, 0, e->st>>>(e->W, nullptr, e->n, r, e->ld, r, tmp.p);
        DN_LAUNCH_CHECK();
        DN_COUNT_LAUNCH(1);
        src = tmp.p;
    }
    DN_TRY(download(out, src, sizeof(float) * (size_t)(e->n * r), e->device, e->st));
    return check_kernel_status(e);
}

int dnpeff_get_h(dnpeff_engine* e, float* out) {
    DN_TRY(check_ready(e, true));
    DeviceGuard g(e->device);
    ArenaScope arena_scope(&e->arena);
    const int r = e->p.rank;
    if (e->ms > 0) {
        DevBuf<float> tmp2;
        float* t = e->WA;  // free between iterations
        if (!t) {
            DN_TRY(tmp2.alloc((size_t)(e->ms * r)));
            t = tmp2.p;
        }
        // Local column j is internal row inv_perm[j]; gathered and transposed in one pass.  Into page-locked memory
        // a large H goes in four parts of its components, each on its way while the next is transposed.
        const size_t bytes = sizeof(float) * (size_t)(e->ms * r);
        const bool parts = bytes >= ((size_t)64 << 20) && r >= 64 && !host_pageable(out);
        const int step = parts ? (r / 4 + 31) / 32 * 32 : r;
        cudaEvent_t done[4] = {nullptr, nullptr, nullptr, nullptr};
        cudaError_t ce = cudaSuccess;
        if (parts && !e->up) ce = StreamCache::get().take(e->device, &e->up);
        for (int c = 0; c * step < r && ce == cudaSuccess; c++) {
            const int64_t c0 = (int64_t)c * step, n = std::min<int64_t>(step, r - c0);
            k_gather_transpose<<<kNumSMs * 8, dim3(32, 8), 0, e->st>>>(e->H + c0, e->inv_perm, e->ms, n, e->ld, t + c0 * e->ms);
            ce = cudaGetLastError();
            DN_COUNT_LAUNCH(1);
            if (!parts) continue;
            if (ce == cudaSuccess) ce = cudaEventCreateWithFlags(&done[c], cudaEventDisableTiming);
            if (ce == cudaSuccess) ce = cudaEventRecord(done[c], e->st);
            if (ce == cudaSuccess) ce = cudaStreamWaitEvent(e->up, done[c], 0);
            if (ce == cudaSuccess)
                ce = cudaMemcpyAsync(out + c0 * e->ms, t + c0 * e->ms, sizeof(float) * (size_t)(n * e->ms),
                                     cudaMemcpyDeviceToHost, e->up);
        }
        if (parts && e->up) {
            const cudaError_t we = cudaStreamSynchronize(e->up);
            if (ce == cudaSuccess) ce = we;
        }
        for (cudaEvent_t d : done)
            if (d) cudaEventDestroy(d);
        DN_CUDA(ce);
        if (!parts) DN_TRY(download(out, t, bytes, e->device, e->st));
        DN_TRY(check_kernel_status(e));
    }
    return DNPEFF_OK;
}

int dnpeff_nccl_unique_id(void* id128) {
    if (!id128) return fail(DNPEFF_ERR_INVALID, "null argument");
    DN_TRY(nccl_load());
    static_assert(sizeof(ncclUniqueId) == 128, "ncclUniqueId is expected to be 128 bytes");
    ncclUniqueId id;
    DN_NCCL(nccl_api().GetUniqueId(&id));
    memcpy(id128, &id, 128);
    return DNPEFF_OK;
}

int dnpeff_comm_init(dnpeff_engine* e, const void* id128, int comm_rank, int comm_size) {
    if (!e || !id128) return fail(DNPEFF_ERR_INVALID, "null argument");
    if (comm_size != e->p.n_shards || comm_rank != e->p.shard_index)
        return fail(DNPEFF_ERR_INVALID, "communicator rank/size must equal shard_index/n_shards");
    DeviceGuard g(e->device);
    ArenaScope arena_scope(&e->arena);
    DN_TRY(nccl_load());
    ncclUniqueId id;
    memcpy(&id, id128, 128);
    DN_NCCL(nccl_api().CommInitRank(&e->comm, comm_size, id, comm_rank));
    e->comm_rank = comm_rank;
    e->comm_size = comm_size;
    e->a_sq_global = -1.0;
    // NCCL connects its channels on the first collective (hundreds of ms): do that
    // here, as part of joining, not inside the first iteration
    // ... and the point-to-point channels the row-sliced loader uses: NCCL opens as many
    // channels per peer as a transfer's size calls for, the first time it is that large,
    // so the first exchange here is of the loader's order of size (4 MB per peer), not a
    // token one
    const size_t kWarm = (size_t)1 << 20;  // floats per peer and direction
    DevBuf<float> one;
    DN_TRY(one.alloc_zero(32 + 2 * kWarm * (size_t)comm_size, e->st));
    DN_NCCL(nccl_api().AllReduce(one.p, one.p, 32, ncclFloat, ncclSum, e->comm, e->st));
    int gs = DNPEFF_OK;
    DN_NCCL(nccl_api().GroupStart());
    for (int d = 0; d < comm_size; d++) {
        if (d == comm_rank) continue;
        DN_NCCL_IN_GROUP(gs, nccl_api().Send(one.p + 32 + kWarm * (size_t)d, kWarm, ncclFloat, d, e->comm, e->st));
        DN_NCCL_IN_GROUP(gs, nccl_api().Recv(one.p + 32 + kWarm * (size_t)(comm_size + d), kWarm, ncclFloat, d, e->comm,
                                             e->st));
    }
    DN_NCCL(nccl_api().GroupEnd());
    DN_TRY(gs);
    DN_CUDA(cudaStreamSynchronize(e->st));
    return DNPEFF_OK;
}

int dnpeff_step_w(dnpeff_engine* e) {
    DN_TRY(check_ready(e, true));
    DeviceGuard g(e->device);
    if (e->p.n_shards > 1 && e->comm_size != e->p.n_shards)
        return fail(DNPEFF_ERR_INVALID, "sharded engine without a communicator: call dnpeff_comm_init");
    return step_w(e);
}

int dnpeff_step_h(dnpeff_engine* e) {
    DN_TRY(check_ready(e, true));
    DeviceGuard g(e->device);
    return step_h(e);
}

int dnpeff_synchronize(dnpeff_engine* e) {
    if (!e) return fail(DNPEFF_ERR_INVALID, "null engine");
    DeviceGuard g(e->device);
    return check_kernel_status(e);
}

int dnpeff_loss(dnpeff_engine* e, double* out) {
    DN_TRY(check_ready(e, true));
    if (!out) return fail(DNPEFF_ERR_INVALID, "null argument");
    DeviceGuard g(e->device);
    if (e->p.n_shards > 1 && e->comm_size != e->p.n_shards)
        return fail(DNPEFF_ERR_INVALID, "sharded engine without a communicator: call dnpeff_comm_init");
    return loss_from_current(e, true, out);
}

int dnpeff_run(dnpeff_engine* e, int32_t iters, int32_t log_every) { return dnpeff_run_steps(e, 0, iters, log_every); }

int dnpeff_run_steps(dnpeff_engine* e, int32_t first_step, int32_t iters, int32_t log_every) {
    DN_TRY(check_ready(e, true));
    DeviceGuard g(e->device);
    if (e->p.n_shards > 1 && e->comm_size != e->p.n_shards)
        return fail(DNPEFF_ERR_INVALID, "sharded engine without a communicator: call dnpeff_comm_init");
    if (first_step < 0) return fail(DNPEFF_ERR_INVALID, "negative first step");
    auto t0 = std::chrono::high_resolution_clock::now();
    bool small = small_problem(e) && iters > 1;
    for (int step = first_step; step < first_step + iters; step++) {
        int made = 0;
        if (small) {
            // as far as the next log line
            int stretch = first_step + iters - step;
            if (log_every > 0) stretch = std::min(stretch, log_every - step % log_every);
            DN_TRY(run_small(e, stretch, &made));
            small = made == stretch;  // refused: the kernels of the large path do it
        }
        if (made == 0) {
            DN_TRY(step_w(e));
            DN_TRY(step_h(e));
            made = 1;
        }
        step += made - 1;
        // "step N: <loss> [<ms> ms/step]" every log_every steps, loss time
        // excluded from the rate (multi_mu_dense_factors_nmf1.h:187-201).
        if (log_every > 0 && (step + 1) % log_every == 0) {
            DN_CUDA(cudaStreamSynchronize(e->st));
            auto t1 = std::chrono::high_resolution_clock::now();
            double ms = std::chrono::duration<double, std::milli>(t1 - t0).count();
            double loss = 0;
            DN_TRY(loss_from_current(e, true, &loss));
            if (e->comm_rank == 0) {
                printf("step %d: %g [%g ms/step]\n", step + 1, loss, ms / (double)log_every);
                fflush(stdout);
            }
            t0 = std::chrono::high_resolution_clock::now();
        }
    }
    return DNPEFF_OK;
}

int dnpeff_fit_w_only(dnpeff_engine* e, int32_t iters, double* loss) {
    DN_TRY(check_ready(e, true));
    DeviceGuard g(e->device);
    if (e->p.n_shards > 1 && e->comm_size != e->p.n_shards)
        return fail(DNPEFF_ERR_INVALID, "sharded engine without a communicator: call dnpeff_comm_init");
    bool split = false;
    DN_TRY(compute_ah_hh(e, &split));
    if (e->timing) {
        for (int it = 0; it < iters; it++) DN_TRY(update_w(e, split || it > 0, 1));  // each step timed by itself
    } else {
        // a launch makes as many steps as take a few milliseconds on one row tile
        for (int it = 0; it < iters; it += kFitSteps) DN_TRY(update_w(e, split || it > 0, std::min(kFitSteps, iters - it)));
    }
    if (loss) DN_TRY(loss_from_current(e, false, loss));
    return DNPEFF_OK;
}

int dnpeff_enable_timing(dnpeff_engine* e, int enable) {
    if (!e) return fail(DNPEFF_ERR_INVALID, "null engine");
    e->timing = enable != 0;
    return DNPEFF_OK;
}

int dnpeff_get_timing(dnpeff_engine* e, double ms_total[DNPEFF_N_TIMERS], int64_t launches[DNPEFF_N_TIMERS]) {
    if (!e) return fail(DNPEFF_ERR_INVALID, "null engine");
    DeviceGuard g(e->device);
    DN_CUDA(cudaStreamSynchronize(e->st));
    for (auto& r : e->regions) {
        float ms = 0.f;
        if (cudaEventElapsedTime(&ms, r.a, r.b) == cudaSuccess) {
            e->t_ms[r.id] += ms;
            e->t_n[r.id] += 1;
        }
        e->ev_pool.push_back(r.a);
        e->ev_pool.push_back(r.b);
    }
    e->regions.clear();
    for (int i = 0; i < DNPEFF_N_TIMERS; i++) {
        if (ms_total) ms_total[i] = e->t_ms[i];
        if (launches) launches[i] = e->t_n[i];
        e->t_ms[i] = 0;
        e->t_n[i] = 0;
    }
    return DNPEFF_OK;
}

int dnpeff_launch_count(dnpeff_engine* e, int64_t* out) {
    if (!e || !out) return fail(DNPEFF_ERR_INVALID, "null argument");
    *out = launch_counter() - e->launches0;
    return DNPEFF_OK;
}

// ---- single kernels ---------------------------------------------------------
int dnpeff_op_spmm(const float* vals, const int32_t* ind, const int64_t* ptr, int64_t rows,
                   const float* D, int32_t r, float* out, void* stream) {
    if (rows < 0 || r <= 0) return fail(DNPEFF_ERR_INVALID, "bad shape");
    cudaStream_t st = (cudaStream_t)stream;
    SpmmPlan plan;
    plan.n_short = rows;
    DevBuf<int32_t> long_list;
    DevBuf<int> n_long;
    if (spmm_fast_rank(r) && rows > 0) {
        DN_TRY(long_list.alloc((size_t)rows));
        DN_TRY(n_long.alloc_zero(1, st));
        DN_TRY(spmm_list_long(ptr, 0, rows, long_list.p, n_long.p, st));
        DN_CUDA(cudaMemcpyAsync(&plan.n_long, n_long.p, sizeof(int), cudaMemcpyDeviceToHost, st));
        DN_CUDA(cudaStreamSynchronize(st));
        plan.long_list = long_list.p;
        plan.n_short = rows - plan.n_long;
    }
    int s = spmm_dispatch(vals, ind, ptr, rows, D, r, out, plan, st);
    if (long_list.p) cudaStreamSynchronize(st);  // the list is released on return
    return s;
}

int dnpeff_op_gram(const float* X, int64_t rows, int32_t r, float* G, void* stream) {
    if (rows < 0 || r <= 0) return fail(DNPEFF_ERR_INVALID, "bad shape");
    float* scratch = nullptr;
    int* err = nullptr;
    DN_TRY(op_scratch(gram_any_scratch(rows, r), &scratch));
    DN_TRY(op_err_word(&err));
    DN_TRY(gram_any(X, rows, r, G, nullptr, scratch, err, (cudaStream_t)stream));
    return op_check_err(err, (cudaStream_t)stream);
}

int dnpeff_op_mu_update(float* X, const float* Num, const float* G, int64_t rows, int32_t r,
                        float eps, void* stream) {
    if (rows < 0 || r <= 0) return fail(DNPEFF_ERR_INVALID, "bad shape");
    float* scratch = nullptr;
    int* err = nullptr;
    DN_TRY(op_scratch(2 * (size_t)r * r, &scratch));
    DN_TRY(op_err_word(&err));
    DN_TRY(mu_update_any(X, Num, G, rows, r, eps, scratch, false, err, (cudaStream_t)stream));
    return op_check_err(err, (cudaStream_t)stream);
}

// The projection with its own scratch (released on return; the call synchronises).
static int hoyer_run(float* W, int64_t n, int32_t r, float l1, float l2, int32_t rule, int32_t max_passes,
                     int32_t* passes, int32_t* converged, cudaStream_t st) {
    if (n < 0 || r <= 0) return fail(DNPEFF_ERR_INVALID, "bad shape");
    if (!(l1 > 0.f) || !(l2 > 0.f)) return fail(DNPEFF_ERR_INVALID, "the L1 and L2 norms must be positive");
    if (rule != 0 && rule != 1) return fail(DNPEFF_ERR_INVALID, "alpha_rule must be 0 or 1");
    if (max_passes <= 0) max_passes = (int32_t)std::min<int64_t>(n + 1, INT32_MAX);  // a pass zeroes >= 1 entry per active column
    int np = 0, conv = 1;
    if (n > 0) {
        HoyerPlan plan = hoyer_plan(n, r);
        DevBuf<unsigned char> scratch;
        DN_TRY(scratch.alloc(plan.bytes));
        int* h_count = nullptr;
        DN_CUDA(cudaHostAlloc((void**)&h_count, sizeof(int), cudaHostAllocDefault));
        int s = hoyer_project(W, n, r, l1, l2, rule, max_passes, scratch.p, plan, h_count, &np, &conv, st);
        cudaStreamSynchronize(st);
        cudaFreeHost(h_count);
        if (s != DNPEFF_OK) return s;
    }
    if (passes) *passes = np;
    if (converged) *converged = conv;
    return DNPEFF_OK;
}

int dnpeff_op_hoyer_project(float* W, int64_t n, int32_t r, float l1_norm, float l2_norm, int32_t alpha_rule,
                            int32_t max_passes, int32_t* passes, int32_t* converged, void* stream) {
    return hoyer_run(W, n, r, l1_norm, l2_norm, alpha_rule, max_passes, passes, converged, (cudaStream_t)stream);
}

int dnpeff_sparsify_w(dnpeff_engine* e, float l1_norm, float l2_norm, int32_t alpha_rule, int32_t* passes,
                      int32_t* converged) {
    DN_TRY(check_ready(e, true));
    DeviceGuard g(e->device);
    ArenaScope arena_scope(&e->arena);
    const int r = e->p.rank;
    if (e->ld == r || e->n <= 0)
        return hoyer_run(e->W, e->n, r, l1_norm, l2_norm, alpha_rule, 0, passes, converged, e->st);
    // the projection takes contiguous rows
    DevBuf<float> tmp;
    DN_TRY(tmp.alloc((size_t)(e->n * r)));
    k_gather_rows<<<kNumSMs * 8, 256, 0, e->st>>>(e->W, nullptr, e->n, r, e->ld, r, tmp.p);
    DN_LAUNCH_CHECK();
    DN_TRY(hoyer_run(tmp.p, e->n, r, l1_norm, l2_norm, alpha_rule, 0, passes, converged, e->st));
    k_gather_rows<<<kNumSMs * 8, 256, 0, e->st>>>(tmp.p, nullptr, e->n, r, r, e->ld, e->W);
    DN_LAUNCH_CHECK();
    DN_COUNT_LAUNCH(2);
    DN_CUDA(cudaStreamSynchronize(e->st));
    return DNPEFF_OK;
}

int dnpeff_op_block_product(const float* X, int64_t M, int64_t K, const float* Y, int32_t r, float* C,
                            void* stream) {
    if (M < 0 || K < 0 || r <= 0) return fail(DNPEFF_ERR_INVALID, "bad shape");
    if (!block_tc_ok(r)) return fail(DNPEFF_ERR_UNSUPPORTED, "rank must be 32, 64, 96, 128, 256, 384 or 512");
    if (M == 0) return DNPEFF_OK;
    cudaStream_t st = (cudaStream_t)stream;
    if (K == 0) {
        DN_CUDA(cudaMemsetAsync(C, 0, sizeof(float) * (size_t)(M * r), st));
        return DNPEFF_OK;
    }
    BlockTcPlan p = block_tc_plan(M, K, r);
    DevBuf<float> partial;
    DevBuf<__half> xb, ysplit;
    DevBuf<uint32_t> maxima;  // of the rows of X, then of the columns of Y (two sets)
    DevBuf<unsigned long long> sums;
    DevBuf<unsigned char> again;
    DN_TRY(xb.alloc(p.x_halves));
    DN_TRY(ysplit.alloc(p.ysplit_halves));
    DN_TRY(partial.alloc(p.partial_floats));
    DN_TRY(maxima.alloc_zero(p.xmax_words + 2 * (size_t)r, st));
    DN_TRY(sums.alloc(p.xmax_words));
    DN_TRY(again.alloc_zero((size_t)M, st));
    int* err = nullptr;
    DN_TRY(op_err_word(&err));
    uint32_t* const ymax = maxima.p + p.xmax_words;
    k_block_layout<<<(unsigned)(p.m_tiles * 16), 256, 0, st>>>(X, M, K, p.m_tiles, p.k_chunks, xb.p, maxima.p,
                                                                   sums.p);
    DN_LAUNCH_CHECK();
    const BlkOperand x = {xb.p, maxima.p, sums.p, {X, nullptr, nullptr, nullptr, nullptr, 0, false}};
    DN_TRY(block_tc_launch(x, p, Y, M, K, r, C, nullptr, again.p, ysplit.p, ymax, ymax + r, partial.p, err, st));
    int s = op_check_err(err, st);
    DN_CUDA(cudaStreamSynchronize(st));  // the scratch buffers are released on return
    return s;
}

}  // extern "C"

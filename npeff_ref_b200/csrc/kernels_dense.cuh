// Dense contractions of the multiplicative update, fp32 on the CUDA cores:
//   gram      G[r,r] = X^T X for a tall X [rows, r]       (H*H^T and W^T*W)
//   mu_update X[i,c] *= Num[i,c] / (sum_t X[i,t] G[t,c] + eps)
//             ((W^T W)*H or W*(H H^T), fused with the elementwise update)
// They replace the four cublasSgemm calls per iteration
// (multi_mu_dense_factors_device_contexts1.h:303,306,322,329) and
// kernelNmfMuUpdate (src/nmf/sparse/kernels.h:24-34).
#pragma once
#include "common.cuh"

namespace dnpeff {

// ---------------------------------------------------------------------------
// Gram: the r x r output is cut into TILE x TILE tiles; only tile pairs
// (ti <= tj) are computed.  The rows of X are cut into slabs; block (pair, slab)
// writes one partial tile to scratch; k_gram_reduce adds the slabs in index
// order in double and mirrors the lower triangle.  Fixed order => repeatable.
constexpr int kGramBK = 16;

__host__ __device__ inline int gram_pair_index(int ti, int tj, int ntile) {
    return ti * ntile - ti * (ti - 1) / 2 + (tj - ti);
}

template <int TILE>
__device__ __forceinline__ void gram_load_stage(const float* __restrict__ X, int64_t kb,
                                                int64_t row1, int r, int col0, bool vec_ok,
                                                float (*S)[TILE]) {
    constexpr int PER = TILE * kGramBK / 256;  // floats per thread
    if (vec_ok) {
#pragma unroll
        for (int i = 0; i < PER / 4; i++) {
            int e = threadIdx.x + 256 * i;
            int rr = e / (TILE / 4), c4 = e % (TILE / 4);
            int64_t row = kb + rr;
            int col = col0 + c4 * 4;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (row < row1 && col < r) v = __ldg((const float4*)(X + row * r + col));
            *(float4*)&S[rr][c4 * 4] = v;
        }
    } else {
#pragma unroll
        for (int i = 0; i < PER; i++) {
            int e = threadIdx.x + 256 * i;
            int rr = e / TILE, c = e % TILE;
            int64_t row = kb + rr;
            int col = col0 + c;
            S[rr][c] = (row < row1 && col < r) ? __ldg(X + row * r + col) : 0.f;
        }
    }
}

template <int TILE>
__global__ void __launch_bounds__(256)
k_gram_partial(const float* __restrict__ X, int64_t rows, int r, int ntile, int64_t rows_per_slab,
               float* __restrict__ partial) {
    constexpr int M = TILE / 16;
    __shared__ __align__(16) float As[kGramBK][TILE];
    __shared__ __align__(16) float Bs[kGramBK][TILE];
    int ti = 0, tj = 0;
    {
        int rem = blockIdx.x;
        for (ti = 0; ti < ntile; ti++) {
            int len = ntile - ti;
            if (rem < len) { tj = ti + rem; break; }
            rem -= len;
        }
    }
    const bool diag = (ti == tj);
    const bool vec_ok = (r % 4) == 0;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    int64_t row0 = (int64_t)blockIdx.y * rows_per_slab;
    int64_t row1 = row0 + rows_per_slab < rows ? row0 + rows_per_slab : rows;
    float acc[M][M];
#pragma unroll
    for (int i = 0; i < M; i++)
#pragma unroll
        for (int j = 0; j < M; j++) acc[i][j] = 0.f;

    for (int64_t kb = row0; kb < row1; kb += kGramBK) {
        gram_load_stage<TILE>(X, kb, row1, r, ti * TILE, vec_ok, As);
        if (!diag) gram_load_stage<TILE>(X, kb, row1, r, tj * TILE, vec_ok, Bs);
        __syncthreads();
        float (*Bp)[TILE] = diag ? As : Bs;
#pragma unroll
        for (int kk = 0; kk < kGramBK; kk++) {
            float a[M], b[M];
            if constexpr (M == 8) {
                *(float4*)&a[0] = *(const float4*)&As[kk][ty * 4];
                *(float4*)&a[4] = *(const float4*)&As[kk][TILE / 2 + ty * 4];
                *(float4*)&b[0] = *(const float4*)&Bp[kk][tx * 4];
                *(float4*)&b[4] = *(const float4*)&Bp[kk][TILE / 2 + tx * 4];
            } else {
                *(float4*)&a[0] = *(const float4*)&As[kk][ty * 4];
                *(float4*)&b[0] = *(const float4*)&Bp[kk][tx * 4];
            }
#pragma unroll
            for (int i = 0; i < M; i++)
#pragma unroll
                for (int j = 0; j < M; j++) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        __syncthreads();
    }
    float* out = partial + ((int64_t)blockIdx.y * gridDim.x + blockIdx.x) * (TILE * TILE);
#pragma unroll
    for (int i = 0; i < M; i++) {
        int ri = (M == 8 && i >= 4) ? (TILE / 2 + ty * 4 + i - 4) : (ty * 4 + i);
#pragma unroll
        for (int j = 0; j < M; j += 4) {
            int cj = (M == 8 && j >= 4) ? (TILE / 2 + tx * 4) : (tx * 4);
            *(float4*)&out[ri * TILE + cj] =
                make_float4(acc[i][j], acc[i][j + 1], acc[i][j + 2], acc[i][j + 3]);
        }
    }
}

// The update's division, as one step of iterative refinement of an approximate quotient (the
// residual correction of Wilkinson's "Rounding Errors in Algebraic Processes" for the scalar
// equation t q = n): q0 = n * r with r ~ 1/t good to 2^-23, residual n - t q0 by one fused
// multiply-add, corrected by r times the residual.  q0 is off by at most 1.5 * 2^-23, the
// correction by as much of itself, so the sum before its final rounding is within 2^-44 of n/t:
// the result is within 0.5 + 2^-20 units in the last place.  The IEEE division ends a basic
// block, so that a thread's divisions run one after the other (about 75 clocks apiece in a role
// with two warps per scheduler: 1.11 ms for the mean update of configuration 2 against 1.03);
// these interleave.  It needs t below 2^100 or so (else r is flushed), |n| >= 2^-100 (else the
// residual loses bits) and a finite quotient: callers check a batch afterwards -- a quotient
// that is infinite or NaN, or r or a dividend other than zero below 2^-100 -- and do the whole
// batch again with quot_careful.  Outside these checks only quotients below 2^-126 can be less
// accurate: within 1.5 * 2^-149.
__device__ __forceinline__ float quot_refined(float n, float t, float& r) {
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(t));
    const float q = __fmul_rn(n, r);
    return __fmaf_rn(__fmaf_rn(-t, q, n), r, q);
}

// What a batch of quotients has to be redone for: chk is a sum of 0 * q, r_min the smallest reciprocal,
// lowest the smallest 2 * bits(n) - 1 (the sign dropped, and zero the largest of all).
__device__ __forceinline__ bool quot_doubtful(float chk, float r_min, uint32_t lowest) {
    return !(chk == 0.f) || !(r_min >= 7.888609e-31f) || lowest < 2u * (27u << 23) - 1u;  // 2^-100
}

// n / t in a doubtful batch.  Most are in doubt for a dividend below 2^-100 (factor entries on their
// way to zero, and with heavy-tailed values many at once): those go by 2^60 times the dividend, which is exact and so is the way
// back unless the quotient is subnormal.  Members that were not in doubt come out bit for bit as they were.  What is left -- divisors
// above 2^99, quotients that are not finite or would be subnormal on the way back -- takes the IEEE division, whose slow path is a call
// (458 x 2551, rank 96, heavy-tailed values: an update of 25 rows took 8 us for 3.5).  The bound of quot_refined holds for all operands.
__device__ __forceinline__ float quot_careful(float n, float t) {
    constexpr float k2p60 = 1152921504606846976.f;
    const bool tiny = 2u * __float_as_uint(n) - 1u < 2u * (27u << 23) - 1u, common = t <= 6.338253e29f;  // 2^99
    float r;
    const float q = quot_refined(tiny ? __fmul_rn(n, k2p60) : n, t, r);
    const float least = tiny ? 1.355253e-20f : 0.f;  // 2^-66: the quotient is not subnormal
    if (!(common && fabsf(q) >= least && __fmul_rn(q, 0.f) == 0.f)) return __fdiv_rn(n, t);
    return tiny ? __fmul_rn(q, 1.f / k2p60) : q;
}

// hi = x with the 13 low mantissa bits cleared (what the tensor core would read
// of x anyway), lo = x - hi (exact) rounded to a tf32 value in magnitude.  Integer
// and FP32-pipe instructions only: cvt.rna.tf32.f32 runs at a quarter of their
// rate and, at two per operand value, was the staging threads' largest cost.
__device__ __forceinline__ void tf32_halves(float x, float& hi, float& lo) {
    hi = __uint_as_float(__float_as_uint(x) & 0xFFFFE000u);
    lo = __uint_as_float((__float_as_uint(x - hi) + 0x1000u) & 0xFFFFE000u);
}

// Element (n, k) of a small matrix, split, in the layout the tensor-core update kernel copies it from (k_tc_split_g).
__device__ __forceinline__ void gsplit_store(float* __restrict__ Gsplit, int r, int n, int k, float x) {
    float hi, lo;
    tf32_halves(x, hi, lo);
    const size_t off = (size_t)(k / 32) * 2 * r * 32 + ((size_t)(n / 8) * 8 + (k % 32) / 4) * 32 + (n % 8) * 4 + (k % 4);
    Gsplit[off] = hi;
    Gsplit[off + (size_t)r * 32] = lo;
}

// G[a,b] = sum over slabs of the partial tile element, in double and in a fixed order: a block
// takes 32 elements of the upper triangle, lane group y = thread / 32 the slabs y, y + 8, ...,
// and the eight sums are added in order.  One thread per element, summing up to 148 slabs by
// itself, took 13 to 20 us of latency (64 KB of partials at rank 32, 9.7 MB at 128); 3 to 5 this
// way.  The lower triangle is a copy, so that the result is symmetric bit for bit.  Gsplit (or
// NULL): the same matrix split for the update kernel, which saves that a launch.
// A partial (of one tile) may hold 1 << fold Gram matrices on its diagonal, all of them to be added.
static __global__ void __launch_bounds__(256)
k_gram_reduce(const float* __restrict__ partial, int nslab, int npairs, int ntile, int tile, int r,
              float* __restrict__ G, float* __restrict__ Gsplit, int fold) {
    __shared__ double sums[8][32];
    grid_wait();
    const int x = threadIdx.x & 31, y = threadIdx.x >> 5;
    const int idx = blockIdx.x * 32 + x;
    const int a = idx / r, b = idx % r;
    const bool mine = idx < r * r && a <= b;
    if (!__syncthreads_or(mine ? 1 : 0)) return;
    double s = 0.0;
    if (mine) {
        const int pair = gram_pair_index(a / tile, b / tile, ntile);
        const float* p = partial + (int64_t)pair * (tile * tile) + (a % tile) * tile + b % tile;
        const int64_t stride = (int64_t)npairs * (tile * tile);
#pragma unroll 4
        for (int sl = y; sl < nslab << fold; sl += 8) s += (double)p[(sl >> fold) * stride + (sl & ((1 << fold) - 1)) * (r * tile + r)];
    }
    sums[y][x] = s;
    __syncthreads();
    if (y != 0 || !mine) return;
#pragma unroll
    for (int k = 1; k < 8; k++) s += sums[k][x];
    const float g = (float)s;
    G[a * r + b] = g;
    if (a != b) G[b * r + a] = g;
    if (Gsplit) {
        gsplit_store(Gsplit, r, a, b, g);
        if (a != b) gsplit_store(Gsplit, r, b, a, g);
    }
}

inline int gram_reduce_launch(const float* partial, int nslab, int npairs, int ntile, int tile, int r, float* G,
                              float* Gsplit, cudaStream_t st, int fold = 0) {
    return launch_overlapped(k_gram_reduce, dim3((unsigned)ceil_div((int64_t)r * r, 32)), 256, 0, st, partial, nslab, npairs, ntile,
                             tile, r, G, Gsplit, fold);
}

struct GramPlan {
    int tile, ntile, npairs, nslab;
    int64_t rows_per_slab;
    size_t scratch_floats;
};

inline GramPlan gram_plan(int64_t rows, int r) {
    GramPlan g;
    g.tile = (r > 64) ? 128 : 64;
    g.ntile = (int)ceil_div(r, g.tile);
    g.npairs = g.ntile * (g.ntile + 1) / 2;
    int64_t want = ceil_div(rows > 0 ? rows : 1, 512);
    int64_t cap = (4 * kNumSMs) / g.npairs;  // about 4 blocks per SM over all pairs
    if (cap < 1) cap = 1;
    g.nslab = (int)(want < cap ? want : cap);
    if (g.nslab < 1) g.nslab = 1;
    g.rows_per_slab = ceil_div(rows > 0 ? rows : 1, g.nslab);
    g.rows_per_slab = ceil_div(g.rows_per_slab, kGramBK) * kGramBK;
    g.nslab = (int)ceil_div(rows > 0 ? rows : 1, g.rows_per_slab);
    g.scratch_floats = (size_t)g.nslab * g.npairs * g.tile * g.tile;
    return g;
}

// scratch must hold g.scratch_floats floats.
inline int gram_launch_plan(const float* X, int64_t rows, int r, float* G, float* scratch,
                            const GramPlan& g, cudaStream_t st) {
    dim3 grid(g.npairs, g.nslab);
    if (g.tile == 128)
        k_gram_partial<128><<<grid, 256, 0, st>>>(X, rows, r, g.ntile, g.rows_per_slab, scratch);
    else
        k_gram_partial<64><<<grid, 256, 0, st>>>(X, rows, r, g.ntile, g.rows_per_slab, scratch);
    DN_LAUNCH_CHECK();
    DN_COUNT_LAUNCH(1);
    DN_TRY(gram_reduce_launch(scratch, g.nslab, g.npairs, g.ntile, g.tile, r, G, nullptr, st));
    return DNPEFF_OK;
}

// scratch must hold gram_plan(rows, r).scratch_floats floats.
inline int gram_launch(const float* X, int64_t rows, int r, float* G, float* scratch,
                       cudaStream_t st) {
    return gram_launch_plan(X, rows, r, G, scratch, gram_plan(rows, r), st);
}

// ---------------------------------------------------------------------------
// mu_update: a block owns TR = 16384/RP whole rows of X (RP = r rounded up to
// 32..512).  It first stages its rows, transposed, in shared memory -- after
// that nothing reads those rows from global memory again, so the update can be
// written in place -- then runs a TR x RP x r SGEMM against G streamed in
// 16-row chunks, and finishes with the elementwise rule
//     t = den + eps;  q = num / t;  x = x * q      (kernels.h:31-33 order).
constexpr int kMuKC = 16;

template <int RP>
__global__ void __launch_bounds__(256)
k_mu_update(float* __restrict__ X, const float* __restrict__ Num, const float* __restrict__ G,
            int64_t rows, int r, float eps) {
    constexpr int TR = 16384 / RP;
    constexpr int TX = RP / 8;
    extern __shared__ __align__(16) float smem[];
    float (*XsT)[TR] = (float (*)[TR])smem;                    // [RP][TR]
    float (*Gs)[RP] = (float (*)[RP])(smem + (size_t)RP * TR);  // [kMuKC][RP]
    const int tx = threadIdx.x % TX, ty = threadIdx.x / TX;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int r4 = r / 4;
    const int64_t row0 = (int64_t)blockIdx.x * TR;

    // stage X rows transposed: lane <-> row, so the shared stores hit 32 banks
    for (int rg = 0; rg < TR / 32; rg++) {
        int rl = rg * 32 + lane;
        int64_t row = row0 + rl;
        for (int kq = 2 * w; kq < r4; kq += 16) {
#pragma unroll
            for (int h = 0; h < 2; h++) {
                int q = kq + h;
                if (q < r4) {
                    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (row < rows) v = *(const float4*)(X + row * r + q * 4);
                    XsT[q * 4 + 0][rl] = v.x;
                    XsT[q * 4 + 1][rl] = v.y;
                    XsT[q * 4 + 2][rl] = v.z;
                    XsT[q * 4 + 3][rl] = v.w;
                }
            }
        }
    }

    float acc[8][8];
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
        for (int j = 0; j < 8; j++) acc[i][j] = 0.f;

    for (int k0 = 0; k0 < r; k0 += kMuKC) {
        __syncthreads();  // X staged (first pass) / previous chunk consumed
        for (int e = threadIdx.x; e < kMuKC * (RP / 4); e += 256) {
            int kk = e / (RP / 4), c4 = e % (RP / 4);
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (k0 + kk < r && c4 < r4) v = __ldg((const float4*)(G + (int64_t)(k0 + kk) * r + c4 * 4));
            *(float4*)&Gs[kk][c4 * 4] = v;
        }
        __syncthreads();
        int kmax = (r - k0) < kMuKC ? (r - k0) : kMuKC;
#pragma unroll 4
        for (int kk = 0; kk < kmax; kk++) {
            float a[8], b[8];
            *(float4*)&a[0] = *(const float4*)&XsT[k0 + kk][ty * 8];
            *(float4*)&a[4] = *(const float4*)&XsT[k0 + kk][ty * 8 + 4];
            *(float4*)&b[0] = *(const float4*)&Gs[kk][tx * 4];
            *(float4*)&b[4] = *(const float4*)&Gs[kk][RP / 2 + tx * 4];
#pragma unroll
            for (int i = 0; i < 8; i++)
#pragma unroll
                for (int j = 0; j < 8; j++) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
    }

#pragma unroll
    for (int i = 0; i < 8; i++) {
        int rl = ty * 8 + i;
        int64_t row = row0 + rl;
        if (row >= rows) continue;
#pragma unroll
        for (int h = 0; h < 2; h++) {
            int c = h * (RP / 2) + tx * 4;
            if (c >= r) continue;
            float4 nu = __ldcs((const float4*)(Num + row * r + c));
            float4 o;
            o.x = XsT[c + 0][rl] * __fdiv_rn(nu.x, __fadd_rn(acc[i][h * 4 + 0], eps));
            o.y = XsT[c + 1][rl] * __fdiv_rn(nu.y, __fadd_rn(acc[i][h * 4 + 1], eps));
            o.z = XsT[c + 2][rl] * __fdiv_rn(nu.z, __fadd_rn(acc[i][h * 4 + 2], eps));
            o.w = XsT[c + 3][rl] * __fdiv_rn(nu.w, __fadd_rn(acc[i][h * 4 + 3], eps));
            *(float4*)(X + row * r + c) = o;
        }
    }
}

// Any rank: one warp per row, the row cached in shared memory (r floats per warp).
static __global__ void k_mu_update_generic(float* __restrict__ X, const float* __restrict__ Num,
                                    const float* __restrict__ G, int64_t rows, int r, float eps) {
    extern __shared__ float xs_all[];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    float* xs = xs_all + (size_t)w * r;
    int64_t row = (int64_t)blockIdx.x * (blockDim.x >> 5) + w;
    if (row >= rows) return;
    for (int c = lane; c < r; c += 32) xs[c] = X[row * r + c];
    __syncwarp();
    for (int c = lane; c < r; c += 32) {
        float den = 0.f;
        for (int t = 0; t < r; t++) den = fmaf(xs[t], G[(int64_t)t * r + c], den);
        X[row * r + c] = xs[c] * __fdiv_rn(Num[row * r + c], __fadd_rn(den, eps));
    }
}

template <int RP>
inline int mu_update_launch_t(float* X, const float* Num, const float* G, int64_t rows, int r,
                              float eps, cudaStream_t st) {
    constexpr int TR = 16384 / RP;
    size_t smem = ((size_t)RP * TR + (size_t)kMuKC * RP) * sizeof(float);
    // per device, so set on every call rather than once per process
    DN_CUDA(cudaFuncSetAttribute(k_mu_update<RP>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)smem));
    k_mu_update<RP><<<(unsigned)ceil_div(rows, TR), 256, smem, st>>>(X, Num, G, rows, r, eps);
    DN_LAUNCH_CHECK();
    DN_COUNT_LAUNCH(1);
    return DNPEFF_OK;
}

inline int mu_update_launch(float* X, const float* Num, const float* G, int64_t rows, int r,
                            float eps, cudaStream_t st) {
    if (rows <= 0) return DNPEFF_OK;
    if (r % 4 == 0 && r <= 512) {
        if (r <= 32) return mu_update_launch_t<32>(X, Num, G, rows, r, eps, st);
        if (r <= 64) return mu_update_launch_t<64>(X, Num, G, rows, r, eps, st);
        if (r <= 128) return mu_update_launch_t<128>(X, Num, G, rows, r, eps, st);
        if (r <= 256) return mu_update_launch_t<256>(X, Num, G, rows, r, eps, st);
        return mu_update_launch_t<512>(X, Num, G, rows, r, eps, st);
    }
    size_t smem = (size_t)8 * r * sizeof(float);
    if (smem > 48 * 1024) return fail(DNPEFF_ERR_UNSUPPORTED, "rank %d too large", r);
    k_mu_update_generic<<<(unsigned)ceil_div(rows, 8), 256, smem, st>>>(X, Num, G, rows, r, eps);
    DN_LAUNCH_CHECK();
    DN_COUNT_LAUNCH(1);
    return DNPEFF_OK;
}

// Many updates of the rows of X with the same numerators and G (the coefficient fit) at the narrow strides:
// rows are independent given G, so a block makes all `steps` of its rows without leaving the SM.  A thread owns
// a column: its column of G lies in registers, the rows of X in shared memory, read as broadcasts (one
// 16-byte read feeds four multiply-adds of a warp, the rate at which an SM issues both).  The tensor-core kernel
// needs 6 to 11 us a step for its chain of copy, split, MMA and drain whatever the rows; 500 rows at rank 32 take
// 0.11 us a step here, 2000 at rank 128 2.6.
__host__ __device__ constexpr int fit_threads(int ld) { return ld == 96 ? 192 : 256; }
template <int LD, int K>
__global__ void __launch_bounds__(fit_threads(LD), 1)
k_fit_steps(float* __restrict__ X, const float* __restrict__ Num, const float* __restrict__ G, int64_t rows, int steps, float eps) {
    constexpr int kGroups = fit_threads(LD) / LD, kRows = kGroups * K;
    __shared__ __align__(16) float xs[2][kRows][LD];
    const int c = threadIdx.x % LD, grp = threadIdx.x / LD;
    grid_wait();
    float g[LD], x[K], num[K];
#pragma unroll
    for (int t = 0; t < LD; t++) g[t] = __ldg(G + t * LD + c);
    const int64_t row0 = (int64_t)blockIdx.x * kRows + grp * K;
#pragma unroll
    for (int k = 0; k < K; k++) {
        x[k] = num[k] = 0.f;
        if (row0 + k < rows) {
            x[k] = X[(row0 + k) * LD + c];
            num[k] = Num[(row0 + k) * LD + c];
        }
        xs[0][grp * K + k][c] = x[k];
    }
    for (int s = 0; s < steps; s++) {
        if (LD == 32) __syncwarp();  // a row is one warp's
        else __syncthreads();
        const float* const xr = xs[s & 1][grp * K];
        float d[K][2];
#pragma unroll
        for (int k = 0; k < K; k++) d[k][0] = d[k][1] = 0.f;
#pragma unroll
        for (int t = 0; t < LD; t += 4) {
#pragma unroll
            for (int k = 0; k < K; k++) {
                const float4 v = *(const float4*)(xr + k * LD + t);
                d[k][0] = fmaf(v.x, g[t], d[k][0]);
                d[k][1] = fmaf(v.y, g[t + 1], d[k][1]);
                d[k][0] = fmaf(v.z, g[t + 2], d[k][0]);
                d[k][1] = fmaf(v.w, g[t + 3], d[k][1]);
            }
        }
#pragma unroll
        for (int k = 0; k < K; k++) {
            // t = den + eps; q = num / t; x = x * q (reference order, kernels.h:31-33)
            const float t = __fadd_rn(d[k][0] + d[k][1], eps);
            float rc;
            float q = quot_refined(num[k], t, rc);
            if (quot_doubtful(__fmul_rn(q, 0.f), rc, 2u * __float_as_uint(num[k]) - 1u)) q = quot_careful(num[k], t);
            x[k] *= q;
            xs[(s + 1) & 1][grp * K + k][c] = x[k];
        }
    }
#pragma unroll
    for (int k = 0; k < K; k++)
        if (row0 + k < rows) X[(row0 + k) * LD + c] = x[k];
}

template <int LD>
inline int fit_steps_launch_t(float* X, const float* Num, const float* G, int64_t rows, int steps, float eps, cudaStream_t st) {
    constexpr int kGroups = fit_threads(LD) / LD;
    auto launch = [&](auto kernel, int k) {
        return launch_overlapped(kernel, dim3((unsigned)ceil_div(rows, (int64_t)kGroups * k)), fit_threads(LD), 0, st, X, Num, G,
                                 rows, steps, eps);
    };
    // rows per thread: as few as give every SM one block, at most 4
    if (rows <= (int64_t)kNumSMs * kGroups) return launch(k_fit_steps<LD, 1>, 1);
    if (rows <= (int64_t)kNumSMs * kGroups * 2) return launch(k_fit_steps<LD, 2>, 2);
    return launch(k_fit_steps<LD, 4>, 4);
}
inline int fit_steps_launch(float* X, const float* Num, const float* G, int64_t rows, int r, int steps, float eps,
                            cudaStream_t st) {
    switch (r) {
        case 32: return fit_steps_launch_t<32>(X, Num, G, rows, steps, eps, st);
        case 64: return fit_steps_launch_t<64>(X, Num, G, rows, steps, eps, st);
        case 96: return fit_steps_launch_t<96>(X, Num, G, rows, steps, eps, st);
        default: return fit_steps_launch_t<128>(X, Num, G, rows, steps, eps, st);
    }
}

}  // namespace dnpeff

// Small problems: whole stretches of iterations in one launch.
//
// A matrix with a few hundred thousand stored entries needs 10 to 50 us of work per iteration, and
// the kernels of the large path -- fourteen launches per iteration, each with a pipeline of
// copies, tensor-core runs and drains to fill and empty -- take 100 to 150 us for it whatever its
// size.  Here one cooperative launch makes many iterations: a persistent block per SM, everything
// L2-resident, the contractions on the CUDA cores (strides 32 and 64) or on mma.sync fragments (96 and
// 128), four grid-wide barriers per iteration:
//
//   A  numerators of W: A * H^T, flat over the stored entries | H H^T from the blocks' partials
//   B  W *= num / (W HH + eps), row tiles; each block's partial of W^T W on the way
//   C  numerators of H: A^T * W                               | W^T W from the partials
//   D  H *= num / (H WW + eps); each block's partial of H H^T
//
// us per iteration of A's and C's products, their Gram sums, B and D, each with its barrier (block 0's clock):
// 64 x 1612, stride 32, 6144 entries: 2.7, 2.7, 2.1, 7.2, 7.4; 2048 x 65536, 32, 8.4 M: 72, 73, 2.4, 8.7, 22 (14.9 TB/s
// of gathered rows); 1777 x 43231, 32 (rank 20), 0.83 M: 9.7, 10.7, 2.1, 7.7, 17.6; 300 x 9000, 128, 0.45 M: 19.3, 19.2,
// 6.3, 9.2, 21.1 (11.9 TB/s).
//
// Sparse products.  The stored entries are cut into units of L consecutive entries, one per lane
// group (LD / 4 lanes, a float4 of the factor row each); a unit adds up its entries row by row.
// The sum of a row that starts inside the unit goes to the row's place, the sum of one that
// started earlier to the unit's carry slot, and whoever reads a row adds the carries of the units
// that begin inside it, in order.  So a row of two thousand entries and two thousand rows of one
// entry take the same time, and the result does not depend on timing.
//
// Factors and numerators change during the launch: they are read with ld.global.cg (L2); the
// matrix does not and goes through L1.  Barrier waits are bounded: a block whose wait runs out
// sets the error word and an abort flag, and all blocks leave.
#pragma once
#include "common.cuh"
#include "kernels_dense.cuh"  // quot_refined

namespace dnpeff {

enum : int { kErrGridTimeout = 32 };
// Threads of a block (one per SM): the gathers want as many as the registers allow, the wide
// ranks up to eight Gram fragments each.  A tile of a factor has at most 8 elements per thread.
__host__ __device__ constexpr int small_threads(int ld) { return ld <= 64 ? 1024 : 512; }
__host__ __device__ constexpr int small_tile_most(int ld) { return ld == 96 ? 32 : 8 * small_threads(ld) / ld; }

// Gathers in flight per unit: the wide strides have fewer warps and registers to spare (300 x 9000, rank 128: 80 -> 75 us
// an iteration).
__host__ __device__ constexpr int small_batch(int ld) { return ld <= 64 ? 8 : 16; }

struct SmallSide {            // one of the two half iterations
    const float* vals;        // stored entries, by output row
    const int32_t* ind;       // factor row of each entry
    const int32_t* row_of;    // output row of each entry
    const int64_t* ptr;       // row offsets
    uint32_t entries, unit;   // number of entries; entries per unit (L, a multiple of small_batch)
    int64_t rows;             // output rows
    int tile_rows;            // rows per tile of the update (a multiple of 4)
    float* X;                 // factor that is updated [rows][LD]
    const float* D;           // factor that is gathered [*][LD]
    float* num;               // numerators [rows][LD]
    float* carry;             // [units][LD]
    float* G;                 // Gram matrix of D's factor, [LD][LD]
    float* partial_in;        // its partials, one per block
    float* partial_out;       // partials of the Gram of X, for the other side
};

struct SmallArgs {
    SmallSide w, h;           // .w updates W from H, .h updates H from W
    int iters, r4;            // iterations; float4 per factor row that are not padding
    float eps;
    unsigned int* barrier;    // arrivals, and the abort flag behind them
    uint32_t wait_limit;
    int* err;
};

// All blocks; false once a wait ran out anywhere.
__device__ __forceinline__ bool small_grid_barrier(const SmallArgs& a, unsigned int target) {
    __shared__ int ok_s;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned int seen = 0;
        int ok = 0;
        __threadfence();
        atomicAdd(a.barrier, 1u);
        for (uint32_t spin = 0; spin < a.wait_limit; spin++) {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(a.barrier) : "memory");
            if (seen >= target) { ok = 1; break; }
            if ((spin & 63u) == 63u && *(volatile unsigned int*)(a.barrier + 1)) break;
        }
        if (!ok) {
            *(volatile unsigned int*)(a.barrier + 1) = 1u;
            atomicOr(a.err, kErrGridTimeout);
        }
        __threadfence();
        ok_s = ok;
    }
    __syncthreads();
    return ok_s != 0;
}

template <int LD>
__device__ __forceinline__ void small_products(const SmallSide& s, int r4) {
    constexpr int kQuads = LD / 4;
    constexpr int kLanes = kQuads <= 8 ? 8 : (kQuads <= 16 ? 16 : 32);  // lanes of a unit
    constexpr int kUnits = 32 / kLanes;                                // units of a warp
    constexpr int kB = small_batch(LD);
    const int lane = threadIdx.x & 31, q = lane % kLanes;
    const uint32_t warp = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;  // few units spread over all SMs
    const uint32_t n_warps = (gridDim.x * small_threads(LD)) >> 5;
    const uint32_t n_units = (s.entries + s.unit - 1) / s.unit;
    const float4* D4 = (const float4*)s.D;
    const bool real = q < r4;
    for (uint32_t u0 = warp * kUnits; u0 < n_units; u0 += n_warps * kUnits) {
        const uint32_t u = u0 + lane / kLanes;
        const uint32_t beg = u < n_units ? u * s.unit : 0, end = u < n_units ? min(s.entries, beg + s.unit) : 0;
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        int cur = -1;
        // where the sum of the current row goes
        float4* dst = nullptr;
        // lane q < kB of the unit holds entry p + q; the next ones are asked for one batch ahead
        float v = 0.f, vn = 0.f;
        int j = 0, jn = 0, i = -1, in_ = -1;
        auto fetch = [&](uint32_t p, float& fv, int& fj, int& fi) {
            fv = 0.f;
            fj = 0;
            fi = -1;
            if (q < kB && p + q < end) {
                fv = __ldg(s.vals + p + q);
                fj = __ldg(s.ind + p + q);
                fi = __ldg(s.row_of + p + q);
            }
        };
        fetch(beg, v, j, i);
        const int before = (beg > 0 && beg < end) ? __ldg(s.row_of + beg - 1) : -1;
        for (uint32_t off = 0; off < s.unit; off += kB) {  // the same trips for every unit of the warp
            const uint32_t p = beg + off;
            if (!__any_sync(0xffffffffu, p < end)) break;
            fetch(p + kB, vn, jn, in_);
            float4 h[kB];
#pragma unroll
            for (int t = 0; t < kB; t++) {
                const int jj = __shfl_sync(0xffffffffu, j, t, kLanes);
                h[t] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (real && p + t < end) h[t] = __ldcg(D4 + (int64_t)jj * kQuads + q);
            }
#pragma unroll
            for (int t = 0; t < kB; t++) {
                const float vv = __shfl_sync(0xffffffffu, v, t, kLanes);
                const int row = __shfl_sync(0xffffffffu, i, t, kLanes);
                if (row >= 0 && row != cur) {
                    if (cur >= 0 && q < kQuads) __stcg(dst, acc);
                    acc = make_float4(0.f, 0.f, 0.f, 0.f);
                    dst = (cur < 0 && row == before ? (float4*)s.carry + (int64_t)u * kQuads
                                                    : (float4*)s.num + (int64_t)row * kQuads) + q;
                    cur = row;
                }
                acc.x = fmaf(vv, h[t].x, acc.x);
                acc.y = fmaf(vv, h[t].y, acc.y);
                acc.z = fmaf(vv, h[t].z, acc.z);
                acc.w = fmaf(vv, h[t].w, acc.w);
            }
            v = vn;
            j = jn;
            i = in_;
        }
        if (cur >= 0 && q < kQuads) __stcg(dst, acc);
    }
}

// G[e] for the elements of this block: 32 consecutive ones at a time, the partials in a fixed order
// and in double.  red: [warps][32] doubles.
template <int LD>
__device__ __forceinline__ void small_gram_reduce(const SmallSide& s, double* red) {
    constexpr int kWarps = small_threads(LD) / 32;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int g = blockIdx.x; g < LD * LD / 32; g += gridDim.x) {
        const int e = g * 32 + lane;
        float v[(kNumSMs + kWarps - 1) / kWarps];  // all loads before the first sum
#pragma unroll
        for (int k = 0; k < (kNumSMs + kWarps - 1) / kWarps; k++)
            v[k] = w + k * kWarps < kNumSMs ? __ldcg(s.partial_in + (int64_t)(w + k * kWarps) * LD * LD + e) : 0.f;
        double t = 0.0;
#pragma unroll
        for (int k = 0; k < (kNumSMs + kWarps - 1) / kWarps; k++) t += (double)v[k];
        red[w * 32 + lane] = t;
        __syncthreads();
        if (w == 0) {
#pragma unroll
            for (int k = 1; k < kWarps; k++) t += red[k * 32 + lane];
            __stcg(s.G + e, (float)t);
        }
        __syncthreads();
    }
}

// K consecutive floats at p (aligned as K allows).
template <int K>
__device__ __forceinline__ void small_lds(const float* p, float (&v)[K]) {
    if constexpr (K % 4 == 0) {
#pragma unroll
        for (int k = 0; k < K; k += 4) {
            const float4 x = *(const float4*)(p + k);
            v[k] = x.x; v[k + 1] = x.y; v[k + 2] = x.z; v[k + 3] = x.w;
        }
    } else {
#pragma unroll
        for (int k = 0; k < K; k += 2) {
            const float2 x = *(const float2*)(p + k);
            v[k] = x.x; v[k + 1] = x.y;
        }
    }
}

// The update of one side at the narrow strides (32, 64), on CUDA cores: tile by tile (kUpdate), and
// this block's partial of the Gram matrix of the result (want_gram).  Groups of 256 threads sum every kGroups-th row of a tile, each thread a
// square of (LD / 16)^2 elements.  What a tile needs from L2 is asked for while the tile before
// it is worked on (row offsets and X, then the numerators).  Gs: [LD][LD], Xs: [rows][LD + 4].
template <int LD, bool kUpdate>
__device__ __forceinline__ void small_update_fma(const SmallSide& s, float eps, bool want_gram, float* Gs) {
    float* const Xs = Gs + LD * LD;
    constexpr int kThreads = small_threads(LD), kGroups = kThreads / 256;
    constexpr int kQuads = LD / 4, kLd = LD + 4, kT = LD / 16;
    const int tid = threadIdx.x;
    if (kUpdate) {
        for (int e = tid; e < LD * LD / 4; e += kThreads) ((float4*)Gs)[e] = __ldcg((const float4*)s.G + e);
    }
    float acc[kT][kT];
#pragma unroll
    for (int x = 0; x < kT; x++)
#pragma unroll
        for (int y = 0; y < kT; y++) acc[x][y] = 0.f;
    const int group = tid >> 8, ty = (tid >> 4) & 15, tx = tid & 15;
    const int64_t n_tiles = (s.rows + s.tile_rows - 1) / s.tile_rows;
    // an item is two rows x four columns of a tile; at most one per thread
    const int pair = tid / kQuads, c = tid % kQuads;
    float4 xr[2], num[2];      // of this thread's item
    uint32_t edge[3];          // row offsets of its two rows
    auto rows_of = [&](int64_t tile) {
        const int64_t left = s.rows - tile * s.tile_rows;
        return tile < n_tiles ? (int)(left < s.tile_rows ? left : s.tile_rows) : 0;
    };
    auto ask_x = [&](int64_t tile) {
        const int rows = rows_of(tile);
        const int64_t row = tile * s.tile_rows + 2 * pair;
#pragma unroll
        for (int k = 0; k < 2; k++) {
            xr[k] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (2 * pair + k < rows) xr[k] = __ldcg((const float4*)s.X + (row + k) * kQuads + c);
        }
        if (kUpdate) {
#pragma unroll
            for (int k = 0; k < 3; k++) edge[k] = 2 * pair < rows && 2 * pair + k <= rows ? (uint32_t)__ldg(s.ptr + row + k) : 0u;
            if (2 * pair + 1 == rows) edge[2] = edge[1];
        }
    };
    auto ask_num = [&](int64_t tile) {
        const int64_t row = tile * s.tile_rows + 2 * pair;
#pragma unroll
        for (int k = 0; k < 2; k++) {
            num[k] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (edge[k + 1] > edge[k]) num[k] = __ldcg((const float4*)s.num + (row + k) * kQuads + c);
        }
    };
    ask_x(blockIdx.x);
    if (kUpdate) ask_num(blockIdx.x);
    for (int64_t tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
        const int64_t row0 = tile * s.tile_rows;
        const int rows = rows_of(tile);
        const bool item = 2 * pair < rows;
        __syncthreads();  // the previous tile's Gram is done with Xs
        if (item) {
#pragma unroll
            for (int k = 0; k < 2; k++)
                if (2 * pair + k < rows) *(float4*)(Xs + (2 * pair + k) * kLd + c * 4) = xr[k];
        }
        __syncthreads();
        if (kUpdate) {
            constexpr int kBatch = 8;
            if (item) {
                // the pieces of a row that later units hold: those that begin inside it
#pragma unroll
                for (int k = 0; k < 2; k++) {
                    if (edge[k + 1] > edge[k]) {
                        const uint32_t u1 = (edge[k + 1] - 1) / s.unit;
                        for (uint32_t u = edge[k] / s.unit + 1; u <= u1; u += kBatch) {
                            float4 x[kBatch];  // in flight together
#pragma unroll
                            for (int b = 0; b < kBatch; b++) {
                                x[b] = make_float4(0.f, 0.f, 0.f, 0.f);
                                if (u + b <= u1) x[b] = __ldcg((const float4*)s.carry + (int64_t)(u + b) * kQuads + c);
                            }
#pragma unroll
                            for (int b = 0; b < kBatch; b++) {
                                num[k].x += x[b].x; num[k].y += x[b].y; num[k].z += x[b].z; num[k].w += x[b].w;
                            }
                        }
                    }
                }
            }
            ask_x(tile + gridDim.x);
            if (item) {
                const float* x0 = Xs + 2 * pair * kLd;
                const float* x1 = 2 * pair + 1 < rows ? x0 + kLd : x0;
                float4 d0 = make_float4(0.f, 0.f, 0.f, 0.f), d1 = d0;
#pragma unroll 2
                for (int t = 0; t < LD; t += 4) {
                    float a[4], b[4];
                    small_lds<4>(x0 + t, a);
                    small_lds<4>(x1 + t, b);
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        const float4 g = *(const float4*)(Gs + (t + k) * LD + c * 4);
                        d0.x = fmaf(a[k], g.x, d0.x); d0.y = fmaf(a[k], g.y, d0.y);
                        d0.z = fmaf(a[k], g.z, d0.z); d0.w = fmaf(a[k], g.w, d0.w);
                        d1.x = fmaf(b[k], g.x, d1.x); d1.y = fmaf(b[k], g.y, d1.y);
                        d1.z = fmaf(b[k], g.z, d1.z); d1.w = fmaf(b[k], g.w, d1.w);
                    }
                }
                // t = den + eps; q = num / t; x = x * q (reference order, kernels.h:31-33).  The IEEE
                // division would leave its fast path for every zero numerator, those of the padding
                // columns first of all: quot_refined, with its checks, as in k_mu_update_ws.
                const float4 xa = *(const float4*)(x0 + c * 4), xb = *(const float4*)(x1 + c * 4);
                const float xs[8] = {xa.x, xa.y, xa.z, xa.w, xb.x, xb.y, xb.z, xb.w};
                const float ns[8] = {num[0].x, num[0].y, num[0].z, num[0].w, num[1].x, num[1].y, num[1].z, num[1].w};
                const float ds[8] = {d0.x, d0.y, d0.z, d0.w, d1.x, d1.y, d1.z, d1.w};
                float q[8], chk = 0.f, r_min = 1.0f;
                uint32_t lowest = 0xffffffffu;
#pragma unroll
                for (int k = 0; k < 8; k++) {
                    float rc;
                    q[k] = quot_refined(ns[k], __fadd_rn(ds[k], eps), rc);
                    chk = __fmaf_rn(q[k], 0.f, chk);
                    lowest = min(lowest, 2u * __float_as_uint(ns[k]) - 1u);
                    r_min = fminf(r_min, rc);
                }
                if (quot_doubtful(chk, r_min, lowest)) {
#pragma unroll 1
                    for (int k = 0; k < 8; k++) {
                        // registers picked without indexing the arrays dynamically
                        float n = ns[0], d = ds[0];
#pragma unroll
                        for (int m = 1; m < 8; m++) {
                            n = k == m ? ns[m] : n;
                            d = k == m ? ds[m] : d;
                        }
                        const float e = __fdiv_rn(n, __fadd_rn(d, eps));
#pragma unroll
                        for (int m = 0; m < 8; m++) q[m] = k == m ? e : q[m];
                    }
                }
                num[0] = make_float4(xs[0] * q[0], xs[1] * q[1], xs[2] * q[2], xs[3] * q[3]);
                num[1] = make_float4(xs[4] * q[4], xs[5] * q[5], xs[6] * q[6], xs[7] * q[7]);
            }
            __syncthreads();  // every thread has read its rows of Xs
            if (item) {
#pragma unroll
                for (int k = 0; k < 2; k++) {
                    if (2 * pair + k < rows) {
                        __stcg((float4*)s.X + (row0 + 2 * pair + k) * kQuads + c, num[k]);
                        *(float4*)(Xs + (2 * pair + k) * kLd + c * 4) = num[k];
                    }
                }
            }
            ask_num(tile + gridDim.x);
            __syncthreads();
        } else {
            ask_x(tile + gridDim.x);
        }
        if (want_gram) {
            for (int rr = group; rr < rows; rr += kGroups) {
                float a[kT], b[kT];
                small_lds<kT>(Xs + rr * kLd + ty * kT, a);
                small_lds<kT>(Xs + rr * kLd + tx * kT, b);
#pragma unroll
                for (int i = 0; i < kT; i++)
#pragma unroll
                    for (int k = 0; k < kT; k++) acc[i][k] = fmaf(a[i], b[k], acc[i][k]);
            }
        }
    }
    if (want_gram) {
        // the groups' squares are added in order in Gs, which is not needed any more
        for (int g = 0; g < kGroups; g++) {
            __syncthreads();
            if (group != g) continue;
#pragma unroll
            for (int i = 0; i < kT; i++)
#pragma unroll
                for (int k = 0; k < kT; k++) {
                    float* p = Gs + (ty * kT + i) * LD + tx * kT + k;
                    *p = g == 0 ? acc[i][k] : *p + acc[i][k];
                }
        }
        __syncthreads();
        float4* out = (float4*)(s.partial_out + (int64_t)blockIdx.x * LD * LD);
        for (int e = tid; e < LD * LD / 4; e += kThreads) __stcg(out + e, ((const float4*)Gs)[e]);
    }
}

// D (16 x 8, fp32) += A (16 x 8) * B (8 x 8), both tf32.  With g = lane / 4 and t = lane % 4 a lane holds
// A(g, t), A(g + 8, t), A(g, t + 4), A(g + 8, t + 4); B(t, g), B(t + 4, g); D(g, 2t), D(g, 2t + 1), D(g + 8, 2t), D(g + 8, 2t + 1).
// (The small fragments of mma.sync fit a tile that is gone in a few microseconds and lives in
// shared memory anyway.  At the wide strides they halve what the CUDA cores' contractions, bound by
// their shared-memory reads, take: 300 x 9000, rank 128: 100 -> 80 us an iteration.  At 32 and 64 the
// splitting of the operands eats that up: 35 against 32 us at 1777 x 43303, rank 20.)
__device__ __forceinline__ void small_mma(float (&d)[4], const float (&a)[4], const float (&b)[2]) {
    asm volatile(
        "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(__float_as_uint(a[0])), "r"(__float_as_uint(a[1])), "r"(__float_as_uint(a[2])), "r"(__float_as_uint(a[3])),
          "r"(__float_as_uint(b[0])), "r"(__float_as_uint(b[1])));
}
// The same to fp32 accuracy from the hi and lo halves.
__device__ __forceinline__ void small_mma3(float (&d)[4], const float (&ah)[4], const float (&al)[4], const float (&bh)[2],
                                           const float (&bl)[2]) {
    small_mma(d, al, bh);
    small_mma(d, ah, bl);
    small_mma(d, ah, bh);
}
__device__ __forceinline__ void small_split_store(float* hi, float* lo, const float4& x) {
    float4 h, l;
    tf32_halves(x.x, h.x, l.x);
    tf32_halves(x.y, h.y, l.y);
    tf32_halves(x.z, h.z, l.z);
    tf32_halves(x.w, h.w, l.w);
    *(float4*)hi = h;
    *(float4*)lo = l;
}

// The update of one side at the wide strides (96, 128): tile by tile (kUpdate), and this block's
// partial of the Gram matrix of the result (want_gram).  Both contractions run on tensor-core fragments of operands split in
// shared memory (3xTF32), 64 values of K at a time: longer sums come out low, the tensor core
// truncates.  Both are bound by the shared-memory reads of their fragments, so the strides keep
// those free of bank conflicts (LD + 4 for G, LD + 8 for the Gram's reads of X along rows) and a
// warp holds several fragments: 16 rows x 16 columns of a tile's denominators, 16 x 32 of the Gram.
// What a tile needs from L2 is asked for while the tile before it is worked on (row offsets and X,
// then the numerators).
// smem: G hi | G lo ([LD][LD + 4] each, symmetric), X hi | X lo ([rows][LD + 8] each).
template <int LD, bool kUpdate>
__device__ __forceinline__ void small_update_mma(const SmallSide& s, float eps, bool want_gram, float* smem) {
    constexpr int kThreads = small_threads(LD), kWarps = kThreads / 32, kMost = small_tile_most(LD);
    constexpr int kQuads = LD / 4, kLdG = LD + 4, kLd = LD + 8;
    constexpr int kN = 4, kPieces = (LD / 16) * (LD / 32), kMine = (kPieces + kWarps - 1) / kWarps;
    constexpr int kXs = (kMost * kQuads + kThreads - 1) / kThreads;  // float4 of X per thread
    float* const Gh = smem;
    float* const Gl = Gh + LD * kLdG;
    float* const Xh = Gl + LD * kLdG;
    float* const Xl = Xh + kMost * kLd;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, g = lane >> 2, t = lane & 3;
    if (kUpdate) {
        for (int e = tid; e < LD * kQuads; e += kThreads)
            small_split_store(Gh + (e / kQuads) * kLdG + (e % kQuads) * 4, Gl + (e / kQuads) * kLdG + (e % kQuads) * 4,
                              __ldcg((const float4*)s.G + e));
    }
    float acc[kMine][kN][4];
#pragma unroll
    for (int f = 0; f < kMine; f++)
#pragma unroll
        for (int h = 0; h < kN; h++)
#pragma unroll
            for (int k = 0; k < 4; k++) acc[f][h][k] = 0.f;
    const int64_t n_tiles = (s.rows + s.tile_rows - 1) / s.tile_rows;
    const int r0 = (w / (LD / 16)) * 16 + g, c0 = (w % (LD / 16)) * 16 + 2 * t;  // this lane's rows r0, r0 + 8; columns c0, c0 + 8 (+ 1)
    float4 xr[kXs];
    float2 num[2][2];          // [row][column pair]
    uint32_t edge[2][2];       // [row][begin, end] of its entries
    auto rows_of = [&](int64_t tile) {
        const int64_t left = s.rows - tile * s.tile_rows;
        return tile < n_tiles ? (int)(left < s.tile_rows ? left : s.tile_rows) : 0;
    };
    auto ask_x = [&](int64_t tile) {
        const int rows = rows_of(tile);
        const int64_t row0 = tile * s.tile_rows;
#pragma unroll
        for (int k = 0; k < kXs; k++) {
            const int e = tid + k * kThreads;
            xr[k] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (e < rows * kQuads) xr[k] = __ldcg((const float4*)s.X + row0 * kQuads + e);
        }
        if (kUpdate) {
#pragma unroll
            for (int k = 0; k < 2; k++) {
                edge[k][0] = edge[k][1] = 0u;
                if (r0 + 8 * k < rows) {
                    edge[k][0] = (uint32_t)__ldg(s.ptr + row0 + r0 + 8 * k);
                    edge[k][1] = (uint32_t)__ldg(s.ptr + row0 + r0 + 8 * k + 1);
                }
            }
        }
    };
    auto ask_num = [&](int64_t tile) {
        const float* p = s.num + (tile * s.tile_rows + r0) * LD + c0;
#pragma unroll
        for (int k = 0; k < 2; k++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                num[k][h] = make_float2(0.f, 0.f);
                if (edge[k][1] > edge[k][0]) num[k][h] = __ldcg((const float2*)(p + 8 * k * LD + 8 * h));
            }
    };
    ask_x(blockIdx.x);
    if (kUpdate) ask_num(blockIdx.x);
    for (int64_t tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
        const int64_t row0 = tile * s.tile_rows;
        const int rows = rows_of(tile), rows16 = (rows + 15) & ~15;
        __syncthreads();  // the previous tile's Gram is done with X
#pragma unroll
        for (int k = 0; k < kXs; k++) {
            const int e = tid + k * kThreads;
            if (e < rows16 * kQuads) {  // rows past the end: zero
                const int o = (e / kQuads) * kLd + (e % kQuads) * 4;
                small_split_store(Xh + o, Xl + o, xr[k]);
            }
        }
        __syncthreads();
        if (kUpdate) {
            const bool item = (w / (LD / 16)) * 16 < rows;  // uniform per warp
            constexpr int kBatch = 4;
            if (item) {
                // the pieces of a row that later units hold: those that begin inside it
                uint32_t u[2], u1[2];
#pragma unroll
                for (int k = 0; k < 2; k++) {
                    u[k] = 1;
                    u1[k] = 0;
                    if (edge[k][1] > edge[k][0]) {
                        u[k] = edge[k][0] / s.unit + 1;
                        u1[k] = (edge[k][1] - 1) / s.unit;
                    }
                }
                while (u[0] <= u1[0] || u[1] <= u1[1]) {
                    float2 x[2][2][kBatch];  // in flight together
#pragma unroll
                    for (int k = 0; k < 2; k++)
#pragma unroll
                        for (int h = 0; h < 2; h++)
#pragma unroll
                            for (int b = 0; b < kBatch; b++) {
                                x[k][h][b] = make_float2(0.f, 0.f);
                                if (u[k] + b <= u1[k])
                                    x[k][h][b] = __ldcg((const float2*)(s.carry + (int64_t)(u[k] + b) * LD + c0 + 8 * h));
                            }
#pragma unroll
                    for (int k = 0; k < 2; k++) {
#pragma unroll
                        for (int h = 0; h < 2; h++)
#pragma unroll
                            for (int b = 0; b < kBatch; b++) {
                                num[k][h].x += x[k][h][b].x;
                                num[k][h].y += x[k][h][b].y;
                            }
                        u[k] += kBatch;
                    }
                }
            }
            ask_x(tile + gridDim.x);
            if (item) {
                float2 xv[2][2];  // X itself: the halves in shared memory hold 22 of its bits
#pragma unroll
                for (int k = 0; k < 2; k++)
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        xv[k][h] = make_float2(0.f, 0.f);
                        if (r0 + 8 * k < rows) xv[k][h] = __ldcg((const float2*)(s.X + (row0 + r0 + 8 * k) * LD + c0 + 8 * h));
                    }
                float d[2][4];
#pragma unroll
                for (int h = 0; h < 2; h++)
#pragma unroll
                    for (int k = 0; k < 4; k++) d[h][k] = 0.f;
                const float* xh = Xh + r0 * kLd + t;
                const float* xl = Xl + r0 * kLd + t;
                const int gn = (w % (LD / 16)) * 16 + g;  // row of G = column n of the fragment
#pragma unroll
                for (int k64 = 0; k64 < LD; k64 += 64) {
                    float q[2][4];
#pragma unroll
                    for (int h = 0; h < 2; h++)
#pragma unroll
                        for (int k = 0; k < 4; k++) q[h][k] = 0.f;
#pragma unroll 2
                    for (int k0 = k64; k0 < (LD < k64 + 64 ? LD : k64 + 64); k0 += 8) {
                        const float ah[4] = {xh[k0], xh[8 * kLd + k0], xh[k0 + 4], xh[8 * kLd + k0 + 4]};
                        const float al[4] = {xl[k0], xl[8 * kLd + k0], xl[k0 + 4], xl[8 * kLd + k0 + 4]};
#pragma unroll
                        for (int h = 0; h < 2; h++) {
                            const int o = (gn + 8 * h) * kLdG + k0 + t;
                            const float bh[2] = {Gh[o], Gh[o + 4]}, bl[2] = {Gl[o], Gl[o + 4]};
                            small_mma3(q[h], ah, al, bh, bl);
                        }
                    }
#pragma unroll
                    for (int h = 0; h < 2; h++)
#pragma unroll
                        for (int k = 0; k < 4; k++) d[h][k] += q[h][k];
                }
                // t = den + eps; q = num / t; x = x * q (reference order, kernels.h:31-33).  The IEEE
                // division would leave its fast path for every zero numerator, those of the padding
                // columns first of all: quot_refined, with its checks, as in k_mu_update_ws.
                float q[8], chk = 0.f, r_min = 1.0f;
                uint32_t lowest = 0xffffffffu;
#pragma unroll
                for (int k = 0; k < 8; k++) {  // k = 4 h + 2 row + column
                    const float2 n2 = num[(k >> 1) & 1][k >> 2];
                    const float n = (k & 1) ? n2.y : n2.x;
                    float rc;
                    q[k] = quot_refined(n, __fadd_rn(d[k >> 2][k & 3], eps), rc);
                    chk = __fmaf_rn(q[k], 0.f, chk);
                    lowest = min(lowest, 2u * __float_as_uint(n) - 1u);
                    r_min = fminf(r_min, rc);
                }
                if (quot_doubtful(chk, r_min, lowest)) {
#pragma unroll
                    for (int k = 0; k < 8; k++) {
                        const float2 n2 = num[(k >> 1) & 1][k >> 2];
                        q[k] = __fdiv_rn((k & 1) ? n2.y : n2.x, __fadd_rn(d[k >> 2][k & 3], eps));
                    }
                }
#pragma unroll
                for (int k = 0; k < 2; k++)
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        num[k][h] = make_float2(xv[k][h].x * q[4 * h + 2 * k], xv[k][h].y * q[4 * h + 2 * k + 1]);
                    }
            }
            __syncthreads();  // every warp has read its rows of X
            if (item) {
#pragma unroll
                for (int k = 0; k < 2; k++)
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        const int o = (r0 + 8 * k) * kLd + c0 + 8 * h;
                        if (r0 + 8 * k < rows) {
                            __stcg((float2*)(s.X + (row0 + r0 + 8 * k) * LD + c0 + 8 * h), num[k][h]);
                            float2 hi, lo;
                            tf32_halves(num[k][h].x, hi.x, lo.x);
                            tf32_halves(num[k][h].y, hi.y, lo.y);
                            *(float2*)(Xh + o) = hi;
                            *(float2*)(Xl + o) = lo;
                        }
                    }
            }
            ask_num(tile + gridDim.x);
            __syncthreads();
        } else {
            ask_x(tile + gridDim.x);
        }
        if (want_gram) {
#pragma unroll
            for (int f = 0; f < kMine; f++) {
                const int piece = w + f * kWarps;
                if (piece < kPieces) {
                    const int m = (piece / (LD / 32)) * 16 + g, n = (piece % (LD / 32)) * 32 + g;
                    for (int k64 = 0; k64 < rows16; k64 += 64) {
                        float q[kN][4];
#pragma unroll
                        for (int h = 0; h < kN; h++)
#pragma unroll
                            for (int k = 0; k < 4; k++) q[h][k] = 0.f;
                        const int last = rows16 < k64 + 64 ? rows16 : k64 + 64;
#pragma unroll 1
                        for (int k0 = k64; k0 < last; k0 += 8) {
                            const int o = (k0 + t) * kLd;
                            const float ah[4] = {Xh[o + m], Xh[o + m + 8], Xh[o + 4 * kLd + m], Xh[o + 4 * kLd + m + 8]};
                            const float al[4] = {Xl[o + m], Xl[o + m + 8], Xl[o + 4 * kLd + m], Xl[o + 4 * kLd + m + 8]};
#pragma unroll
                            for (int h = 0; h < kN; h++) {
                                const float bh[2] = {Xh[o + n + 8 * h], Xh[o + 4 * kLd + n + 8 * h]};
                                const float bl[2] = {Xl[o + n + 8 * h], Xl[o + 4 * kLd + n + 8 * h]};
                                small_mma3(q[h], ah, al, bh, bl);
                            }
                        }
#pragma unroll
                        for (int h = 0; h < kN; h++)
#pragma unroll
                            for (int k = 0; k < 4; k++) acc[f][h][k] += q[h][k];
                    }
                }
            }
        }
    }
    if (want_gram) {
#pragma unroll
        for (int f = 0; f < kMine; f++) {
            const int piece = w + f * kWarps;
            if (piece >= kPieces) continue;
            float* p = s.partial_out + (int64_t)blockIdx.x * LD * LD + ((piece / (LD / 32)) * 16 + g) * LD +
                       (piece % (LD / 32)) * 32 + 2 * t;
#pragma unroll
            for (int h = 0; h < kN; h++) {
                __stcg((float2*)(p + 8 * h), make_float2(acc[f][h][0], acc[f][h][1]));
                __stcg((float2*)(p + 8 * h + 8 * LD), make_float2(acc[f][h][2], acc[f][h][3]));
            }
        }
    }
}

template <int LD, bool kUpdate>
__device__ __forceinline__ void small_update(const SmallSide& s, float eps, bool want_gram, float* smem) {
    if constexpr (LD <= 64) small_update_fma<LD, kUpdate>(s, eps, want_gram, smem);
    else small_update_mma<LD, kUpdate>(s, eps, want_gram, smem);
}

template <int LD>
__global__ void __launch_bounds__(small_threads(LD), 1) k_small_run(const SmallArgs a) {
    extern __shared__ __align__(16) float small_smem[];
    __shared__ double red[small_threads(LD)];
    unsigned int target = 0;
    // the partials of H H^T for the first W update
    small_update<LD, false>(a.h, a.eps, true, small_smem);
    if (!small_grid_barrier(a, target += gridDim.x)) return;
    for (int it = 0; it < a.iters; it++) {
        small_gram_reduce<LD>(a.w, red);
        small_products<LD>(a.w, a.r4);
        if (!small_grid_barrier(a, target += gridDim.x)) return;
        small_update<LD, true>(a.w, a.eps, true, small_smem);
        if (!small_grid_barrier(a, target += gridDim.x)) return;
        small_gram_reduce<LD>(a.h, red);
        small_products<LD>(a.h, a.r4);
        if (!small_grid_barrier(a, target += gridDim.x)) return;
        small_update<LD, true>(a.h, a.eps, it + 1 < a.iters, small_smem);
        if (it + 1 < a.iters && !small_grid_barrier(a, target += gridDim.x)) return;
    }
}

// row_of[p] = i for the entries p of row i; one warp per row.
static __global__ void k_small_row_of(const int64_t* __restrict__ ptr, int64_t rows, int32_t* __restrict__ row_of) {
    const int64_t warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < rows; i += warps)
        for (int64_t p = ptr[i] + (threadIdx.x & 31); p < ptr[i + 1]; p += 32) row_of[p] = (int32_t)i;
}

inline bool small_rank_ok(int ld) { return ld == 32 || ld == 64 || ld == 96 || ld == 128; }

inline size_t small_smem_bytes(int ld) {
    const size_t rows = (size_t)small_tile_most(ld), n = (size_t)ld;
    return sizeof(float) * (ld <= 64 ? n * n + rows * (n + 4) : 2 * (n * (n + 4) + rows * (n + 8)));
}

// Entries per unit so that every lane group of the grid has one.
inline uint32_t small_unit(int64_t entries, int ld) {
    const int lanes = ld <= 32 ? 8 : (ld <= 64 ? 16 : 32);
    const int64_t groups = (int64_t)kNumSMs * (small_threads(ld) / lanes);
    const int b = small_batch(ld);
    return (uint32_t)std::max<int64_t>(b, (ceil_div(entries, groups) + b - 1) / b * b);
}
// Rows per tile: every block the same number of tiles, none larger than a block can hold.
inline int small_tile_rows(int64_t rows, int ld) {
    const int64_t most = small_tile_most(ld);
    const int64_t per_block = ceil_div(rows, kNumSMs), rounds = ceil_div(per_block, most);
    return (int)std::max<int64_t>(4, (ceil_div(per_block, rounds) + 3) / 4 * 4);
}

// Whether these launches beat the large path.  An iteration takes about 20 us (barriers, and the
// latency of the four phases), two gathers of a factor row per stored entry at 15 TB/s (12 at the wide strides;
// measured: 14.9 and 11.9) and the two contractions at what shared memory delivers to the cores.  The large path
// takes 65 to 105 us plus the same gathers a little slower, but contracts on the tensor cores: even near
// 230 us in all at stride 32 (3000 x 60000 x 4000 values: 233 either way; half of them 136 against 175),
// 160 at 64 (2000 x 40000 x 2000: 182 against 167; 500 x 20000 x 2000: 75 against 109) and 130 above
// (rank 128, 1000 x 20000 x 1500: 177 against 152; 300 x 9000 x 1500: 75 against 104).
inline bool small_pays(int64_t nnz, int64_t rows, int r4, int ld) {
    const double gather = 2.0 * (double)nnz * 16.0 * r4 / (ld <= 64 ? 15.0e6 : 12.0e6);
    const double contract = (double)rows * ld * ld / (ld <= 64 ? 5.0e6 : 10.0e6);
    return contract < 60.0 && 20.0 + gather + contract < (ld <= 32 ? 230.0 : (ld <= 64 ? 160.0 : 130.0));
}

// All blocks have to be on the GPU together: where the process may not use that many SMs (a share of an MPS
// server, for one) the runtime refuses the launch, and *made says so; nothing has run then.
// refuse: as if it had.
template <int LD>
inline int small_launch_t(SmallArgs& a, cudaStream_t st, bool refuse, bool* made) {
    DN_CUDA(cudaFuncSetAttribute(k_small_run<LD>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)small_smem_bytes(LD)));
    void* args[] = {&a};
    const cudaError_t e = refuse ? cudaErrorCooperativeLaunchTooLarge
                                 : cudaLaunchCooperativeKernel((void*)k_small_run<LD>, dim3(kNumSMs), dim3(small_threads(LD)), args,
                                                               small_smem_bytes(LD), st);
    *made = e != cudaErrorCooperativeLaunchTooLarge;
    if (!*made) {
        cudaGetLastError();
        return DNPEFF_OK;
    }
    DN_CUDA(e);
    DN_COUNT_LAUNCH(1);
    return DNPEFF_OK;
}
inline int small_launch(SmallArgs& a, int ld, cudaStream_t st, bool refuse, bool* made) {
    DN_CUDA(cudaMemsetAsync(a.barrier, 0, 2 * sizeof(unsigned int), st));
    switch (ld) {
        case 32: return small_launch_t<32>(a, st, refuse, made);
        case 64: return small_launch_t<64>(a, st, refuse, made);
        case 96: return small_launch_t<96>(a, st, refuse, made);
        default: return small_launch_t<128>(a, st, refuse, made);
    }
}

}  // namespace dnpeff

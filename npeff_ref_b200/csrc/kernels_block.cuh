// Dense block product  C[M x r] = X[M x K] * Y[K x r]  (r a multiple of 32 up to 128, or of 128 up to
// 512) on the tensor cores (tcgen05.mma, fp16 operands in two halves, fp32 accumulation).
//
// The popular columns of A form a block that is far from sparse, so that block is kept a
// second time as a dense matrix and its share of both sparse products runs
// on the tensor cores:  A*H^T gets X = A_pop (rows of A x popular columns),
// Y = the popular rows of H;  A^T*W gets X = A_pop^T, Y = W.
//
// Precision.  Every operand x, scaled by a power of two that brings the largest magnitude of its row of X
// (its column of Y) into [2^14, 2^15), is split into hi = fp16(x) and lo = fp16((x - hi) * 2^11), both
// rounded to nearest: within 2^-24 of x while the scaled value is at least 2^-12 (a 2^-27th of the largest),
// within 2^-36 (2^-51 of the largest) below.  hi*hi and hi*lo + lo*hi go to accumulators of their own, the
// second counting 2^-11; lo*lo is left out.  Measured against float64, sums of 20000 terms: 1.1e-7 where a
// quarter of X is stored (with tf32 halves, truncated, in one accumulator: 5.3e-7).
// Values below 2^-12 ("faint") matter only where a sum consists of little else, and there they must not be
// lost: a numerator that comes out zero would hold its factor entry at zero for good.  Rows of X and
// columns of Y with faint values are marked, and where such a row or column meets a sum so small that the
// representation could be off by 2^-23 of it, the row of C is computed again from the values themselves
// (blk_faint, blk_repair_row).
//
// Layouts.  X is split when the matrix is loaded (4 bytes per element, as fp32), in blocks of 128
// rows x 64 K-values, block (tile, chunk) at (tile * k_chunks + chunk) * 32 KB: [hi | lo], each in the
// K-major core matrices (8 rows x 8 K-values, 128 bytes) that the MMA reads (blk_canon).  Y
// is split once per product (k_split_y), in chunks of 64 K-values in the same layout
// [hi r*64 | lo r*64].  A block of X and a chunk of Y arrive by one bulk copy each and are used as they
// are.  (Splitting X in the kernel, through registers into TMEM, took 2100 clocks a run for the MMAs' 770:
// two thirds of them in the hand-over between copies, splitting warps and MMAs.)
//
// What bounds it: the stream of X, 4 bytes per element.  20000 x 16384 x 128: 267 us, 4.9 TB/s; with tf32
// halves split in the kernel 370 us, bound by the tensor pipe at the clock that the power limit left.
//
// Runs.  The tensor core accumulates hi*hi over 64 K-values (4 MMAs) into one of two TMEM
// accumulators; the drainers add each finished run into fp32 registers (the tensor core truncates, see
// kernels_tc.cuh).  The cross terms are 2^-12 of the sum and of either sign: their accumulator is
// drained once, at the end of the item.
//
// Roles in a block of 11 warps, meeting only through mbarriers:
//   warps 0-7   drainers: thread = tile row (w%4)*32 + lane; accumulator columns [64*(w/4), +64) of
//               each finished run are added into registers
//   warp 8      issues hi*hi, warp 9 the cross terms: no accumulator is written by MMAs of two threads, and
//               while one is held up by the tensor-core queue the other waits for the next run's
//               operands, so barrier latency stays off the tensor core's path
//   warp 10     lane 0 issues the bulk copies
// `abort` ends every role's loop once any bounded wait ran out.
//
// Work item = (K split s, row tile t, panel p of 128 columns of Y), id = (s * m_tiles + t) * panels + p: the
// blocks running at one time read the same chunks of Y (L2 hits), and the panels of a tile share
// its blocks of X in L2 instead of reading them from HBM once per panel.  With one split an item's
// result goes to C; else to partial[s][p][tile rows][pn], and k_block_reduce adds the splits in index order.
//
// TMEM columns: two hi*hi accumulators and the one of the cross terms, buf_cols each.
#pragma once
#include <cuda_fp16.h>

#include <type_traits>

#include "kernels_tc.cuh"

namespace dnpeff {

constexpr int kBlkStages = 5;      // most runs in flight: 32 KB of X and 256 r bytes of Y each, 3 of them at r = 128
constexpr int kBlkThreads = (8 + 3) * 32;

// Element (row, k) of an fp16 operand of 64 K-values.
__host__ __device__ __forceinline__ int blk_canon(int row, int k) {
    return ((row >> 3) * 8 + (k >> 3)) * 64 + (row & 7) * 8 + (k & 7);
}
constexpr int kBlkHalf = 128 * kBlkKC;     // fp16 values of either half of a block of X
constexpr int kBlkHalves = 2 * kBlkHalf;

// D fp32, A and B fp16, both K-major, M x N.
__device__ __forceinline__ uint32_t tc_idesc_f16(int M, int N) {
    return (1u << 4) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}
__device__ __forceinline__ void tc_mma_f16(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void bulk_copy(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}

// The power of two that brings a row's or column's largest magnitude (its bits; 0: nothing stored) into
// [2^14, 2^15), and its reciprocal.  Held to [2^-114, 2^113], so that both, and 2^11 times the first, are normal.
__device__ __forceinline__ float blk_scale(uint32_t max_bits) {
    const uint32_t e = (max_bits >> 23) & 255u;
    return __uint_as_float((e < 28u ? 240u : 268u - e) << 23);
}
__device__ __forceinline__ float blk_unscale(uint32_t max_bits) {
    const uint32_t e = (max_bits >> 23) & 255u;
    return __uint_as_float((e < 28u ? 14u : e - 14u) << 23);
}
constexpr float kBlkLoScale = 2048.f;  // of the lo halves

// Marks in the sign bit of a maximum's word: the row (column) holds values other than zero that are below
// kBlkFaint once they are scaled.
constexpr uint32_t kBlkMark = 0x80000000u;
constexpr float kBlkFaint = 1.f / 4096.f;

// v, a product of scaled operands, with both scalings taken out: the smaller factor first, since v is at
// least 1 or of no consequence (below) and neither step then leaves the range of fp32 unless the result does.
__device__ __forceinline__ float blk_unscaled(float v, uint32_t row_word, uint32_t col_word) {
    const float a = blk_unscale(row_word), b = blk_unscale(col_word);
    return v * fminf(a, b) * fmaxf(a, b);
}
// Whether v, a scaled sum, may be off by more than 2^-23 of itself for what the halves do not hold.  A faint
// value of Y is off by 2^-36 at most, one of X by 2^-35 (k_block_split) and meets 2^15 at most:
// 2^-36 * sum |x| + 2^-35 * 2^15 * (faint values of the row) in all, that is 2^-36 times `row_sum`, which
// k_block_split and k_block_layout add up as sum |x| + 2^16 * (faint values).
constexpr unsigned long long kBlkFaintWeight = 65536;
__device__ __forceinline__ bool blk_faint(float v, uint32_t row_word, uint32_t col_word, float row_sum) {
    return ((row_word | col_word) & kBlkMark) && fabsf(v) < row_sum * (1.f / 8192.f);
}
// Two values times s as fp16 pairs: hi, and lo (s2 = s * 2^11).
__device__ __forceinline__ void blk_split2(float x, float y, float s, float s2, uint32_t& hi, uint32_t& lo) {
    const __half2 h = __floats2half2_rn(x * s, y * s);
    const float2 f = __half22float2(h);
    const __half2 l = __floats2half2_rn(fmaf(f.x, -kBlkLoScale, x * s2), fmaf(f.y, -kBlkLoScale, y * s2));
    hi = *(const uint32_t*)&h;
    lo = *(const uint32_t*)&l;
}
__device__ __forceinline__ void blk_split8(const float (&v)[8], uint32_t max_bits, uint4& hi, uint4& lo) {
    const float s = blk_scale(max_bits), s2 = s * kBlkLoScale;
    blk_split2(v[0], v[1], s, s2, hi.x, lo.x);
    blk_split2(v[2], v[3], s, s2, hi.y, lo.y);
    blk_split2(v[4], v[5], s, s2, hi.z, lo.z);
    blk_split2(v[6], v[7], s, s2, hi.w, lo.w);
}

// How many of eight values are faint under the scale s.
__device__ __forceinline__ uint32_t blk_count_faint(const float (&v)[8], float s) {
    uint32_t n = 0;
#pragma unroll
    for (int t = 0; t < 8; t++) n += v[t] != 0.f && fabsf(v[t] * s) < kBlkFaint ? 1u : 0u;
    return n;
}

// Whether any of them is, under the scale of the maximum's word: the smallest magnitude other than zero (2 * bits - 1
// drops the sign and makes zero the largest) against the power of two that the scale takes to kBlkFaint.
__device__ __forceinline__ bool blk_any_faint(const float (&v)[8], uint32_t word) {
    uint32_t least = 0xffffffffu;
#pragma unroll
    for (int t = 0; t < 8; t++) least = min(least, 2u * __float_as_uint(v[t]) - 1u);
    return least < 2u * __float_as_uint(kBlkFaint * blk_unscale(word)) - 1u;
}

// The smallest lo half for values other than zero that both halves would lose.
__device__ __forceinline__ uint32_t blk_lost2(float x, float y, uint32_t hi, uint32_t lo) {
    const uint32_t some = hi | lo;
    return (x != 0.f && !(some & 0x7fffu) ? 1u : 0u) | (y != 0.f && !(some & 0x7fff0000u) ? 0x10000u : 0u);
}

// ymax[c] = bits of the largest magnitude in column c of Y (K rows, r columns); zero before.
__global__ void __launch_bounds__(256)
k_col_max(const float* __restrict__ Y, int64_t K, int r, uint32_t* __restrict__ ymax) {
    __shared__ uint32_t best[512];
    for (int c = threadIdx.x; c < r; c += 256) best[c] = 0u;
    __syncthreads();
    grid_wait();
    const int quads = r >> 2, per = 256 / quads, q = threadIdx.x % quads, g = threadIdx.x / quads;
    if (g < per) {
        uint32_t m[4] = {0u, 0u, 0u, 0u};
        const int64_t step = (int64_t)gridDim.x * per;
        auto take = [&](const float4& v) {
            m[0] = max(m[0], __float_as_uint(v.x) & 0x7fffffffu);
            m[1] = max(m[1], __float_as_uint(v.y) & 0x7fffffffu);
            m[2] = max(m[2], __float_as_uint(v.z) & 0x7fffffffu);
            m[3] = max(m[3], __float_as_uint(v.w) & 0x7fffffffu);
        };
        const float4* Y4 = (const float4*)Y + q;
        int64_t k = (int64_t)blockIdx.x * per + g;
        for (; k + 3 * step < K; k += 4 * step) {  // four loads in flight
            const float4 a = Y4[k * quads], b = Y4[(k + step) * quads], c = Y4[(k + 2 * step) * quads],
                         d = Y4[(k + 3 * step) * quads];
            take(a); take(b); take(c); take(d);
        }
        for (; k < K; k += step) take(Y4[k * quads]);
#pragma unroll
        for (int j = 0; j < 4; j++)
            if (m[j]) atomicMax(&best[4 * q + j], m[j]);
    }
    __syncthreads();
    for (int c = threadIdx.x; c < r; c += 256)
        if (best[c]) atomicMax(&ymax[c], best[c]);
}

// Y (K rows, r columns) in panels of pn columns -> per panel and chunk of 64 K-values
// [hi pn*64 | lo pn*64] fp16 in core matrices of 8 columns x 8 K-values; rows K..64*k_chunks are zero.
// One thread per (panel, K octet, column).  Marks columns with faint values.  Clears `clear` (r words) for the next product.
__global__ void k_split_y(const float* __restrict__ Y, int64_t K, int r, int pn, int64_t k_chunks, uint32_t* ymax,
                          uint32_t* __restrict__ clear, __half* __restrict__ Ysplit) {
    const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    grid_wait();
    if (idx < r) clear[idx] = 0u;
    if (idx >= k_chunks * 8 * r) return;
    const int col = (int)(idx % r), panel = col / pn, n = col - panel * pn;
    const int64_t ko = idx / r;  // octet of K values
    float v[8];
#pragma unroll
    for (int j = 0; j < 8; j++) v[j] = ko * 8 + j < K ? Y[(ko * 8 + j) * r + col] : 0.f;
    uint4 hi, lo;
    const uint32_t most = ymax[col];
    blk_split8(v, most, hi, lo);
    if (blk_any_faint(v, most) && !(__ldcg(ymax + col) & kBlkMark)) atomicOr(ymax + col, kBlkMark);
    const int64_t c = ko / 8;
    __half* base = Ysplit + (panel * k_chunks + c) * (2 * 64) * pn + blk_canon(n, (int)(ko % 8) * 8);
    *(uint4*)base = hi;
    *(uint4*)(base + 64 * pn) = lo;
}

__device__ __forceinline__ float4 blk_unscaled4(const float4& v, uint32_t row_word, const uint4& m) {
    return make_float4(blk_unscaled(v.x, row_word, m.x), blk_unscaled(v.y, row_word, m.y), blk_unscaled(v.z, row_word, m.z),
                       blk_unscaled(v.w, row_word, m.w));
}
// Whether one of four sums at `at` wants computing again.
__device__ __forceinline__ bool blk_again(const float4& v, uint32_t row_word, const uint4& m,
                                          const unsigned long long* __restrict__ sum, const float* __restrict__ keep, int64_t at) {
    if (!((row_word | m.x | m.y | m.z | m.w) & kBlkMark)) return false;
    const float row_sum = (float)__ldg(sum);
    const bool a = blk_faint(v.x, row_word, m.x, row_sum), b = blk_faint(v.y, row_word, m.y, row_sum),
               c = blk_faint(v.z, row_word, m.z, row_sum), d = blk_faint(v.w, row_word, m.w, row_sum);
    if (!(a || b || c || d)) return false;
    if (!keep) return true;
    const float4 k = *(const float4*)(keep + at);
    return (a && k.x != 0.f) || (b && k.y != 0.f) || (c && k.z != 0.f) || (d && k.w != 0.f);
}

// What the last step of a product needs beside its sums: the operands' scaling, and where rows that want
// computing again are noted.  keep (or null): the factor whose numerators C holds, of C's shape; where it is
// zero, so is its update whatever the numerator.
struct BlkFinish {
    const uint32_t* row_max;
    const uint32_t* col_max;
    const unsigned long long* row_sum;
    const float* keep;
    unsigned char* again;  // one byte per row of C (k_block_tc alone notes them)
};

// r: columns of a panel.  direct: C, with row stride ldc -- or null, and `fin` is not used.
__global__ void __launch_bounds__(kBlkThreads, 1)
k_block_tc(const __half* __restrict__ X, int64_t m_tiles, int64_t k_chunks, const __half* __restrict__ Ysplit, int r,
           int panels, int n_split, int64_t chunks_per_split, int stages, float* __restrict__ partial, uint32_t buf_cols,
           float* __restrict__ direct, int64_t rows, int ldc, const BlkFinish fin, uint32_t wait_limit, int* __restrict__ err) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t full[kBlkStages], free_[kBlkStages];
    __shared__ __align__(8) uint64_t acc_done[2], acc_free[2];
    __shared__ __align__(8) uint64_t cross_done, cross_free, drained[2];
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_flag;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    constexpr uint32_t kXBytes = kBlkHalves * 2u;
    const uint32_t y_bytes = (uint32_t)r * kBlkKC * 4u;
    const uint32_t stage_bytes = kXBytes + y_bytes;
    const uint32_t tmem_cols = tc_tmem_pow2(3 * buf_cols);
    volatile int* abort = &abort_flag;

    if (w == 0) tc_alloc(&tmem_slot, tmem_cols);
    if (tid == 32) {
        for (int i = 0; i < stages; i++) {
            mbar_init(&full[i], 1);
            mbar_init(&free_[i], 2);  // both issuers
        }
        for (int i = 0; i < 2; i++) {
            mbar_init(&acc_done[i], 1);
            mbar_init(&acc_free[i], 8);
            mbar_init(&drained[i], 1);
        }
        mbar_init(&cross_done, 1);
        mbar_init(&cross_free, 8);
        abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    grid_wait();
    const uint32_t tmem = tmem_slot;
    const uint32_t tmem_cross = tmem + 2 * buf_cols;

    BlkCursor cur;
    cur.n_items = m_tiles * n_split * panels;
    cur.m_tiles = m_tiles;
    cur.panels = panels;
    cur.k_chunks = k_chunks;
    cur.chunks_per_split = chunks_per_split;
    cur.stride = (int)gridDim.x;
    cur.open(blockIdx.x);

    if (w < 8) {
        // ---- drainers
        const int q = w & 3, ch = w >> 2;
        const int xrow = q * 32 + lane;
        const uint32_t lane_base = (uint32_t)(q * 32) << 16;
        float acc[64];
#pragma unroll
        for (int j = 0; j < 64; j++) acc[j] = 0.f;
        uint32_t items = 0;
        for (uint32_t it = 0; cur.valid(); cur.next(), it++) {
            if (!warp_wait_or_abort(&acc_done[it & 1u], (it >> 1) & 1u, abort, lane, wait_limit)) break;
            tc_fence_after();
            const uint32_t src = tmem + (it & 1u) * buf_cols + lane_base + (uint32_t)(ch * 64);
#pragma unroll
            for (int g = 0; g < 2; g++) {
                if (ch * 64 + g * 32 < r) {  // uniform per warp
                    float v[32];
                    tc_ld32(src + 32u * g, v);
                    tc_ld_wait();
#pragma unroll
                    for (int j = 0; j < 32; j++) acc[g * 32 + j] += v[j];
                }
            }
            tc_fence_before();
            if (lane == 0) mbar_arrive(&acc_free[it & 1u]);
            if (cur.last_of_item()) {
                if (!warp_wait_or_abort(&cross_done, items & 1u, abort, lane, wait_limit)) break;
                items++;
                tc_fence_after();
                const int64_t row = cur.tile * 128 + xrow;
                const int col0 = cur.panel * r + ch * 64;
                const bool store = !direct || row < rows;
                uint32_t row_word = 0u;
                bool again = false;
                if (direct && store) row_word = __ldg(fin.row_max + row);
                float* dst = direct ? direct + row * ldc + col0
                                    : partial + (((cur.split * panels + cur.panel) * m_tiles + cur.tile) * 128 + xrow) * (int64_t)r + ch * 64;
#pragma unroll
                for (int g = 0; g < 4; g++) {
                    if (ch * 64 + g * 16 < r) {
                        float v[16];
                        tc_ld16(tmem_cross + lane_base + (uint32_t)(ch * 64 + 16 * g), v);
                        tc_ld_wait();
#pragma unroll
                        for (int j = 0; j < 16; j++) v[j] = fmaf(v[j], 1.f / kBlkLoScale, acc[g * 16 + j]);
#pragma unroll
                        for (int j = 0; j < 16; j += 4) {
                            float4 x = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
                            if (direct) {
                                const int col = col0 + g * 16 + j;
                                const uint4 m = __ldg((const uint4*)(fin.col_max + col));
                                again = again || (store && blk_again(x, row_word, m, fin.row_sum + row, fin.keep, row * ldc + col));
                                x = blk_unscaled4(x, row_word, m);
                            }
                            if (store) *(float4*)(dst + g * 16 + j) = x;
                        }
                    }
                }
                if (again) fin.again[row] = 1;
                tc_fence_before();
                if (lane == 0) mbar_arrive(&cross_free);
#pragma unroll
                for (int j = 0; j < 64; j++) acc[j] = 0.f;
            }
        }
    } else if (w < 10) {
        // ---- MMA issuers: warp 8 hi*hi, warp 9 the cross terms
        auto issue = [&](auto cross_tag) {
            constexpr bool cross = decltype(cross_tag)::value;
            const uint32_t idesc = tc_idesc_f16(128, r);
            // stage 0, hi halves, K-step 0; the others differ in the start-address field only
            // (16-byte units; a K-step is two core matrices)
            const uint32_t smem0 = smem_u32(smem_raw);
            const uint64_t descx = tc_smem_desc(smem0, 128, 128u * (kBlkKC / 8));
            const uint64_t descy = tc_smem_desc(smem0 + kXBytes, 128, 128u * (kBlkKC / 8));
            const uint32_t stage_u = stage_bytes >> 4, half_y = y_bytes >> 5;
            constexpr uint32_t half_x = kXBytes >> 5;
            uint32_t items = 0, sx = 0, ring = 0;
            for (uint32_t it = 0; cur.valid(); cur.next(), it++) {
                const uint32_t e = it & 1u;
                const bool first = cur.first_of_item(), last = cur.last_of_item();
                if (!cross && it >= 2 && !mbar_wait_or_abort<true>(&acc_free[e], ((it >> 1) & 1u) ^ 1u, abort, wait_limit)) break;
                if (cross && first && items > 0 && !mbar_wait_or_abort<true>(&cross_free, (items - 1u) & 1u, abort, wait_limit)) break;
                if (!mbar_wait_or_abort<true>(&full[sx], ring, abort, wait_limit)) break;
                tc_fence_after();
                const uint64_t dx = descx + sx * stage_u, dy = descy + sx * stage_u;
#pragma unroll
                for (int ks = 0; ks < 4; ks++) {
                    const uint64_t ah = dx + 16u * ks, al = ah + half_x, bh = dy + 16u * ks, bl = bh + half_y;
                    if (cross) {
                        tc_mma_f16(tmem_cross, al, bh, idesc, ks == 0 && first ? 0u : 1u);
                        tc_mma_f16(tmem_cross, ah, bl, idesc, 1u);
                    } else {
                        tc_mma_f16(tmem + e * buf_cols, ah, bh, idesc, ks == 0 ? 0u : 1u);
                    }
                }
                if (!cross) tc_commit(&acc_done[e]);
                if (cross && last) {
                    tc_commit(&cross_done);
                    items++;
                }
                tc_commit(&free_[sx]);
                if (++sx == (uint32_t)stages) {
                    sx = 0;
                    ring ^= 1u;
                }
            }
            // Nothing this thread issued may still be running when the block frees its
            // TMEM and shared memory (waited for with the full limit).
            tc_commit(&drained[cross ? 1 : 0]);
            if (!mbar_wait(&drained[cross ? 1 : 0], 0u)) *abort = 1;
        };
        if (tc_elect()) {
            if (w == 8) issue(std::false_type());
            else issue(std::true_type());
        }
    } else if (lane == 0) {
        // ---- bulk copies: a block of X and a chunk of Y per run
        uint32_t j = 0, sx = 0, ring = 0;  // runs whose copies were issued; their stage, and how often it was used
        for (; cur.valid(); cur.next(), j++) {
            if (ring > 0 && !mbar_wait_or_abort<false>(&free_[sx], (ring - 1u) & 1u, abort, wait_limit)) break;
            unsigned char* dst = smem_raw + (size_t)sx * stage_bytes;
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(&full[sx])),
                         "r"(stage_bytes)
                         : "memory");
            bulk_copy(dst, X + (cur.tile * k_chunks + cur.c) * kBlkHalves, kXBytes, &full[sx]);
            bulk_copy(dst + kXBytes, Ysplit + (cur.panel * k_chunks + cur.c) * (int64_t)(2 * kBlkKC) * r, y_bytes, &full[sx]);
            if (++sx == (uint32_t)stages) {
                sx = 0;
                ring++;
            }
        }
        if (*abort) {
            // gave up: let the copies already issued land before the shared memory
            // is released (bounded waits; the parity of a stage's latest copy)
            for (uint32_t k = (j > (uint32_t)stages ? j - stages : 0); k < j; k++)
                mbar_wait(&full[k % stages], (k / stages) & 1u);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (tid == 0 && abort_flag) atomicOr(err, kErrTcTimeout);
    if (w == 0) tc_dealloc(tmem, tmem_cols);
}

// The popular block of A written in fp32 where its blocks of X1 will lie, row-major inside a block
// (zeroed before; k_block_split turns it into X1 proper).  One warp per row; hot_len[row * stride] =
// entries of the row that lie in popular columns (they come first in the bucketed
// row, with internal column ids < n_hot).  xmax[row]: bits of its largest magnitude;
// colmax[column] (zeroed before): of the column's, over all calls.
__global__ void k_fill_blocks(const float* __restrict__ vals, const int32_t* __restrict__ col,
                              const int64_t* __restrict__ rowptr, const uint32_t* __restrict__ hot_len,
                              int stride, int64_t row_begin, int64_t n_rows, int64_t chunks1,
                              float* __restrict__ X1, uint32_t* __restrict__ xmax, uint32_t* colmax) {
    const int lane = threadIdx.x & 31;
    const int64_t warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t i = row_begin + (((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5); i < n_rows; i += warps) {
        const int64_t beg = rowptr[i], end = beg + hot_len[i * stride];
        float* const x = X1 + (i >> 7) * chunks1 * kBlkHalf + (i & 127) * kBlkKC;
        uint32_t most = 0u;
        for (int64_t p = beg + lane; p < end; p += 32) {
            const int j = col[p];
            const float v = vals[p];
            const uint32_t b = __float_as_uint(v) & 0x7fffffffu;
            most = max(most, b);
            // few entries are the largest so far of their column (a stale value only asks once too often)
            if (__ldca(colmax + j) < b) atomicMax(colmax + j, b);
            x[(int64_t)(j / kBlkKC) * kBlkHalf + j % kBlkKC] = v;
        }
        most = __reduce_max_sync(0xffffffffu, most);
        if (lane == 0) xmax[i] = most;
    }
}

// A block of X1 from fp32 into its halves, in place, and its transpose into X2.  Block (it, c1) of the
// grid takes rows 128 it.. and columns 64 c1.. through shared memory; blocks past the last chunk of X1 write
// the zeros that pad X2's last tile (X2 needs no clearing).  max1, max2: largest magnitudes of the rows of
// either, marked here; sum1, sum2 (zero before): their row_sum (blk_faint), in whole numbers, so that the
// order of the additions does not matter.  Reads 4 bytes and writes 8 per element.  256 threads; 8
// consecutive ones write a core matrix.
// A value that both halves in X2 would lose is left there as their smallest, 2^-35: blk_repair_row
// has to see that there is one, and looks it up.
__global__ void __launch_bounds__(256)
k_block_split(__half* __restrict__ X1, uint32_t* max1, unsigned long long* sum1, int64_t chunks1, __half* __restrict__ X2,
              uint32_t* max2, unsigned long long* sum2, int64_t chunks2) {
    __shared__ float sq[128][kBlkKC + 1];
    __shared__ uint32_t part1[2][128], part2[4][kBlkKC];  // of the sums, by octets that one warp holds
    const int64_t it = blockIdx.x, c1 = blockIdx.y;
    const int lane = threadIdx.x & 31;
    __half* const x1 = X1 + (it * chunks1 + c1) * kBlkHalves;
    const bool stored = c1 < chunks1;
#pragma unroll
    for (int e = threadIdx.x; e < 128 * (kBlkKC / 4); e += 256) {
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (stored) v = ((const float4*)x1)[e];
        float* d = &sq[e / (kBlkKC / 4)][4 * (e % (kBlkKC / 4))];
        d[0] = v.x; d[1] = v.y; d[2] = v.z; d[3] = v.w;
    }
    __syncthreads();
    // of the eight values of a lane and of the lanes 8, 16 and 24 further on
    auto sum_of_octets = [&](const float (&v)[8], uint32_t word) {
        const float s = blk_scale(word);
        float sum = 0.f;
#pragma unroll
        for (int t = 0; t < 8; t++) sum += fabsf(v[t] * s);
        // 24 bits of sum (32 values below 2^15, rounded up by octets), then the faint ones
        uint32_t q = min(__float2uint_ru(sum), 8u << 15) + (blk_count_faint(v, s) << 24);
        q += __shfl_xor_sync(0xffffffffu, q, 8);
        return q + __shfl_xor_sync(0xffffffffu, q, 16);
    };
    if (stored) {
#pragma unroll
        for (int e = threadIdx.x; e < 128 * 8; e += 256) {  // (row, octet of columns)
            const int row = (e >> 6) * 8 + (e & 7), ko = (e >> 3) & 7;
            float v[8];
#pragma unroll
            for (int t = 0; t < 8; t++) v[t] = sq[row][8 * ko + t];
            uint4 hi, lo;
            const uint32_t word = __ldcg(max1 + it * 128 + row);
            blk_split8(v, word, hi, lo);
            *(uint4*)(x1 + blk_canon(row, 8 * ko)) = hi;
            *(uint4*)(x1 + kBlkHalf + blk_canon(row, 8 * ko)) = lo;
            const uint32_t q = sum_of_octets(v, word);
            if (lane < 8) part1[ko >> 2][row] = q;
        }
    }
#pragma unroll
    for (int e = threadIdx.x; e < 64 * 16; e += 256) {  // (column, octet of rows)
        const int ko = (e >> 3) & 7, io = ko + 8 * (e >> 9), j = ((e >> 6) & 7) * 8 + (e & 7);
        const int64_t c2 = 2 * it + (io >> 3);
        float v[8];
#pragma unroll
        for (int t = 0; t < 8; t++) v[t] = sq[8 * io + t][j];
        const int row2 = (int)(c1 & 1) * 64 + j;
        const uint32_t word = __ldcg(max2 + (c1 >> 1) * 128 + row2);
        const uint32_t q = sum_of_octets(v, word);
        if (lane < 8) part2[io >> 2][j] = q;
        if (c2 >= chunks2) continue;
        uint4 hi, lo;
        blk_split8(v, word, hi, lo);
        lo.x |= blk_lost2(v[0], v[1], hi.x, lo.x);
        lo.y |= blk_lost2(v[2], v[3], hi.y, lo.y);
        lo.z |= blk_lost2(v[4], v[5], hi.z, lo.z);
        lo.w |= blk_lost2(v[6], v[7], hi.w, lo.w);
        __half* const x2 = X2 + ((c1 >> 1) * chunks2 + c2) * kBlkHalves + blk_canon(row2, 8 * ko);
        *(uint4*)x2 = hi;
        *(uint4*)(x2 + kBlkHalf) = lo;
    }
    __syncthreads();
    if (!stored) return;
    const int t = threadIdx.x;
    if (t < 128 + kBlkKC) {
        const bool row = t < 128;
        const int j = t - 128;
        const int64_t at = row ? it * 128 + t : c1 * kBlkKC + j;
        const uint32_t parts[4] = {row ? part1[0][t] : part2[0][j], row ? part1[1][t] : part2[1][j], row ? 0u : part2[2][j],
                                   row ? 0u : part2[3][j]};
        unsigned long long q = 0;
        bool faint = false;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            q += (parts[k] & 0xffffffu) + (parts[k] >> 24) * kBlkFaintWeight;
            faint = faint || (parts[k] >> 24);
        }
        if (q) atomicAdd((row ? sum1 : sum2) + at, q);
        if (faint && !(__ldcg((row ? max1 : max2) + at) & kBlkMark)) atomicOr((row ? max1 : max2) + at, kBlkMark);
    }
}

// A row-major dense X (M x K) split into the blocked layout of k_block_tc (zero
// padding included): one warp per row of the blocked matrix.  xmax, xsum: as k_block_split leaves them.
__global__ void k_block_layout(const float* __restrict__ X, int64_t M, int64_t K, int64_t m_tiles, int64_t k_chunks,
                               __half* __restrict__ Xb, uint32_t* __restrict__ xmax, unsigned long long* __restrict__ xsum) {
    const int lane = threadIdx.x & 31;
    const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (i >= m_tiles * 128) return;
    uint32_t most = 0u;
    for (int64_t k = lane; i < M && k < K; k += 32) most = max(most, __float_as_uint(X[i * K + k]) & 0x7fffffffu);
    most = __reduce_max_sync(0xffffffffu, most);
    __half* const x = Xb + (i >> 7) * k_chunks * kBlkHalves;
    const float s = blk_scale(most);
    unsigned long long sum = 0, faint = 0;
    for (int64_t ko = lane; ko < k_chunks * 8; ko += 32) {
        float v[8], octet = 0.f;
#pragma unroll
        for (int t = 0; t < 8; t++) {
            v[t] = i < M && ko * 8 + t < K ? X[i * K + ko * 8 + t] : 0.f;
            octet += fabsf(v[t] * s);
        }
        sum += __float2uint_ru(octet);
        faint += blk_count_faint(v, s);
        uint4 hi, lo;
        blk_split8(v, most, hi, lo);
        __half* const d = x + (ko >> 3) * kBlkHalves + blk_canon((int)(i & 127), (int)(ko & 7) * 8);
        *(uint4*)d = hi;
        *(uint4*)(d + kBlkHalf) = lo;
    }
    sum += faint * kBlkFaintWeight;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        sum += __shfl_xor_sync(0xffffffffu, sum, o);
        faint += __shfl_xor_sync(0xffffffffu, faint, o);
    }
    if (lane == 0) {
        xmax[i] = most | (faint ? kBlkMark : 0u);
        xsum[i] = sum;
    }
}

// Where the values of X are kept as they are: as a row-major matrix, or as the stored entries of the
// popular columns in the rows of A, that is the rows of X or (`columns`) its columns.
struct BlkValues {
    const float* dense;        // K values per row of X, or null:
    const float* vals;
    const int32_t* col;        // internal column ids
    const int64_t* rowptr;
    const uint32_t* hot_len;   // entries of a row of A in popular columns (they come first), every `stride` words
    int stride;
    bool columns;
};

// What computing a row of C = X * Y again takes: X's blocks with the words of its rows, its values, Y, and C (M x r).
struct BlkRepair {
    const __half* X;
    const uint32_t* xmax;
    int64_t k_chunks;
    BlkValues values;
    const float* Y;
    int64_t M, K;
    int r;
    float* C;
};
constexpr int kRepairThreads = 256, kRepairBatch = 8;
struct BlkRepairSums {
    double of[512];  // (one set that the warps add to in turn: 32 KB for a set each would be the space that the gathers' L1 has)
};

// Row i of C by a block of kRepairThreads, from the values of X as they are, products and sums in double: what the
// halves lose of faint values is in this row too much (blk_faint).  There is hardly ever one.  Where there
// are many it is bound by latency: every popular column of 20000 x 4194304 at rank 128 computed again
// takes 75 to 85 ms, the sparse product of the same entries 12; entries that are this small last a few updates only.
// With `columns` the stored entries of a row of X are found through its halves, and the faint ones among them in
// the row of A.
__device__ __forceinline__ void blk_repair_row(const BlkRepair& a, int64_t i, BlkRepairSums& sums) {
    constexpr int kWarps = kRepairThreads / 32;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, quads = a.r >> 2;
    double acc[4][4];
#pragma unroll
    for (int q = 0; q < 4; q++)
#pragma unroll
        for (int t = 0; t < 4; t++) acc[q][t] = 0.0;
    int64_t beg = 0, end = a.K;
    if (!a.values.dense && !a.values.columns) {
        beg = a.values.rowptr[i];
        end = beg + a.values.hot_len[i * a.values.stride];
    }
    const float back = blk_unscale(a.xmax[i]);
    for (int64_t p0 = beg + w * 32; p0 < end; p0 += kRepairThreads) {
        const int64_t p = p0 + lane;
        int64_t k = p;
        float v = 0.f;
        if (p < end) {
            if (a.values.dense) {
                v = a.values.dense[i * a.K + p];
            } else if (!a.values.columns) {
                k = a.values.col[p];
                v = a.values.vals[p];
            } else {
                const __half* x = a.X + ((i >> 7) * a.k_chunks + (p >> 6)) * kBlkHalves + blk_canon((int)(i & 127), (int)(p & 63));
                v = fmaf(__half2float(x[kBlkHalf]), 1.f / kBlkLoScale, __half2float(x[0]));
            }
        }
        if (!a.values.dense && a.values.columns) {
            uint32_t ask = __ballot_sync(0xffffffffu, v != 0.f && fabsf(v) < kBlkFaint);
            v *= back;
            while (ask) {
                const int src = __ffs(ask) - 1;
                ask &= ask - 1;
                const int64_t row = __shfl_sync(0xffffffffu, k, src), first = a.values.rowptr[row];
                const int64_t last = first + a.values.hot_len[row * a.values.stride];
                for (int64_t q = first; q < last; q += 32 * kRepairBatch) {
                    int found = -1;
#pragma unroll
                    for (int b = 0; b < kRepairBatch; b++) {
                        const int64_t at = q + 32 * b + lane;
                        if (at < last && a.values.col[at] == i) found = b;
                    }
                    const uint32_t hit = __ballot_sync(0xffffffffu, found >= 0);
                    if (!hit) continue;
                    const int by = __ffs(hit) - 1;
                    const int b = __shfl_sync(0xffffffffu, found, by);
                    if (lane == src) v = a.values.vals[q + 32 * b + by];
                    break;
                }
            }
        }
        uint32_t live = __ballot_sync(0xffffffffu, v != 0.f);
        while (live) {
            double x[kRepairBatch];  // that many entries at a time, so that their rows of Y are on the way together
            int64_t at[kRepairBatch];
            int m = 0;
#pragma unroll
            for (int b = 0; b < kRepairBatch; b++) {
                const int src = live ? __ffs(live) - 1 : 0;
                x[b] = (double)__shfl_sync(0xffffffffu, v, src);
                at[b] = __shfl_sync(0xffffffffu, k, src) * quads;
                m += live ? 1 : 0;
                live &= live - 1;
            }
#pragma unroll
            for (int q = 0; q < 4; q++) {
                if (32 * q >= quads) continue;
                const int c = lane + 32 * q;
                float4 f[kRepairBatch];
#pragma unroll
                for (int b = 0; b < kRepairBatch; b++) {
                    f[b] = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (b < m && c < quads) f[b] = __ldg((const float4*)a.Y + at[b] + c);
                }
#pragma unroll
                for (int b = 0; b < kRepairBatch; b++) {
                    if (b >= m) continue;
                    acc[q][0] = fma(x[b], (double)f[b].x, acc[q][0]);
                    acc[q][1] = fma(x[b], (double)f[b].y, acc[q][1]);
                    acc[q][2] = fma(x[b], (double)f[b].z, acc[q][2]);
                    acc[q][3] = fma(x[b], (double)f[b].w, acc[q][3]);
                }
            }
        }
    }
    for (int turn = 0; turn < kWarps; turn++) {
        if (w == turn) {
#pragma unroll
            for (int q = 0; q < 4; q++)
                if (lane + 32 * q < quads)
#pragma unroll
                    for (int t = 0; t < 4; t++) {
                        double* const s = sums.of + 4 * (lane + 32 * q) + t;
                        *s = turn == 0 ? acc[q][t] : *s + acc[q][t];
                    }
        }
        __syncthreads();
    }
    for (int c = tid; c < a.r; c += kRepairThreads) a.C[i * a.r + c] = (float)sums.of[c];
    __syncthreads();
}

// The rows whose byte in `again` is set (it is cleared); the launch costs a product 3.5 us (3001 x 100003, rank 50),
// so that products of several splits leave it to k_block_reduce.
__global__ void __launch_bounds__(kRepairThreads, 2) k_block_repair(const BlkRepair a, unsigned char* __restrict__ again) {
    constexpr int kWarps = kRepairThreads / 32;
    __shared__ int64_t list[kRepairThreads];
    __shared__ int listed;
    __shared__ BlkRepairSums sums;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    grid_wait();
    // 32 consecutive rows per warp and round
    for (int64_t g0 = (int64_t)blockIdx.x * kWarps; g0 * 32 < a.M; g0 += (int64_t)gridDim.x * kWarps) {
        if (tid == 0) listed = 0;
        __syncthreads();
        const int64_t mine = (g0 + w) * 32 + lane;
        if (mine < a.M && again[mine]) {
            again[mine] = 0;
            list[atomicAdd(&listed, 1)] = mine;  // (in any order: the rows do not depend on one another)
        }
        __syncthreads();
        const int n = listed;
        for (int l = 0; l < n; l++) blk_repair_row(a, list[l], sums);
        __syncthreads();  // (the list is read before it is started anew)
    }
}

// C[i][:] (r / 4 float4 each) = sum over splits s (in index order) of partial[s][panel][i][:],
// with the operands' scaling taken out.  A block takes whole rows, 256 / (r / 4) of them, and computes those again that want it.
__global__ void __launch_bounds__(kRepairThreads, 4)
k_block_reduce(const float* __restrict__ partial, int n_split, int64_t rows_pad, int pn4, const BlkFinish fin, const BlkRepair a) {
    __shared__ BlkRepairSums sums;
    __shared__ bool again[32];
    const int r4 = a.r >> 2, mine = threadIdx.x / r4, c = threadIdx.x - mine * r4, per = kRepairThreads / r4;
    const int64_t first = (int64_t)blockIdx.x * per, i = first + mine;
    if (threadIdx.x < 32) again[threadIdx.x] = false;
    grid_wait();
    bool want = false;
    float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
    const bool real = mine < per && i < a.M;
    if (real) {
        const int panel = c / pn4;
        const float4* p = (const float4*)partial + (panel * rows_pad + i) * pn4 + (c - panel * pn4);
        const uint32_t row_word = __ldg(fin.row_max + i);
        const uint4 m = __ldg((const uint4*)fin.col_max + c);
        t = p[0];
        for (int s = 1; s < n_split; s++) {
            const float4 b = p[(int64_t)s * rows_pad * r4];
            t.x += b.x; t.y += b.y; t.z += b.z; t.w += b.w;
        }
        want = blk_again(t, row_word, m, fin.row_sum + i, fin.keep, 4 * (i * r4 + c));
        ((float4*)a.C)[i * r4 + c] = blk_unscaled4(t, row_word, m);
    }
    if (!__syncthreads_or(want)) return;
    if (want) again[mine] = true;
    __syncthreads();
    for (int l = 0; l < per; l++)
        if (again[l]) blk_repair_row(a, first + l, sums);
}

// Ranks up to 128 in one panel; 256, 384 and 512 as panels of 128 columns of Y and C.
inline bool block_tc_ok(int r) {
    return (r >= 32 && r <= kTcMaxN && (r % 32) == 0) || (r > 128 && r <= 512 && (r % 128) == 0);
}
inline int block_tc_panel(int r) { return r <= 128 ? r : 128; }

struct BlockTcPlan {
    int64_t m_tiles, k_chunks, chunks_per_split;
    int n_split, panels;
    size_t x_halves, xmax_words, ysplit_halves, partial_floats;
};

// Row tiles x panels x K splits should fill whole waves of kNumSMs blocks.
inline BlockTcPlan block_tc_plan(int64_t M, int64_t K, int r) {
    BlockTcPlan p;
    p.m_tiles = ceil_div(std::max<int64_t>(M, 1), 128);
    p.k_chunks = ceil_div(std::max<int64_t>(K, 1), kBlkKC);
    p.panels = r / block_tc_panel(r);
    int best = 1;
    double best_eff = 0.0;
    for (int s = 1; s <= 16; s++) {
        if (s > 1 && p.k_chunks / s < 8) break;
        int64_t items = p.m_tiles * p.panels * s;
        double eff = (double)items / (double)(ceil_div(items, kNumSMs) * kNumSMs);
        if (eff > best_eff + 0.02) { best_eff = eff; best = s; }
    }
    p.chunks_per_split = ceil_div(p.k_chunks, best);
    p.n_split = (int)ceil_div(p.k_chunks, p.chunks_per_split);
    p.x_halves = (size_t)p.m_tiles * (size_t)p.k_chunks * kBlkHalves;
    p.xmax_words = (size_t)p.m_tiles * 128;
    p.ysplit_halves = (size_t)p.k_chunks * 2 * kBlkKC * (size_t)r;
    p.partial_floats = p.n_split > 1 ? (size_t)p.n_split * (size_t)p.m_tiles * 128 * (size_t)r : 4;
    return p;
}

// X of a product: its blocks, the words and sums of its rows (BlkFinish), and its values.
struct BlkOperand {
    const __half* blocks;
    const uint32_t* max;
    const unsigned long long* sum;
    BlkValues values;
};

// C (M x r, overwritten) = X * Y.  Y row-major K x r.  keep: as in BlkFinish.  again: M bytes, zero before and after.
// ymax: r words, zero before the call; ymax_next: r words that are zero after it, for the next one.
inline int block_tc_launch(const BlkOperand& X, const BlockTcPlan& p, const float* Y, int64_t M, int64_t K, int r, float* C,
                           const float* keep, unsigned char* again, __half* ysplit, uint32_t* ymax, uint32_t* ymax_next,
                           float* partial, int* err, cudaStream_t st, uint32_t wait_limit = kTiledSpinLimit) {
    if (M <= 0) return DNPEFF_OK;
    const int pn = block_tc_panel(r);
    const size_t stage = (size_t)kBlkHalves * 2 + (size_t)pn * kBlkKC * 4;
    const int stages = (int)std::min<size_t>(kBlkStages, (size_t)220 * 1024 / stage);
    const size_t smem = stages * stage;  // 172 KB or more: one block per SM
    DN_CUDA(cudaFuncSetAttribute(k_block_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    // four rows of Y per thread (one round of loads), or more where two blocks per SM do not cover them
    const int64_t per = 256 / (r / 4);
    DN_TRY(launch_overlapped(k_col_max, dim3((unsigned)std::min<int64_t>(2 * kNumSMs, ceil_div(std::max<int64_t>(K, 1), per * 4))),
                             256, 0, st, Y, K, r, ymax));
    DN_TRY(launch_overlapped(k_split_y, dim3((unsigned)ceil_div(p.k_chunks * 8 * r, 256)), 256, 0, st, Y, K, r, pn, p.k_chunks,
                             ymax, ymax_next, ysplit));
    const BlkFinish fin = {X.max, ymax, X.sum, keep, again};
    const int64_t items = p.m_tiles * p.n_split * p.panels;
    DN_TRY(launch_overlapped(k_block_tc, dim3((unsigned)std::min<int64_t>(items, (int64_t)kNumSMs)), kBlkThreads, smem, st, X.blocks,
                             p.m_tiles, p.k_chunks, ysplit, pn, p.panels, p.n_split, p.chunks_per_split, stages, partial,
                             tc_tmem_cols(pn), p.n_split > 1 ? (float*)nullptr : C, M, r, fin, wait_limit, err));
    const BlkRepair repair = {X.blocks, X.max, p.k_chunks, X.values, Y, M, K, r, C};
    if (p.n_split > 1)
        return launch_overlapped(k_block_reduce, dim3((unsigned)ceil_div(M, kRepairThreads / (r / 4))), kRepairThreads, 0, st, partial,
                                 p.n_split, p.m_tiles * 128, pn / 4, fin, repair);
    return launch_overlapped(k_block_repair, dim3((unsigned)std::min<int64_t>(ceil_div(M, kRepairThreads), 2 * kNumSMs)), kRepairThreads, 0,
                             st, repair, again);
}

}  // namespace dnpeff

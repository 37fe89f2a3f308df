// Small problems: whole stretches of iterations in one launch.
//
// A matrix with a few hundred thousand stored entries needs 10 to 50 us of work per iteration, and
// the kernels of the large path -- fourteen launches per iteration, each with a pipeline of
// copies, tensor-core runs and drains to fill and empty -- take 100 to 150 us for it whatever its
// size.  Here one cooperative launch makes many iterations: a persistent block per SM, everything
// L2-resident, two grid-wide barriers per iteration, one behind each half:
//
//   W *= (A H^T) / (W (H H^T) + eps), and the blocks' partials of W^T W
//   H *= (A^T W) / (H (W^T W) + eps), and the blocks' partials of H H^T
//
// Workers.  A half is cut into contiguous pieces, one per worker (a group of 512 threads; a block holds
// one or two), so that entries to gather and rows to update weigh the same in each (k_small_cuts).  A
// worker gathers the numerators of its rows tile by tile into shared memory and updates the tile right
// there, so numerators never go through L2 and no barrier stands between product and update; where a
// block holds two workers one gathers while the other computes.  Only rows that are a good part of a worker's
// share are cut: the workers behind write their piece of the sum to a carry, and raise a flag that the
// owner of the row waits for.  Few workers take part where there is little work: a barrier, and the
// summing of the partials, cost more with more of them.
//
// The Gram matrix of the factor that is gathered comes as one partial per block of the half before.  Few
// partials are summed by every worker for itself (narrow strides).  Many are summed chunk by chunk, each chunk by one
// worker, before it turns to its product; the result is first needed behind the first tile's product, where
// a counter says that all chunks are there.
//
// Sparse products.  The entries of a tile are cut into equal units, one per lane group (LD / 4 lanes, a
// float4 of the factor row each: with two float4 a lane and rows of 128 bytes every load would touch eight lines for
// four, 1.2 times the time); a unit adds up its entries row by row, in runs of at most kSmallRun.  The sum of a row that starts
// inside the unit goes to the row's place, the sum of one that started earlier to the unit's carry slot,
// and whoever reads a row adds the carries of the units that begin inside it, in order.  So a row of two
// thousand entries and two thousand rows of one entry take the same time, and the result does not depend
// on timing.
//
// Contractions.  Strides 32 and 64: on the CUDA cores, a thread two rows x four columns.  96 and 128: on tcgen05,
// transposed, so that a thread has a column: (X G)^T = G X^T with G in TMEM and the tile's rows as the other
// operand, and X^T X with X^T in TMEM, in tf32 halves and in runs of at most 64 values of K as in kernels_tc.cuh.
//
// Factors change during the launch: they are read with ld.global.cg (L2); the matrix does not and goes
// through L1.  All waits are bounded: a block whose wait runs out sets the error word and an abort flag,
// and all blocks leave.
#pragma once
#include "common.cuh"
#include "kernels_dense.cuh"  // quot_refined
#include "kernels_tc.cuh"     // tcgen05 wrappers

namespace dnpeff {

enum : int { kErrGridTimeout = 32 };

// What a stride takes: the gathers want as many threads as the registers allow (kB gathers of 16 bytes each in flight),
// the wide strides registers for their columns.
template <int LD>
struct SmallShape {
    static constexpr bool kWide = LD > 64;
    static constexpr int kT = 512;                             // threads of a worker
    static constexpr int kWorkers = kWide ? 1 : 2;             // of a block
    static constexpr int kThreads = kT * kWorkers;
    static constexpr int kWarps = kT / 32;
    static constexpr int kQuads = LD / 4;                      // float4 of a factor row
    static constexpr int kLanes = kQuads <= 8 ? 8 : (kQuads <= 16 ? 16 : 32);  // lanes of a unit, a float4 each
    static constexpr int kUnits = kT / kLanes;
    static constexpr int kB = kWide ? 16 : 8;                  // entries of a unit in flight
    static constexpr int kTile = kWide ? 64 : 2 * kT / kQuads; // rows of a tile, at most
    static constexpr int kLdN = LD + 4;                        // row strides in shared memory: numerators,
    static constexpr int kLdX = LD + 4;                        // and X
    static constexpr int kSub = kWide ? 1 : kT / (kQuads * kQuads);  // threads of a square of the Gram matrix on CUDA cores
    static constexpr int kVec = kWide ? 4 : 1;                 // elements per lane of a chunk of G
    static constexpr int kChunks = LD * LD / (32 * kVec);
    // a worker's shared memory, in floats: G, and X (wide: the operand in shared memory, X or X^T in halves) | numerators |
    // carries, the last one of the piece of another worker's row | sums of the Gram matrix (narrow) | row offsets, of either
    // side's first tile and of two more | the rows' carries
    static constexpr int kOffsets = (kTile + 4) / 4 * 4;
    static constexpr int kG = 0, kX = kG + (kWide ? 0 : LD * LD), kN = kX + (kWide ? 2 * kTile * LD : kTile * kLdX),
                         kC = kN + kTile * kLdN, kS = kC + (kUnits + 1) * LD, kP = kS + (kWide ? 0 : LD * LD),
                         kR = kP + 4 * kOffsets, kFloats = kR + kTile;
    static_assert(2 * kWarps * 32 * kVec <= kS - kN, "the chunk sums (doubles) go over numerators and carries");
    // Dynamic shared memory of a block.  A block of the wide strides holds all of its SM's TMEM and waits for blocks on other SMs: of two
    // launches (of two engines) that shared SMs, each could hold TMEM that the other waits for.  So it takes more than half of an SM's
    // 228 KB, whatever its registers are.
    static constexpr size_t kNeeds = sizeof(float) * kFloats * kWorkers, kSmem = kWide && kNeeds < 120 * 1024 ? 120 * 1024 : kNeeds;
    static_assert(!kWide || 2 * kSmem > 228 * 1024, "one block per SM");
    static_assert(kSmem <= 226 * 1024, "and the static arrays beside it");
};

// Wide strides, TMEM columns: G as hi | lo, then the runs of either product, then X^T as hi | lo.
template <int LD>
struct SmallTmem {
    static constexpr uint32_t kG = 0, kD = 2 * LD, kX = kD + 2 * SmallShape<LD>::kTile, kUsed = kX + 2 * SmallShape<LD>::kTile, kColumns = 512;
    static_assert(kUsed <= kColumns && LD <= 2 * SmallShape<LD>::kTile, "512 columns in all");
};

struct SmallCut {
    uint32_t row, entry;      // first row of the worker; first entry (before the row's own: the rest of the row before)
};

struct SmallSide {            // one of the two half iterations
    const float* vals;        // stored entries, by output row
    const int32_t* ind;       // factor row of each entry
    const int64_t* ptr;       // row offsets
    const SmallCut* cuts;     // [workers + 1]
    uint32_t workers;
    float* X;                 // factor that is updated [rows][LD]
    const float* D;           // factor that is gathered [*][LD]
    float* carry;             // [workers][LD]: pieces of rows that other workers own
    unsigned int* flag;       // [workers]: the iteration whose piece is there
    float* G;                 // Gram matrix of D, [LD][LD], and
    unsigned int* ready;      // the chunks of it that have been summed
    const float* partial_in;  // its partials
    int partials;
    float* partial_out;       // partials of the Gram matrix of X, for the other side
};

struct SmallArgs {
    SmallSide side[2];        // 0 updates W from H, 1 updates H from W
    int iters, r4;            // iterations; float4 per factor row that are not padding
    float eps;
    unsigned int* barrier;    // arrivals, and the abort flag behind them
    uint32_t wait_limit;
    int* err;
};

__device__ __forceinline__ unsigned int small_acquire(const unsigned int* p) {
    unsigned int v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Until *p >= target; false once a wait ran out anywhere.
__device__ __forceinline__ bool small_wait(const SmallArgs& a, const unsigned int* p, unsigned int target) {
    for (uint32_t spin = 0; spin < a.wait_limit; spin++) {
        if (small_acquire(p) >= target) return true;
        if ((spin & 63u) == 63u && *(volatile unsigned int*)(a.barrier + 1)) return false;
    }
    *(volatile unsigned int*)(a.barrier + 1) = 1u;
    atomicOr(a.err, kErrGridTimeout);
    return false;
}
__device__ __forceinline__ void small_arrive(unsigned int* p) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(p) : "memory");
}

// All blocks; false once a wait ran out anywhere.
__device__ __forceinline__ bool small_grid_barrier(const SmallArgs& a, unsigned int target) {
    __shared__ int ok_s;
    __syncthreads();
    if (threadIdx.x == 0) {
        small_arrive(a.barrier);
        ok_s = small_wait(a, a.barrier, target);
    }
    __syncthreads();
    return ok_s != 0;
}

// The threads of one worker.
template <int LD>
__device__ __forceinline__ void small_sync(int worker) {
    if constexpr (SmallShape<LD>::kWorkers == 1) __syncthreads();
    else asm volatile("bar.sync %0, %1;" ::"r"(worker + 1), "n"(SmallShape<LD>::kT) : "memory");
}

// What a tile of a worker is.
struct SmallTile {
    uint32_t e0, e1;          // its entries: those before the first row's own belong to a row that another worker owns ("head")
    uint32_t unit;            // entries per lane group, and
    float inv;                // the reciprocal
    uint32_t row0;            // its first row
    int rows;
    uint32_t next, last_end;  // of the last row: the worker that holds its next piece (0: it is whole), and its end
    int last;                 // of the worker's tiles
};

// acc += v * h, two columns at a time.
__device__ __forceinline__ void small_fma2(float2& acc, float v, float2 h) {
    unsigned long long d, x, y;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(acc.x), "f"(acc.y));
    asm("mov.b64 %0, {%1, %1};" : "=l"(x) : "f"(v));
    asm("mov.b64 %0, {%1, %2};" : "=l"(y) : "f"(h.x), "f"(h.y));
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(x), "l"(y));
    asm("mov.b64 {%0, %1}, %2;" : "=f"(acc.x), "=f"(acc.y) : "l"(d));
}
struct SmallSum {             // of a unit's row: this lane's float4
    float2 x[2];
    __device__ __forceinline__ void clear() { x[0] = x[1] = make_float2(0.f, 0.f); }
    __device__ __forceinline__ void add(float v, const float4& a) {
        small_fma2(x[0], v, make_float2(a.x, a.y));
        small_fma2(x[1], v, make_float2(a.z, a.w));
    }
    __device__ __forceinline__ void add(const SmallSum& s) {
        small_fma2(x[0], 1.f, s.x[0]);
        small_fma2(x[1], 1.f, s.x[1]);
    }
};

// A unit adds up runs of at most this many entries, and then the runs: where a worker's tile has 10^5 entries its units have thousands,
// and one chain of them is off by 2^-24 times the square root of their number.  Numerators of W against float64 (rms after two updates; one
// chain, runs of 64): 8000 x 600000 x 4000 values, rank 32, 7.2e-7, 1.2e-7; 17000 x 200000 x 1800 8.6e-7, 1.4e-7; on the large path
// 5.1e-7 and 5.2e-7.  us an iteration: 693, 704 and 571, 578; 500 x 600000 x 20000 349, 356; 2048 x 65536 x 4096 160.7, 161.8;
// 300 x 9000 x 1500, rank 128, 59.4, 59.4.  (The loop counts down: a register less, 1 % at 32 and 64 and 2 at 96 and 128.)
constexpr uint32_t kSmallRun = 64;

// Where the units of a tile whose entries begin at e0 begin.
template <int LD>
__device__ __forceinline__ uint32_t small_base(uint32_t e0) { return e0 / SmallShape<LD>::kB * SmallShape<LD>::kB; }

// The numerators of a tile.  sp[0 .. rows]: the rows' offsets, clipped to the worker's end.
template <int LD>
__device__ __forceinline__ void small_gather(const SmallSide& s, const SmallTile& tl, const uint32_t* sp, float* N, float* C, int r4, int t) {
    using S = SmallShape<LD>;
    constexpr int kB = S::kB, kLanes = S::kLanes, kQuads = S::kQuads;
    const int q = t % kLanes, g = t / kLanes;
    const uint32_t unit = tl.unit;
    // units begin at whole sectors of the entries' arrays
    uint32_t p = small_base<LD>(tl.e0) + g * unit;
    const uint32_t beg = max(tl.e0, p), end = min(tl.e1, p + unit);
    if (!__any_sync(0xffffffffu, beg < end)) return;
    // lanes without a column of their own (the padding of the rank) read a column that is read anyway
    const bool real = q < r4;
    const float4* const D4 = (const float4*)s.D + (real ? q : 0);
    // lane q < kB of the unit holds entry p + q and its row (-1: the head); the next entries are asked for one batch ahead
    float v = 0.f, vn = 0.f;
    uint32_t j = 0, jn = 0;
    int i = -1;
    auto fetch = [&](uint32_t at, float& fv, uint32_t& fj) {
        fv = 0.f;
        fj = 0;
        if (q < kB && at + q >= beg && at + q < end) {
            fv = __ldg(s.vals + at + q);
            fj = (uint32_t)__ldg(s.ind + at + q) * kQuads;
        }
    };
    fetch(p, v, j);
    // the row of the first entry: the last one that starts at or before it
    for (int lo = 0, n = tl.rows; n > 0;) {
        const int half = n >> 1;
        if (sp[lo + half] <= beg) {
            i = lo + half;
            lo += half + 1;
            n -= half + 1;
        } else {
            n = half;
        }
    }
    // where the sum of the unit's first row goes: the carry where the row started earlier
    float* dst = ((i >= 0 ? sp[i] : tl.e0) < beg ? C + g * LD : (i >= 0 ? N + i * S::kLdN : C + S::kUnits * LD)) + 4 * q;
    bool started = false;
    uint32_t i_end = tl.rows > 0 ? sp[i + 1] : tl.e1;
    SmallSum acc, runs;  // of the row: the present run of entries, and the runs before
    acc.clear();
    runs.clear();
    constexpr uint32_t kFirst = kLanes == 8 ? 0x01010101u : (kLanes == 16 ? 0x00010001u : 1u);  // the first lanes of a warp's units
    static_assert(kSmallRun % kB == 0, "a run ends with a batch");
    for (uint32_t left = unit; left != 0; left -= kB, p += kB) {  // the same trips for every unit of the warp
        if (left % kSmallRun == 0) {
            runs.add(acc);
            acc.clear();
        }
        const bool in = q < kB && p + q >= beg && p + q < end;
        float4 h[kB];
        fetch(p + kB, vn, jn);
        if (__all_sync(0xffffffffu, p >= beg && p + kB <= end)) {
#pragma unroll
            for (int k = 0; k < kB; k++) h[k] = __ldcg(D4 + __shfl_sync(0xffffffffu, j, k, kLanes));
        } else {
            // the first unit's begin, the last one's end
            if (!__any_sync(0xffffffffu, p < end)) break;
#pragma unroll
            for (int k = 0; k < kB; k++) {
                const uint32_t jj = __shfl_sync(0xffffffffu, j, k, kLanes);
                h[k] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (p + k >= beg && p + k < end) h[k] = __ldcg(D4 + jj);
            }
        }
        while (in && i_end <= p + q) {
            i++;
            i_end = sp[i + 1];
        }
        // lanes whose entry is the last of its row in the unit
        const uint32_t lasts = __ballot_sync(0xffffffffu, in && (p + q + 1 == i_end || p + q + 1 == end));
        if (lasts == 0) {
#pragma unroll
            for (int k = 0; k < kB; k++) acc.add(__shfl_sync(0xffffffffu, v, k, kLanes), h[k]);
        } else {
#pragma unroll
            for (int k = 0; k < kB; k++) {
                acc.add(__shfl_sync(0xffffffffu, v, k, kLanes), h[k]);
                if (lasts & (kFirst << k)) {  // in some unit of the warp
                    const int row = __shfl_sync(0xffffffffu, i, k, kLanes);
                    if (lasts >> ((threadIdx.x & 31u) - q + k) & 1u) {
                        if (started) dst = N + row * S::kLdN + 4 * q;
                        acc.add(runs);
                        runs.clear();
                        if (q < kQuads) *(float4*)dst = real ? make_float4(acc.x[0].x, acc.x[0].y, acc.x[1].x, acc.x[1].y) : make_float4(0.f, 0.f, 0.f, 0.f);
                        started = true;
                        acc.clear();
                    }
                }
            }
        }
        v = vn;
        j = jn;
    }
}

// x / unit (at most some hundred), by a reciprocal and a step up or down.
__device__ __forceinline__ uint32_t small_unit_of(uint32_t x, uint32_t unit, float inv) {
    uint32_t u = (uint32_t)((float)x * inv);
    if (u * unit > x) u--;
    if ((u + 1) * unit <= x) u++;
    return u;
}
// The units that hold a piece of a row (entries [beg, end) of the tile) in their carries, those that begin inside it: first | last << 16.
constexpr uint32_t kSmallEmpty = 0xffffu;  // no entries in the tile
template <int LD>
__device__ __forceinline__ uint32_t small_carries_of(const SmallTile& tl, uint32_t beg, uint32_t end) {
    if (beg >= end) return kSmallEmpty;
    const uint32_t base = small_base<LD>(tl.e0);
    return (small_unit_of(beg - base, tl.unit, tl.inv) + 1) | small_unit_of(end - 1 - base, tl.unit, tl.inv) << 16;
}
__device__ __forceinline__ void small_add(float4& x, const float4& y) {
    x.x += y.x;
    x.y += y.y;
    x.z += y.z;
    x.w += y.w;
}
__device__ __forceinline__ void small_add(float& x, float y) { x += y; }
// x: columns c .. of the row.
template <int LD, typename F>
__device__ __forceinline__ void small_add_carries(F& x, const float* C, uint32_t carries, int c) {
    const uint32_t last = carries >> 16;
#pragma unroll 4
    for (uint32_t u = carries & 0xffffu; u <= last; u++) small_add(x, *(const F*)(C + u * LD + c));
}
// Adds the pieces that the workers from `next` on hold of a row whose entries end at `end`.
template <int LD, typename F>
__device__ __forceinline__ void small_add_pieces(F& x, const SmallArgs& a, const SmallSide& s, uint32_t next, uint32_t end,
                                                 unsigned int epoch, int c) {
    for (bool more = true; more; next++) {
        if (!small_wait(a, s.flag + next, epoch)) return;
        small_add(x, __ldcg((const F*)(s.carry + (int64_t)next * LD + c)));
        more = next + 1 < s.workers && __ldg(&s.cuts[next + 1].entry) < end;
    }
}

// Few partials (8 at stride 32, 2 at 64): the worker sums all of G for itself.  In a fixed order and in double, as below.  (us an iteration
// at 8 and at 32 or 64 allowed: 64 x 2048 x 96 values, rank 32, 16.1, 17.3; 185 x 2695 x 150, rank 12, with 64 of them 16.9, 27.4.)
template <int LD>
__device__ __forceinline__ bool small_gram_direct(int partials) { return !SmallShape<LD>::kWide && partials * LD * LD <= 8192; }
template <int LD>
__device__ __forceinline__ void small_gram_sum_all(const SmallSide& s, int t, float* G) {
    for (int e = t; e < LD * LD / 2; e += SmallShape<LD>::kT) {
        double x = 0.0, y = 0.0;
#pragma unroll 8
        for (int k = 0; k < s.partials; k++) {
            const float2 v = __ldcg((const float2*)(s.partial_in + (int64_t)k * LD * LD) + e);
            x += (double)v.x;
            y += (double)v.y;
        }
        ((float2*)G)[e] = make_float2((float)x, (float)y);
    }
}
// Many: the chunks of this worker, the partials of a chunk over its warps.  red: [warps][32 * kVec] doubles.
template <int LD>
__device__ __forceinline__ void small_gram_chunks(const SmallSide& s, int worker, int t, double* red) {
    using S = SmallShape<LD>;
    constexpr int kV = S::kVec, kLoads = (kNumSMs + S::kWarps - 1) / S::kWarps;
    const int lane = t & 31, w = t >> 5;
    for (int g = worker * gridDim.x + blockIdx.x; g < S::kChunks; g += gridDim.x * S::kWorkers) {
        const int e = (g * 32 + lane) * kV;
        double sum[kV];
        if constexpr (kV == 1) {
            float v[kLoads];  // all loads before the first sum
#pragma unroll
            for (int k = 0; k < kLoads; k++)
                v[k] = w + k * S::kWarps < s.partials ? __ldcg(s.partial_in + (int64_t)(w + k * S::kWarps) * LD * LD + e) : 0.f;
            sum[0] = 0.0;
#pragma unroll
            for (int k = 0; k < kLoads; k++) sum[0] += (double)v[k];
        } else {
            float4 v[kLoads];
#pragma unroll
            for (int k = 0; k < kLoads; k++) {
                v[k] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (w + k * S::kWarps < s.partials)
                    v[k] = __ldcg((const float4*)(s.partial_in + (int64_t)(w + k * S::kWarps) * LD * LD + e));
            }
#pragma unroll
            for (int i = 0; i < kV; i++) sum[i] = 0.0;
#pragma unroll
            for (int k = 0; k < kLoads; k++) {
                sum[0] += (double)v[k].x;
                sum[1] += (double)v[k].y;
                sum[2] += (double)v[k].z;
                sum[3] += (double)v[k].w;
            }
        }
        small_sync<LD>(worker);  // the chunk before has been read
#pragma unroll
        for (int i = 0; i < kV; i++) red[(w * kV + i) * 32 + lane] = sum[i];
        small_sync<LD>(worker);
        if (w < kV) {  // warp i adds up the lanes' i-th elements
            double x = 0.0;
#pragma unroll
            for (int k = 0; k < S::kWarps; k++) x += red[(k * kV + w) * 32 + lane];
            __stcg(s.G + (g * 32 + lane) * kV + w, (float)x);
            __syncwarp();
            if (lane == 0) small_arrive(s.ready);
        }
    }
}

// K consecutive floats at p (aligned as K allows).
template <int K>
__device__ __forceinline__ void small_lds(const float* p, float (&v)[K]) {
#pragma unroll
    for (int k = 0; k < K; k += 4) {
        const float4 x = *(const float4*)(p + k);
        v[k] = x.x; v[k + 1] = x.y; v[k + 2] = x.z; v[k + 3] = x.w;
    }
}

__device__ __forceinline__ void small_copy16(float* dst, const float* src) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}

// The numerators of columns c .. of row k of the tile.
template <int LD, typename F>
__device__ __forceinline__ F small_numerator(const SmallArgs& a, const SmallSide& s, const SmallTile& tl, const float* N, const float* C,
                                             const uint32_t* carries, unsigned int epoch, int k, int c) {
    F x = F();
    const uint32_t cr = carries[k];
    if (cr != kSmallEmpty) {
        x = *(const F*)(N + k * SmallShape<LD>::kLdN + c);
        small_add_carries<LD>(x, C, cr, c);
    }
    if (tl.next != 0 && k == tl.rows - 1) small_add_pieces<LD>(x, a, s, tl.next, tl.last_end, epoch, c);
    return x;
}

// Wide strides.  Warp w has TMEM lanes 32 (w % 4) ..: a thread has column c = 32 (w % 4) + lane of the factor, and of a tile the
// R rows from R (w / 4) on: 8, or 16 in tiles of more than 32.

// G, the whole matrix, into TMEM.  It is symmetric, so that a thread's row can be read as a column.
template <int LD>
__device__ __forceinline__ void small_load_g(const float* g, uint32_t tmem, int t) {
    constexpr int kPer = LD / 4;  // values of K per thread
    const int w = t >> 5, c = 32 * (w & 3) + (t & 31), k0 = kPer * (w >> 2);
    if (32 * (w & 3) >= LD) return;
    float x[kPer];
#pragma unroll
    for (int k = 0; k < kPer; k++) x[k] = __ldcg(g + (k0 + k) * LD + c);
    const uint32_t at = tmem + SmallTmem<LD>::kG + ((uint32_t)(32 * (w & 3)) << 16) + (uint32_t)k0;
#pragma unroll
    for (int k = 0; k < kPer; k += 8) {
        float4 h0, l0, h1, l1;
        tf32_split(make_float4(x[k], x[k + 1], x[k + 2], x[k + 3]), h0, l0);
        tf32_split(make_float4(x[k + 4], x[k + 5], x[k + 6], x[k + 7]), h1, l1);
        tc_st8(at + k, h0, h1);
        tc_st8(at + LD + k, l0, l1);
    }
    tc_st_wait();
}

// The tile's rows of X into shared memory, as the operand of G X^T: per 32 columns the hi and the lo half of kTile rows.
template <int LD>
__device__ __forceinline__ void small_load_x(const SmallSide& s, const SmallTile& tl, float* X, int t) {
    using S = SmallShape<LD>;
    for (int e = t; e < (tl.rows + 7) / 8 * 8 * S::kQuads; e += S::kT) {
        const int row = e % 8 + e / (8 * S::kQuads) * 8, quad = e / 8 % S::kQuads;
        float4 x = make_float4(0.f, 0.f, 0.f, 0.f), hi, lo;
        if (row < tl.rows) x = __ldcg((const float4*)s.X + (int64_t)(tl.row0 + row) * S::kQuads + quad);
        tf32_split(x, hi, lo);
        float* p = X + quad / 8 * (2 * S::kTile * 32) + tc_canon(row, quad % 8 * 4);
        *(float4*)p = hi;
        *(float4*)(p + S::kTile * 32) = lo;
    }
    fence_async_smem();
}

// One run of either product: d (+)= A B over the K-steps [k0, k1), hi * hi last (see k_gram_tc).  a: the operand in TMEM, hi, and
// lo_columns behind it lo; b: the one in shared memory, whose rows are `rows`.
__device__ __forceinline__ void small_mma_run(uint32_t d, uint32_t a, uint32_t lo_columns, const float* b, int rows, int k0, int k1,
                                              uint32_t idesc) {
    const uint64_t desc0 = tc_smem_desc(smem_u32(b), 128, 1024);
    const uint32_t half = (uint32_t)rows * 8u, chunk = 2 * half;  // 16-byte units: 32 values of K
    for (int k = k0; k < k1; k++) {
        const uint64_t bh = desc0 + (uint32_t)(k / 4) * chunk + 16u * (uint32_t)(k % 4);
        tc_mma_tf32_ta(d, a + lo_columns + 8u * k, bh, idesc, k == k0 ? 0u : 1u);
        tc_mma_tf32_ta(d, a + 8u * k, bh + half, idesc, 1u);
    }
    for (int k = k0; k < k1; k++)
        tc_mma_tf32_ta(d, a + 8u * k, desc0 + (uint32_t)(k / 4) * chunk + 16u * (uint32_t)(k % 4), idesc, 1u);
}
// G X^T in two runs (one thread).
template <int LD>
__device__ __forceinline__ void small_mma_gx(uint32_t tmem, const float* X, uint64_t* bar) {
    constexpr int kRows = SmallShape<LD>::kTile;
    const uint32_t idesc = tc_idesc_tf32(128, kRows);
    small_mma_run(tmem + SmallTmem<LD>::kD, tmem + SmallTmem<LD>::kG, LD, X, kRows, 0, 8, idesc);
    small_mma_run(tmem + SmallTmem<LD>::kD + kRows, tmem + SmallTmem<LD>::kG, LD, X, kRows, 8, LD / 8, idesc);
    tc_commit(bar);
}

// The new values of this thread's column: rows past the tile's end are zero.  mma_wait: until G X^T is there.
template <int LD, int R, typename Wait>
__device__ __forceinline__ void small_update_tc(const SmallArgs& a, const SmallSide& s, const SmallTile& tl, uint32_t tmem, const float* N,
                                                const float* C, const uint32_t* carries, unsigned int epoch, int t, float (&x)[R],
                                                Wait mma_wait) {
    using S = SmallShape<LD>;
    const int w = t >> 5, c = 32 * (w & 3) + (t & 31), j0 = R * (w >> 2);
    const bool mine = 32 * (w & 3) < LD && j0 < tl.rows;  // uniform per warp
    float* const out = s.X + (int64_t)(tl.row0 + j0) * LD + c;
    float n[R], d[R], e[R];
#pragma unroll
    for (int j = 0; j < R; j++) x[j] = mine && j0 + j < tl.rows ? __ldcg(out + j * LD) : 0.f;
#pragma unroll
    for (int j = 0; j < R; j++)
        n[j] = mine && j0 + j < tl.rows ? small_numerator<LD, float>(a, s, tl, N, C, carries, epoch, j0 + j, c) : 0.f;
    mma_wait();
    if (!mine) return;
    const uint32_t at = tmem + SmallTmem<LD>::kD + ((uint32_t)(32 * (w & 3)) << 16) + (uint32_t)j0;
    if constexpr (R == 16) {
        tc_ld16(at, d);
        tc_ld16(at + S::kTile, e);
    } else {
        tc_ld8(at, d);
        tc_ld8(at + S::kTile, e);
    }
    tc_ld_wait();
#pragma unroll
    for (int j = 0; j < R; j++) d[j] += e[j];
    float q[R], chk = 0.f, r_min = 1.0f;
    uint32_t lowest = 0xffffffffu;
#pragma unroll
    for (int j = 0; j < R; j++) {
        // t = den + eps; q = num / t; x = x * q (reference order, kernels.h:31-33), as in k_mu_update_ws
        d[j] = j0 + j < tl.rows ? __fadd_rn(d[j], a.eps) : 1.f;
        float rc;
        q[j] = quot_refined(n[j], d[j], rc);
        chk = __fmaf_rn(q[j], 0.f, chk);
        lowest = min(lowest, 2u * __float_as_uint(n[j]) - 1u);
        r_min = fminf(r_min, rc);
    }
    if (quot_doubtful(chk, r_min, lowest)) {
#pragma unroll
        for (int j = 0; j < R; j++) q[j] = quot_careful(n[j], d[j]);
    }
#pragma unroll
    for (int j = 0; j < R; j++) {
        x[j] *= q[j];
        if (j0 + j < tl.rows) __stcg(out + j * LD, x[j]);
    }
}

// X^T of the tile, from the threads' columns, as both operands of the Gram matrix.
template <int LD, int R>
__device__ __forceinline__ void small_store_xt(const float (&x)[R], uint32_t tmem, float* X, int t) {
    const int w = t >> 5, c = 32 * (w & 3) + (t & 31), j0 = R * (w >> 2);
    if (32 * (w & 3) < LD) {
        const uint32_t at = tmem + SmallTmem<LD>::kX + ((uint32_t)(32 * (w & 3)) << 16) + (uint32_t)j0;
        float* p = X + j0 / 32 * (2 * LD * 32) + tc_canon(c, j0 % 32);
#pragma unroll
        for (int j = 0; j < R; j += 8) {
            float4 h0, l0, h1, l1;
            tf32_split(make_float4(x[j], x[j + 1], x[j + 2], x[j + 3]), h0, l0);
            tf32_split(make_float4(x[j + 4], x[j + 5], x[j + 6], x[j + 7]), h1, l1);
            tc_st8(at + j, h0, h1);
            tc_st8(at + SmallShape<LD>::kTile + j, l0, l1);
            *(float4*)(p + j * 8) = h0;
            *(float4*)(p + j * 8 + 32) = h1;
            *(float4*)(p + LD * 32 + j * 8) = l0;
            *(float4*)(p + LD * 32 + j * 8 + 32) = l1;
        }
        fence_async_smem();
        tc_st_wait();
    }
}

// The update of a tile (update; else its rows as they are) and, where the Gram matrix is wanted, X^T as its operands.
template <int LD, int R, typename Wait>
__device__ __forceinline__ void small_tile_tc(const SmallArgs& a, const SmallSide& s, const SmallTile& tl, uint32_t tmem, float* X,
                                              const float* N, const float* C, const uint32_t* carries, unsigned int epoch, int t,
                                              bool update, bool want_gram, Wait mma_wait) {
    float x[R];
    if (update) {
        small_update_tc<LD, R>(a, s, tl, tmem, N, C, carries, epoch, t, x, mma_wait);
    } else {
        const int w = t >> 5, c = 32 * (w & 3) + (t & 31);
#pragma unroll
        for (int j = 0; j < R; j++) {
            const int row = R * (w >> 2) + j;
            x[j] = row < tl.rows && c < LD ? __ldcg(s.X + (int64_t)(tl.row0 + row) * LD + c) : 0.f;
        }
    }
    if (want_gram) small_store_xt<LD, R>(x, tmem, X, t);
}

// The update of a tile at the narrow strides (32, 64), on CUDA cores: a thread makes two rows x four columns.
template <int LD>
__device__ __forceinline__ void small_update_fma(const SmallArgs& a, const SmallSide& s, const SmallTile& tl, const float* G, float* X,
                                                 const float* N, const float* C, const uint32_t* carries, unsigned int epoch, int t) {
    using S = SmallShape<LD>;
    constexpr int kQuads = S::kQuads, kLd = S::kLdX;
    const int pair = t / kQuads, c = t % kQuads;
    const bool item = 2 * pair < tl.rows, two = 2 * pair + 1 < tl.rows;
    float* x0 = X + 2 * pair * kLd;
    float* x1 = two ? x0 + kLd : x0;
    float4 num[2];
    if (item) {
        num[0] = small_numerator<LD, float4>(a, s, tl, N, C, carries, epoch, 2 * pair, 4 * c);
        num[1] = two ? small_numerator<LD, float4>(a, s, tl, N, C, carries, epoch, 2 * pair + 1, 4 * c) : make_float4(0.f, 0.f, 0.f, 0.f);
        float4 d0 = make_float4(0.f, 0.f, 0.f, 0.f), d1 = d0;
#pragma unroll 2
        for (int k0 = 0; k0 < LD; k0 += 4) {
            float u[4], v[4];
            small_lds<4>(x0 + k0, u);
            small_lds<4>(x1 + k0, v);
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const float4 g = *(const float4*)(G + (k0 + k) * LD + c * 4);
                d0.x = fmaf(u[k], g.x, d0.x); d0.y = fmaf(u[k], g.y, d0.y);
                d0.z = fmaf(u[k], g.z, d0.z); d0.w = fmaf(u[k], g.w, d0.w);
                d1.x = fmaf(v[k], g.x, d1.x); d1.y = fmaf(v[k], g.y, d1.y);
                d1.z = fmaf(v[k], g.z, d1.z); d1.w = fmaf(v[k], g.w, d1.w);
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
            q[k] = quot_refined(ns[k], __fadd_rn(ds[k], a.eps), rc);
            chk = __fmaf_rn(q[k], 0.f, chk);
            lowest = min(lowest, 2u * __float_as_uint(ns[k]) - 1u);
            r_min = fminf(r_min, rc);
        }
        if (quot_doubtful(chk, r_min, lowest)) {
#pragma unroll
            for (int k = 0; k < 8; k++) q[k] = quot_careful(ns[k], __fadd_rn(ds[k], a.eps));
        }
        num[0] = make_float4(xs[0] * q[0], xs[1] * q[1], xs[2] * q[2], xs[3] * q[3]);
        num[1] = make_float4(xs[4] * q[4], xs[5] * q[5], xs[6] * q[6], xs[7] * q[7]);
    }
    __syncwarp();  // the threads of a row are of one warp: all have read it
    if (item) {
        float4* out = (float4*)s.X + (int64_t)(tl.row0 + 2 * pair) * kQuads + c;
        __stcg(out, num[0]);
        *(float4*)(x0 + c * 4) = num[0];
        if (two) {
            __stcg(out + kQuads, num[1]);
            *(float4*)(x1 + c * 4) = num[1];
        }
    }
}

// The tile's part of the Gram matrix at the narrow strides: kSub neighbouring threads sum a square of 4 x 4, each over every kSub-th
// row, and share out the adding up.  The sums stay in shared memory (registers belong to the gathers).
template <int LD>
__device__ __forceinline__ void small_gram_fma(float* sums, bool first, const float* X, int rows, int t) {
    using S = SmallShape<LD>;
    constexpr int kSub = S::kSub;
    float2 acc[8];  // row major
#pragma unroll
    for (int i = 0; i < 8; i++) acc[i] = make_float2(0.f, 0.f);
    const int sub = t % kSub, ty = t / kSub / S::kQuads, tx = t / kSub % S::kQuads;
#pragma unroll 2
    for (int k = sub; k < rows; k += kSub) {
        const float4 u = *(const float4*)(X + k * S::kLdX + ty * 4), v = *(const float4*)(X + k * S::kLdX + tx * 4);
        const float2 v0 = make_float2(v.x, v.y), v1 = make_float2(v.z, v.w);
        small_fma2(acc[0], u.x, v0); small_fma2(acc[1], u.x, v1);
        small_fma2(acc[2], u.y, v0); small_fma2(acc[3], u.y, v1);
        small_fma2(acc[4], u.z, v0); small_fma2(acc[5], u.z, v1);
        small_fma2(acc[6], u.w, v0); small_fma2(acc[7], u.w, v1);
    }
    // halve what a thread holds and double what is in it, kSub times
    int lo = 0;
#pragma unroll
    for (int d = 1, n = 8; d < kSub; d *= 2, n /= 2) {
        const bool up = sub & d;
#pragma unroll
        for (int i = 0; i < n / 2; i++) {
            const float2 keep = up ? acc[i + n / 2] : acc[i], give = up ? acc[i] : acc[i + n / 2];
            acc[i].x = keep.x + __shfl_xor_sync(0xffffffffu, give.x, d);
            acc[i].y = keep.y + __shfl_xor_sync(0xffffffffu, give.y, d);
        }
        lo += up ? n / 2 : 0;
    }
#pragma unroll
    for (int i = 0; i < 8 / kSub; i++) {
        const int e = 2 * (lo + i);
        float2* p = (float2*)(sums + (ty * 4 + e / 4) * LD + tx * 4 + e % 4);
        float2 x = acc[i];
        if (!first) {
            const float2 y = *p;
            x.x += y.x;
            x.y += y.y;
        }
        *p = x;
    }
}

// A tile of a worker from its first row and entry on.
template <int LD>
__device__ __forceinline__ void small_tile(SmallTile& tl, const SmallSide& s, const SmallCut* cut, uint32_t wk, uint32_t row0, uint32_t e0,
                                           const uint32_t* sp) {
    using S = SmallShape<LD>;
    tl.row0 = row0;
    tl.rows = min(S::kTile, (int)(cut[1].row - row0));
    tl.last = row0 + tl.rows == cut[1].row;
    tl.e0 = e0;
    tl.e1 = tl.rows > 0 ? sp[tl.rows] : cut[1].entry;
    const uint32_t unit = (max(tl.e1 - small_base<LD>(e0), 1u) + S::kUnits - 1) / S::kUnits;
    tl.unit = (unit + S::kB - 1) / S::kB * S::kB;
    tl.inv = 1.0f / (float)tl.unit;
    tl.next = tl.last_end = 0;
    if (tl.last && tl.rows > 0) {
        tl.last_end = (uint32_t)__ldg(s.ptr + cut[1].row);
        if (tl.last_end > cut[1].entry) tl.next = wk + 1;
    }
}

// The state between the gathers is in shared memory: registers belong to them.
template <int LD>
__global__ void __launch_bounds__(SmallShape<LD>::kThreads, 1) k_small_run(const __grid_constant__ SmallArgs a) {
    using S = SmallShape<LD>;
    using T = SmallTmem<S::kWide ? LD : 128>;
    extern __shared__ __align__(128) float small_smem[];
    __shared__ SmallCut cuts[S::kWorkers][2][2];
    __shared__ SmallTile tiles[S::kWorkers][4];  // either side's first tile, and two that the others take in turn
    __shared__ __align__(8) uint64_t mma_done;
    __shared__ uint32_t tmem_slot;
    const int worker = threadIdx.x / S::kT, t = threadIdx.x % S::kT;
    const uint32_t wk = (uint32_t)worker * gridDim.x + blockIdx.x;
    float* const base = small_smem + worker * S::kFloats;
    float* const G = base + S::kG;
    float* const X = base + S::kX;
    float* const N = base + S::kN;
    float* const C = base + S::kC;
    float* const sums = base + S::kS;
    uint32_t* const offsets = (uint32_t*)(base + S::kP);
    uint32_t* const carries = (uint32_t*)(base + S::kR);
    if (S::kWide) {
        if (threadIdx.x < 32) tc_alloc(&tmem_slot, T::kColumns);
        if (threadIdx.x == 32) {
            mbar_init(&mma_done, 1);
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
    }
    // what does not change: the cuts, and either side's first tile with its row offsets
    for (int sd = 0; sd < 2; sd++) {
        const SmallSide& s = a.side[sd];
        if (wk >= s.workers) continue;
        const SmallCut cut0 = s.cuts[wk], cut1 = s.cuts[wk + 1];
        const int rows = min((int)(cut1.row - cut0.row), S::kTile);
        for (int k = t; k <= rows; k += S::kT) offsets[sd * S::kOffsets + k] = min((uint32_t)__ldg(s.ptr + cut0.row + k), cut1.entry);
        small_sync<LD>(worker);
        if (t == 0) {
            cuts[worker][sd][0] = cut0;
            cuts[worker][sd][1] = cut1;
            small_tile<LD>(tiles[worker][sd], s, cuts[worker][sd], wk, cut0.row, cut0.entry, offsets + sd * S::kOffsets);
        }
    }
    if (S::kWide) tc_fence_before();
    __syncthreads();
    uint32_t tmem = 0, runs = 0;  // wide strides: TMEM, and the commits that mma_done has seen
    if (S::kWide) {
        tc_fence_after();
        tmem = tmem_slot;
    }
    // all threads, behind an MMA's commit
    auto mma_wait = [&]() {
        if (!mbar_wait(&mma_done, runs & 1u)) {
            *(volatile unsigned int*)(a.barrier + 1) = 1u;
            atomicOr(a.err, kErrTcTimeout);
        }
        runs++;
        tc_fence_after();
    };
    // W, H, W, H ...; before them the partials of H H^T for the first W update.  One piece of code: instructions too come
    // through a cache (64 x 2048 at rank 32 with the code three times: 24 us an iteration for 19).
    for (int half = -1; half < 2 * a.iters; half++) {
        const SmallSide& s = a.side[half & 1];
        const unsigned int epoch = (unsigned int)(half >> 1) + 1;
        const bool want_gram = half + 1 < 2 * a.iters;
        float acc[S::kWide ? 32 : 1];  // wide strides: of row c of the Gram matrix, columns 32 (w / 4) ..
        if (S::kWide) {
#pragma unroll
            for (int i = 0; i < (S::kWide ? 32 : 1); i++) acc[i] = 0.f;
        }
        if (half >= 0) {
            if (!small_gram_direct<LD>(s.partials)) small_gram_chunks<LD>(s, worker, t, (double*)N);
            else if (wk < s.workers) small_gram_sum_all<LD>(s, t, G);
        }
        for (int slot = half & 1, more = wk < s.workers; more;) {
            const bool first = slot < 2;
            const SmallTile& tl = tiles[worker][slot];
            const uint32_t* const sp = offsets + slot * S::kOffsets;
            const int slot_next = slot == 2 ? 3 : 2;
            small_sync<LD>(worker);  // the tile before is done with shared memory
            if constexpr (!S::kWide) {
                for (int e = t; e < tl.rows * S::kQuads; e += S::kT)
                    small_copy16(X + (e / S::kQuads) * S::kLdX + (e % S::kQuads) * 4, s.X + ((int64_t)tl.row0 * S::kQuads + e) * 4);
                asm volatile("cp.async.commit_group;" ::: "memory");
            }
            if (half >= 0) {
                // the next tile's row offsets
                if (!tl.last && t <= min(S::kTile, (int)(cuts[worker][half & 1][1].row - tl.row0) - S::kTile)) {
                    const uint32_t d = (uint32_t)__cvta_generic_to_shared(offsets + slot_next * S::kOffsets + t);
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(s.ptr + tl.row0 + S::kTile + t) : "memory");
                }
                if (t < tl.rows) carries[t] = small_carries_of<LD>(tl, sp[t], sp[t + 1]);
                if constexpr (S::kWide) {
                    small_load_x<LD>(s, tl, X, t);
                    if (!first) {  // G is there: the tensor cores work while the warps gather
                        tc_fence_before();
                        small_sync<LD>(worker);
                        if (t < 32 && tc_elect()) {
                            tc_fence_after();
                            small_mma_gx<LD>(tmem, X, &mma_done);
                        }
                        __syncwarp();
                    }
                }
                small_gather<LD>(s, tl, sp, N, C, a.r4, t);
                asm volatile("cp.async.wait_all;" ::: "memory");
                if (first && t == 0 && !small_gram_direct<LD>(s.partials)) small_wait(a, s.ready, epoch * (S::kChunks * S::kVec));
                small_sync<LD>(worker);
                if (first) {
                    // the piece of the row before
                    const uint32_t head = tl.rows > 0 ? sp[0] : tl.e1;
                    const int lane = t & 31;
                    if (t / 32 == S::kWarps - 1 && head > tl.e0) {
                        if (lane < S::kQuads) {
                            float4 x = *(const float4*)(C + S::kUnits * LD + 4 * lane);
                            small_add_carries<LD>(x, C, small_carries_of<LD>(tl, tl.e0, head), 4 * lane);
                            __stcg((float4*)s.carry + (int64_t)wk * S::kQuads + lane, x);
                        }
                        __syncwarp();
                        if (lane == 0) asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(s.flag + wk), "r"(epoch) : "memory");
                    }
                    if constexpr (S::kWide) {
                        small_load_g<LD>(s.G, tmem, t);
                        tc_fence_before();
                        small_sync<LD>(worker);
                        if (t < 32 && tc_elect()) {
                            tc_fence_after();
                            small_mma_gx<LD>(tmem, X, &mma_done);
                        }
                        __syncwarp();
                    } else if (!small_gram_direct<LD>(s.partials)) {
                        for (int e = t; e < LD * S::kQuads; e += S::kT) ((float4*)G)[e] = __ldcg((const float4*)s.G + e);
                        small_sync<LD>(worker);
                    }
                }
            }
            if constexpr (S::kWide) {
                const int w = t >> 5;
                if (tl.rows <= 32) small_tile_tc<LD, 8>(a, s, tl, tmem, X, N, C, carries, epoch, t, half >= 0, want_gram, mma_wait);
                else small_tile_tc<LD, 16>(a, s, tl, tmem, X, N, C, carries, epoch, t, half >= 0, want_gram, mma_wait);
                if (want_gram) {
                    tc_fence_before();
                    small_sync<LD>(worker);
                    if (t < 32 && tc_elect()) {
                        tc_fence_after();
                        small_mma_run(tmem + T::kD, tmem + T::kX, S::kTile, X, LD, 0, (tl.rows + 7) / 8, tc_idesc_tf32(128, LD));
                        tc_commit(&mma_done);
                    }
                    __syncwarp();
                    mma_wait();
                    if (32 * (w >> 2) < LD) {
                        float d[32];
                        tc_ld32(tmem + T::kD + ((uint32_t)(32 * (w & 3)) << 16) + (uint32_t)(32 * (w >> 2)), d);
                        tc_ld_wait();
                        if (tl.rows > 0) {
#pragma unroll
                            for (int i = 0; i < 32; i++) acc[i] += d[i];
                        }
                    }
                }
                tc_fence_before();
            } else {
                if (half >= 0) small_update_fma<LD>(a, s, tl, G, X, N, C, carries, epoch, t);
                else asm volatile("cp.async.wait_all;" ::: "memory");
                if (want_gram) {
                    small_sync<LD>(worker);
                    small_gram_fma<LD>(sums, first, X, tl.rows, t);
                }
            }
            more = !tl.last;
            if (more && t == 0) {
                const SmallCut* cut = cuts[worker][half & 1];
                uint32_t* const spn = offsets + slot_next * S::kOffsets;
                const int rows = min(S::kTile, (int)(cut[1].row - tl.row0) - S::kTile);
                spn[rows] = min(spn[rows], cut[1].entry);  // (the low words of the offsets: entries fit)
                small_tile<LD>(tiles[worker][slot_next], s, cut, wk, tl.row0 + tl.rows, tl.e1, spn);
            }
            slot = slot_next;
        }
        if (!want_gram) break;
        float* const out = s.partial_out + (int64_t)blockIdx.x * LD * LD;
        if constexpr (S::kWide) {
            const int w = t >> 5, c = 32 * (w & 3) + (t & 31);
            if (wk < s.workers && 32 * (w & 3) < LD && 32 * (w >> 2) < LD) {
#pragma unroll
                for (int i = 0; i < 32; i++) __stcg(out + (32 * (w >> 2) + i) * LD + c, acc[i]);  // symmetric
            }
        } else {
            __syncthreads();
            if (blockIdx.x < s.workers) {
                // the sums of the block's workers, in order
                const bool two = blockIdx.x + gridDim.x < s.workers;
                const float4* const p = (const float4*)(small_smem + S::kS);
                for (int e = threadIdx.x; e < LD * LD / 4; e += S::kThreads) {
                    float4 x = p[e];
                    if (two) small_add(x, p[e + S::kFloats / 4]);
                    __stcg((float4*)out + e, x);
                }
            }
        }
        if (!small_grid_barrier(a, (unsigned int)(half + 2) * gridDim.x)) break;
    }
    if (S::kWide) {
        tc_fence_before();
        __syncthreads();
        if (threadIdx.x < 32) tc_dealloc(tmem, T::kColumns);
    }
}

// Where the workers' pieces begin.  A piece weighs its entries, and row_cost of them for each of its rows.
// A row is cut where a piece ends inside it only if it weighs an eighth of a piece or more; else the nearer end of it.
static __global__ void k_small_cuts(const int64_t* __restrict__ ptr, uint32_t rows, uint32_t row_cost, uint32_t workers,
                                    SmallCut* __restrict__ cuts) {
    const uint32_t w = blockIdx.x * blockDim.x + threadIdx.x;
    if (w > workers) return;
    if (w == workers) {
        cuts[w] = {rows, (uint32_t)ptr[rows]};
        return;
    }
    const uint64_t total = (uint64_t)ptr[rows] + (uint64_t)rows * row_cost, at = total * w / workers;
    uint32_t lo = 0, n = rows;  // the last row that begins at or before `at`
    while (n > 1) {
        const uint32_t half = n >> 1;
        if ((uint64_t)ptr[lo + half] + (uint64_t)(lo + half) * row_cost <= at) {
            lo += half;
            n -= half;
        } else {
            n = half;
        }
    }
    const uint32_t beg = (uint32_t)ptr[lo], len = (uint32_t)ptr[lo + 1] - beg;
    const uint64_t in = at - ((uint64_t)beg + (uint64_t)lo * row_cost);
    constexpr uint32_t kLeast = 32;  // entries of a piece of a row
    if ((uint64_t)(len + row_cost) * 8 * workers < total) {
        cuts[w] = 2 * in < len + row_cost ? SmallCut{lo, beg} : SmallCut{lo + 1, beg + len};
    } else if (in < row_cost + kLeast) {
        cuts[w] = {lo, beg};
    } else {
        const uint32_t e = (uint32_t)(in - row_cost);
        cuts[w] = e + kLeast > len ? SmallCut{lo + 1, beg + len} : SmallCut{lo + 1, beg + e};
    }
}

inline bool small_rank_ok(int ld) { return ld == 32 || ld == 64 || ld == 96 || ld == 128; }

inline int small_workers_per_block(int ld) { return ld > 64 ? 1 : 2; }

// What updating a row takes, in gathers of a factor row (us per iteration at half, this and 1.5 times this: 2048 x 65536 x 4096
// values, rank 32, 175, 162, 163; 1738 x 186396 x 3055, 32, 168, 152, 154; 300 x 9000 x 1500, 128, 62, 59, 62; 832 x 11990 x 1199, 94, 97, 87, 91).
inline uint32_t small_row_cost(int ld) { return (uint32_t)(ld <= 64 ? 8 + ld / 2 : 4 + ld / 3); }

// Workers of a side: as many as there are, but each with the work of 600 gathers, or 384 at the wide strides, whose tiles take time by
// runs of 16 rows (us an iteration at these and at 1024: 185 x 2695 x 150 values, rank 12, 16.9, 17.3; 64 x 2048 x 96, rank 32,
// 16.1, 15.6, and 20 or more from 1500 on; 400 x 8000 x 300, 32, 969 x 6722 x 400, 33, and 458 x 2551 x 300, 96, even).
inline int small_workers(int64_t rows, int64_t entries, int ld) {
    const int64_t cost = entries + rows * small_row_cost(ld);
    const int64_t most = (int64_t)kNumSMs * small_workers_per_block(ld);
    return (int)std::min(most, std::max<int64_t>(1, cost / (ld > 64 ? 384 : 600)));
}

// Whether these launches beat the large path.  An iteration takes about 15 us, two gathers of a factor row per stored entry, and the two
// contractions.  The large path takes 65 to 105 us plus the same gathers, but does the popular columns densely and contracts at the
// tensor cores' full rate.  us an iteration here and there:
//   stride 32: 8000 x 600000 x 4000 values 702, 763; 500 x 600000 x 20000 355, 468; 17000 x 200000 x 1800 560, 571; 3000 x 60000 x 4000
//              214, 237; 20000 x 50000 x 1500 507, 454; 5000 x 20000 x 3000 245, 227
//   64: 2000 x 40000 x 2000 165, 171; 1000 x 200000 x 2000 221, 228; 5000 x 50000 x 1000 204, 195; 3001 x 100003 x 2047 280, 250
//   96: 12000 x 12000 x 150 140, 165; 200 x 100000 x 3000 146, 170; 3060 x 80340 x 368 163, 170; 1500 x 60000 x 1500 215, 208
//   128: 800 x 40000 x 1000 118, 173; 200 x 100000 x 3000 161, 185; 4000 x 40000 x 300 144, 162; 828 x 74164 x 8240 523, 289
// popular: stored entries in popular columns; block: elements of the dense block.
inline bool small_pays(int64_t nnz, int64_t rows, int ld, int64_t popular, int64_t block) {
    if (ld == 32) {
        // Here large problems can gain too, and what decides is how dense the popular columns are.  us per million gathers, per MB of
        // the dense block and per MB of factors and numerators, from fourteen shapes (here within 3 % with the 1.04 below, there 8, but
        // for the least): the large path where the two are about even.
        const double gathers = 2e-6 * (double)nnz, factors = 384e-6 * (double)rows;
        const double here = 7.5 * gathers + 0.84 * factors;
        const double there = 73.0 + 6.8 * 2e-6 * (double)(nnz - popular) + 0.18 * 8e-6 * (double)block + 1.47 * factors;
        return nnz <= (1 << 26) && rows <= (1 << 22) && 1.04 * here < there;  // (not looked at beyond)
    }
    // bytes gathered per us (a lane group takes whole strides), elements contracted per us, and where the large path takes over
    const double gather = ld == 64 ? 15.0e6 : (ld == 96 ? 11.0e6 : 12.0e6);
    const double contract = ld == 64 ? 6.5e6 : (ld == 96 ? 10.0e6 : 20.0e6);
    const double line = ld == 64 ? 205.0 : (ld == 96 ? 166.0 : 155.0);
    return 15.0 + 8.0 * ld * (double)nnz / gather + (double)rows * ld * ld / contract < line;
}

// All blocks have to be on the GPU together: where the process may not use that many SMs (a share of an MPS
// server, for one) the runtime refuses the launch, and *made says so; nothing has run then.
// refuse: as if it had.
template <int LD>
inline int small_launch_t(SmallArgs& a, int blocks, cudaStream_t st, bool refuse, bool* made) {
    using S = SmallShape<LD>;
    DN_CUDA(cudaFuncSetAttribute(k_small_run<LD>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::kSmem));
    void* args[] = {&a};
    const cudaError_t e = refuse ? cudaErrorCooperativeLaunchTooLarge
                                 : cudaLaunchCooperativeKernel((void*)k_small_run<LD>, dim3((unsigned)blocks), dim3(S::kThreads), args, S::kSmem, st);
    *made = e != cudaErrorCooperativeLaunchTooLarge;
    if (!*made) {
        cudaGetLastError();
        return DNPEFF_OK;
    }
    DN_CUDA(e);
    DN_COUNT_LAUNCH(1);
    return DNPEFF_OK;
}
// sync_words: the words that the launch counts in (a.barrier first), cleared here.
inline int small_launch(SmallArgs& a, int ld, size_t sync_words, cudaStream_t st, bool refuse, bool* made) {
    DN_CUDA(cudaMemsetAsync(a.barrier, 0, sync_words * sizeof(unsigned int), st));
    // (at the wide strides also a block for every chunk of the Gram matrices)
    const uint32_t chunks = ld > 64 ? (uint32_t)(ld * ld / 128) : 1;
    const int blocks = (int)std::min<uint32_t>(kNumSMs, std::max(chunks, std::max(a.side[0].workers, a.side[1].workers)));
    a.side[0].partials = (int)std::min<uint32_t>(a.side[1].workers, (uint32_t)blocks);
    a.side[1].partials = (int)std::min<uint32_t>(a.side[0].workers, (uint32_t)blocks);
    switch (ld) {
        case 32: return small_launch_t<32>(a, blocks, st, refuse, made);
        case 64: return small_launch_t<64>(a, blocks, st, refuse, made);
        case 96: return small_launch_t<96>(a, blocks, st, refuse, made);
        default: return small_launch_t<128>(a, blocks, st, refuse, made);
    }
}

}  // namespace dnpeff

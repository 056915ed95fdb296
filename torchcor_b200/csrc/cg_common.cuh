// Grid-barrier and reduction helpers shared by the persistent CG kernels.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "tcb200.h"

namespace tcb {
namespace cgk {

constexpr int kCgThreads = 512;
constexpr int kCgWarps = kCgThreads / 32;
constexpr int kMinSlicesPerBlock = 2 * kCgWarps;
constexpr int kMaxBlocks = 2048;
constexpr uint64_t kBarrierTimeoutNs = 2000000000ull;  // 2 s: a wait that long means a lost block

// Limits of the bounded device waits (grid barriers, bulk-copy mbarriers).
// In normal runs: the 2 s timeout and nothing else.  The failure-detection
// tests set TCB_TEST_WAIT_STALL (wait_limit() in api.cu): then the timeout is
// 10 ms and either every grid barrier waits for one arrival more than the grid
// has ("grid") or the first bulk copies of the batched kernels' first warp or
// block are not made while their mbarrier still expects the bytes ("copy"), so
// that a wait runs out, the error word is set and every block returns.
struct WaitLimit {
    uint64_t timeout_ns;
    uint32_t extra_arrivals;
    uint32_t drop_first_copy;
};

__device__ __forceinline__ uint64_t globaltimer() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Grid-wide barrier with a bounded wait.  bar[2] counts arrivals and only ever
// grows (modulo 2^32); bar[3] is its value between launches, which every block
// reads as it starts and block 0 writes as it ends.  A block arrives with an add
// that returns nothing and polls the same word until all have: a fence, an add and a
// poll, where a counter with a generation beside it took two round trips more (the
// add's result, and the last arrival's second add).  On B200 the last arrival is
// seen after 1.3 us, before 2.6.
struct GridWait {
    uint32_t* word;
    uint32_t target;
    int32_t* err;
    WaitLimit lim;
};
__device__ __forceinline__ GridWait grid_wait_begin(uint32_t* bar, int32_t* err, const WaitLimit& w) {
    return GridWait{bar + 2, bar[3], err, w};
}
// (a launch whose wait ran out leaves its error word set, and nothing runs after that)
__device__ __forceinline__ void grid_wait_end(const GridWait& g, uint32_t* bar) {
    if (blockIdx.x == 0 && threadIdx.x == 0) bar[3] = g.target;
}

// One thread's part; false if the wait ran past the limit or, while waiting, another
// block recorded an error (reading the error word after every barrier would cost a
// round trip; a block that gave up is missing at the next one).
__device__ __forceinline__ bool grid_arrive_and_wait(const GridWait& g) {
    asm volatile("fence.acq_rel.gpu;" ::: "memory");   // the block's writes before its arrival
    asm volatile("red.relaxed.gpu.global.add.u32 [%0], 1;" ::"l"(g.word) : "memory");
    const uint32_t target = g.target + g.lim.extra_arrivals;
    uint64_t t0 = 0;
    for (int spin = 1;; ++spin) {
        uint32_t v;
        asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(g.word) : "memory");
        if ((int32_t)(v - target) >= 0) break;
        if ((spin & 31) == 0) {
            if (*(volatile int32_t*)g.err != 0) return false;
            const uint64_t now = globaltimer();
            if (t0 == 0) t0 = now;
            if (now - t0 > g.lim.timeout_ns) {
                atomicCAS(g.err, 0, TCB_ETIMEOUT);
                return false;
            }
        }
    }
    asm volatile("fence.acq_rel.gpu;" ::: "memory");
    return true;
}

// Every block's earlier writes are visible to every block after it; false: return.
__device__ __forceinline__ bool grid_barrier(GridWait& g) {
    __syncthreads();
    g.target += gridDim.x;
    int bad = 0;
    if (threadIdx.x == 0) bad = !grid_arrive_and_wait(g);
    return !__syncthreads_or(bad);
}

// The barrier with the totals over all threads of NV (4 or 8) float64 values, in
// sh.total[0..NV) after it.  A warp's values are added by halving exchanges (each step
// hands half of the values to the partner lane), the warps' by warp 0; after the
// barrier warp j adds the blocks' value j.  parts: NV * SLOTS doubles, at least
// gridDim.x slots; two alternating sets of them.
template <int NV>
struct GridSums {
    double part[kCgWarps][NV];
    double total[NV];
};
// every warp: its lanes' values into sh.part[warp]
template <int NV>
__device__ __forceinline__ void fold_warps(const double (&v)[NV], GridSums<NV>& sh) {
    static_assert(NV == 4 || NV == 8, "exchange pattern");
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double a[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) a[i] = v[i];
    int bit = 16;
#pragma unroll
    for (int half = NV / 2; half > 0; half >>= 1, bit >>= 1) {
        const bool up = lane & bit;
#pragma unroll
        for (int i = 0; i < half; ++i) {
            const double give = up ? a[i] : a[i + half], mine = up ? a[i + half] : a[i];
            a[i] = mine + __shfl_xor_sync(0xffffffffu, give, bit);
        }
    }
#pragma unroll
    for (; bit > 0; bit >>= 1) a[0] += __shfl_xor_sync(0xffffffffu, a[0], bit);
    // value (bits 4, 3[, 2] of the lane) is complete in every lane
    if ((lane & (32 / NV - 1)) == 0) sh.part[warp][lane / (32 / NV)] = a[0];
}
// one warp, after the block has met: the block's value lane % NV, in every lane
template <int NV>
__device__ __forceinline__ double fold_block(const GridSums<NV>& sh) {
    constexpr int kPer = kCgWarps * NV / 32;   // warps a lane adds
    const int lane = threadIdx.x & 31, q = lane % NV, w = lane / NV * kPer;
    double t = sh.part[w][q];
#pragma unroll
    for (int j = 1; j < kPer; ++j) t += sh.part[w + j][q];
#pragma unroll
    for (int o = NV; o < 32; o <<= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    return t;
}
template <int NV, int SLOTS>
__device__ __forceinline__ bool grid_barrier_sums(const double (&v)[NV], GridSums<NV>& sh, double* parts, GridWait& g) {
    static_assert(SLOTS % 32 == 0, "whole strides");
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    fold_warps<NV>(v, sh);
    __syncthreads();
    g.target += gridDim.x;
    int bad = 0;
    if (warp == 0) {
        const double t = fold_block<NV>(sh);
        if (lane < NV) parts[lane * SLOTS + blockIdx.x] = t;
        __syncwarp();
        if (lane == 0) bad = !grid_arrive_and_wait(g);
    }
    if (__syncthreads_or(bad)) return false;
    if (warp < NV) {
        double t[SLOTS / 32];
#pragma unroll
        for (int k = 0; k < SLOTS / 32; ++k) {
            const int i = lane + 32 * k;
            t[k] = i < (int)gridDim.x ? __ldcg(parts + warp * SLOTS + i) : 0.0;
        }
        double sum = 0.0;
#pragma unroll
        for (int k = 0; k < SLOTS / 32; ++k) sum += t[k];
        sum = warp_sum(sum);
        if (lane == 0) sh.total[warp] = sum;
    }
    __syncthreads();
    return true;
}

// Block partial of NV float64 values -> parts[blockIdx.x * NV + i] (fixed order).
template <int NV>
__device__ __forceinline__ void block_partial(double (&v)[NV], double* parts, double* sh) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        double t = warp_sum(v[i]);
        if (lane == 0) sh[warp * NV + i] = t;
    }
    __syncthreads();
    if (warp == 0) {
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            double t = lane < kCgWarps ? sh[lane * NV + i] : 0.0;
            t = warp_sum(t);
            if (lane == 0) parts[blockIdx.x * NV + i] = t;
        }
    }
}

// Sum of all blocks' partials; every block computes the same value.  Each lane
// adds the partials of blocks lane, lane + 32, ... in that order; the loads of
// eight strides are issued before their adds, so a lane waits for one L2 round
// trip per eight strides instead of one per stride (same sums, bit for bit).
template <int NV>
__device__ __forceinline__ void grid_total(const double* parts, double (&out)[NV], double* sh) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warp == 0) {
        constexpr int kBatch = 8;
        double acc[NV];
#pragma unroll
        for (int i = 0; i < NV; ++i) acc[i] = 0.0;
        const unsigned nb = gridDim.x;
        unsigned b = lane;
        for (; b + 32 * (kBatch - 1) < nb; b += 32 * kBatch) {
            double t[kBatch][NV];
#pragma unroll
            for (int k = 0; k < kBatch; ++k)
#pragma unroll
                for (int i = 0; i < NV; ++i) t[k][i] = __ldcg(parts + (b + 32 * k) * NV + i);
#pragma unroll
            for (int k = 0; k < kBatch; ++k)
#pragma unroll
                for (int i = 0; i < NV; ++i) acc[i] += t[k][i];
        }
        for (; b < nb; b += 32)
#pragma unroll
            for (int i = 0; i < NV; ++i) acc[i] += __ldcg(parts + b * NV + i);
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            acc[i] = warp_sum(acc[i]);
            if (lane == 0) sh[i] = acc[i];
        }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < NV; ++i) out[i] = sh[i];
}

}  // namespace cgk
}  // namespace tcb

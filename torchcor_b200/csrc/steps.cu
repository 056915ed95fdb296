// Many time steps of one simulation in one persistent cooperative launch.
//
// Small and middle-sized meshes are bound by latency: launches, grid barriers
// and the chain column -> neighbour -> sum.  Here one launch runs a whole
// stretch of steps (ionic update, right-hand side, Jacobi-PCG of
// torchcor/core/solver.py:40-76) and keeps what the steps share on chip: a block
// owns a contiguous range of rows; the solution, the CG vectors, the rows'
// columns and matrix values and (where it fits) the ionic state stay in its shared
// memory from step to step.  Blocks exchange
// one 16-byte record per row through L2: {b', u, x0} for the right-hand side and
// {r, p, A p, 1/diag} between CG passes; records of the block's own rows are
// read from shared memory.
//
// Grid barriers: a step needs one after the ionic update, one after the
// right-hand side (z of the neighbours) and one per CG pass.
//  * Arrivals are counted in a word that only grows, so a barrier is a fence, an
//    add without a result and a poll.  (Every block polling a flag word of every
//    other one, with the partial sums in the words, has a round trip less but
//    measured 4.7 us at 148 blocks: they all read the same lines.)
//  * One barrier per CG pass: the sums a pass takes over r, p and A p give alpha
//    and, by the identities
//      |z'|^2 = |z|^2 - 2 alpha (D r, D A p) + alpha^2 |D A p|^2,
//      (r', z') = (r, z) - 2 alpha (z, A p) + alpha^2 (A p, D A p),
//    the stopping test and beta of the same pass (float64 throughout; every pass
//    sums r and z anew, so nothing accumulates).  The next pass forms r', z' and p'
//    of its own and its neighbours' rows from the records with the same roundings.
//
// What bounds it: the chain of latencies of a step (three grid barriers of about
// 1.7 us, one of them with the sums 2.3 us; the ionic update's table reads 1-3 us;
// column, gather and sum of a row 1-2 us a pass), not bytes.  Measured on B200, us a
// step with x CG iterations, the two launches of a step replayed as a CUDA graph ->
// here: TTP cube 1,000 nodes (1.15) 26 -> 10.7 (a cluster); MS cube 9,261 (0.4) 34.9 -> 12.1; TTP
// cube 50,653 (1) 43.1 -> 17.7, 117,649 (0.8) 48.6 -> 26.0; CRN shell 40,962 (1) 36.6
// -> 15.8, 163,842 (1) 51.7 -> 31.8.  The line to the two-launch form lies where the
// matrix no longer fits (about 170,000 nodes of a tetrahedral mesh): reading it from
// L2 instead, 262,144 nodes took 59.9 us here and 49.1 in two launches.
//
// The smallest meshes run as one thread-block cluster instead of a grid: its barrier
// is the hardware's, sums and neighbours' records travel through distributed shared
// memory and nothing goes through L2.  (A neighbour in the block itself is read the
// same way: telling it apart with a predicate took half as long again.)
//
// Sums inside a row run in the order of the other CG kernels (M b' and K u in
// float32, A x0 and A p in float64); sums over rows are float64 in an order that
// depends on the launch shape only.
#include <cuda_runtime.h>
#include <math.h>

#include <algorithm>
#include <type_traits>
#include <vector>

#include "cg_common.cuh"
#include "ionic_crn.cuh"
#include "ionic_ms.cuh"
#include "ionic_node.cuh"
#include "ionic_ttp.cuh"
#include "mono.cuh"
#include "tcb_internal.h"

namespace tcb {
int validate_mono(const tcb_mono* m);
namespace {

using namespace cgk;

constexpr int kThreads = kCgThreads;
constexpr int kWarps = kCgWarps;
constexpr int kSums = 8;                  // sums of a CG pass (see pass_sums)
constexpr int kSlots = 160;               // most blocks of a launch
constexpr size_t kHeadBytes = 256;        // barrier words
constexpr size_t kPartBytes = 2 * (size_t)kSums * kSlots * sizeof(double);

// no ionic update: b' comes from the caller (tcb_mono_cg_run)
struct GivenRhs {
    static constexpr bool kIonic = false;
};
template <class M, class Q>
struct Ionic {
    static constexpr bool kIonic = true;
    static constexpr int kStates = M::kStates;
    using Model = M;
    using Policy = Q;
    typename M::C c;
    typename M::Tables T;
};

struct StepsPlan {
    int32_t n_steps, blocks, cluster;              // cluster: the blocks are one cluster
    int32_t cap_rows, cap_entries;                 // rows and matrix entries a block has at most
    int32_t smem_bytes, held_at, state_at;         // byte offsets of the matrix and the state (0: not held)
    uint32_t* bar;                                 // barrier words (GridWait)
    double* parts;                                 // [2 parities][kSums][kSlots] block sums
    float4* rec[2];                                // per-row records, n_pad each
};

// alpha as a pair of float32 (high and low part) for advance()
struct Alpha {
    float hi, lo;
};
__device__ __forceinline__ Alpha split(double alpha) {
    Alpha a;
    a.hi = (float)alpha;
    a.lo = (float)(alpha - (double)a.hi);
    return a;
}

// r' = r - alpha A p, z' = D r', p' = z' + beta p of a row from its record
// {r, p, A p, 1/diag}.  Every row that needs p' of a neighbour forms it, so the
// conversions to float64 that r' would take (8.5 cycles of a scheduler each, three for
// r' alone) weigh more than the sum: r' is taken from the exact product and sum in
// float32 pairs instead (Dekker 1971, Knuth's two-sum), right to about 2^-46 of
// |r| + |alpha A p| before its one rounding.  z' is one rounding of an exact product in
// either form.  Against the same kernel with r' formed in float64, the errors of 24
// extracellular recoveries (cubes of 2,197 to 195,112 nodes) and 13 runs against 64 bits
// are equal (ratios 1.000, spread 0.001), and the pairs are faster: recovery of 68,921
// nodes 12.8 -> 11.8 ms, CRN shell 40,962 18.1 -> 16.9, TTP cube 50,653 19.8 -> 19.2.
__device__ __forceinline__ void advance(const float4& f, const Alpha& alpha, float beta, float& r, float& z, float& p) {
    const float h = __fmul_rn(alpha.hi, f.z);
    const float l = __fmaf_rn(alpha.lo, f.z, __fmaf_rn(alpha.hi, f.z, -h));
    const float s = __fsub_rn(f.x, h);
    const float t = __fsub_rn(s, f.x);
    const float e = __fsub_rn(__fsub_rn(f.x, __fsub_rn(s, t)), __fadd_rn(h, t));
    r = __fadd_rn(s, __fsub_rn(e, l));
    z = __fmul_rn(f.w, r);
    p = __fmaf_rn(beta, f.y, z);
}

// The sums of one CG pass for a row.  All are of the unrounded D r and D A p: where
// |z'| is far below |z| the identities cancel, and sums over the rounded z beside
// unrounded products would leave 1e-5 of |z'|^2.
__device__ __forceinline__ void pass_sums(double (&s)[kSums], float r, float p, float ap, float di) {
    const double d_ap = (double)ap, d_r = (double)r, dap = (double)di * d_ap, dr = (double)di * d_r;
    s[0] += (double)p * d_ap;
    s[1] += dr * d_ap;
    s[2] += dap * d_ap;
    s[3] += dr * dap;
    s[4] += dap * dap;
    s[5] += dr * d_r;
    s[6] += dr * dr;
}

// copy `bytes` (a multiple of 64; both sides 16-byte aligned) into shared memory, whole block
__device__ __forceinline__ void hold(void* dst, const void* src, size_t bytes) {
    for (size_t i = threadIdx.x; i < bytes / 16; i += kThreads)
        static_cast<uint4*>(dst)[i] = static_cast<const uint4*>(src)[i];
}

// Address in the cluster's shared memory of what is at `local` in this block's.
__device__ __forceinline__ uint32_t peer_address(const void* local, uint32_t rank) {
    uint32_t a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((uint32_t)__cvta_generic_to_shared(local)), "r"(rank));
    return a;
}
__device__ __forceinline__ void peer_load(float& v, uint32_t a) {
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a));
}
__device__ __forceinline__ void peer_load(float4& v, uint32_t a) {
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a));
}
__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}

// The block's part of the matrix in shared memory and where its neighbours' values
// are.  CL: the blocks are one cluster, and a column is (block << 16 | row of the block).
template <typename IDX, bool CL>
struct Rows {
    const std::conditional_t<CL, uint32_t, IDX>* col;   // int16: column - row; int32: column
    const float *m, *k, *a;
    int row0, rows;
    float cm;
    __device__ __forceinline__ int column(int e, int i) const {
        return !CL && sizeof(IDX) == 2 ? row0 + i + (int)col[e] : (int)col[e];
    }
    // a neighbour's value: from the shared memory of its block (CL); else the block's own rows from
    // shared memory, others through L1
    template <class T>
    __device__ __forceinline__ T value(const T* own, const T* all, int c) const {
        if constexpr (CL) {
            T v;
            peer_load(v, peer_address(own + (c & 0xffff), (uint32_t)c >> 16));
            return v;
        }
        const int l = c - row0;
        const T* p = (unsigned)l < (unsigned)rows ? own + l : all + c;
        return *p;
    }
};

// grid_barrier_sums among the blocks of one cluster: warp 0 hands the block's sums to
// every block, and each adds them in block order.
constexpr int kMaxCluster = 16;
struct ClusterSums {
    double from[2][kMaxCluster][kSums];
};
__device__ __forceinline__ void cluster_barrier_sums(double (&v)[kSums], GridSums<kSums>& sh, ClusterSums& cs, int parity) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nb = (int)gridDim.x;
    fold_warps<kSums>(v, sh);
    __syncthreads();
    if (warp == 0) {
        const double t = fold_block<kSums>(sh);   // value lane % kSums, in every lane
        for (int r = lane / kSums; r < nb; r += 32 / kSums)
            asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(peer_address(&cs.from[parity][blockIdx.x][lane % kSums], (uint32_t)r)),
                         "d"(t)
                         : "memory");
    }
    cluster_barrier();
    if (warp < kSums) {
        double t = lane < nb ? cs.from[parity][lane][warp] : 0.0;
#pragma unroll
        for (int o = kMaxCluster / 2; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (lane == 0) sh.total[warp] = t;
    }
    __syncthreads();
}

// Entries 0 .. w-1 of a row, C at a time, without branches: entries past the end
// repeat the last one with a coefficient of zero.  All C gathers are in flight
// before the first is used.
template <int C, bool ASPLIT, typename IDX, bool CL>
__device__ __forceinline__ void row_rhs(const Rows<IDX, CL>& R, const float4* own, const float4* all, int base, int w, int i,
                                        float& mb, float& ku, double& ax) {
    for (int k0 = 0; k0 < w; k0 += C) {
        float4 q[C];
#pragma unroll
        for (int j = 0; j < C; ++j) q[j] = R.value(own, all, R.column(base + min(k0 + j, w - 1) * TCB_SLICE, i));
#pragma unroll
        for (int j = 0; j < C; ++j) {
            const bool ok = k0 + j < w;
            const int e = base + min(k0 + j, w - 1) * TCB_SLICE;
            const float m = ok ? R.m[e] : 0.0f, k = ok ? R.k[e] : 0.0f;
            float a;
            if constexpr (ASPLIT) a = __fadd_rn(__fmul_rn(m, R.cm), k);
            else a = ok ? R.a[e] : 0.0f;
            mb = __fmaf_rn(m, q[j].x, mb);
            ku = __fmaf_rn(k, q[j].y, ku);
            ax += (double)a * (double)q[j].z;
        }
    }
}

template <bool ASPLIT, typename IDX, bool CL>
__device__ __forceinline__ float coefficient(const Rows<IDX, CL>& R, int e) {
    if constexpr (ASPLIT) return __fadd_rn(__fmul_rn(R.m[e], R.cm), R.k[e]);
    else return R.a[e];
}

template <int C, bool ASPLIT, typename IDX, bool CL>
__device__ __forceinline__ double row_first(const Rows<IDX, CL>& R, const float* own, const float* all, int base, int w, int i) {
    double acc = 0.0;
    for (int k0 = 0; k0 < w; k0 += C) {
        float z[C];
#pragma unroll
        for (int j = 0; j < C; ++j) z[j] = R.value(own, all, R.column(base + min(k0 + j, w - 1) * TCB_SLICE, i));
#pragma unroll
        for (int j = 0; j < C; ++j) {
            const float a = coefficient<ASPLIT>(R, base + min(k0 + j, w - 1) * TCB_SLICE);
            acc += (double)(k0 + j < w ? a : 0.0f) * (double)z[j];
        }
    }
    return acc;
}

template <int C, bool ASPLIT, typename IDX, bool CL>
__device__ __forceinline__ double row_next(const Rows<IDX, CL>& R, const float4* own, const float4* all, int base, int w, int i,
                                           const Alpha& alpha, float beta) {
    double acc = 0.0;
    for (int k0 = 0; k0 < w; k0 += C) {
        float4 f[C];
#pragma unroll
        for (int j = 0; j < C; ++j) f[j] = R.value(own, all, R.column(base + min(k0 + j, w - 1) * TCB_SLICE, i));
#pragma unroll
        for (int j = 0; j < C; ++j) {
            const float a = coefficient<ASPLIT>(R, base + min(k0 + j, w - 1) * TCB_SLICE);
            float r, z, p;
            advance(f[j], alpha, beta, r, z, p);
            acc += (double)(k0 + j < w ? a : 0.0f) * (double)p;
        }
    }
    return acc;
}

template <typename IDX, bool ASPLIT, bool CL, class ION>
__global__ void __launch_bounds__(kThreads, 1) mono_steps_kernel(MonoDev d, const IDX* __restrict__ col, StepsPlan pl,
                                                                 ION ion) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ GridSums<kSums> sh;
    __shared__ std::conditional_t<CL, ClusterSums, char> cs;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t s_begin = (int64_t)blockIdx.x * d.n_slices / gridDim.x;
    const int64_t s_end = (int64_t)(blockIdx.x + 1) * d.n_slices / gridDim.x;
    const int slices = (int)(s_end - s_begin);
    const int row0 = (int)s_begin * TCB_SLICE;
    const int rows = (int)((d.n < s_end * TCB_SLICE ? d.n : s_end * TCB_SLICE) - row0);
    int32_t* err = d.counter + 1;
    const int first_step = d.counter[0];
    GridWait g = grid_wait_begin(pl.bar, err, d.wait);
    int parity = 0;
    if (*(volatile int32_t*)err != 0) return;

    // ---- shared memory (steps_layout): records, solutions, z, slice offsets, matrix, ionic state
    const int cap = pl.cap_rows;
    float4* rec0 = reinterpret_cast<float4*>(smem);
    float4* rec1 = rec0 + cap;
    float* sx = reinterpret_cast<float*>(rec1 + cap);
    float* sxp = sx + cap;
    float* sz = sxp + cap;
    int* off = reinterpret_cast<int*>(sz + cap);
    unsigned char* held = smem + pl.held_at;
    const size_t vals = (size_t)pl.cap_entries * 4;
    float* sm = reinterpret_cast<float*>(held);
    float* sk = reinterpret_cast<float*>(held + vals);
    float* sa = ASPLIT ? sk : reinterpret_cast<float*>(held + 2 * vals);
    using COL = std::conditional_t<CL, uint32_t, IDX>;
    COL* sc = reinterpret_cast<COL*>(held + (ASPLIT ? 2 : 3) * vals);
    float* ss = reinterpret_cast<float*>(smem + pl.state_at);
    const int64_t e0 = d.slice_ptr[s_begin];
    const size_t ent = (size_t)(d.slice_ptr[s_end] - e0);   // multiple of 32, at most cap_entries
    if constexpr (!CL) hold(sc, col + e0, ent * sizeof(IDX));
    hold(sm, d.mv + e0, ent * 4);
    hold(sk, d.kv + e0, ent * 4);
    if (!ASPLIT) hold(sa, d.av + e0, ent * 4);
    const bool state_held = pl.state_at != 0;
    if constexpr (ION::kIonic) {
        if (state_held)
            for (int k = 0; k < ION::kStates; ++k)
                for (int i = threadIdx.x; i < rows; i += kThreads) ss[k * cap + i] = d.state[k * d.n_pad + row0 + i];
    }
    for (int i = threadIdx.x; i <= slices; i += kThreads) off[i] = (int)(d.slice_ptr[s_begin + i] - e0);
    for (int i = threadIdx.x; i < rows; i += kThreads) {
        sx[i] = d.x[ring_cur(first_step) * d.n_pad + row0 + i];
        sxp[i] = d.x[ring_prev(first_step) * d.n_pad + row0 + i];
        rec0[i].w = d.dinv[row0 + i];
    }
    __syncthreads();
    if constexpr (CL) {
        // columns as (block, row of the block): block b has the slices from b*S/nb on
        const uint32_t S = (uint32_t)d.n_slices, nb = gridDim.x;
        for (int s = warp; s < slices; s += kWarps)
            for (int e = off[s] + lane; e < off[s + 1]; e += TCB_SLICE) {
                const uint32_t c = (uint32_t)(row0 + s * TCB_SLICE + lane + (int)col[e0 + e]);
                const uint32_t b = ((c / TCB_SLICE + 1) * nb - 1) / S;
                sc[e] = b << 16 | (c - b * S / nb * TCB_SLICE);
            }
    }

    const Rows<IDX, CL> R{sc, sm, sk, sa, row0, rows, d.cm};
    const bool lg = d.linear_guess != 0;
    float* zg = d.r;
    float4* q4 = pl.rec[1];        // {b', u, x0, -}; read before the first pass that writes rec[1]
    const int last_step = first_step + pl.n_steps;
    const double stop_a = d.a_tol > 0.0 ? d.a_tol * d.a_tol : 0.0;
    // (the barriers of a cluster are the hardware's and need no limit)
    auto barrier = [&] {
        if constexpr (CL) {
            cluster_barrier();
            return true;
        } else {
            return grid_barrier(g);
        }
    };
    auto barrier_sums = [&](double (&v)[kSums]) {
        parity ^= 1;
        if constexpr (CL) {
            cluster_barrier_sums(v, sh, cs, parity);
            return true;
        } else {
            return grid_barrier_sums<kSums, kSlots>(v, sh, pl.parts + (size_t)parity * kSums * kSlots, g);
        }
    };
    for (int n = first_step; n < last_step; ++n) {
        // ---- ionic update of the block's rows, b', guess (monodomain.py:117-128, solver.py:35-38)
        {
            StepView sv;
            if constexpr (ION::kIonic) sv = step_view(d, n);
            for (int i = threadIdx.x; i < rows; i += kThreads) {
                const float u = sx[i];
                float bp;
                if constexpr (ION::kIonic) {
                    using M = typename ION::Model;
                    using Q = typename ION::Policy;
                    const int row = row0 + i;
                    if (sv.do_atrt) at_rt_update(u, sv.t_prev, d.at, d.rt, row);
                    if (sv.snap) sv.snap[row] = u;
                    float s[M::kStates];
                    if (state_held) {
#pragma unroll
                        for (int k = 0; k < M::kStates; ++k) s[k] = ss[k * cap + i];
                    } else {
#pragma unroll
                        for (int k = 0; k < M::kStates; ++k) s[k] = d.state[k * d.n_pad + row];
                    }
                    const float dV = M::template step<Q>(u, s, ion.c, ion.T, M::node_g(ion.c, d.node_params, d.n_pad, row));
                    if (state_held) {
#pragma unroll
                        for (int k = 0; k < M::kStates; ++k) ss[k * cap + i] = s[k];
                    } else {
#pragma unroll
                        for (int k = 0; k < M::kStates; ++k) d.state[k * d.n_pad + row] = s[k];
                    }
                    bp = u * d.cm + d.dt * Q::div(dV, 100.0f);
                    if (sv.smask) {
                        const uint32_t bits = d.stim_bits[row] & sv.smask;
                        if (bits) bp = bp + d.dt * Q::div(stim_sum(d, sv.smask, bits), 100.0f);
                    }
                } else {
                    bp = d.bp[row0 + i];
                }
                const float4 q = make_float4(bp, u, lg ? 2.0f * u - sxp[i] : u, 0.0f);
                rec1[i] = q;
                if constexpr (!CL) q4[row0 + i] = q;
            }
        }
        if (!barrier()) return;

        // ---- right-hand side, r0, z0 (monodomain.py:130-131, solver.py:46-55)
        double sums[kSums];
#pragma unroll
        for (int j = 0; j < kSums; ++j) sums[j] = 0.0;
        for (int s = warp; s < slices; s += kWarps) {
            const int i = s * TCB_SLICE + lane;
            if (i >= rows) continue;
            const int base = off[s] + lane, w = (off[s + 1] - off[s]) / TCB_SLICE;
            float mb = 0.0f, ku = 0.0f;
            double ax = 0.0;
            if (w <= 8) row_rhs<8, ASPLIT>(R, rec1, q4, base, w, i, mb, ku, ax);
            else row_rhs<16, ASPLIT>(R, rec1, q4, base, w, i, mb, ku, ax);
            const float4 own = rec1[i];
            sxp[i] = own.y;
            sx[i] = own.z;
            const float rhs = mb - ku;
            const float di = rec0[i].w;
            const float r = (float)((double)rhs - ax);
            const float z = __fmul_rn(di, r);
            rec0[i].x = r;
            sz[i] = z;
            if constexpr (!CL) zg[row0 + i] = z;
            const double db = (double)di * (double)rhs;
            sums[7] += db * db;
        }
        if (!barrier()) return;

        int it = 0;
        Alpha alpha = {0.0f, 0.0f};
        double stop_b = 0.0;   // (r_tol |D b|)^2
        bool zero_stops = false;
        float beta = 0.0f;
        while (it < d.max_iter) {
            // ---- p, A p; the sums that give alpha, beta and the stopping test
            float4* rout = (it & 1) ? rec1 : rec0;
            const float4* rin = (it & 1) ? rec0 : rec1;
            float4* gout = pl.rec[it & 1];
            const float4* gin = pl.rec[(it & 1) ^ 1];
            for (int s = warp; s < slices; s += kWarps) {
                const int i = s * TCB_SLICE + lane;
                if (i >= rows) continue;
                const int base = off[s] + lane, w = (off[s + 1] - off[s]) / TCB_SLICE;
                float r, z, p, ap, di;
                if (it == 0) {
                    r = rec0[i].x;
                    di = rec0[i].w;
                    p = z = sz[i];
                    ap = (float)(w <= 8 ? row_first<8, ASPLIT>(R, sz, zg, base, w, i)
                                        : row_first<16, ASPLIT>(R, sz, zg, base, w, i));
                } else {
                    const float4 f = rin[i];
                    di = f.w;
                    advance(f, alpha, beta, r, z, p);
                    ap = (float)(w <= 8 ? row_next<8, ASPLIT>(R, rin, gin, base, w, i, alpha, beta)
                                        : row_next<16, ASPLIT>(R, rin, gin, base, w, i, alpha, beta));
                }
                pass_sums(sums, r, p, ap, di);
                const float4 out = make_float4(r, p, ap, di);
                rout[i] = out;
                if constexpr (!CL) gout[row0 + i] = out;
            }
            if (!barrier_sums(sums)) return;
            const double rz = sh.total[5];
            if (it == 0) {
                stop_b = d.r_tol > 0.0 ? d.r_tol * d.r_tol * sh.total[7] : 0.0;
                zero_stops = d.a_tol > 0.0 || (d.r_tol > 0.0 && sh.total[7] > 0.0);
            }
            const double al = rz / sh.total[0];
            alpha = split(al);
            double zz = sh.total[6] - al * (2.0 * sh.total[3] - al * sh.total[4]);
            if (zz < 0.0) zz = 0.0;
            const double rz1 = rz - al * (2.0 * sh.total[1] - al * sh.total[2]);
            for (int s = warp; s < slices; s += kWarps) {
                const int i = s * TCB_SLICE + lane;
                if (i < rows) sx[i] = (float)((double)sx[i] + al * (double)rout[i].y);
            }
            // |z'| below a_tol or r_tol |D b| (solver.py:66-69), squared
            if (zz < stop_a || zz < stop_b || (zz == 0.0 && zero_stops)) break;
            beta = (float)(rz1 / rz);
            ++it;
#pragma unroll
            for (int j = 0; j < kSums; ++j) sums[j] = 0.0;
        }
        // the last three solutions of the stretch go to the ring (the next launch
        // needs two of them; a shorter stretch leaves the older slots as they are)
        if (n >= last_step - 3) {
            float* xout = d.x + ring_next(n) * d.n_pad + row0;
            for (int s = warp; s < slices; s += kWarps) {
                const int i = s * TCB_SLICE + lane;
                if (i < rows) xout[i] = sx[i];
            }
        }
        if (blockIdx.x == 0 && threadIdx.x == 0) d.step_iters[n] = it;
    }
    if constexpr (ION::kIonic) {
        if (state_held)
            for (int k = 0; k < ION::kStates; ++k)
                for (int i = threadIdx.x; i < rows; i += kThreads) d.state[k * d.n_pad + row0 + i] = ss[k * cap + i];
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        d.counter[0] = last_step;
    }
    if constexpr (!CL) grid_wait_end(g, pl.bar);
}

// ---------------------------------------------------------------- launch
struct StepsInfo {
    int sms = 0, max_smem = 0;
};
StepsInfo steps_info() {
    static PerDevice<StepsInfo> infos;
    return infos.get([](StepsInfo& si, int dev) {
        if (cudaDeviceGetAttribute(&si.max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess ||
            cudaDeviceGetAttribute(&si.sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
            return false;
        si.max_smem -= (int)(sizeof(GridSums<kSums>) + sizeof(ClusterSums)) + 1024;
        return true;
    });
}

constexpr int kMinSlices = 8;              // slices a block has at least
constexpr int kHoldStateFrom = 4;          // shorter launches update the ionic state where it is
constexpr int64_t kStepsPerLaunch = 128;   // about a millisecond or a few: other streams get their turn
// Meshes of up to this many slices (4,608 nodes) run as one cluster of at most 16
// blocks.  us a step with x CG iterations, grid -> cluster: TTP cube 1,000 nodes (1.15)
// 14.4 -> 10.7, 2,197 (2.1) 18.7 -> 14.1, 4,096 (1.75) 19.3 -> 15.6; beyond, the rows of a
// block weigh more than the barriers: 6,859 (1.4) 17.3 -> 19.0, MS 9,261 (0) 10.1 -> 12.5.
constexpr int kClusterSlices = 144;
constexpr int32_t kClusterWork = 1 << 30;  // tcb_mono.work_entries: entries are counted for a cluster's blocks

bool aligned16(const void* p) { return ((uintptr_t)p & 15u) == 0; }

int64_t steps_blocks(const MonoDev& d, bool cluster) {
    const int64_t nb = std::max<int64_t>(ceil_div(d.n_slices, kMinSlices), 1);
    if (!cluster) return std::min<int64_t>(nb, std::max(1, std::min(steps_info().sms, kSlots)));
    int64_t p = 1;
    while (p < nb && p < kMaxCluster) p *= 2;
    return std::min(p, d.n_slices);
}

// Shared memory of a block with at most `entries` matrix entries; false where it
// does not fit (the matrix has to; the ionic state stays in global memory if need be).
bool steps_layout(const MonoDev& d, int64_t blocks, int64_t entries, int states, bool cluster, StepsPlan* pl) {
    const size_t max = (size_t)steps_info().max_smem;
    auto up = [](size_t b) { return (b + 127) / 128 * 128; };
    const int64_t cap = ceil_div(d.n_slices, blocks) * TCB_SLICE;
    const size_t fixed = (size_t)cap * 44 + up((size_t)(cap / TCB_SLICE + 1) * 4);
    const size_t per_entry = (d.a_split ? 8 : 12) + (d.dcol && !cluster ? 2 : 4);
    const size_t matrix = up((size_t)entries * per_entry), state = (size_t)cap * 4 * states;
    if (cap > 16384 || entries > (1 << 20) || fixed + matrix > max) return false;
    pl->blocks = (int)blocks;
    pl->cluster = cluster;
    pl->cap_rows = (int)cap;
    pl->cap_entries = (int)entries;
    pl->held_at = (int)fixed;
    pl->state_at = states > 0 && fixed + matrix + state <= max ? (int)(fixed + matrix) : 0;
    pl->smem_bytes = (int)(fixed + matrix + (pl->state_at ? state : 0));
    return true;
}

// false where the step-by-step launches run instead
bool steps_plan(const tcb_mono* m, const MonoDev& d, bool ionic, int states, StepsPlan* pl) {
    if (!m->work || m->work_entries <= 0 || m->fused_step != 0 || cg_forced_fallback()) return false;
    const bool as_cluster = (m->work_entries & kClusterWork) != 0;
    // the blocks counted for a cluster also run as a grid: where the cluster form is not compiled (ionic
    // steps whose A is not M Cm + K': theta 0.25, TTP cube 1,000 nodes 8.7 us a step against 17.9 in two
    // launches, 4,096 nodes 18.9 against 35.4; a grid of its own would have 18 blocks instead of 16 at
    // most), and for the tests that let a grid barrier's wait run out
    const bool cluster = as_cluster && (d.a_split || !ionic) && d.wait.extra_arrivals == 0;
    if (!steps_layout(d, steps_blocks(d, as_cluster), m->work_entries & ~kClusterWork, states, cluster, pl)) return false;
    unsigned char* w = static_cast<unsigned char*>(m->work);
    pl->bar = reinterpret_cast<uint32_t*>(w);
    pl->parts = reinterpret_cast<double*>(w + kHeadBytes);
    pl->rec[0] = reinterpret_cast<float4*>(w + kHeadBytes + kPartBytes);
    pl->rec[1] = pl->rec[0] + d.n_pad;
    return true;
}

template <typename IDX, bool ASPLIT, bool CL, class ION>
int launch(const MonoDev& d, const IDX* col, const StepsPlan& pl, const ION& ion, cudaStream_t s) {
    static PerDevice<bool> configured;
    const void* fn = (const void*)mono_steps_kernel<IDX, ASPLIT, CL, ION>;
    const bool ok = configured.get([fn](bool& done, int) {
        return done = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, steps_info().max_smem) == cudaSuccess &&
                      (!CL || cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess);
    });
    if (!ok) {
        const cudaError_t e = cudaGetLastError();
        return cuda_fail(e != cudaSuccess ? e : cudaErrorUnknown, "steps kernel attributes");
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)pl.blocks);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = (size_t)pl.smem_bytes;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    if (CL) {   // one cluster: its blocks run together by themselves
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = (unsigned)pl.blocks;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    } else {
        attr[0].id = cudaLaunchAttributeCooperative;
        attr[0].val.cooperative = 1;
    }
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    void* args[] = {const_cast<MonoDev*>(&d), &col, const_cast<StepsPlan*>(&pl), const_cast<ION*>(&ion)};
    cudaError_t e = cudaLaunchKernelExC(&cfg, fn, args);
    if (e != cudaSuccess) return cuda_fail(e, "steps kernel launch");
    return 1;
}

template <class ION>
int launch_any(const MonoDev& d, const StepsPlan& pl, const ION& ion, cudaStream_t s) {
    if (pl.cluster) {
        if constexpr (!ION::kIonic)
            if (!d.a_split) return launch<int16_t, false, true, ION>(d, d.dcol, pl, ion, s);
        return launch<int16_t, true, true, ION>(d, d.dcol, pl, ion, s);
    }
    if (d.dcol)
        return d.a_split ? launch<int16_t, true, false, ION>(d, d.dcol, pl, ion, s)
                         : launch<int16_t, false, false, ION>(d, d.dcol, pl, ion, s);
    return d.a_split ? launch<int32_t, true, false, ION>(d, d.col, pl, ion, s)
                     : launch<int32_t, false, false, ION>(d, d.col, pl, ion, s);
}

template <class M, class Q>
int launch_model(const tcb_mono* m, const MonoDev& d, const StepsPlan& pl, cudaStream_t s) {
    Ionic<M, Q> ion;
    ion.c = M::derive(m->params);
    ion.T = M::tables(m->tables, m->params);
    return launch_any(d, pl, ion, s);
}

// whether the device takes a cluster of kMaxCluster blocks with all of the shared memory
bool cluster_fits() {
    static PerDevice<bool> fits;
    return fits.get([](bool& fit, int) {
        const void* fn = (const void*)mono_steps_kernel<int16_t, true, true, GivenRhs>;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(kMaxCluster);
        cfg.blockDim = dim3(kThreads);
        cfg.dynamicSmemBytes = (size_t)steps_info().max_smem;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = kMaxCluster;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int clusters = 0;
        fit = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, steps_info().max_smem) == cudaSuccess &&
              cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
              cudaOccupancyMaxActiveClusters(&clusters, fn, &cfg) == cudaSuccess && clusters >= 1;
        if (!fit) cudaGetLastError();
        return true;
    });
}

}  // namespace

// Steps [counter, counter + n_steps) as persistent launches of up to kStepsPerLaunch steps:
// 1 = launched, 0 = not applicable (the caller launches step by step), < 0 = error
int launch_steps(const tcb_mono* m, const MonoDev& d, int64_t n_steps, bool ionic, cudaStream_t s) {
    StepsPlan pl;
    constexpr int kStates[4] = {0, MS::kStates, TTP::kStates, CRN::kStates};
    if (ionic && (m->model < TCB_MODEL_MS || m->model > TCB_MODEL_CRN)) return 0;
    if (!steps_plan(m, d, ionic, ionic ? kStates[m->model] : 0, &pl)) return 0;
    int32_t count, v, b, fast = 0, staged;
    if (ionic) {
        // the chosen instance's division policy
        const int st = tcb_ionic_variant(m->model, m->ionic_variant, &count, &v, &b, &fast, &staged);
        if (st) return st;
    }
    for (int64_t done = 0; done < n_steps; done += kStepsPerLaunch) {
        pl.n_steps = (int)std::min(kStepsPerLaunch, n_steps - done);
        if (pl.n_steps < kHoldStateFrom && pl.state_at) {
            pl.smem_bytes = pl.state_at;
            pl.state_at = 0;
        }
        int st;
        if (!ionic) st = launch_any(d, pl, GivenRhs{}, s);
        else if (m->model == TCB_MODEL_MS) st = launch_model<MS, QExact>(m, d, pl, s);
        else if (m->model == TCB_MODEL_TTP) st = fast ? launch_model<TTP, QFast>(m, d, pl, s) : launch_model<TTP, QExact>(m, d, pl, s);
        else st = fast ? launch_model<CRN, QFast>(m, d, pl, s) : launch_model<CRN, QExact>(m, d, pl, s);
        if (st != 1) return st;
    }
    return 1;
}

}  // namespace tcb

// `host_slices`: slice_ptr on the host, or null (read from the device on `stream`, which is synchronised)
static int64_t work_bytes(const tcb_mono* m, const int64_t* host_slices, int32_t* entries, cudaStream_t s) {
    using namespace tcb;
    const int st = validate_mono(m);
    if (st) return st;
    if (!entries) return fail(TCB_EINVAL, "tcb_mono_work_bytes: null output");
    *entries = 0;
    const MonoDev d = make_dev(m);
    StepsPlan pl;
    // (16-byte copies of the matrix; nothing to ask the device for where even one entry a row would not fit)
    if (m->fused_step != 0 || cg_forced_fallback() || !aligned16(d.dcol ? (const void*)d.dcol : (const void*)d.col) ||
        !aligned16(d.mv) || !aligned16(d.kv) || !aligned16(d.av))
        return 0;
    const int64_t grid = steps_blocks(d, false);
    if (!steps_layout(d, grid, TCB_SLICE * ceil_div(d.n_slices, grid), 0, false, &pl)) return 0;
    std::vector<int64_t> copy;
    if (!host_slices) {
        copy.resize((size_t)d.n_slices + 1);
        TCB_CHECK_CUDA(cudaMemcpyAsync(copy.data(), d.slice_ptr, copy.size() * sizeof(int64_t), cudaMemcpyDeviceToHost, s));
        TCB_CHECK_CUDA(cudaStreamSynchronize(s));
    }
    const int64_t* sp = host_slices ? host_slices : copy.data();
    auto most = [&](int64_t nb) {
        int64_t e = 0;
        for (int64_t b = 0; b < nb; ++b) e = std::max(e, sp[(b + 1) * d.n_slices / nb] - sp[b * d.n_slices / nb]);
        return e;
    };
    if (d.dcol && d.n_slices <= kClusterSlices && cluster_fits()) {
        const int64_t nb = steps_blocks(d, true), e = most(nb);
        if (steps_layout(d, nb, e, 0, true, &pl)) *entries = (int32_t)e | kClusterWork;
    }
    if (*entries == 0) {
        const int64_t e = most(grid);
        if (!steps_layout(d, grid, e, 0, false, &pl)) return 0;
        *entries = (int32_t)e;
    }
    return (int64_t)(kHeadBytes + kPartBytes + 2 * (size_t)m->n_pad * sizeof(float4));
}

extern "C" int64_t tcb_mono_work_bytes(const tcb_mono* m, int32_t* entries, void* stream) {
    return work_bytes(m, nullptr, entries, tcb::as_stream(stream));
}

extern "C" int64_t tcb_mono_work_bytes_host(const tcb_mono* m, const int64_t* slice_ptr, int32_t* entries) {
    if (!slice_ptr) return tcb::fail(TCB_EINVAL, "tcb_mono_work_bytes_host: null slice_ptr");
    return work_bytes(m, slice_ptr, entries, nullptr);
}

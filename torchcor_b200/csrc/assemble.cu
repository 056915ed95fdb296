// P1 assembly on the device: element matrices, deterministic gather into CSR
// values, the monodomain system values and the sliced-ELL repack.
//
// Element kernels follow torchcor/core/assemble.py (Matrices3D :148-248,
// Matrices3DSurface :99-145).  The reference forms the local matrices in the
// simulation dtype with batched LU-based det/inv; here each element is one
// thread working in float64 from the float32 coordinates (closed-form
// determinant and adjugate), rounded to float32 once at the end.
#include <cuda_runtime.h>

#include "tcb_internal.h"

namespace {

constexpr int kThreads = 256;

// sigma = st*I + ((sl - st)*f_a)*f_b in float32, as conductivity.py:64-67
// (the outer product there is a batched matmul of single products).
__device__ inline void conductivity_tensor(float sl, float st, const float* f, double s[3][3]) {
    float d = sl - st;
    for (int a = 0; a < 3; ++a)
        for (int b = 0; b < 3; ++b) {
            float o = __fmul_rn(__fmul_rn(d, f[a]), f[b]);
            float v = __fadd_rn(a == b ? st : 0.0f, o);
            s[a][b] = (double)v;
        }
}

// a / b rounded once, from r = 1 / b rounded to nearest: the product's remainder is exact in a fused
// multiply-add and corrects it (Markstein 1990, "Computation of elementary functions on the IBM RISC
// System/6000 processor"; nothing over- or underflows for float32 coordinates, and a determinant of
// zero makes all of K NaN either way).  Nine quotients of one determinant: 3.1 million elements take
// 90 us, with nine divisions 172, with products by r left as they are, which moved 2 of 94 million
// values of K by an ulp, 92.
__device__ __forceinline__ double quotient(double a, double b, double r) {
    const double q = a * r;
    return fma(fma(-q, b, a), r, q);
}

__global__ void tet_local_kernel(const float* __restrict__ nodes, const int32_t* __restrict__ elems, int64_t E,
                                 const float* __restrict__ sl, const float* __restrict__ st,
                                 const float* __restrict__ fib, float* __restrict__ ke, float* __restrict__ mw) {
    int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= E) return;
    // 16-byte accesses where the arrays allow them: 4-byte stores 64 bytes apart cost an
    // L2 sector operation each (222 us against 75 us at 3.1 million elements)
    const bool wide = (((uintptr_t)elems | (uintptr_t)ke) & 15u) == 0;
    int4 el;
    if (wide) el = reinterpret_cast<const int4*>(elems)[e];
    else el = make_int4(elems[e * 4], elems[e * 4 + 1], elems[e * 4 + 2], elems[e * 4 + 3]);
    double x[4][3];
    for (int a = 0; a < 4; ++a) {
        const int32_t v = a == 0 ? el.x : a == 1 ? el.y : a == 2 ? el.z : el.w;
        for (int c = 0; c < 3; ++c) x[a][c] = (double)nodes[(int64_t)v * 3 + c];
    }
    // J[:, c] = x_{c+1} - x_0  (assemble.py:163-169)
    double J[3][3];
    for (int r = 0; r < 3; ++r)
        for (int c = 0; c < 3; ++c) J[r][c] = x[c + 1][r] - x[0][r];
    double C00 = J[1][1] * J[2][2] - J[1][2] * J[2][1];
    double C01 = J[1][2] * J[2][0] - J[1][0] * J[2][2];
    double C02 = J[1][0] * J[2][1] - J[1][1] * J[2][0];
    double det = J[0][0] * C00 + J[0][1] * C01 + J[0][2] * C02;
    // inverse = adj / det
    const double rdet = 1.0 / det;
    double inv[3][3];
    inv[0][0] = quotient(C00, det, rdet);
    inv[1][0] = quotient(C01, det, rdet);
    inv[2][0] = quotient(C02, det, rdet);
    inv[0][1] = quotient(J[0][2] * J[2][1] - J[0][1] * J[2][2], det, rdet);
    inv[1][1] = quotient(J[0][0] * J[2][2] - J[0][2] * J[2][0], det, rdet);
    inv[2][1] = quotient(J[0][1] * J[2][0] - J[0][0] * J[2][1], det, rdet);
    inv[0][2] = quotient(J[0][1] * J[1][2] - J[0][2] * J[1][1], det, rdet);
    inv[1][2] = quotient(J[0][2] * J[1][0] - J[0][0] * J[1][2], det, rdet);
    inv[2][2] = quotient(J[0][0] * J[1][1] - J[0][1] * J[1][0], det, rdet);
    // G = dN @ inv(J): row 0 = -(sum of rows), row a = inv row a-1
    double G[4][3];
    for (int c = 0; c < 3; ++c) {
        G[1][c] = inv[0][c];
        G[2][c] = inv[1][c];
        G[3][c] = inv[2][c];
        G[0][c] = -(inv[0][c] + inv[1][c] + inv[2][c]);
    }
    double s[3][3];
    conductivity_tensor(sl[e], st[e], fib + e * 3, s);
    double adet = fabs(det);
    // vol = |det([1|X])|/6 equals |det J|/6 (assemble.py:194-200); Me = vol/20 * (1 + delta)
    float vol = __fdiv_rn((float)adet, 6.0f);
    mw[e] = __fdiv_rn(vol, 20.0f);
    double scale = adet / 6.0;
    double GS[4][3];
    for (int a = 0; a < 4; ++a)
        for (int c = 0; c < 3; ++c) GS[a][c] = G[a][0] * s[0][c] + G[a][1] * s[1][c] + G[a][2] * s[2][c];
    for (int a = 0; a < 4; ++a) {
        float o[4];
        for (int b = 0; b < 4; ++b) {
            double v = GS[a][0] * G[b][0] + GS[a][1] * G[b][1] + GS[a][2] * G[b][2];
            o[b] = (float)(scale * v);
        }
        if (wide) reinterpret_cast<float4*>(ke)[e * 4 + a] = make_float4(o[0], o[1], o[2], o[3]);
        else
            for (int b = 0; b < 4; ++b) ke[e * 16 + a * 4 + b] = o[b];
    }
}

__global__ void tri_local_kernel(const float* __restrict__ nodes, const int32_t* __restrict__ elems, int64_t E,
                                 const float* __restrict__ sl, const float* __restrict__ st,
                                 const float* __restrict__ fib, float* __restrict__ ke, float* __restrict__ mw) {
    int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= E) return;
    double x[3][3];
    for (int a = 0; a < 3; ++a) {
        int32_t v = elems[e * 3 + a];
        for (int c = 0; c < 3; ++c) x[a][c] = (double)nodes[(int64_t)v * 3 + c];
    }
    double u1[3], u2[3];
    for (int c = 0; c < 3; ++c) {
        u1[c] = x[1][c] - x[0][c];
        u2[c] = x[2][c] - x[0][c];
    }
    // area = |u1 x u2| / 2 (assemble.py:123-130); Me = area/12 * (1 + delta)
    double cr0 = u1[1] * u2[2] - u1[2] * u2[1];
    double cr1 = u1[2] * u2[0] - u1[0] * u2[2];
    double cr2 = u1[0] * u2[1] - u1[1] * u2[0];
    float area = (float)(0.5 * sqrt(cr0 * cr0 + cr1 * cr1 + cr2 * cr2));
    mw[e] = __fdiv_rn(area, 12.0f);
    // in-plane orthonormal frame (assemble.py:103-113)
    double n1 = sqrt(u1[0] * u1[0] + u1[1] * u1[1] + u1[2] * u1[2]);
    double al[3] = {u1[0] / n1, u1[1] / n1, u1[2] / n1};
    double pr = u2[0] * al[0] + u2[1] * al[1] + u2[2] * al[2];
    double be[3] = {u2[0] - pr * al[0], u2[1] - pr * al[1], u2[2] - pr * al[2]};
    double n2 = sqrt(be[0] * be[0] + be[1] * be[1] + be[2] * be[2]);
    for (int c = 0; c < 3; ++c) be[c] /= n2;
    double s[3][3];
    conductivity_tensor(sl[e], st[e], fib + e * 3, s);
    // sigma2 = R sigma R^T (2x2), R rows = (alpha, beta)  (assemble.py:134)
    const double* R[2] = {al, be};
    double s2[2][2];
    for (int i = 0; i < 2; ++i)
        for (int j = 0; j < 2; ++j) {
            double acc = 0.0;
            for (int a = 0; a < 3; ++a)
                for (int b = 0; b < 3; ++b) acc += R[i][a] * s[a][b] * R[j][b];
            s2[i][j] = acc;
        }
    // J = R X^T dN: columns are the edges in the local frame (assemble.py:115-121)
    double J[2][2];
    J[0][0] = al[0] * u1[0] + al[1] * u1[1] + al[2] * u1[2];
    J[1][0] = be[0] * u1[0] + be[1] * u1[1] + be[2] * u1[2];
    J[0][1] = al[0] * u2[0] + al[1] * u2[1] + al[2] * u2[2];
    J[1][1] = be[0] * u2[0] + be[1] * u2[1] + be[2] * u2[2];
    double det = J[0][0] * J[1][1] - J[0][1] * J[1][0];
    double inv[2][2] = {{J[1][1] / det, -J[0][1] / det}, {-J[1][0] / det, J[0][0] / det}};
    double G[3][2];
    for (int c = 0; c < 2; ++c) {
        G[1][c] = inv[0][c];
        G[2][c] = inv[1][c];
        G[0][c] = -(inv[0][c] + inv[1][c]);
    }
    double scale = 0.5 * det;  // signed, as assemble.py:143
    for (int a = 0; a < 3; ++a)
        for (int b = 0; b < 3; ++b) {
            double v = 0.0;
            for (int i = 0; i < 2; ++i)
                for (int j = 0; j < 2; ++j) v += G[a][i] * s2[i][j] * G[b][j];
            ke[e * 9 + a * 3 + b] = (float)(scale * v);
        }
}

// Values of 256 consecutive slots: the block loads their contributions, which are
// consecutive too, into shared memory (kWindow at a time, every thread some of them),
// then each slot adds its own in float32 in the reference COO order.  A thread that
// followed its own list in global memory kept its warp for the longest one (the
// diagonal's, 24 contributions in a cube, against 3 on average).
constexpr int kWindow = 2048;
template <int K>
__global__ void __launch_bounds__(kThreads) gather_kernel(const int32_t* __restrict__ slot_ptr, const int32_t* __restrict__ slot_src,
                                                          int64_t nnz, const float* __restrict__ ke, const float* __restrict__ mw,
                                                          float* __restrict__ kval, float* __restrict__ mval) {
    __shared__ float2 sh[kWindow];
    const int64_t s0 = (int64_t)blockIdx.x * kThreads, s = s0 + threadIdx.x;
    const int64_t s1 = s0 + kThreads < nnz ? s0 + kThreads : nnz;
    const int32_t c0 = slot_ptr[s0], c1 = slot_ptr[s1];
    const int32_t q0 = s < nnz ? slot_ptr[s] : c1, q1 = s < nnz ? slot_ptr[s + 1] : c1;
    float ks = 0.0f, ms = 0.0f;
    // (offsets within a window: up to 2^31 - 2 contributions, an int32 beyond the last one would overflow)
    for (int64_t w0 = c0; w0 < c1; w0 += kWindow) {
        const int32_t len = c1 - w0 < kWindow ? (int32_t)(c1 - w0) : kWindow;
        const int32_t* from = slot_src + w0;
#pragma unroll 4
        for (int32_t i = (int32_t)threadIdx.x; i < len; i += kThreads) {
            const int32_t src = from[i], e = src / (K * K), ab = src - e * (K * K);
            const float m = mw[e];
            sh[i] = make_float2(ke[src], (ab / K == ab % K) ? __fmul_rn(m, 2.0f) : m);
        }
        __syncthreads();
        const int32_t i0 = (int32_t)(q0 - w0), i1 = q1 - w0 < len ? (int32_t)(q1 - w0) : len;
        for (int32_t i = i0 > 0 ? i0 : 0; i < i1; ++i) {
            const float2 v = sh[i];
            ks = i == i0 ? v.x : __fadd_rn(ks, v.x);
            ms = i == i0 ? v.y : __fadd_rn(ms, v.y);
        }
        __syncthreads();
    }
    if (s < nnz) {
        kval[s] = ks;
        mval[s] = ms;
    }
}

// Four consecutive entries a thread, moved as 16-byte vectors where all arrays are so aligned
// (8.0 M entries 40 -> 21 us).
__global__ void system_kernel(int64_t nnz, float* __restrict__ kval, const float* __restrict__ mval, float chi,
                              float cm, float dt, float theta, float rhs_scale, float* __restrict__ aval,
                              float* __restrict__ krhs, int32_t* a_split, bool aligned) {
    const int64_t s = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * 4;
    if (s >= nnz) return;
    bool same = true;
    auto entry = [&](float& k, float m, float& a, float& kr) {
        k = __fdiv_rn(k, chi);                                // K / chi   (monodomain.py:93)
        const float mc = __fmul_rn(m, cm);
        a = __fadd_rn(mc, __fmul_rn(__fmul_rn(k, dt), theta));  // :96
        kr = __fmul_rn(k, rhs_scale);                         // ((1-theta)*dt)*K  (:131)
        same = same && __fadd_rn(mc, kr) == a;
    };
    if (aligned && s + 4 <= nnz) {
        float4 k = *reinterpret_cast<const float4*>(kval + s), a, kr;
        const float4 m = *reinterpret_cast<const float4*>(mval + s);
        entry(k.x, m.x, a.x, kr.x);
        entry(k.y, m.y, a.y, kr.y);
        entry(k.z, m.z, a.z, kr.z);
        entry(k.w, m.w, a.w, kr.w);
        *reinterpret_cast<float4*>(kval + s) = k;
        *reinterpret_cast<float4*>(aval + s) = a;
        *reinterpret_cast<float4*>(krhs + s) = kr;
    } else {
        for (int64_t i = s; i < nnz && i < s + 4; ++i) {
            float k = kval[i], a, kr;
            entry(k, mval[i], a, kr);
            kval[i] = k;
            aval[i] = a;
            krhs[i] = kr;
        }
    }
    if (a_split && !same) atomicAnd(a_split, 0);
}

__global__ void jacobi_kernel(int64_t n, int64_t n_pad, const int32_t* __restrict__ diag,
                              const float* __restrict__ aval, float* __restrict__ dinv) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_pad) return;
    const int32_t s = i < n ? diag[i] : -1;
    dinv[i] = s >= 0 ? __fdiv_rn(1.0f, aval[s]) : 0.0f;   // preconditioner.py:27; 0 for a node in no element
}

struct SellVals {
    const float* in[4];
    float* out[4];
};

// One warp a slice.  Its rows are consecutive in the CSR arrays, so the warp copies
// them to shared memory as they lie (coalesced, the columns and all values of an
// entry in flight together) and writes the columns of the slice from there.
// Slices of more than kPackCap entries are read row by row.
constexpr int kPackWarps = 4, kPackCap = 640;
__global__ void __launch_bounds__(kPackWarps * 32) sell_pack_kernel(int64_t n_rows, int64_t n_slices, const int32_t* __restrict__ rowptr,
                                                                    const int32_t* __restrict__ col, const int64_t* __restrict__ slice_ptr,
                                                                    int nv, SellVals v, int32_t* __restrict__ scol) {
    __shared__ uint32_t sh[kPackWarps][4][kPackCap];   // columns and up to three values
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t s = (int64_t)blockIdx.x * kPackWarps + warp;
    if (s >= n_slices) return;
    const int64_t row = s * TCB_SLICE + lane;
    const int64_t base = slice_ptr[s];
    const int32_t w = (int32_t)((slice_ptr[s + 1] - base) / TCB_SLICE);
    const int32_t b = rowptr[row < n_rows ? row : n_rows];
    const int32_t len = row < n_rows ? rowptr[row + 1] - b : 0;
    const int32_t first = __shfl_sync(0xffffffffu, b, 0);
    const int32_t total = __shfl_sync(0xffffffffu, b + len, 31) - first;
    const int32_t pad = (int32_t)(row < n_rows ? row : 0);
    if (total <= kPackCap && nv == 3) {
        const int32_t* c = col + first;
        const float *v0 = v.in[0] + first, *v1 = v.in[1] + first, *v2 = v.in[2] + first;
#pragma unroll 4
        for (int i = lane; i < total; i += 32) {
            sh[warp][0][i] = (uint32_t)c[i];
            sh[warp][1][i] = __float_as_uint(v0[i]);
            sh[warp][2][i] = __float_as_uint(v1[i]);
            sh[warp][3][i] = __float_as_uint(v2[i]);
        }
        __syncwarp();
#pragma unroll 4
        for (int32_t k = 0; k < w; ++k) {
            const int64_t e = base + (int64_t)k * TCB_SLICE + lane;
            const int q = b - first + k;
            const bool real = k < len;
            scol[e] = real ? (int32_t)sh[warp][0][q] : pad;
            v.out[0][e] = real ? __uint_as_float(sh[warp][1][q]) : 0.0f;
            v.out[1][e] = real ? __uint_as_float(sh[warp][2][q]) : 0.0f;
            v.out[2][e] = real ? __uint_as_float(sh[warp][3][q]) : 0.0f;
        }
        return;
    }
    for (int32_t k = 0; k < w; ++k) {
        const int64_t e = base + (int64_t)k * TCB_SLICE + lane;
        const bool real = k < len;
        scol[e] = real ? col[b + k] : pad;
        for (int j = 0; j < nv; ++j) v.out[j][e] = real ? v.in[j][b + k] : 0.0f;
    }
}

__global__ void sell_delta_kernel(int64_t n_rows, int64_t n_slices, const int64_t* __restrict__ slice_ptr,
                                  const int32_t* __restrict__ scol, int16_t* __restrict__ delta, int32_t* max_abs) {
    int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    int64_t s = t / TCB_SLICE;
    int lane = (int)(t % TCB_SLICE);
    if (s >= n_slices) return;
    int64_t row = s * TCB_SLICE + lane;
    int64_t base = slice_ptr[s];
    int32_t w = (int32_t)((slice_ptr[s + 1] - base) / TCB_SLICE);
    int32_t m = 0;
    for (int32_t k = 0; k < w; ++k) {
        int64_t e = base + (int64_t)k * TCB_SLICE + lane;
        int64_t dlt = row < n_rows ? (int64_t)scol[e] - row : 0;
        int64_t a = dlt < 0 ? -dlt : dlt;
        if (a > m) m = a > INT32_MAX ? INT32_MAX : (int32_t)a;
        delta[e] = (int16_t)(a < 32768 ? dlt : 0);
    }
    atomicMax(max_abs, m);   // integer maximum: order-independent
}

inline unsigned blocks_for(int64_t n) { return (unsigned)tcb::ceil_div(n, kThreads); }

}  // namespace

extern "C" int tcb_assemble_local(int32_t k, const float* nodes, const int32_t* elems, int64_t E, const float* sl,
                                  const float* st, const float* fibres, float* ke, float* mw, void* stream) {
    if ((k != 3 && k != 4) || !nodes || !elems || !sl || !st || !fibres || !ke || !mw || E <= 0)
        return tcb::fail(TCB_EINVAL, "tcb_assemble_local: bad arguments");
    cudaStream_t s = tcb::as_stream(stream);
    if (k == 4)
        tet_local_kernel<<<blocks_for(E), kThreads, 0, s>>>(nodes, elems, E, sl, st, fibres, ke, mw);
    else
        tri_local_kernel<<<blocks_for(E), kThreads, 0, s>>>(nodes, elems, E, sl, st, fibres, ke, mw);
    TCB_CHECK_LAUNCH("element kernel");
    return TCB_OK;
}

extern "C" int tcb_assemble_gather(int32_t k, const int32_t* slot_ptr, const int32_t* slot_src, int64_t nnz,
                                   const float* ke, const float* mw, float* k_val, float* m_val, void* stream) {
    if ((k != 3 && k != 4) || !slot_ptr || !slot_src || !ke || !mw || !k_val || !m_val || nnz <= 0)
        return tcb::fail(TCB_EINVAL, "tcb_assemble_gather: bad arguments");
    cudaStream_t s = tcb::as_stream(stream);
    if (k == 4)
        gather_kernel<4><<<blocks_for(nnz), kThreads, 0, s>>>(slot_ptr, slot_src, nnz, ke, mw, k_val, m_val);
    else
        gather_kernel<3><<<blocks_for(nnz), kThreads, 0, s>>>(slot_ptr, slot_src, nnz, ke, mw, k_val, m_val);
    TCB_CHECK_LAUNCH("gather kernel");
    return TCB_OK;
}

extern "C" int tcb_assemble_system(int64_t nnz, int64_t n, int64_t n_pad, const int32_t* diag, float* k_val,
                                   const float* m_val, double chi, double cm, double dt, double theta, float* a_val,
                                   float* k_rhs, float* d_inv, int32_t* a_split, void* stream) {
    if (!diag || !k_val || !m_val || !a_val || !k_rhs || !d_inv || nnz <= 0 || n <= 0 || n_pad < n)
        return tcb::fail(TCB_EINVAL, "tcb_assemble_system: bad arguments");
    cudaStream_t s = tcb::as_stream(stream);
    // Python-level scalars meet float32 tensors: each is rounded to float32 first
    const bool aligned = (((uintptr_t)k_val | (uintptr_t)m_val | (uintptr_t)a_val | (uintptr_t)k_rhs) & 15u) == 0;
    system_kernel<<<blocks_for(tcb::ceil_div(nnz, 4)), kThreads, 0, s>>>(nnz, k_val, m_val, (float)chi, (float)cm, (float)dt,
                                                                         (float)theta, (float)((1.0 - theta) * dt), a_val,
                                                                         k_rhs, a_split, aligned);
    TCB_CHECK_LAUNCH("system kernel");
    jacobi_kernel<<<blocks_for(n_pad), kThreads, 0, s>>>(n, n_pad, diag, a_val, d_inv);
    TCB_CHECK_LAUNCH("jacobi kernel");
    return TCB_OK;
}

extern "C" int tcb_sell_delta(int64_t n_rows, const int64_t* slice_ptr, int64_t n_slices, const int32_t* sell_col,
                              int16_t* delta, int32_t* max_abs, void* stream) {
    if (!slice_ptr || !sell_col || !delta || !max_abs || n_rows <= 0 || n_slices != tcb::ceil_div(n_rows, TCB_SLICE))
        return tcb::fail(TCB_EINVAL, "tcb_sell_delta: bad arguments");
    sell_delta_kernel<<<blocks_for(n_slices * TCB_SLICE), kThreads, 0, tcb::as_stream(stream)>>>(
        n_rows, n_slices, slice_ptr, sell_col, delta, max_abs);
    TCB_CHECK_LAUNCH("sell delta kernel");
    return TCB_OK;
}

extern "C" int tcb_sell_pack(int64_t n_rows, const int32_t* rowptr, const int32_t* col, const int64_t* slice_ptr,
                             int64_t n_slices, int32_t n_vals, const float* const* vals, int32_t* sell_col,
                             float* const* sell_vals, void* stream) {
    if (!rowptr || !col || !slice_ptr || !sell_col || n_vals < 0 || n_vals > 4 || n_rows <= 0 ||
        n_slices != tcb::ceil_div(n_rows, TCB_SLICE))
        return tcb::fail(TCB_EINVAL, "tcb_sell_pack: bad arguments");
    SellVals v{};
    for (int j = 0; j < n_vals; ++j) {
        if (!vals[j] || !sell_vals[j]) return tcb::fail(TCB_EINVAL, "tcb_sell_pack: null value array");
        v.in[j] = vals[j];
        v.out[j] = sell_vals[j];
    }
    cudaStream_t s = tcb::as_stream(stream);
    sell_pack_kernel<<<(unsigned)tcb::ceil_div(n_slices, kPackWarps), kPackWarps * 32, 0, s>>>(n_rows, n_slices, rowptr, col, slice_ptr,
                                                                           n_vals, v, sell_col);
    TCB_CHECK_LAUNCH("sell pack kernel");
    return TCB_OK;
}

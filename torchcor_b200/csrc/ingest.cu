// Mesh ingest on the device: openCARP text tables parsed on the GPU and the CSR
// pattern + scatter map built on the GPU (the role of torchcor/core/mesh.py:26-63
// and of the COO construction + coalesce in torchcor/core/assemble.py:217-248).
//
// Text: the file's bytes are copied to the device once; the newline positions
// are found with a three-pass count / scan / write; one thread per row parses
// its whitespace-separated fields.  Decimal -> double is correctly rounded, so
// it is the double np.loadtxt reads: with a significand m <= 2^53 and
// |exponent| <= 22 both m and 10^|e| are exact doubles and one IEEE multiply or
// divide rounds once (Clinger 1990); larger significands (up to 19 digits) use
// exact integer arithmetic -- m * 10^e for e <= 19 (128-bit product), and
// m / 10^k = (m / 5^k) * 2^-k for k <= 54 (long division, round-half-even on the
// quotient with the remainder as sticky bit).  Rows outside these paths (more than 19 significant digits, other
// exponents, malformed fields) are counted in `bad`; the caller then parses the
// file on the host instead.
//
// Pattern: every element corner is put into its node's segment; one warp per row
// expands them into the row's contributions (column, position in the reference's
// COO list (a*k + b)*E + e), sorts and compacts them: the unique columns are the CSR
// columns and, for each slot, its contributions in COO order -- the host builder's
// output, bit for bit.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "tcb_internal.h"

namespace tcb {
namespace {

constexpr int kThreads = 256;
constexpr int kBytesPerThread = 32;
constexpr int kRowCap = 1024;          // entries one row may have in the device pattern build
constexpr int kSortWarps = 4;
constexpr int kScanThreads = 1024;

// ---------------------------------------------------------------- newlines
__device__ __forceinline__ int count_nl(const char* t, int64_t b, int64_t e) {
    int c = 0;
    for (int64_t i = b; i < e; ++i) c += t[i] == '\n';
    return c;
}

__global__ void nl_count_kernel(const char* __restrict__ t, int64_t n, int64_t* __restrict__ block_cnt) {
    __shared__ int sh[kThreads];
    const int64_t b = ((int64_t)blockIdx.x * kThreads + threadIdx.x) * kBytesPerThread;
    const int64_t e = b + kBytesPerThread < n ? b + kBytesPerThread : n;
    sh[threadIdx.x] = b < n ? count_nl(t, b, e) : 0;
    __syncthreads();
    for (int s = kThreads / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s) sh[threadIdx.x] += sh[threadIdx.x + s];
        __syncthreads();
    }
    if (threadIdx.x == 0) block_cnt[blockIdx.x] = sh[0];
}

// ---------------------------------------------------------------- exclusive scans
// Counts (times mul) -> int64 offsets with the total behind the last one; in place
// where input and output are the same int64 array.  A block takes kScanTile values,
// kScanItems consecutive ones a thread.  Up to kScanOneBlock values one block walks the
// tiles with a running carry; more take two launches (tile sums, then the tiles, each
// adding the sums before its own; beyond kScanThreads tiles a launch between them scans the sums),
// so that 531,441 counts take 11 us (14 with the third launch) instead of the 820 us one block
// took value by value with a barrier per doubling.
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;
constexpr int64_t kScanOneBlock = 4 * kScanTile;

// exclusive prefix of v over the block; `total` = the block's sum.  sh: 33 values.
__device__ __forceinline__ int64_t block_prefix(int64_t v, int64_t* sh, int64_t& total) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int64_t inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int64_t y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
    }
    if (lane == 31) sh[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        const int64_t w = sh[lane];
        int64_t x = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int64_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        sh[lane] = x - w;
        if (lane == 31) sh[32] = x;
    }
    __syncthreads();
    const int64_t r = sh[warp] + inc - v;
    total = sh[32];
    __syncthreads();
    return r;
}

// offsets of the tile at `base`, on top of `carry`; returns the tile's sum
template <typename T>
__device__ __forceinline__ int64_t scan_tile(const T* v, int64_t* out, int64_t n, int64_t mul, int64_t base, int64_t carry,
                                             int64_t* sh) {
    int64_t x[kScanItems], sum = 0;
#pragma unroll
    for (int j = 0; j < kScanItems; ++j) {
        const int64_t i = base + threadIdx.x * kScanItems + j;
        x[j] = i < n ? (int64_t)v[i] * mul : 0;
        sum += x[j];
    }
    int64_t total;
    int64_t at = carry + block_prefix(sum, sh, total);
#pragma unroll
    for (int j = 0; j < kScanItems; ++j) {
        const int64_t i = base + threadIdx.x * kScanItems + j;
        if (i < n) out[i] = at;
        at += x[j];
    }
    return total;
}

template <typename T>
__global__ void __launch_bounds__(kScanThreads) scan_block_kernel(const T* v, int64_t* out, int64_t n, int64_t mul, int64_t* total) {
    __shared__ int64_t sh[33];
    int64_t carry = 0;
    for (int64_t base = 0; base < n; base += kScanTile) carry += scan_tile(v, out, n, mul, base, carry, sh);
    if (threadIdx.x == 0 && total) *total = carry;
}

template <typename T>
__global__ void __launch_bounds__(kScanThreads) scan_sums_kernel(const T* v, int64_t n, int64_t mul, int64_t* sums) {
    __shared__ int64_t sh[33];
    const int64_t base = (int64_t)blockIdx.x * kScanTile;
    int64_t sum = 0;
    for (int j = 0; j < kScanItems; ++j) {
        const int64_t i = base + j * kScanThreads + threadIdx.x;
        if (i < n) sum += (int64_t)v[i] * mul;
    }
    int64_t total;
    block_prefix(sum, sh, total);
    if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

// A tile's carry: CARRY = false: sums[tile], scanned before; true: every block adds the sums of the tiles
// before its own (up to kScanThreads tiles), the last one also gives the total.
template <typename T, bool CARRY>
__global__ void __launch_bounds__(kScanThreads) scan_tiles_kernel(const T* v, int64_t* out, int64_t n, int64_t mul, const int64_t* sums,
                                                                  int64_t* total) {
    __shared__ int64_t sh[33];
    int64_t carry = 0;
    if constexpr (CARRY) block_prefix(threadIdx.x < blockIdx.x ? sums[threadIdx.x] : 0, sh, carry);
    else carry = sums[blockIdx.x];
    const int64_t sum = scan_tile(v, out, n, mul, (int64_t)blockIdx.x * kScanTile, carry, sh);
    if (CARRY && total && blockIdx.x + 1 == gridDim.x && threadIdx.x == 0) *total = carry + sum;
}

inline int64_t scan_tiles(int64_t n) { return (n + kScanTile - 1) / kScanTile; }

// out[0..n): offsets, *total: the sum (both on the device); tmp: scan_tiles(n) values of its own
template <typename T>
int scan(const T* v, int64_t* out, int64_t n, int64_t mul, int64_t* total, int64_t* tmp, cudaStream_t s) {
    if (n <= kScanOneBlock || !tmp) {
        scan_block_kernel<T><<<1, kScanThreads, 0, s>>>(v, out, n, mul, total);
    } else {
        const unsigned nb = (unsigned)scan_tiles(n);
        scan_sums_kernel<T><<<nb, kScanThreads, 0, s>>>(v, n, mul, tmp);
        if (nb <= kScanThreads) {
            scan_tiles_kernel<T, true><<<nb, kScanThreads, 0, s>>>(v, out, n, mul, tmp, total);
        } else {
            scan_block_kernel<int64_t><<<1, kScanThreads, 0, s>>>(tmp, tmp, nb, 1, total);
            scan_tiles_kernel<T, false><<<nb, kScanThreads, 0, s>>>(v, out, n, mul, tmp, total);
        }
    }
    TCB_CHECK_LAUNCH("scan kernel");
    return TCB_OK;
}

__global__ void nl_write_kernel(const char* __restrict__ t, int64_t n, const int64_t* __restrict__ block_off,
                                int64_t* __restrict__ pos) {
    __shared__ int sh[kThreads];
    const int64_t b = ((int64_t)blockIdx.x * kThreads + threadIdx.x) * kBytesPerThread;
    const int64_t e = b + kBytesPerThread < n ? b + kBytesPerThread : n;
    const int c = b < n ? count_nl(t, b, e) : 0;
    sh[threadIdx.x] = c;
    __syncthreads();
    for (int o = 1; o < kThreads; o <<= 1) {
        const int y = threadIdx.x >= o ? sh[threadIdx.x - o] : 0;
        __syncthreads();
        sh[threadIdx.x] += y;
        __syncthreads();
    }
    int64_t w = block_off[blockIdx.x] + sh[threadIdx.x] - c;
    for (int64_t i = b; i < e; ++i)
        if (t[i] == '\n') pos[w++] = i;
}

// ---------------------------------------------------------------- fields
__device__ __forceinline__ bool is_space(char c) { return c == ' ' || c == '\t' || c == '\r' || c == '\v' || c == '\f'; }

__device__ const double kPow10[23] = {1e0,  1e1,  1e2,  1e3,  1e4,  1e5,  1e6,  1e7,  1e8,  1e9,  1e10, 1e11,
                                      1e12, 1e13, 1e14, 1e15, 1e16, 1e17, 1e18, 1e19, 1e20, 1e21, 1e22};

// Correctly rounded double of an unsigned 128-bit value times 2^scale (round
// half to even; `sticky` marks a nonzero remainder below the value's last bit).
__device__ double round_u128(unsigned __int128 v, int scale, bool sticky) {
    const uint64_t hi = (uint64_t)(v >> 64), lo = (uint64_t)v;
    const int len = hi ? 128 - __clzll((long long)hi) : 64 - __clzll((long long)lo);
    if (len <= 53) return ldexp((double)(uint64_t)v, scale);   // exact (sticky cannot occur: no bits dropped)
    const int sh = len - 53;
    uint64_t m = (uint64_t)(v >> sh);
    const unsigned __int128 rb = v & ((((unsigned __int128)1) << sh) - 1);
    const unsigned __int128 half = ((unsigned __int128)1) << (sh - 1);
    const bool up = rb > half || (rb == half && (sticky || (m & 1)));
    if (up) ++m;
    return ldexp((double)m, scale + sh);   // m <= 2^53: exact conversion, exact scaling
}

__device__ const uint64_t kPow10u[20] = {1ull, 10ull, 100ull, 1000ull, 10000ull, 100000ull, 1000000ull,
                                         10000000ull, 100000000ull, 1000000000ull, 10000000000ull,
                                         100000000000ull, 1000000000000ull, 10000000000000ull,
                                         100000000000000ull, 1000000000000000ull, 10000000000000000ull,
                                         100000000000000000ull, 1000000000000000000ull,
                                         10000000000000000000ull};

// parse one decimal field [p, e); false if malformed or outside the exact range
// (more than 19 significant digits, or an exponent the paths below do not cover)
__device__ bool parse_double(const char* p, const char* e, double* out) {
    bool neg = false;
    if (p < e && (*p == '+' || *p == '-')) neg = *p++ == '-';
    uint64_t m = 0;
    int digits = 0, exp10 = 0;
    bool any = false, dropped = false;
    for (; p < e && *p >= '0' && *p <= '9'; ++p) {
        any = true;
        if (m == 0 && *p == '0') continue;
        if (digits < 19) {
            m = m * 10 + (uint64_t)(*p - '0');
            ++digits;
        } else {
            ++exp10;
            dropped |= *p != '0';
        }
    }
    if (p < e && *p == '.') {
        ++p;
        for (; p < e && *p >= '0' && *p <= '9'; ++p) {
            any = true;
            if (m == 0 && *p == '0') {
                --exp10;
                continue;
            }
            if (digits < 19) {
                m = m * 10 + (uint64_t)(*p - '0');
                ++digits;
                --exp10;
            } else {
                dropped |= *p != '0';
            }
        }
    }
    if (!any) return false;
    if (p < e && (*p == 'e' || *p == 'E')) {
        ++p;
        bool eneg = false;
        if (p < e && (*p == '+' || *p == '-')) eneg = *p++ == '-';
        int x = 0;
        bool ed = false;
        for (; p < e && *p >= '0' && *p <= '9'; ++p) {
            ed = true;
            if (x < 100000) x = x * 10 + (*p - '0');
        }
        if (!ed) return false;
        exp10 += eneg ? -x : x;
    }
    if (p != e || dropped) return false;
    double v;
    if (m == 0) {
        v = 0.0;
    } else if (m <= (1ull << 53) && exp10 >= -22 && exp10 <= 22) {
        // m and 10^|e| are exact doubles: one correctly rounded operation
        v = exp10 < 0 ? __ddiv_rn((double)m, kPow10[-exp10]) : __dmul_rn((double)m, kPow10[exp10]);
    } else if (exp10 >= 0 && exp10 <= 19) {
        v = round_u128((unsigned __int128)m * kPow10u[exp10], 0, false);   // < 2^128, exact product
    } else if (exp10 < 0 && exp10 >= -54) {
        // m / 10^k = (m / 5^k) * 2^-k: long division of m * 2^s by 5^k (< 2^126), s chosen
        // for a quotient of 56..57 bits, then one rounding with the remainder as sticky bit
        const int k = -exp10;
        unsigned __int128 p5 = 1;
        for (int i = 0; i < k; ++i) p5 *= 5;
        const uint64_t phi = (uint64_t)(p5 >> 64), plo = (uint64_t)p5;
        const int plen = phi ? 128 - __clzll((long long)phi) : 64 - __clzll((long long)plo);
        const int mlen = 64 - __clzll((long long)m);
        int sh = 56 + plen - mlen;
        if (sh < 0) sh = 0;
        const int len = mlen + sh;   // bits of m * 2^s (<= 182)
        unsigned __int128 r = 0;
        uint64_t q = 0;
        for (int i = len - 1; i >= 0; --i) {
            r = (r << 1) | (i >= sh ? (m >> (i - sh)) & 1ull : 0ull);   // r < 5^k < 2^127 before the shift
            q <<= 1;
            if (r >= p5) {
                r -= p5;
                q |= 1ull;
            }
        }
        v = round_u128(q, -sh - k, r != 0);
    } else {
        return false;
    }
    *out = neg ? -v : v;
    return true;
}

__device__ bool parse_int(const char* p, const char* e, int64_t* out) {
    bool neg = false;
    if (p < e && (*p == '+' || *p == '-')) neg = *p++ == '-';
    if (p >= e) return false;
    int64_t v = 0;
    for (; p < e; ++p) {
        if (*p < '0' || *p > '9' || v > (INT64_MAX - 9) / 10) return false;
        v = v * 10 + (*p - '0');
    }
    *out = neg ? -v : v;
    return true;
}

__global__ void parse_kernel(const char* __restrict__ t, int64_t n, const int64_t* __restrict__ nl, int64_t n_nl,
                             int64_t first_line, int64_t rows, int skip, int cols, int as_int, void* __restrict__ out,
                             int64_t* __restrict__ bad) {
    const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= rows) return;
    const int64_t line = first_line + r;
    if (line > n_nl) {   // no such line
        atomicAdd((unsigned long long*)bad, 1ull);
        return;
    }
    const int64_t lb = line == 0 ? 0 : nl[line - 1] + 1;
    const int64_t le = line < n_nl ? nl[line] : n;
    const char* p = t + lb;
    const char* end = t + le;
    int field = 0;
    bool ok = true;
    while (ok) {
        while (p < end && is_space(*p)) ++p;
        if (p >= end) break;
        const char* q = p;
        while (q < end && !is_space(*q)) ++q;
        if (field >= skip) {
            const int c = field - skip;
            if (c >= cols) {
                ok = false;
                break;
            }
            if (as_int) ok = parse_int(p, q, static_cast<int64_t*>(out) + r * cols + c);
            else ok = parse_double(p, q, static_cast<double*>(out) + r * cols + c);
        }
        ++field;
        p = q;
    }
    if (!ok || field != skip + cols) atomicAdd((unsigned long long*)bad, 1ull);
}

// ---------------------------------------------------------------- pattern
__global__ void pattern_count_kernel(const int32_t* __restrict__ el, int64_t E, int k, int64_t N,
                                     int32_t* __restrict__ row_cnt, int32_t* __restrict__ err) {
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= E) return;
    for (int a = 0; a < k; ++a) {
        const int32_t v = el[e * k + a];
        if (v < 0 || v >= N) {
            atomicExch(err, 1);
            return;
        }
        atomicAdd(row_cnt + v, 1);
    }
}

// The two halves of the 64-bit keys' buffer, row_off + i a row's i-th word in each: `src` gets the
// contributions in their final order (flat element-matrix indices e*k*k + a*k + b), so
// that the emit kernel need not read them again; `list` holds the row's element corners
// (e*k + a, any order) until the sort, then its distinct columns.
struct KeyHalves {
    uint32_t* src;
    uint32_t* list;
};

inline KeyHalves key_halves(uint64_t* keys, int64_t E, int k) {
    uint32_t* p = reinterpret_cast<uint32_t*>(keys);
    return {p, p + (int64_t)k * k * E};
}

__global__ void pattern_fill_kernel(const int32_t* __restrict__ el, int64_t E, int k, int64_t N, const int64_t* __restrict__ row_off,
                                    int32_t* __restrict__ fill, uint32_t* __restrict__ list) {
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= E) return;
    for (int a = 0; a < k; ++a) {
        const int32_t row = el[e * k + a];
        if (row < 0 || row >= N) return;   // recorded by the count
        list[row_off[row] + atomicAdd(fill + row, 1)] = (uint32_t)(e * k + a);
    }
}

// A distinct column in `list`: its distance from the row (23 bits) above its first contribution's
// place in the row (8 bits).  Rows of the shared-memory sort have the column itself with the top
// bit set, and the top bit of `src` at the first contribution of a column.
constexpr int kStartBits = 8;
constexpr int32_t kFar = 1 << 22;
constexpr uint32_t kRestRow = 0x80000000u, kFirstOfColumn = 0x80000000u;

// Ascending bitonic sort of G*R keys in the registers of G lanes, key r of a lane at lane*R + r.  A merge
// starts by comparing mirrored places, so every exchange goes the same way: the lower place keeps
// the smaller key.
template <int G, int R>
__device__ __forceinline__ void group_sort(uint32_t (&key)[R]) {
    const int lane = threadIdx.x & (G - 1);
#pragma unroll
    for (int size = 2; size <= G * R; size <<= 1) {
        if (size <= R) {
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const int q = r ^ (size - 1);
                if (q < r) continue;
                const uint32_t x = key[r], y = key[q];
                key[r] = min(x, y);
                key[q] = max(x, y);
            }
        } else {
            const bool lower = (lane & (size / R / 2)) == 0;
            uint32_t o[R];
#pragma unroll
            for (int r = 0; r < R; ++r) o[r] = __shfl_xor_sync(0xffffffffu, key[R - 1 - r], size / R - 1);
#pragma unroll
            for (int r = 0; r < R; ++r) key[r] = lower ? min(key[r], o[r]) : max(key[r], o[r]);
        }
#pragma unroll
        for (int stride = size >> 2; stride > 0; stride >>= 1) {
            if (stride >= R) {
                const bool lower = (lane & (stride / R)) == 0;
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const uint32_t o = __shfl_xor_sync(0xffffffffu, key[r], stride / R);
                    key[r] = lower ? min(key[r], o) : max(key[r], o);
                }
            } else {
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    if (r & stride) continue;
                    const uint32_t x = key[r], y = key[r | stride];
                    key[r] = min(x, y);
                    key[r | stride] = max(x, y);
                }
            }
        }
    }
}

// G lanes sort a row's contributions in registers (the other groups of the warp their own rows'):
// its element corners first, A a lane (so that a corner's rank orders elements as the
// reference's COO list does), then one 32-bit key per contribution, (column - row, a*k + b,
// corner rank); a lane's first keys are those of its own corners.  shared: G*A words of the group.
// false (nothing written) if a column is too far from the row for the key's 23 (up to 32
// corners) or 22 bits, or the group has no row (`active`).
template <int G, int A, int K>
__device__ __forceinline__ bool sort_row(bool active, const int32_t* __restrict__ el, int64_t row, int deg, uint32_t* __restrict__ src,
                                         uint32_t* __restrict__ list, int32_t* uniq, uint32_t* shared) {
    constexpr uint32_t k = K;
    constexpr int R = 4 * A;   // (a triangle's fourth key is padding)
    constexpr int kRankBits = G * A <= 32 ? 5 : 6, kLow = 4 + kRankBits;
    constexpr int kHalf = 1 << (31 - kLow);   // |column - row| below this
    static_assert(G * A <= 1 << kRankBits && kHalf <= kFar && G * R <= 1 << kStartBits, "fields of the keys");
    const int lane = threadIdx.x & (G - 1);
    const int cnt = deg * K;
    uint32_t corner[A];
#pragma unroll
    for (int r = 0; r < A; ++r) corner[r] = lane * A + r < deg ? list[lane * A + r] : 0xffffffffu;
    group_sort<G, A>(corner);
    const bool wide = K == 4 && (reinterpret_cast<uintptr_t>(el) & 15) == 0;
    uint32_t key[R];
    bool ok = active;
#pragma unroll
    for (int r = 0; r < A; ++r) {
        const int j = lane * A + r;
        const uint32_t e = corner[r] / k, a = corner[r] - e * k;
        int32_t v[4] = {};
        if (j < deg) {
            if (wide) {
                const int4 q = *reinterpret_cast<const int4*>(el + (size_t)e * k);
                v[0] = q.x, v[1] = q.y, v[2] = q.z, v[3] = q.w;
            } else {
#pragma unroll
                for (int b = 0; b < K; ++b) v[b] = el[(size_t)e * k + b];
            }
        }
        shared[j] = e * (k * k);
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            key[r * 4 + b] = 0xffffffffu;
            if (b < K && j < deg) {
                const int64_t d = (int64_t)v[b] - row;
                ok = ok && d > -kHalf && d < kHalf - 1;   // (kHalf - 1 with all low bits set would be the padding)
                key[r * 4 + b] = ((uint32_t)(int32_t)(d + kHalf) << kLow) | ((a * k + b) << kRankBits) | (uint32_t)j;
            }
        }
    }
    group_sort<G, R>(key);
    const uint32_t last = __shfl_up_sync(0xffffffffu, key[R - 1], 1, G);
    const unsigned group = G == 32 ? 0xffffffffu : ((1u << (G & 31)) - 1) << (threadIdx.x & 31 & ~(G - 1));
    ok = (__ballot_sync(0xffffffffu, ok) & group) == group;   // (also orders `shared`)
    __syncwarp();
    bool first[R];
    int u = 0;
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int p = lane * R + r;
        first[r] = p < cnt && (p == 0 || (key[r] >> kLow) != ((r ? key[r - 1] : last) >> kLow));
        u += first[r];
    }
    int at = u;
#pragma unroll
    for (int o = 1; o < G; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, at, o, G);
        if (lane >= o) at += v;
    }
    if (!ok) return false;
    if (lane == G - 1) *uniq = at;
    at -= u;
#pragma unroll
    for (int r = 0; r < R; ++r)
        if (first[r]) list[at++] = (((key[r] >> kLow) + (kFar - kHalf)) << kStartBits) | (uint32_t)(lane * R + r);
    // (a tetrahedron's four contributions keep the places of a row in multiples of four)
    const bool wide_out = K == 4 && (reinterpret_cast<uintptr_t>(src) & 15) == 0;
#pragma unroll
    for (int r = 0; r < R; r += 4) {
        const int p = lane * R + r;
        if (p >= cnt) break;
        uint32_t out[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const uint32_t v = key[r + q];
            out[q] = shared[v & (G * A - 1)] + ((v >> kRankBits) & 15);
        }
        if (wide_out) {
            *reinterpret_cast<uint4*>(src + p) = make_uint4(out[0], out[1], out[2], out[3]);
        } else {
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (p + q < cnt) src[p + q] = out[q];
        }
    }
    return true;
}

// Rows of up to 64 corners whose columns are near enough (all rows of meshes below two
// million nodes); the others go to `rest` (rest[0] counts).  Four rows a warp, 8 lanes each, where
// they have up to 32 corners, else a warp a row.  Bound by the exchanges: of the 28 steps of a
// 128-key sort 6 leave a lane's 16 registers with 8 lanes a row, 15 with a warp a row and 4
// registers, and a shuffle costs as much issue as four other instructions.
// Measured on B200: 531,441 nodes, 50 M contributions, a warp a row 378 -> 297 us (482 with exchanges that
// selected a direction and 8-byte keys written back); the whole pattern 633 -> 554 us, of a
// level-8 icosphere (655,362 nodes) 454 -> 309 us, of a 20-cube even (140, launches).
template <int K>
__global__ void __launch_bounds__(256) pattern_sort_kernel(const int32_t* __restrict__ el, const int64_t* __restrict__ row_off, int64_t N,
                                                           KeyHalves keys, int32_t* __restrict__ uniq, int64_t* __restrict__ rest) {
    constexpr int G = 8, kRows = 32 / G;
    __shared__ uint32_t shared[8][128];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t row0 = ((int64_t)blockIdx.x * 8 + warp) * kRows;
    if (row0 >= N) return;
    const int64_t row = row0 + lane / G;
    const bool in = row < N;
    const int64_t b = in ? row_off[row] : 0;
    const int64_t deg64 = in ? (row_off[row + 1] - b) / K : 0;
    const bool small = in && deg64 <= 32;
    const int deg = small ? (int)deg64 : 0;
    int most = deg;
#pragma unroll
    for (int o = G; o < 32; o <<= 1) most = max(most, __shfl_xor_sync(0xffffffffu, most, o));
    uint32_t* mine = shared[warp] + lane / G * 32;
    bool done;
    if (most <= 8) done = sort_row<G, 1, K>(small, el, row, deg, keys.src + b, keys.list + b, uniq + row, mine);
    else if (most <= 16) done = sort_row<G, 2, K>(small, el, row, deg, keys.src + b, keys.list + b, uniq + row, mine);
    else done = sort_row<G, 4, K>(small, el, row, deg, keys.src + b, keys.list + b, uniq + row, mine);
    unsigned large = __ballot_sync(0xffffffffu, in && deg64 > 32 && deg64 <= 64 && lane % G == 0);
    while (large) {
        const int from = __ffs(large) - 1;
        large &= large - 1;
        const int64_t r = row0 + from / G, rb = __shfl_sync(0xffffffffu, b, from);
        const int rd = __shfl_sync(0xffffffffu, (int)deg64, from);
        __syncwarp();   // the words of the sort before have been read
        const bool ok = sort_row<32, 2, K>(true, el, r, rd, keys.src + rb, keys.list + rb, uniq + r, shared[warp]);
        if (lane / G == from / G) done = ok;
    }
    if (in && !done && lane % G == 0)
        rest[1 + atomicAdd(reinterpret_cast<unsigned long long*>(rest), 1ull)] = row;
}

// The remaining rows: 64-bit keys (column, COO order) sorted in shared memory, one warp a row
__global__ void pattern_rest_kernel(const int32_t* __restrict__ el, int64_t E, int k, const int64_t* __restrict__ row_off,
                                    KeyHalves keys, int32_t* __restrict__ uniq, const int64_t* __restrict__ rest,
                                    int32_t* __restrict__ err) {
    __shared__ uint64_t sh[kSortWarps][kRowCap];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t n = rest[0];
    for (int64_t q = (int64_t)blockIdx.x * kSortWarps + warp; q < n; q += (int64_t)gridDim.x * kSortWarps) {
        const int64_t row = rest[1 + q], b = row_off[row];
        const int64_t cnt64 = row_off[row + 1] - b;
        if (cnt64 > kRowCap) {
            if (lane == 0) {
                atomicExch(err, 2);
                uniq[row] = 0;
            }
            continue;
        }
        const int cnt = (int)cnt64;
        int p2 = 1;
        while (p2 < cnt) p2 <<= 1;
        uint64_t* s = sh[warp];
        for (int i = lane; i < p2; i += 32) {
            uint64_t v = ~0ull;
            if (i < cnt) {
                const int64_t corner = keys.list[b + i / k], e = corner / k, a = corner - e * k, c = i % k;
                v = ((uint64_t)(uint32_t)el[e * k + c] << 32) | ((uint64_t)(a * k + c) * (uint64_t)E + (uint64_t)e);
            }
            s[i] = v;
        }
        __syncwarp();
        for (int size = 2; size <= p2; size <<= 1)
            for (int stride = size >> 1; stride > 0; stride >>= 1) {
                for (int i = lane; i < p2; i += 32) {
                    const int j = i ^ stride;
                    if (j > i) {
                        const bool up = (i & size) == 0;
                        const uint64_t x = s[i], y = s[j];
                        if ((x > y) == up) {
                            s[i] = y;
                            s[j] = x;
                        }
                    }
                }
                __syncwarp();
            }
        int u = 0;
        for (int i0 = 0; i0 < cnt; i0 += 32) {
            const int i = i0 + lane;
            const uint64_t v = i < cnt ? s[i] : 0ull;
            const bool first = i < cnt && (i == 0 || (v >> 32) != (s[i - 1] >> 32));
            const unsigned m = __ballot_sync(0xffffffffu, first);
            const uint64_t order = v & 0xffffffffull, ab = order / (uint64_t)E, e = order - ab * (uint64_t)E;
            if (i < cnt) keys.src[b + i] = (first ? kFirstOfColumn : 0u) | (uint32_t)(e * k * k + ab);
            if (first) keys.list[b + u + __popc(m & ((1u << lane) - 1))] = kRestRow | (uint32_t)(v >> 32);
            u += __popc(m);
        }
        if (lane == 0) uniq[row] = u;
        __syncwarp();
    }
}

// CSR columns, slot boundaries and the diagonal slot, half a warp a row (a cube's interior rows have
// 15 columns): it reads the 15, not the 96 contributions, which are in place (531,441 nodes: 145 -> 55 us).
// `src` is rewritten only in rows that the shared-memory sort left flagged.
__global__ void __launch_bounds__(256) pattern_emit_kernel(const int64_t* __restrict__ row_off, const int64_t* __restrict__ rowptr64,
                                                           int64_t N, const uint32_t* __restrict__ list,
                                                           int32_t* __restrict__ rowptr, int32_t* __restrict__ col,
                                                           int32_t* __restrict__ slot_ptr, int32_t* __restrict__ src,
                                                           int32_t* __restrict__ diag) {
    const int lane = threadIdx.x & 15;
    const int64_t row = (int64_t)blockIdx.x * (blockDim.x >> 4) + (threadIdx.x >> 4);
    if (row >= N) return;
    const int64_t b = row_off[row], w = rowptr64[row];
    const int u = (int)(rowptr64[row + 1] - w);
    if (lane == 0) rowptr[row] = (int32_t)w;
    if (u == 0 && lane == 0) diag[row] = -1;   // a node in no element
    bool flagged = false;
    for (int i = lane; i < u; i += 16) {
        const uint32_t v = list[b + i];
        flagged = (v & kRestRow) != 0;
        int32_t c = (int32_t)(v & ~kRestRow);
        if (!flagged) {
            c = (int32_t)row + (int32_t)(v >> kStartBits) - kFar;
            slot_ptr[w + i] = (int32_t)(b + (v & ((1u << kStartBits) - 1)));
        }
        col[w + i] = c;
        if (c == row) diag[row] = (int32_t)(w + i);
    }
    const unsigned half = 0xffffu << (threadIdx.x & 16);
    if (!__any_sync(half, flagged)) return;
    const int64_t end = row_off[row + 1];
    int64_t j = w;
    for (int64_t q0 = b; q0 < end; q0 += 16) {
        const int64_t q = q0 + lane;
        const uint32_t v = q < end ? (uint32_t)src[q] : 0u;
        const bool first = (v & kFirstOfColumn) != 0;
        const unsigned m = __ballot_sync(half, first) >> (threadIdx.x & 16);
        if (first) {
            slot_ptr[j + __popc(m & ((1u << lane) - 1))] = (int32_t)q;
            src[q] = (int32_t)(v & ~kFirstOfColumn);
        }
        j += __popc(m);
    }
}

__global__ void pattern_tail_kernel(const int64_t* rp64, const int64_t* ro, int64_t n, int32_t* rp, int32_t* sp) {
    rp[n] = (int32_t)rp64[n];
    sp[rp64[n]] = (int32_t)ro[n];
}

// one warp per slice: its widest row
__global__ void __launch_bounds__(256) slice_width_kernel(const int32_t* __restrict__ rowptr, int64_t n_rows, int64_t n_slices, int64_t* __restrict__ width) {
    const int64_t s = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (s >= n_slices) return;
    const int64_t r = s * TCB_SLICE + (threadIdx.x & 31);
    int w = r < n_rows ? rowptr[r + 1] - rowptr[r] : 0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) w = max(w, __shfl_xor_sync(0xffffffffu, w, o));
    if ((threadIdx.x & 31) == 0) width[s] = w;
}

inline unsigned blocks(int64_t n, int per) { return (unsigned)((n + per - 1) / per); }

}  // namespace
}  // namespace tcb

using namespace tcb;

extern "C" int64_t tcb_text_scratch(int64_t n_bytes) {
    if (n_bytes < 0) return -1;
    return (int64_t)blocks(n_bytes, kThreads * kBytesPerThread) + 1;
}

extern "C" int tcb_text_newlines(const char* text, int64_t n_bytes, int64_t* scratch, int64_t* pos, int64_t cap,
                                 int64_t* count, void* stream) {
    if (!text || !scratch || !count || n_bytes <= 0 || (pos && cap < 0))
        return fail(TCB_EINVAL, "tcb_text_newlines: bad arguments");
    cudaStream_t s = as_stream(stream);
    const unsigned nb = blocks(n_bytes, kThreads * kBytesPerThread);
    nl_count_kernel<<<nb, kThreads, 0, s>>>(text, n_bytes, scratch);
    TCB_CHECK_LAUNCH("newline count kernel");
    int st = scan(scratch, scratch, nb, 1, scratch + nb, (int64_t*)nullptr, s);
    if (st) return st;
    int64_t total = 0;
    TCB_CHECK_CUDA(cudaMemcpyAsync(&total, scratch + nb, sizeof total, cudaMemcpyDeviceToHost, s));
    TCB_CHECK_CUDA(cudaStreamSynchronize(s));
    *count = total;
    if (!pos) return TCB_OK;
    if (total > cap) return fail(TCB_ERANGE, "tcb_text_newlines: more newlines than capacity");
    nl_write_kernel<<<nb, kThreads, 0, s>>>(text, n_bytes, scratch, pos);
    TCB_CHECK_LAUNCH("newline write kernel");
    return TCB_OK;
}

extern "C" int tcb_text_parse(const char* text, int64_t n_bytes, const int64_t* nl, int64_t n_nl, int64_t first_line,
                              int64_t rows, int32_t skip, int32_t cols, int32_t as_int, void* out, int64_t* bad,
                              void* stream) {
    if (!text || !out || !bad || n_bytes <= 0 || (n_nl > 0 && !nl) || first_line < 0 || rows < 0 || skip < 0 ||
        cols < 1)
        return fail(TCB_EINVAL, "tcb_text_parse: bad arguments");
    if (rows == 0) return TCB_OK;
    cudaStream_t s = as_stream(stream);
    parse_kernel<<<blocks(rows, kThreads), kThreads, 0, s>>>(text, n_bytes, nl, n_nl, first_line, rows, skip, cols,
                                                             as_int, out, bad);
    TCB_CHECK_LAUNCH("parse kernel");
    return TCB_OK;
}

extern "C" int tcb_pattern_device(const int32_t* elems, int64_t E, int32_t k, int64_t N, int64_t* work,
                                  uint64_t* keys, int32_t* iwork, int64_t* nnz, void* stream) {
    if (!elems || !work || !keys || !iwork || !nnz || E <= 0 || N <= 0 || (k != 3 && k != 4))
        return fail(TCB_EINVAL, "tcb_pattern_device: bad arguments");
    if ((int64_t)k * k * E >= INT32_MAX) return fail(TCB_ERANGE, "too many element contributions for int32");
    cudaStream_t s = as_stream(stream);
    // work: row_off [N+1] | rowptr64 [N+1];  iwork: row counts / fill [N] | uniq [N] | err [1]
    int64_t* row_off = work;
    int64_t* rowptr64 = work + N + 1;
    int32_t* cnt = iwork;
    int32_t* uniq = iwork + N;
    int32_t* err = iwork + 2 * N;
    TCB_CHECK_CUDA(cudaMemsetAsync(iwork, 0, sizeof(int32_t) * (2 * N + 1), s));
    pattern_count_kernel<<<blocks(E, kThreads), kThreads, 0, s>>>(elems, E, k, N, cnt, err);
    TCB_CHECK_LAUNCH("pattern count kernel");
    // rowptr64 is written last: until then it holds the tile sums and the rows left over by the sort
    // (their number, then the rows: at most N + 1 values)
    int st = scan(cnt, row_off, N, k, row_off + N, rowptr64, s);
    if (st) return st;
    TCB_CHECK_CUDA(cudaMemsetAsync(cnt, 0, sizeof(int32_t) * N, s));
    TCB_CHECK_CUDA(cudaMemsetAsync(rowptr64, 0, sizeof(int64_t), s));
    const KeyHalves halves = key_halves(keys, E, k);
    pattern_fill_kernel<<<blocks(E, kThreads), kThreads, 0, s>>>(elems, E, k, N, row_off, cnt, halves.list);
    TCB_CHECK_LAUNCH("pattern fill kernel");
    if (k == 4) pattern_sort_kernel<4><<<blocks(N, 32), 256, 0, s>>>(elems, row_off, N, halves, uniq, rowptr64);
    else pattern_sort_kernel<3><<<blocks(N, 32), 256, 0, s>>>(elems, row_off, N, halves, uniq, rowptr64);
    TCB_CHECK_LAUNCH("pattern sort kernel");
    pattern_rest_kernel<<<(unsigned)std::min<int64_t>(blocks(N, kSortWarps), 592), kSortWarps * 32, 0, s>>>(
        elems, E, k, row_off, halves, uniq, rowptr64, err);
    TCB_CHECK_LAUNCH("pattern rest kernel");
    // (the tile sums of this scan go where the corner counts were: 8-byte aligned, read no more)
    int64_t* tmp = reinterpret_cast<int64_t*>(((uintptr_t)cnt + 7) & ~(uintptr_t)7);
    st = scan(uniq, rowptr64, N, 1, rowptr64 + N, tmp, s);
    if (st) return st;
    int32_t h_err = 0;
    TCB_CHECK_CUDA(cudaMemcpyAsync(&h_err, err, sizeof h_err, cudaMemcpyDeviceToHost, s));
    TCB_CHECK_CUDA(cudaMemcpyAsync(nnz, rowptr64 + N, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
    TCB_CHECK_CUDA(cudaStreamSynchronize(s));
    if (h_err == 1) return fail(TCB_EINVAL, "element node index out of range");
    if (h_err == 2) return fail(TCB_ERANGE, "a node has more than 1024 element contributions (device pattern)");
    if (*nnz >= INT32_MAX) return fail(TCB_ERANGE, "nnz beyond int32");
    return TCB_OK;
}

extern "C" int tcb_pattern_device_emit(const int64_t* work, const uint64_t* keys, int64_t E, int32_t k, int64_t N,
                                       int32_t* rowptr, int32_t* col, int32_t* slot_ptr, int32_t* slot_src,
                                       int32_t* diag, void* stream) {
    if (!work || !keys || !rowptr || !col || !slot_ptr || !slot_src || !diag || E <= 0 || N <= 0 ||
        (k != 3 && k != 4))
        return fail(TCB_EINVAL, "tcb_pattern_device_emit: bad arguments");
    cudaStream_t s = as_stream(stream);
    const int64_t* row_off = work;
    const int64_t* rowptr64 = work + N + 1;
    const KeyHalves halves = key_halves(const_cast<uint64_t*>(keys), E, k);
    if (reinterpret_cast<uint32_t*>(slot_src) != halves.src)
        TCB_CHECK_CUDA(cudaMemcpyAsync(slot_src, halves.src, sizeof(int32_t) * k * k * E, cudaMemcpyDeviceToDevice, s));
    pattern_emit_kernel<<<blocks(N, 16), 256, 0, s>>>(row_off, rowptr64, N, halves.list, rowptr, col, slot_ptr, slot_src, diag);
    TCB_CHECK_LAUNCH("pattern emit kernel");
    pattern_tail_kernel<<<1, 1, 0, s>>>(rowptr64, row_off, N, rowptr, slot_ptr);
    TCB_CHECK_LAUNCH("pattern tail kernel");
    return TCB_OK;
}

extern "C" int64_t tcb_sell_layout_scratch(int64_t n_rows) {
    if (n_rows < 0) return -1;
    const int64_t ns = ceil_div(n_rows, TCB_SLICE);
    return scan_tiles(ns) + 1;
}

// `host` gets the last `n_host` of the offsets (synchronises the stream)
static int sell_layout(const int32_t* rowptr, int64_t n_rows, int64_t* slice_ptr, int64_t* scratch, int64_t* host, int64_t n_host,
                       cudaStream_t s) {
    const int64_t ns = ceil_div(n_rows, TCB_SLICE);
    slice_width_kernel<<<blocks(ns, 8), 256, 0, s>>>(rowptr, n_rows, ns, slice_ptr);
    TCB_CHECK_LAUNCH("slice width kernel");
    const int st = scan(slice_ptr, slice_ptr, ns, TCB_SLICE, slice_ptr + ns, scratch, s);
    if (st) return st;
    TCB_CHECK_CUDA(cudaMemcpyAsync(host, slice_ptr + ns + 1 - n_host, n_host * sizeof(int64_t), cudaMemcpyDeviceToHost, s));
    TCB_CHECK_CUDA(cudaStreamSynchronize(s));
    return TCB_OK;
}

extern "C" int tcb_sell_layout_device(const int32_t* rowptr, int64_t n_rows, int64_t* slice_ptr, int64_t* scratch,
                                      int64_t* n_entries, void* stream) {
    if (!rowptr || !slice_ptr || !scratch || !n_entries || n_rows <= 0)
        return fail(TCB_EINVAL, "tcb_sell_layout_device: bad arguments");
    return sell_layout(rowptr, n_rows, slice_ptr, scratch, n_entries, 1, as_stream(stream));
}

extern "C" int tcb_sell_layout_both(const int32_t* rowptr, int64_t n_rows, int64_t* slice_ptr, int64_t* scratch,
                                    int64_t* host_slice_ptr, void* stream) {
    if (!rowptr || !slice_ptr || !scratch || !host_slice_ptr || n_rows <= 0)
        return fail(TCB_EINVAL, "tcb_sell_layout_both: bad arguments");
    return sell_layout(rowptr, n_rows, slice_ptr, scratch, host_slice_ptr, ceil_div(n_rows, TCB_SLICE) + 1, as_stream(stream));
}

// Batched sign and log|det| of small real matrices, and the gradient of
// log|det| (the reference's fused log-det kernels, csrc/ffi/logdet_cuda.cu:
// forward :187-262 by LU with partial pivoting, backward :264-331 by solving
// A^T X = I), written without cuSolverDx.
//
// Partial pivoting picks the largest |a_rk| of the rows not used yet, the
// lowest current row on ties, as LAPACK's idamax; trailing elements are updated
// by fused multiply-adds in pivot order.  A zero (or not-a-number) pivot column
// marks the matrix singular: sign 0 and log|det| -inf, gradient 0, as the
// reference reports a nonzero factorisation status.  The gradient solves A Y =
// I from the factors (rows of I moved as the factorisation moved them) and
// writes cot * Y^T = cot * A^{-T}.
//
//   small n (lu_rows_max): 4, 8, 16 or 32 lanes per matrix (the next power of
//     two), a row per lane in registers: no row is moved (each lane tracks
//     where its row stands), the pivot row comes by shuffles, and the factors
//     go to shared memory once, for the gradient's substitutions (a column of Y
//     per lane).  Bound by instruction issue: the division and the search for
//     the pivot are most of a small step.  32,768 FP64 matrices of n = 10: a
//     warp per matrix, two lanes in three idle, 126 us (value) and 167 us
//     (gradient); 52 and 73 now.
//   larger n: one warp per matrix in shared memory, row-major with an odd row
//     stride; the trailing block is updated by columns, each lane walking its
//     columns down the rows.
#include "common.cuh"

#include <algorithm>
#include <cmath>
#include <type_traits>
#include <utility>

namespace dnq {

void keep_pool(int device);

namespace {

// ---------------------------------------------------------------------------
// n <= N <= 32: G lanes per matrix, lane = row
// ---------------------------------------------------------------------------
constexpr int kLuWarps = 4;

// f(0), f(1), ..., f(N - 1) with the index a constant of each call: the rows
// stay in registers only if every index into them is one (the compiler leaves
// such loops rolled from N = 10 on).
template <class F, int... I>
__device__ __forceinline__ void static_for_(std::integer_sequence<int, I...>, F&& f) {
    (f(std::integral_constant<int, I>{}), ...);
}
template <int N, class F>
__device__ __forceinline__ void static_for(F&& f) {
    static_for_(std::make_integer_sequence<int, N>{}, f);
}

template <int N>
struct LuGroup {
    static constexpr int G = N <= 4 ? 4 : N <= 8 ? 8 : N <= 16 ? 16 : 32;
    static constexpr int M = 32 / G;   // matrices of a warp
};

// Copies the warp's matrices (cnt of them, contiguous) between global memory
// and the warp's shared buffer, neighbouring lanes on neighbouring values.
template <class T>
__device__ __forceinline__ void lu_copy(T* dst, const T* src, int count, int lane) {
    for (int e = lane; e < count; e += 32) dst[e] = src[e];
}

// LU of the n x n matrix whose row r the group's lane r holds in a[]; lanes r
// >= n hold nothing.  pos: where the lane's row ends up; piv: u_kk in the
// group's lane k; par: parity of the exchanges.  Returns false for a group
// that met a pivot column without a usable value.
template <class T, int N>
__device__ __forceinline__ bool lu_rows(T (&a)[N], int n, int r, int gbase, int& pos, T& piv,
                                        int& par) {
    constexpr int G = LuGroup<N>::G;
    const unsigned gmask = G == 32 ? 0xffffffffu : (1u << (G & 31)) - 1u;
    bool ok = true;
    par = 0;
    pos = r;
    piv = T(0);
    static_for<N>([&](auto step) {
        constexpr int k = decltype(step)::value;
        if (k >= n) return;   // the same for all lanes
        const T v = fabs(a[k]);
        const bool mine = r < n && pos >= k && v > T(-1);   // false for NaN
        T best = mine ? v : T(-1);
        int br = mine ? pos : n;
#pragma unroll
        for (int o = G / 2; o; o >>= 1) {
            const T ov = __shfl_xor_sync(0xffffffffu, best, o);
            const int orow = __shfl_xor_sync(0xffffffffu, br, o);
            if (ov > best || (ov == best && orow < br)) {
                best = ov;
                br = orow;
            }
        }
        ok = ok && br < n && best > T(0);
        const unsigned who = __ballot_sync(0xffffffffu, mine && pos == br) >> gbase & gmask;
        const int src = gbase + (who ? __ffs(who) - 1 : 0);
        const bool is_piv = gbase + r == src && who;
        par ^= br != k;
        // no row is moved in a column without a usable value (br == n), so the
        // positions stay a permutation of the n rows
        if (is_piv) pos = k;
        else if (pos == k && br < n) pos = br;
        const T p = __shfl_sync(0xffffffffu, a[k], src);
        if (r == k) piv = p;
        const bool below = r < n && pos > k;
        const T l = below ? a[k] / p : T(0);
        if (below) a[k] = l;
        static_for<N - k - 1>([&](auto col) {
            constexpr int j = k + 1 + decltype(col)::value;
            const T u = __shfl_sync(0xffffffffu, a[j], src);
            if (below) a[j] = fma(-l, u, a[j]);
        });
    });
    return ok;
}

template <class T, int N>
__global__ void __launch_bounds__(kLuWarps * 32) k_slogdet_rows(const T* A, i64 B, int n, T* sign,
                                                                T* logabs) {
    constexpr int G = LuGroup<N>::G, M = LuGroup<N>::M;
    __shared__ T buf[kLuWarps][M * N * N];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int r = lane & (G - 1), m = lane / G, gbase = m * G;
    const int nn = n * n;
    T* S = buf[w];
    for (i64 b0 = ((i64)blockIdx.x * kLuWarps + w) * M; b0 < B;
         b0 += (i64)gridDim.x * kLuWarps * M) {
        const int cnt = (int)min((i64)M, B - b0);
        __syncwarp();
        lu_copy(S, A + b0 * nn, cnt * nn, lane);
        __syncwarp();
        const bool have = m < cnt && r < n;
        T a[N];
#pragma unroll
        for (int j = 0; j < N; ++j) a[j] = have && j < n ? S[m * nn + r * n + j] : T(0);
        int pos, par;
        T piv;
        const bool ok = lu_rows<T, N>(a, n, r, gbase, pos, piv, par);
        // as the reference: log|u_ii| summed in FP64 in order
        const double d = (double)piv, ad = fabs(d);
        const unsigned gmask = G == 32 ? 0xffffffffu : (1u << (G & 31)) - 1u;
        const bool bad = r < n && (!(ad > 0.0) || !isfinite(ad));
        const bool good =
            ok && ((__ballot_sync(0xffffffffu, bad) >> gbase) & gmask) == 0;
        const unsigned neg = (__ballot_sync(0xffffffffu, r < n && d < 0.0) >> gbase) & gmask;
        const double lg = r < n ? log(ad) : 0.0;
        double la = 0.0;
#pragma unroll
        for (int i = 0; i < N; ++i) {
            if (i >= n) continue;
            la += __shfl_sync(0xffffffffu, lg, gbase + i);
        }
        if (r == 0 && m < cnt) {
            const bool minus = (par + __popc(neg)) & 1;
            sign[b0 + m] = good ? (minus ? T(-1) : T(1)) : T(0);
            logabs[b0 + m] = good ? (T)la : (T)(-INFINITY);
        }
    }
}

template <class T, int N>
__global__ void __launch_bounds__(kLuWarps * 32)
k_slogdet_grad_rows(const T* A, const T* cot, i64 B, int n, T* grad) {
    constexpr int G = LuGroup<N>::G, M = LuGroup<N>::M;
    extern __shared__ __align__(16) unsigned char lu_smem[];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int r = lane & (G - 1), m = lane / G, gbase = m * G;
    const int nn = n * n;
    T* S = reinterpret_cast<T*>(lu_smem) + (size_t)w * M * nn;
    for (i64 b0 = ((i64)blockIdx.x * kLuWarps + w) * M; b0 < B;
         b0 += (i64)gridDim.x * kLuWarps * M) {
        const int cnt = (int)min((i64)M, B - b0);
        __syncwarp();
        lu_copy(S, A + b0 * nn, cnt * nn, lane);
        __syncwarp();
        const bool have = m < cnt && r < n;
        T a[N];
#pragma unroll
        for (int j = 0; j < N; ++j) a[j] = have && j < n ? S[m * nn + r * n + j] : T(0);
        int pos, par;
        T piv;
        const bool ok = lu_rows<T, N>(a, n, r, gbase, pos, piv, par);
        __syncwarp();
        const bool solve = have && ok;   // a singular matrix' gradient is 0
        if (solve) {   // the factors, rows where the exchanges put them
#pragma unroll
            for (int j = 0; j < N; ++j)
                if (j < n) S[m * nn + pos * n + j] = a[j];
        }
        __syncwarp();
        // column r of Y: row r of I stands at row pos
        T y[N] = {};
        const T* F = S + m * nn;
        if (solve) {
            static_for<N>([&](auto row) {   // L z = e (unit diagonal)
                constexpr int i = decltype(row)::value;
                if (i >= n) return;
                T s = i == pos ? T(1) : T(0);
                static_for<i>([&](auto col) {
                    constexpr int j = decltype(col)::value;
                    s = fma(-F[i * n + j], y[j], s);
                });
                y[i] = s;
            });
            static_for<N>([&](auto row) {   // U y = z
                constexpr int i = N - 1 - decltype(row)::value;
                if (i >= n) return;
                T s = y[i];
                static_for<N - 1 - i>([&](auto col) {
                    constexpr int j = i + 1 + decltype(col)::value;
                    if (j < n) s = fma(-F[i * n + j], y[j], s);
                });
                y[i] = s / F[i * n + i];
            });
        }
        __syncwarp();
        if (have) {   // grad[r][j] = cot * (A^-1)[j][r]
            const T g = cot[b0 + m];
#pragma unroll
            for (int j = 0; j < N; ++j)
                if (j < n) S[m * nn + r * n + j] = ok ? g * y[j] : T(0);
        }
        __syncwarp();
        lu_copy(grad + b0 * nn, S, cnt * nn, lane);
    }
}

// ---------------------------------------------------------------------------
// larger n: a warp per matrix in shared memory
// ---------------------------------------------------------------------------
__host__ __device__ inline int lu_stride(int n) { return n | 1; }

template <class T>
__host__ __device__ inline size_t warp_bytes(int n, bool grad) {
    const size_t m = (size_t)n * lu_stride(n) * sizeof(T);
    const size_t b = grad ? 2 * m + (size_t)n * sizeof(int) : m;
    return (b + 15) & ~(size_t)15;
}

template <class T>
__device__ __forceinline__ void load_matrix(T* M, const T* A, int n, int ld, int lane) {
    for (int e = lane; e < n * n; e += 32) M[(e / n) * ld + e % n] = A[e];
}

// In-place LU with partial pivoting of the n x n matrix M (row stride ld).
// Returns false at the first pivot column without a usable value; *swaps is
// the parity of the row exchanges, piv[k] (when given) the row exchanged
// with row k.
template <class T>
__device__ bool lu_warp(T* M, int n, int ld, int lane, int* swaps, int* piv) {
    int par = 0;
    for (int k = 0; k < n; ++k) {
        T best = T(-1);
        int br = n;
        for (int r = k + lane; r < n; r += 32) {
            const T v = fabs(M[r * ld + k]);
            if (v > best) {   // rows ascend per lane: the first maximum stays
                best = v;
                br = r;
            }
        }
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            const T ov = __shfl_xor_sync(0xffffffffu, best, o);
            const int orow = __shfl_xor_sync(0xffffffffu, br, o);
            if (ov > best || (ov == best && orow < br)) {
                best = ov;
                br = orow;
            }
        }
        if (br >= n || !(best > T(0))) {   // warp-uniform after the reduction
            *swaps = par;
            return false;
        }
        if (piv && lane == 0) piv[k] = br;
        if (br != k) {
            par ^= 1;
            for (int c = lane; c < n; c += 32) {
                const T t = M[k * ld + c];
                M[k * ld + c] = M[br * ld + c];
                M[br * ld + c] = t;
            }
        }
        __syncwarp();
        const T p = M[k * ld + k];
        for (int r = k + 1 + lane; r < n; r += 32) M[r * ld + k] = M[r * ld + k] / p;
        __syncwarp();
        for (int c = k + 1 + lane; c < n; c += 32) {
            const T u = M[k * ld + c];
            for (int r = k + 1; r < n; ++r) M[r * ld + c] = fma(-M[r * ld + k], u, M[r * ld + c]);
        }
        __syncwarp();
    }
    *swaps = par;
    return true;
}

template <class T>
__global__ void __launch_bounds__(256) k_slogdet(const T* A, i64 B, int n, T* sign, T* logabs) {
    extern __shared__ __align__(16) unsigned char lu_smem[];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, wpb = blockDim.x >> 5;
    const int ld = lu_stride(n);
    T* M = reinterpret_cast<T*>(lu_smem + (size_t)w * warp_bytes<T>(n, false));
    for (i64 b = blockIdx.x * (i64)wpb + w; b < B; b += (i64)gridDim.x * wpb) {
        load_matrix(M, A + b * (i64)n * n, n, ld, lane);
        __syncwarp();
        int par = 0;
        const bool ok = lu_warp(M, n, ld, lane, &par, (int*)nullptr);
        if (lane == 0) {
            double s = par ? -1.0 : 1.0, la = 0.0;
            bool good = ok;
            for (int i = 0; good && i < n; ++i) {   // as the reference: log|u_ii| summed in FP64
                const double d = (double)M[i * ld + i];
                const double ad = fabs(d);
                if (!(ad > 0.0) || !isfinite(ad)) {
                    good = false;
                    break;
                }
                la += log(ad);
                if (d < 0.0) s = -s;
            }
            sign[b] = good ? (T)s : T(0);
            logabs[b] = good ? (T)la : (T)(-INFINITY);
        }
        __syncwarp();
    }
}

template <class T>
__global__ void __launch_bounds__(256) k_slogdet_grad(const T* A, const T* cot, i64 B, int n,
                                                      T* grad) {
    extern __shared__ __align__(16) unsigned char lu_smem[];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, wpb = blockDim.x >> 5;
    const int ld = lu_stride(n);
    unsigned char* base = lu_smem + (size_t)w * warp_bytes<T>(n, true);
    T* M = reinterpret_cast<T*>(base);
    T* Y = M + (size_t)n * ld;
    int* piv = reinterpret_cast<int*>(Y + (size_t)n * ld);
    const i64 nn = (i64)n * n;
    for (i64 b = blockIdx.x * (i64)wpb + w; b < B; b += (i64)gridDim.x * wpb) {
        load_matrix(M, A + b * nn, n, ld, lane);
        __syncwarp();
        int par = 0;
        const bool ok = lu_warp(M, n, ld, lane, &par, piv);
        T* G = grad + b * nn;
        if (!ok) {
            for (i64 e = lane; e < nn; e += 32) G[e] = T(0);
            __syncwarp();
            continue;
        }
        for (int c = lane; c < n; c += 32) {
            int pos = c;   // row of column c's one after the factorisation's swaps
            for (int k = 0; k < n; ++k) {
                if (piv[k] == pos) pos = k;
                else if (k == pos) pos = piv[k];
            }
            for (int i = 0; i < n; ++i) Y[i * ld + c] = i == pos ? T(1) : T(0);
            for (int i = 1; i < n; ++i) {   // L z = e (unit diagonal)
                T s = Y[i * ld + c];
                for (int j = 0; j < i; ++j) s = fma(-M[i * ld + j], Y[j * ld + c], s);
                Y[i * ld + c] = s;
            }
            for (int i = n - 1; i >= 0; --i) {   // U y = z
                T s = Y[i * ld + c];
                for (int j = i + 1; j < n; ++j) s = fma(-M[i * ld + j], Y[j * ld + c], s);
                Y[i * ld + c] = s / M[i * ld + i];
            }
        }
        __syncwarp();
        const T g = cot[b];
        for (i64 e = lane; e < nn; e += 32) {   // grad[i][j] = cot * (A^-1)[j][i]
            const int i = (int)(e / n), j = (int)(e % n);
            G[e] = g * Y[j * ld + i];
        }
        __syncwarp();
    }
}

// Warps per block from the shared memory each matrix needs (up to 96 KB per
// block), and the launch's dynamic shared memory.
template <class K>
void lu_launch_shape(K kernel, size_t per_warp, i64 B, int device, int& wpb, int& grid,
                     size_t& smem) {
    wpb = (int)std::max<size_t>(1, std::min<size_t>(8, (96 * 1024) / per_warp));
    smem = per_warp * wpb;
    DNQ_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    grid = (int)std::min<i64>((B + wpb - 1) / wpb, (i64)sm_count(device) * 32);
}

// Rows by lanes up to these n; past them the unrolled substitutions no longer
// fit the instruction cache.  Calls of 3e6 values (rows / a warp per matrix,
// us, 28 of each the call itself): value FP64 86 / 105 and FP32 58 / 84 at n =
// 32; gradient FP64 124 / 138 at 16 and 227 / 172 at 24; FP32 97 / 114 at 24
// and 133 / 112 at 32.
template <class T>
constexpr int lu_rows_max(bool grad) {
    return !grad ? 32 : sizeof(T) == 8 ? 16 : 24;
}

// Calls f with the smallest built row count that holds n <= MAX.
template <int MAX, class F>
void with_rows(int n, F f) {
    if (n <= 4) f(std::integral_constant<int, 4>{});
    else if (n <= 6) f(std::integral_constant<int, 6>{});
    else if (n <= 8) f(std::integral_constant<int, 8>{});
    else if (n <= 10) f(std::integral_constant<int, 10>{});
    else if (n <= 12) f(std::integral_constant<int, 12>{});
    else if (n <= 16) f(std::integral_constant<int, 16>{});
    if constexpr (MAX >= 24) {
        if (n > 16 && n <= 20) f(std::integral_constant<int, 20>{});
        else if (n > 20 && n <= 24) f(std::integral_constant<int, 24>{});
    }
    if constexpr (MAX >= 32) {
        if (n > 24) f(std::integral_constant<int, 32>{});
    }
}

template <class T>
void launch_slogdet(const T* a, i64 B, int n, T* sign, T* logabs, int device, cudaStream_t s) {
    const i64 sms = sm_count(device);
    constexpr int kMax = lu_rows_max<T>(false);
    if (n > kMax) {
        int wpb = 0, grid = 0;
        size_t smem = 0;
        lu_launch_shape(k_slogdet<T>, warp_bytes<T>(n, false), B, device, wpb, grid, smem);
        k_slogdet<T><<<grid, wpb * 32, smem, s>>>(a, B, n, sign, logabs);
    } else {
        with_rows<kMax>(n, [&](auto rows) {
            constexpr int N = decltype(rows)::value;
            const i64 per = kLuWarps * LuGroup<N>::M;
            k_slogdet_rows<T, N><<<(unsigned)std::min<i64>((B + per - 1) / per, sms * 64),
                                   kLuWarps * 32, 0, s>>>(a, B, n, sign, logabs);
        });
    }
    DNQ_CHECK_LAUNCH();
}

template <class T>
void launch_slogdet_grad(const T* a, const T* cot, i64 B, int n, T* grad, int device,
                         cudaStream_t s) {
    const i64 sms = sm_count(device);
    constexpr int kMax = lu_rows_max<T>(true);
    if (n > kMax) {
        int wpb = 0, grid = 0;
        size_t smem = 0;
        lu_launch_shape(k_slogdet_grad<T>, warp_bytes<T>(n, true), B, device, wpb, grid, smem);
        k_slogdet_grad<T><<<grid, wpb * 32, smem, s>>>(a, cot, B, n, grad);
    } else {
        with_rows<kMax>(n, [&](auto rows) {
            constexpr int N = decltype(rows)::value;
            const i64 per = kLuWarps * LuGroup<N>::M;
            const size_t smem = (size_t)per * n * n * sizeof(T);   // at most 32 KB
            k_slogdet_grad_rows<T, N><<<(unsigned)std::min<i64>((B + per - 1) / per, sms * 64),
                                        kLuWarps * 32, smem, s>>>(a, cot, B, n, grad);
        });
    }
    DNQ_CHECK_LAUNCH();
}

template <class T>
void run_slogdet(const void* A, i64 B, int n, void* sign, void* logabs, int device,
                 cudaStream_t s) {
    DIn<T> a(static_cast<const T*>(A), (size_t)B * n * n, s);
    const bool dev_s = is_device_ptr(sign), dev_l = is_device_ptr(logabs);
    DBuf<T> ts, tl;
    T* ps = static_cast<T*>(sign);
    T* pl = static_cast<T*>(logabs);
    if (!dev_s) {
        ts.alloc(B, s);
        ps = ts.p;
    }
    if (!dev_l) {
        tl.alloc(B, s);
        pl = tl.p;
    }
    launch_slogdet<T>(a.p, B, n, ps, pl, device, s);
    if (!dev_s) copy_out(static_cast<T*>(sign), ps, B, s);
    if (!dev_l) copy_out(static_cast<T*>(logabs), pl, B, s);
    DNQ_CUDA(cudaStreamSynchronize(s));
}

template <class T>
void run_slogdet_grad(const void* A, const void* cot, i64 B, int n, void* grad, int device,
                      cudaStream_t s) {
    DIn<T> a(static_cast<const T*>(A), (size_t)B * n * n, s);
    DIn<T> c(static_cast<const T*>(cot), (size_t)B, s);
    const bool dev_g = is_device_ptr(grad);
    DBuf<T> tg;
    T* pg = static_cast<T*>(grad);
    if (!dev_g) {
        tg.alloc((size_t)B * n * n, s);
        pg = tg.p;
    }
    launch_slogdet_grad<T>(a.p, c.p, B, n, pg, device, s);
    if (!dev_g) copy_out(static_cast<T*>(grad), pg, (size_t)B * n * n, s);
    DNQ_CUDA(cudaStreamSynchronize(s));
}

// The reference's argument checks (logdet_cuda.cu:92-118).
void check_batch(i64 B, int n, int precision) {
    require(precision == DNQ_F64 || precision == DNQ_F32, DNQ_ERR_INVALID,
            "precision must be DNQ_F64 or DNQ_F32");
    require(n >= 2 && n <= 64, DNQ_ERR_INVALID, "N must be in [2, 64]");
    require(B >= 1 && B <= (i64)0x7fffffff, DNQ_ERR_INVALID, "Batch size out of int32 range");
}

}  // namespace
}  // namespace dnq

using namespace dnq;

extern "C" {

int dnq_slogdet(const void* a, int64_t B, int n, int precision, void* sign, void* logabs,
                int device, void* stream) {
    DNQ_API_BEGIN
    check_batch(B, n, precision);
    require(a && sign && logabs, DNQ_ERR_INVALID, "null argument");
    DeviceGuard g(device);
    keep_pool(device);
    cudaStream_t s = (cudaStream_t)stream;
    if (precision == DNQ_F64) run_slogdet<double>(a, B, n, sign, logabs, device, s);
    else run_slogdet<float>(a, B, n, sign, logabs, device, s);
    DNQ_API_END
}

int dnq_slogdet_grad(const void* a, const void* cot_logabs, int64_t B, int n, int precision,
                     void* grad, int device, void* stream) {
    DNQ_API_BEGIN
    check_batch(B, n, precision);
    require(a && cot_logabs && grad, DNQ_ERR_INVALID, "null argument");
    DeviceGuard g(device);
    keep_pool(device);
    cudaStream_t s = (cudaStream_t)stream;
    if (precision == DNQ_F64) run_slogdet_grad<double>(a, cot_logabs, B, n, grad, device, s);
    else run_slogdet_grad<float>(a, cot_logabs, B, n, grad, device, s);
    DNQ_API_END
}

}  // extern "C"

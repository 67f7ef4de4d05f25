// Plain-arithmetic complex products (the "plain FP32" form and complex128).
//
// Replaces TensorHelpers::MultiplyTensorData (include/jet/TensorHelpers.hpp:
// 128-168), which dispatches row-major CBLAS cgemm/zgemm (m, n > 1),
// cgemv (right labels empty), cgemv^T (left labels empty) and cdotu (both
// empty) with alpha = 1, beta = 0. Here:
//  * gemm_kernel: CTA tiles of 64 x 64 down to 32 x 32 outputs by the shape
//    (kTilesC64), k slices staged by cp.async, 4 FMAs per complex
//    multiply-add. Products whose tiles would leave SMs idle split k into
//    partial sums in the workspace (GemmSplits), reduced in a fixed order.
//  * gemv_rows_kernel (n == 1) / gemv_cols_kernel (m == 1, also DOTU): split
//    over k into partial sums, reduced in a fixed order by reduce_partials
//    (deterministic).
#include <algorithm>
#include <type_traits>
#include <utility>
#include <vector>

#include "common.cuh"

namespace jetgpu {
namespace {

template <typename T> struct C2;
template <> struct C2<float> {
    using type = float2;
};
template <> struct C2<double> {
    using type = double2;
};

// Plain products, C = A B with FP32 or FP64 FMAs, k in increasing order per
// output (re: +a.re b.re, -a.im b.im; im: +a.re b.im, +a.im b.re). Every
// kernel and tile below runs that sequence, so the tile that a shape gets
// never changes the result; only a split of k does.
//
// blockIdx.z = b * splits + s: batch b (operand strides sa, sb, 0 = shared;
// C packed) and k range s (splits > 1: [s kchunk, (s + 1) kchunk), partial
// sums to C + (s * batch + b) * M * N, reduced later). Tiles come in
// row-major order over one grid dimension (N tiles fastest), so M may exceed
// 65535 tiles (2^23 rows).
template <typename V> struct GemmOperands {
    const V *A, *B;
    V *C;
    int64_t M, N, K;   // this CTA's k extent
    int64_t lda;       // A's row length (the whole k)
    int64_t m0, n0;
};

template <typename V, int BM, int BN>
__device__ __forceinline__ GemmOperands<V> GemmBlock(const V *A, const V *B, V *C, int64_t M,
                                                     int64_t N, int64_t K, int64_t sa,
                                                     int64_t sb, int splits, int64_t kchunk)
{
    const int64_t s = (int64_t)blockIdx.z % splits;
    const int64_t bz = (int64_t)blockIdx.z / splits;
    const int64_t batch = (int64_t)gridDim.z / splits;
    const int64_t k_begin = s * kchunk;
    const int64_t k_end = min(K, k_begin + kchunk);
    const int64_t tiles_n = (N + BN - 1) / BN;
    GemmOperands<V> o;
    o.A = A + bz * sa + k_begin;
    o.B = B + bz * sb + k_begin * N;
    o.C = C + (s * batch + bz) * M * N;
    o.M = M;
    o.N = N;
    o.K = k_end > k_begin ? k_end - k_begin : 0;
    o.lda = K;
    o.m0 = ((int64_t)blockIdx.x / tiles_n) * BM;
    o.n0 = ((int64_t)blockIdx.x % tiles_n) * BN;
    return o;
}

// One element by cp.async (zero-filled when !valid: nothing is read).
template <typename V> __device__ __forceinline__ void CpAsyncElem(V *smem, const V *src, bool valid)
{
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(smem);
    const int n = valid ? (int)sizeof(V) : 0; // 0: zero-fill, nothing read
    if constexpr (sizeof(V) == 8)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d), "l"(src), "r"(n)
                     : "memory");
    else
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(n)
                     : "memory");
}

// TX x TY threads, each a TM x TN block of outputs of a (TY TM) x (TX TN) tile.
// The k slices arrive by cp.async through a ring of three stages, two in
// flight, so a CTA alone on its SM does not wait out a memory latency per
// slice (with one slice in registers and one in shared memory that took 2,400
// clocks per 8 k). A thread's rows and columns come in adjacent pairs
// (complex64), so each shared-memory load brings two elements.
// complex64 is bound by FMA issue: the register file feeds about 70 % of the
// FMA pipe (56 TFLOP/s of 80) with three-operand FMAs at this reuse; packed
// FMAs (fma.rn.f32x2) measured 38, and larger tiles (128 x 64, 8 x 8 outputs a
// thread) no more than 64 x 64 while wasting more of the last wave (2187 x
// 2187 in 128 x 64 tiles is 2.07 waves).
// complex128 is bound by the FP64 pipe (1.1 TFLOP/s), whatever the block: 32 x
// 32 tiles waste least on edges and on the last wave. 900 x 770 x 515: 4.14 ->
// 2.60 ms (64 x 64 tiles were 195 CTAs on 152 SMs, 15 % padding).
template <typename T, int TM, int TN, int TX, int TY, int BK, int kMinBlocks>
__global__ void __launch_bounds__(TX *TY, kMinBlocks)
    gemm_kernel(const typename C2<T>::type *__restrict__ A,
                const typename C2<T>::type *__restrict__ B,
                typename C2<T>::type *__restrict__ C, int64_t M, int64_t N, int64_t K, T scale,
                int64_t sa, int64_t sb, int splits, int64_t kchunk)
{
    using V = typename C2<T>::type;
    constexpr int kThreads = TX * TY, BM = TY * TM, BN = TX * TN, NS = 3;
    constexpr int G = 16 / sizeof(V); // adjacent rows (columns) per thread and load
    static_assert(TM % G == 0 && TN % G == 0, "whole pairs");
    static_assert(BM * BK % kThreads == 0 && BN * BK % kThreads == 0, "whole loads");
    struct alignas(16) Pack {
        V v[G];
    };
    __shared__ __align__(16) V As[NS][BK][BM + G];
    __shared__ __align__(16) V Bs[NS][BK][BN];
    const auto o = GemmBlock<V, BM, BN>(A, B, C, M, N, K, sa, sb, splits, kchunk);
    const int tid = threadIdx.x, tx = tid % TX, ty = tid / TX;

    auto load = [&](int st, int64_t t) {
        const int64_t k0 = t * BK;
#pragma unroll
        for (int q = 0; q < BM * BK / kThreads; ++q) {
            const int e = tid + kThreads * q, row = e / BK, col = e % BK;
            const bool ok = o.m0 + row < o.M && k0 + col < o.K;
            CpAsyncElem(&As[st][col][row], ok ? o.A + (o.m0 + row) * o.lda + k0 + col : A, ok);
        }
#pragma unroll
        for (int q = 0; q < BN * BK / kThreads; ++q) {
            const int e = tid + kThreads * q, row = e / BN, col = e % BN;
            const bool ok = k0 + row < o.K && o.n0 + col < o.N;
            CpAsyncElem(&Bs[st][row][col], ok ? o.B + (k0 + row) * o.N + o.n0 + col : B, ok);
        }
    };

    V acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j)
            acc[i][j] = V{0, 0};
    const int64_t ktiles = (o.K + BK - 1) / BK;
    // Every iteration commits one group (empty past the last slice), so
    // wait_group NS - 2 always means "slice t has landed".
#pragma unroll
    for (int q = 0; q < NS - 1; ++q) {
        if (q < ktiles)
            load(q, q);
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    }
    int st = 0;
    for (int64_t t = 0; t < ktiles; ++t) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(NS - 2) : "memory");
        __syncthreads(); // slice t is visible, and slice t - 1 has been read
        if (t + NS - 1 < ktiles)
            load(st == 0 ? NS - 1 : st - 1, t + NS - 1);
        asm volatile("cp.async.commit_group;\n" ::: "memory");
#pragma unroll
        for (int k = 0; k < BK; ++k) {
            V a[TM], b[TN];
#pragma unroll
            for (int i = 0; i < TM; i += G) {
                const Pack w = *reinterpret_cast<const Pack *>(&As[st][k][G * ty + TY * i]);
#pragma unroll
                for (int u = 0; u < G; ++u)
                    a[i + u] = w.v[u];
            }
#pragma unroll
            for (int j = 0; j < TN; j += G) {
                const Pack w = *reinterpret_cast<const Pack *>(&Bs[st][k][G * tx + TX * j]);
#pragma unroll
                for (int u = 0; u < G; ++u)
                    b[j + u] = w.v[u];
            }
#pragma unroll
            for (int i = 0; i < TM; ++i) {
#pragma unroll
                for (int j = 0; j < TN; ++j) {
                    acc[i][j].x = fma(a[i].x, b[j].x, acc[i][j].x);
                    acc[i][j].y = fma(a[i].x, b[j].y, acc[i][j].y);
                }
#pragma unroll
                for (int j = 0; j < TN; ++j) {
                    acc[i][j].x = fma(-a[i].y, b[j].y, acc[i][j].x);
                    acc[i][j].y = fma(a[i].y, b[j].x, acc[i][j].y);
                }
            }
        }
        st = st + 1 == NS ? 0 : st + 1;
    }
    // Whole 16-byte pairs where C's rows allow it.
    const bool vec = o.N % G == 0 && (reinterpret_cast<uintptr_t>(o.C) & 15) == 0;
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int64_t gm = o.m0 + G * ty + TY * (i - i % G) + i % G;
        if (gm >= o.M)
            continue;
#pragma unroll
        for (int j = 0; j < TN; j += G) {
            const int64_t gn = o.n0 + G * tx + TX * j;
            Pack w;
#pragma unroll
            for (int u = 0; u < G; ++u)
                w.v[u] = V{acc[i][j + u].x * scale, acc[i][j + u].y * scale};
            if (vec) {
                if (gn < o.N)
                    *reinterpret_cast<Pack *>(o.C + gm * o.N + gn) = w;
                continue;
            }
#pragma unroll
            for (int u = 0; u < G; ++u)
                if (gn + u < o.N)
                    o.C[gm * o.N + gn + u] = w.v[u];
        }
    }
}

// Compensated (Kahan) running sum: vector-shaped products reduce long k
// ranges in one thread, where plain FP32 accumulation would lose ~log2(k)
// bits; the extra adds are free in these bandwidth-bound kernels.
template <typename T> struct KahanSum {
    T s = 0, c = 0;
    __device__ __forceinline__ void add(T x)
    {
        const T y = x - c;
        const T t = s + y;
        c = (t - s) - y;
        s = t;
    }
};

// y[b, m] (+ partial s) = sum_{k in chunk s} A_b[m, k] x_b[k]. A CTA of 8
// warps covers `rows` rows (8, 4, 2 or 1) with 8 / rows warps per row, which
// interleave the row's k chunk, so few rows still keep every warp streaming.
// Batch b = blockIdx.z (operand strides sa, sb; 0 = shared). Partial s of row
// (b, m) lands at out[(s * batch + b) * M + m].
template <typename T>
__global__ void __launch_bounds__(256)
    gemv_rows_kernel(const typename C2<T>::type *__restrict__ A,
                     const typename C2<T>::type *__restrict__ x,
                     typename C2<T>::type *__restrict__ out, int64_t M,
                     int64_t K, int64_t kchunk, T scale, int64_t sa, int64_t sb, int rows)
{
    using V = typename C2<T>::type;
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const int wpr = 8 / rows; // warps per row
    const int part = warp % wpr;
    const int64_t m = (int64_t)blockIdx.x * rows + warp / wpr;
    const int64_t s = blockIdx.y;
    const int64_t b = blockIdx.z;
    A += b * sa;
    x += b * sb;
    out += (s * gridDim.z + b) * M;
    const int64_t k_begin = s * kchunk;
    const int64_t k_end = min(K, k_begin + kchunk);
    KahanSum<T> sr, si;
    if (m < M) {
        // Four products per compensated add: four loads in flight per thread
        // and a quarter of the compensation work (the sum of four products
        // carries one rounding of the plain FMA chain). Several groups' loads at
        // once, as in gemv_cols_kernel, cost more registers than they hide
        // here: complex64 100 x 3000 6.6 us with one group, 7.1 with two, 8.1
        // with four, 4096 x 4096 26, 30 and 32.
        const int64_t step = wpr * 32;
        int64_t k = k_begin + part * 32 + lane;
        for (; k + 3 * step < k_end; k += 4 * step) {
            V a[4], xv[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                a[u] = A[m * K + k + u * step];
                xv[u] = x[k + u * step];
            }
            T re = a[0].x * xv[0].x - a[0].y * xv[0].y;
            T im = a[0].x * xv[0].y + a[0].y * xv[0].x;
#pragma unroll
            for (int u = 1; u < 4; ++u) {
                re = fma(a[u].x, xv[u].x, fma(-a[u].y, xv[u].y, re));
                im = fma(a[u].x, xv[u].y, fma(a[u].y, xv[u].x, im));
            }
            sr.add(re);
            si.add(im);
        }
        for (; k < k_end; k += step) {
            V a = A[m * K + k], b = x[k];
            sr.add(fma(a.x, b.x, -a.y * b.y));
            si.add(fma(a.x, b.y, a.y * b.x));
        }
    }
    T re = sr.s, im = si.s;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        re += __shfl_xor_sync(0xffffffffu, re, o);
        im += __shfl_xor_sync(0xffffffffu, im, o);
    }
    __shared__ T wre[8], wim[8];
    if (lane == 0) {
        wre[warp] = re;
        wim[warp] = im;
    }
    __syncthreads();
    if (lane == 0 && part == 0 && m < M) {
        for (int w = 1; w < wpr; ++w) { // fixed order: deterministic
            re += wre[warp + w];
            im += wim[warp + w];
        }
        out[m] = V{re * scale, im * scale};
    }
}

// y[b, n] (+ partial s) = sum_{k in chunk s} x_b[k] B_b[k, n]. A CTA of 256
// threads covers `cols` columns (a power of two up to 256) with 256 / cols
// threads per column, which interleave the k chunk: thread t takes column
// t % cols and rows k = t / cols (mod 256 / cols), so consecutive threads read
// consecutive elements of B's rows. `cols` = 1 is the dot product. Batch b =
// blockIdx.z (strides sa, sb; 0 = shared). Partial s of column (b, n) lands at
// out[(s * batch + b) * N + n].
// G: groups of four products whose loads a thread issues at once. A thread of
// a narrow B waits out a memory latency per group: two groups, us against one
// and four, complex64 1 x 256 x 1024 55 (139, 71), 1 x 4096 x 4096 151 (375, 211),
// 81 of 1 x 243 x 243 18.7 (35.0, 19.4); complex128 1 x 4096 x 4096 499 (565).
// complex128 dot products take one: k = 2^22 84 (two 126).
template <typename T, int G>
__global__ void __launch_bounds__(256)
    gemv_cols_kernel(const typename C2<T>::type *__restrict__ x,
                     const typename C2<T>::type *__restrict__ B,
                     typename C2<T>::type *__restrict__ out, int64_t N,
                     int64_t K, int64_t kchunk, T scale, int64_t sa, int64_t sb, int cols)
{
    using V = typename C2<T>::type;
    const int64_t s = blockIdx.y;
    const int64_t b = blockIdx.z;
    const int tk_count = 256 / cols;
    const int tn = threadIdx.x % cols;
    const int tk = threadIdx.x / cols;
    const int64_t n = (int64_t)blockIdx.x * cols + tn;
    const int64_t k_begin = s * kchunk;
    const int64_t k_end = min(K, k_begin + kchunk);
    x += b * sa;
    B += b * sb;
    out += (s * gridDim.z + b) * N;
    KahanSum<T> sr, si;
    if (n < N) {
        // Four products per compensated add, the loads of G groups at once
        // (see gemv_rows_kernel).
        int64_t k = k_begin + tk;
        if constexpr (G > 1)
        for (; k + (4 * G - 1) * (int64_t)tk_count < k_end; k += 4 * G * (int64_t)tk_count) {
            V a[4 * G], v[4 * G];
#pragma unroll
            for (int u = 0; u < 4 * G; ++u) {
                a[u] = x[k + u * tk_count];
                v[u] = B[(k + u * tk_count) * N + n];
            }
#pragma unroll
            for (int g = 0; g < G; ++g) {
                T re = a[4 * g].x * v[4 * g].x - a[4 * g].y * v[4 * g].y;
                T im = a[4 * g].x * v[4 * g].y + a[4 * g].y * v[4 * g].x;
#pragma unroll
                for (int u = 4 * g + 1; u < 4 * g + 4; ++u) {
                    re = fma(a[u].x, v[u].x, fma(-a[u].y, v[u].y, re));
                    im = fma(a[u].x, v[u].y, fma(a[u].y, v[u].x, im));
                }
                sr.add(re);
                si.add(im);
            }
        }
        for (; k + 3 * (int64_t)tk_count < k_end; k += 4 * (int64_t)tk_count) {
            V a[4], v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                a[u] = x[k + u * tk_count];
                v[u] = B[(k + u * tk_count) * N + n];
            }
            T re = a[0].x * v[0].x - a[0].y * v[0].y;
            T im = a[0].x * v[0].y + a[0].y * v[0].x;
#pragma unroll
            for (int u = 1; u < 4; ++u) {
                re = fma(a[u].x, v[u].x, fma(-a[u].y, v[u].y, re));
                im = fma(a[u].x, v[u].y, fma(a[u].y, v[u].x, im));
            }
            sr.add(re);
            si.add(im);
        }
        for (; k < k_end; k += tk_count) {
            V a = x[k], v = B[k * N + n];
            sr.add(fma(a.x, v.x, -a.y * v.y));
            si.add(fma(a.x, v.y, a.y * v.x));
        }
    }
    if (tk_count == 1) {
        if (n < N)
            out[n] = V{sr.s * scale, si.s * scale};
        return;
    }
    __shared__ T pre[256], pim[256];
    pre[threadIdx.x] = sr.s;
    pim[threadIdx.x] = si.s;
    __syncthreads();
    if (tk == 0 && n < N) {
        T re = 0, im = 0;
        for (int j = 0; j < tk_count; ++j) { // fixed order: deterministic
            re += pre[j * cols + tn];
            im += pim[j * cols + tn];
        }
        out[n] = V{re * scale, im * scale};
    }
}

// One k of a small output's tile: lane (rg, cg) adds its TR x TC block, `a` and
// `b` at its values of the k's rows.
template <typename T, int TR, int TC>
__device__ __forceinline__ void SmallMac(typename C2<T>::type (&acc)[TR][TC],
                                         const typename C2<T>::type *as,
                                         const typename C2<T>::type *bs)
{
    using V = typename C2<T>::type;
    constexpr int G = 16 / sizeof(V); // elements per 16-byte shared-memory load
    struct alignas(16) Pack {
        V v[G];
    };
    V a[TR], b[TC];
#pragma unroll
    for (int r = 0; r < TR; r += G) {
        if constexpr (TR % G != 0) {
            a[r] = as[r];
            continue;
        }
        const Pack w = *reinterpret_cast<const Pack *>(as + r);
#pragma unroll
        for (int u = 0; u < G; ++u)
            a[r + u] = w.v[u];
    }
#pragma unroll
    for (int c = 0; c < TC; c += G) {
        if constexpr (TC % G != 0) {
            b[c] = bs[c];
            continue;
        }
        const Pack w = *reinterpret_cast<const Pack *>(bs + c);
#pragma unroll
        for (int u = 0; u < G; ++u)
            b[c + u] = w.v[u];
    }
#pragma unroll
    for (int r = 0; r < TR; ++r) {
#pragma unroll
        for (int c = 0; c < TC; ++c) {
            acc[r][c].x = fma(a[r].x, b[c].x, acc[r][c].x);
            acc[r][c].y = fma(a[r].x, b[c].y, acc[r][c].y);
        }
#pragma unroll
        for (int c = 0; c < TC; ++c) {
            acc[r][c].x = fma(-a[r].y, b[c].y, acc[r][c].x);
            acc[r][c].y = fma(a[r].y, b[c].x, acc[r][c].y);
        }
    }
}

// The eight warps' sums in warp order through `red` (MT x NT), then to C.
template <typename T, int MT, int NT>
__device__ __forceinline__ void SmallFinish(const typename C2<T>::type (&acc)[MT / 4][NT / 8],
                                            typename C2<T>::type *red, typename C2<T>::type *C,
                                            int64_t M, int64_t N, T scale)
{
    using V = typename C2<T>::type;
    constexpr int TR = MT / 4, TC = NT / 8;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int rg = lane >> 3, cg = lane & 7;
    for (int w = 0; w < 8; ++w) {
        if (warp == w) {
#pragma unroll
            for (int r = 0; r < TR; ++r)
#pragma unroll
                for (int c = 0; c < TC; ++c) {
                    V &o = red[(rg * TR + r) * NT + cg * TC + c];
                    if (w == 0)
                        o = acc[r][c];
                    else
                        o = V{o.x + acc[r][c].x, o.y + acc[r][c].y};
                }
        }
        __syncthreads();
    }
    for (int64_t e = tid; e < M * N; e += 256) {
        const V v = red[(e / N) * NT + e % N];
        C[e] = V{v.x * scale, v.y * scale};
    }
}

// Products with a small output and a long k: M <= 16 and N <= 32, or M <= 32
// and N <= 16, with k >= 2048 -- steps that close two large tensors down to a
// few values, such as the 16 x 32 x 2^21 step of the reference's m10 network,
// where gemm_kernel's 32 x 64 tile is three quarters empty and streams 8 k per
// pass with few loads in flight (1.06 ms, 0.76 TB/s). Here one CTA per
// (k range, batch item):
//  * the A (MT x KC, stored k-major) and B (KC x NT) tiles of the range come in
//    by cp.async, double-buffered, elements past M, N or the range zero-filled;
//    KC = 32 (complex64) or 16 (complex128), so each warp has four (two) k per
//    tile between barriers;
//  * the 8 warps split every tile, each lane accumulating an
//    (MT / 4) x (NT / 8) block, so each warp covers the whole output. MT x NT is
//    the smallest of 4 x 8, 8 x 16, 16 x 16, 16 x 32 and 32 x 16 that holds the
//    output (2 x 2 outputs in 16 x 32 tiles cost as much as 512); which k a warp
//    adds does not depend on it;
//  * the warps' sums are added in warp order in shared memory and the k
//    ranges' in the workspace by reduce_partials: a fixed order.
// Bound by FMA issue at 16 x 32 (complex128: by the FP64 pipe), by its barriers
// below. 16 x 32 x 2^21 complex64: 361 -> 253 us with padded rows in the place of
// an XOR per load and with pointers that advance; 2 x 2 x 2^21 350 -> 60;
// complex128 4 x 8 x 2^17 547 -> 49.
template <typename T, int MT, int NT>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 3 : 1)
    gemm_small_kernel(const typename C2<T>::type *__restrict__ A,
                      const typename C2<T>::type *__restrict__ B,
                      typename C2<T>::type *__restrict__ C, int64_t M, int64_t N, int64_t K,
                      T scale, int64_t sa, int64_t sb, int64_t kchunk)
{
    using V = typename C2<T>::type;
    constexpr int TR = MT / 4, TC = NT / 8;
    static_assert((TR == 1 || TR % 2 == 0) && (TC == 1 || TC % 2 == 0), "one or whole pairs");
    constexpr int kSmallKC = sizeof(T) == 4 ? 32 : 16;
    constexpr int NS = 2; // stages (three measured 5 % slower: occupancy, not latency, binds)
    constexpr int G = 16 / sizeof(V); // elements per 16-byte shared-memory load: rows' padding
    // Copies per thread (the smallest tiles leave some threads without).
    constexpr int AP = (MT * kSmallKC + 255) / 256, BP = (NT * kSmallKC + 255) / 256;
    __shared__ __align__(16) V As[NS][kSmallKC][MT + G];
    __shared__ __align__(16) V Bs[NS][kSmallKC][NT];
    __shared__ V red[MT * NT];
    const int64_t s = blockIdx.x, bz = blockIdx.z, batch = gridDim.z;
    A += bz * sa;
    B += bz * sb;
    C += (s * batch + bz) * M * N;
    const int64_t k_begin = s * kchunk;
    const int64_t k_end = min(K, k_begin + kchunk);
    const int64_t tiles = k_end > k_begin ? (k_end - k_begin + kSmallKC - 1) / kSmallKC : 0;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int rg = lane >> 3, cg = lane & 7;

    // This thread's copies of a tile: elements (i, kk) of A, (kk, j) of B, at
    // pointers that advance with the tiles.
    const int a_kk = tid % kSmallKC, a_i = tid / kSmallKC;
    const int b_j = tid % NT, b_kk = tid / NT;
    const V *pa = A + a_i * K + k_begin + a_kk;
    const V *pb = B + (k_begin + b_kk) * N + b_j;
    const int64_t a_step = (int64_t)(256 / kSmallKC) * K, b_step = (int64_t)(256 / NT) * N;
    int64_t left = k_end - k_begin; // k from the next tile to load on
    auto load = [&](int st) {
#pragma unroll
        for (int q = 0; q < AP; ++q) {
            const int i = a_i + q * (256 / kSmallKC);
            const bool ok = i < M && a_kk < left;
            if (MT * kSmallKC >= 256 || i < MT)
                CpAsyncElem(&As[st][a_kk][i], ok ? pa + q * a_step : A, ok);
        }
#pragma unroll
        for (int q = 0; q < BP; ++q) {
            const int kk = b_kk + q * (256 / NT);
            const bool ok = b_j < N && kk < left;
            if (NT * kSmallKC >= 256 || kk < kSmallKC)
                CpAsyncElem(&Bs[st][kk][b_j], ok ? pb + q * b_step : B, ok);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
        pa += kSmallKC;
        pb += (int64_t)kSmallKC * N;
        left -= kSmallKC;
    };

    V acc[TR][TC];
#pragma unroll
    for (int r = 0; r < TR; ++r)
#pragma unroll
        for (int c = 0; c < TC; ++c)
            acc[r][c] = V{0, 0};
    // Every iteration commits one group (empty past the last tile), so
    // wait_group NS - 1 always means "tile t has landed".
    if (tiles > 0)
        load(0);
    int st = 0;
    for (int64_t t = 0; t < tiles; ++t) {
        if (t + 1 < tiles)
            load(st ^ 1);
        else
            asm volatile("cp.async.commit_group;\n" ::: "memory");
        asm volatile("cp.async.wait_group %0;\n" ::"n"(NS - 1) : "memory");
        __syncthreads();
#pragma unroll
        for (int kk = warp; kk < kSmallKC; kk += 8) {
            SmallMac<T, TR, TC>(acc, &As[st][kk][rg * TR], &Bs[st][kk][cg * TC]);
        }
        __syncthreads(); // the next load reuses this stage
        st ^= 1;
    }
    SmallFinish<T, MT, NT>(acc, red, C, M, N, scale);
}

// Small outputs over a long k whose operands' axes are interleaved, read where
// they lie: power-of-2 extents, so an element's place is a permutation of its
// index bits. Transposing both operands first moves each twice more, which is
// half of a closing step's time (16 x 32 x 2^21: two transposes 245 us of 499).
//  * A tile is all of M and N and 2^kClosingLog k: the k bits lowest in A and
//    lowest in B in turn, so both are read in runs of 64 bytes (complex64; a
//    free axis among the low bits lengthens them). Tiles follow the next k
//    bits up, so a CTA's consecutive tiles finish the lines around them.
//  * A thread's copies stand at offsets fixed for the kernel from a base that
//    moves by one addition per tile: from tile t to t + 1 it is the plan's
//    step for the number of trailing ones of t.
//  * In shared memory a k's row is padded by 16 bytes and every eight rows by
//    16 more: copies along the low and along the high k bits then both spread
//    over the banks.
// The product is gemm_small_kernel's, over the k in the tiles' order, and bounds
// it at 16 x 32 outputs (issue of FMAs and the loads that feed a lane's 4 x 4
// block, 32 TFLOP/s; complex128 the FP64 pipe). 16 x 32 x 2^21
// with both transposes before: 499 us, now 268; 4 x 8 x 2^21 reads 3.0 TB/s.
constexpr int kClosingMaxBits = 32;
template <typename T> constexpr int kClosingLog = sizeof(T) == 4 ? 6 : 5;

struct ClosingSide {
    uint32_t src[11]; // element bit (in the order of memory): its offset there,
    uint32_t dst[11]; // ... and in a stage's rows
    uint32_t tile[kClosingMaxBits]; // tile index bit: its offset
    uint32_t step[kClosingMaxBits]; // from tile t to t + 1, by t's trailing ones
};

struct ClosingPlan {
    ClosingSide a, b;
    int tile_bits;
};

// A k's row in shared memory, of `width` elements.
template <typename V> __host__ __device__ __forceinline__ int ClosingRow(int kk, int width)
{
    constexpr int G = 16 / sizeof(V);
    return kk * (width + G) + (kk >> 3) * G;
}

// Where the element bits from `first` on of e place it (bits past the tile's
// are zero in the plan).
__host__ __device__ __forceinline__ void ClosingElement(const ClosingSide &p, int e, int first,
                                                        int last, uint32_t &src, uint32_t &dst)
{
    src = dst = 0;
#pragma unroll
    for (int b = first; b < last; ++b)
        if (e >> b & 1) {
            src += p.src[b];
            dst += p.dst[b];
        }
}

template <typename T, int MT, int NT> constexpr size_t ClosingShared()
{
    using V = typename C2<T>::type;
    constexpr int KC = 1 << kClosingLog<T>, G = 16 / sizeof(V);
    return 2 * (size_t)(KC * (MT + G) + KC / 8 * G + KC * (NT + G) + KC / 8 * G) * sizeof(V);
}

template <typename T, int MT, int NT>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 3 : 1)
    closing_kernel(const typename C2<T>::type *__restrict__ A,
                   const typename C2<T>::type *__restrict__ B, typename C2<T>::type *__restrict__ C,
                   int M, int N, uint32_t tiles, uint32_t per_cta, T scale,
                   const __grid_constant__ ClosingPlan p)
{
    using V = typename C2<T>::type;
    constexpr int TR = MT / 4, TC = NT / 8;
    constexpr int KC = 1 << kClosingLog<T>, G = 16 / sizeof(V);
    constexpr int AP = (MT * KC + 255) / 256, BP = (NT * KC + 255) / 256; // copies per thread
    constexpr int kARows = KC * (MT + G) + KC / 8 * G, kBRows = KC * (NT + G) + KC / 8 * G;
    static_assert(2 * (kARows + kBRows) >= MT * NT, "the sums reuse the stages");
    extern __shared__ __align__(16) unsigned char closing_smem[];
    V *const sm = reinterpret_cast<V *>(closing_smem); // two stages of A rows, B rows
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int rg = lane >> 3, cg = lane & 7;
    const uint32_t t0 = blockIdx.x * per_cta;
    const uint32_t t1 = min(tiles, t0 + per_cta);

    // Rows and columns past M and N stay zero.
    for (int e = tid; e < 2 * (kARows + kBRows); e += 256)
        sm[e] = V{0, 0};
    // This thread's elements are tid + 256 q: the low bits once, q's from the plan.
    uint32_t a_src, a_dst, b_src, b_dst;
    ClosingElement(p.a, tid, 0, 8, a_src, a_dst);
    ClosingElement(p.b, tid, 0, 8, b_src, b_dst);
    const int a_count = M * KC, b_count = N * KC;
    uint32_t a_base = 0, b_base = 0; // of the next tile to load
    for (int b = 0; b < p.tile_bits; ++b)
        if (t0 >> b & 1) {
            a_base += p.a.tile[b];
            b_base += p.b.tile[b];
        }
    auto load = [&](uint32_t t, int st) {
        V *as = sm + st * (kARows + kBRows), *bs = as + kARows;
#pragma unroll
        for (int q = 0; q < AP; ++q)
            if (tid + 256 * q < a_count) {
                uint32_t src, dst;
                ClosingElement(p.a, 256 * q, 8, 11, src, dst);
                CpAsyncElem(as + a_dst + dst, A + (a_base + a_src + src), true);
            }
#pragma unroll
        for (int q = 0; q < BP; ++q)
            if (tid + 256 * q < b_count) {
                uint32_t src, dst;
                ClosingElement(p.b, 256 * q, 8, 11, src, dst);
                CpAsyncElem(bs + b_dst + dst, B + (b_base + b_src + src), true);
            }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
        const int ones = __ffs(~t) - 1;
        a_base += p.a.step[ones];
        b_base += p.b.step[ones];
    };

    V acc[TR][TC];
#pragma unroll
    for (int r = 0; r < TR; ++r)
#pragma unroll
        for (int c = 0; c < TC; ++c)
            acc[r][c] = V{0, 0};
    __syncthreads(); // the zeros are in place
    if (t0 < t1)
        load(t0, 0);
    int st = 0;
    for (uint32_t t = t0; t < t1; ++t) {
        if (t + 1 < t1)
            load(t + 1, st ^ 1);
        else
            asm volatile("cp.async.commit_group;\n" ::: "memory");
        asm volatile("cp.async.wait_group 1;\n" ::: "memory"); // all but the newest group
        __syncthreads();
        const V *as = sm + st * (kARows + kBRows), *bs = as + kARows;
#pragma unroll
        for (int u = 0; u < KC / 8; ++u) {
            const int kk = warp + 8 * u;
            SmallMac<T, TR, TC>(acc, as + ClosingRow<V>(kk, MT) + rg * TR,
                                bs + ClosingRow<V>(kk, NT) + cg * TC);
        }
        __syncthreads(); // the next load reuses this stage
        st ^= 1;
    }
    SmallFinish<T, MT, NT>(acc, sm, C + (int64_t)blockIdx.x * M * N, M, N, scale);
}

// Sums of the k ranges' partial results, accumulated in FP64: the partials
// of a long product can be much larger than their sum (an amplitude is a sum
// of terms of both signs), so FP32 adds here would cost accuracy the k ranges
// kept.
template <typename T>
__global__ void reduce_partials(const typename C2<T>::type *__restrict__ part,
                                typename C2<T>::type *__restrict__ out,
                                int64_t len, int64_t S)
{
    using V = typename C2<T>::type;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < len;
         i += (int64_t)gridDim.x * blockDim.x) {
        double re = 0, im = 0;
        for (int64_t s = 0; s < S; ++s) {
            V v = part[s * len + i];
            re += v.x;
            im += v.y;
        }
        out[i] = V{(T)re, (T)im};
    }
}

// reduce_partials for few outputs over many partial sums (S >= 64): one warp
// per output, lane l adding partials l, l + 32, ... in order (FP64), then a
// fixed shuffle tree -- a fixed order, where one thread per output walked the
// S partials one dependent load at a time (93 us for 512 outputs of 456 k
// ranges).
template <typename T>
__global__ void reduce_partials_warp(const typename C2<T>::type *__restrict__ part,
                                     typename C2<T>::type *__restrict__ out, int64_t len,
                                     int64_t S)
{
    using V = typename C2<T>::type;
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x / 32);
    for (int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / 32; i < len;
         i += warps) {
        double re = 0, im = 0;
#pragma unroll 4
        for (int64_t s = lane; s < S; s += 32) {
            const V v = part[s * len + i];
            re += v.x;
            im += v.y;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            re += __shfl_xor_sync(0xffffffffu, re, o);
            im += __shfl_xor_sync(0xffffffffu, im, o);
        }
        if (lane == 0)
            out[i] = V{(T)re, (T)im};
    }
}

// The sums of a jetgpu_contract product's k ranges, complex64, in range order.
// FP64 adds and conversions bound the kernel above on this GPU (2^18 outputs of
// nine ranges 24 us, their 19 MB in L2): here the running sum is a pair of
// FP32 values, the second adding up the exact rounding errors of the first's
// adds (Knuth's two-sum). Those adds of errors round too: S ranges are off by
// at most (S - 1)^2 2^-48 of the sum of their magnitudes before the last
// rounding. The range is FP32's, so a sum that leaves it on the way, or meets
// an infinity or NaN, is taken again in FP64.
struct PairSum {
    float s = 0, e = 0;
    __device__ __forceinline__ void add(float x)
    {
        const float t = s + x;
        const float b = t - s;
        e += (s - (t - b)) + (x - b);
        s = t;
    }
};

// Ranges [s, last) of output i, in order, the loads of U at once.
template <int U>
__device__ __forceinline__ void AddRanges(const float2 *__restrict__ part, int64_t len, int64_t i,
                                          int64_t s, int64_t last, PairSum &re, PairSum &im)
{
    for (; s + U <= last; s += U) {
        float2 v[U];
#pragma unroll
        for (int u = 0; u < U; ++u)
            v[u] = part[(s + u) * len + i];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            re.add(v[u].x);
            im.add(v[u].y);
        }
    }
    if constexpr (U > 1)
        AddRanges<U / (U > 4 ? 2 : 4)>(part, len, i, s, last, re, im);
}

__device__ __forceinline__ float2 SumOfRanges(const float2 *__restrict__ part, int64_t len,
                                              int64_t i, int64_t S, const PairSum &re,
                                              const PairSum &im)
{
    if (isfinite(re.s) && isfinite(im.s)) // once not finite, a sum stays so
        return make_float2(re.s + re.e, im.s + im.e);
    double x = 0, y = 0;
#pragma unroll 1
    for (int64_t s = 0; s < S; ++s) {
        x += part[s * len + i].x;
        y += part[s * len + i].y;
    }
    return make_float2((float)x, (float)y);
}

__global__ void __launch_bounds__(256)
    sum_partials_kernel(const float2 *__restrict__ part, float2 *__restrict__ out, int64_t len,
                        int64_t S)
{
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < len;
         i += (int64_t)gridDim.x * blockDim.x) {
        PairSum re, im;
        AddRanges<4>(part, len, i, 0, S, re, im);
        out[i] = SumOfRanges(part, len, i, S, re, im);
    }
}

// From kManyRanges ranges on, where one thread per output waits out a memory
// latency per four of them: the warps of a CTA each add a share of the ranges of
// 32 outputs, the first warp their sums in order. us back to back, a thread per
// output / a warp of FP64 adds / these: 289 outputs of 256 ranges 18 / 6 / 4, of
// 1,024 66 / 10 / 8; 4,096 outputs of 256 18 / 14 / 4; 65,536 of 64 8 / 98 / 10.
constexpr uint64_t kManyRanges = 64;
constexpr int kManyWarps = 16;

__global__ void __launch_bounds__(32 * kManyWarps)
    sum_many_kernel(const float2 *__restrict__ part, float2 *__restrict__ out, int64_t len,
                    int64_t S)
{
    __shared__ float4 sums[kManyWarps][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t per = (S + kManyWarps - 1) / kManyWarps;
    for (int64_t i0 = (int64_t)blockIdx.x * 32; i0 < len; i0 += (int64_t)gridDim.x * 32) {
        const int64_t i = i0 + lane;
        PairSum re, im;
        if (i < len)
            AddRanges<8>(part, len, i, min(S, warp * per), min(S, (warp + 1) * per), re, im);
        sums[warp][lane] = make_float4(re.s, re.e, im.s, im.e);
        __syncthreads();
        if (warp == 0 && i < len) {
#pragma unroll
            for (int w = 1; w < kManyWarps; ++w) {
                const float4 q = sums[w][lane];
                re.add(q.x);
                re.e += q.y;
                im.add(q.z);
                im.e += q.w;
            }
            out[i] = SumOfRanges(part, len, i, S, re, im);
        }
        __syncthreads(); // the sums are read
    }
}

// Sums S partial results of `len` elements each into out (a fixed order).
template <typename T>
int ReducePartials(const typename C2<T>::type *part, typename C2<T>::type *out, int64_t len,
                   int64_t S, cudaStream_t stream)
{
    if (S >= 64 && len <= 65536) {
        reduce_partials_warp<T><<<GridFor((len * 32 + 255) / 256, 8), 256, 0, stream>>>(
            part, out, len, S);
        return CheckLaunch("reduce_partials_warp");
    }
    reduce_partials<T><<<GridFor((len + 255) / 256, 4), 256, 0, stream>>>(part, out, len, S);
    return CheckLaunch("reduce_partials");
}

template <typename T>
__global__ void fill_zero(typename C2<T>::type *out, int64_t len)
{
    using V = typename C2<T>::type;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < len;
         i += (int64_t)gridDim.x * blockDim.x)
        out[i] = V{0, 0};
}

// Split-k factor of the matrix product when its tiles (times the batch) do
// not fill the GPU: up to two CTAs per SM, at least 256 k per split, and at
// most 32 MiB of partial sums (out_bytes: the bytes of C).
int64_t GemmSplits(int64_t ctas, int64_t batch, int64_t K, int64_t out_bytes)
{
    const int64_t target = (int64_t)SmCount() * 2;
    if (ctas >= target / 2 || K < 512)
        return 1;
    int64_t s = (target + ctas - 1) / ctas;
    s = min(s, K / 256);
    s = min(s, (int64_t)65535 / (batch > 0 ? batch : 1));
    s = min(s, (int64_t)(32ll << 20) / (out_bytes > 0 ? out_bytes : 1));
    return s < 2 ? 1 : s;
}

// The small-output kernel's tile (MT x NT; 0: the product is not one) and
// its k ranges: one wave of CTAs (the kernel's launch bounds guarantee three
// per SM for complex64, one for complex128; a second, partial wave cost a
// third of the time), at least 1024 k each, at most 32 MiB of partial sums.
inline void SmallTile(int64_t M, int64_t N, int64_t K, int &mt, int &nt)
{
    mt = nt = 0;
    if (K < 2048 || M < 2 || N < 2)
        return;
    if (M <= 4 && N <= 8) {
        mt = 4;
        nt = 8;
    } else if (M <= 8 && N <= 16) {
        mt = 8;
        nt = 16;
    } else if (M <= 16 && N <= 16) {
        mt = nt = 16;
    } else if (M <= 16 && N <= 32) {
        mt = 16;
        nt = 32;
    } else if (M <= 32 && N <= 16) {
        mt = 32;
        nt = 16;
    }
}

int64_t SmallSplits(int64_t batch, int64_t K, int64_t out_bytes, size_t elem_bytes)
{
    int64_t s = (int64_t)SmCount() * (elem_bytes == 8 ? 3 : 1) / (batch > 0 ? batch : 1);
    s = min(s, K / 1024);
    s = min(s, (int64_t)(32ll << 20) / (out_bytes > 0 ? out_bytes : 1));
    return s < 2 ? 1 : s;
}

// The tiles of the matrix product and the measured clocks that one k of a tile
// takes: in a CTA alone on its SM, and as its share of a full SM. A launch
// takes the tile whose busiest SM finishes first: large products 64 x 64, or
// 64 x 32 of 64 threads where 64 x 64 would leave the last wave thin; products
// of few tiles the smaller blocks, whose CTAs finish sooner. Measured against
// 128 x 64 tiles alone: 2187 x 2187 x 729 713 -> 568 us, 512 x 32 x 512 55 ->
// 14, 9 x (81 x 243 x 243) 52 -> 17, 16 x (1024 x 8192 x 16) 456 -> 438, 4096 x
// 4096 x 1024 2,765 -> 2,450.
struct GemmTile {
    int bm, bn;
    double alone, shared;
};
constexpr GemmTile kTilesC64[] = {
    {64, 64, 215, 183}, // 8 x 4 a thread, 128 threads
    {64, 64, 199, 188}, // 4 x 4, 256 threads
    {64, 32, 215, 97},  // 8 x 4, 64 threads
    {64, 32, 122, 105}, // 4 x 2, 256 threads
    {32, 64, 128, 112}, // 2 x 4
    {32, 32, 83, 61},   // 2 x 2
    // Short k only (PickTileC64): no clocks.
    {64, 64, 0, 0}, // 4 x 4, 256 threads, 8 k a slice
    {32, 64, 0, 0}, // 4 x 4, 128 threads, 8 k a slice
};
constexpr int kLongTilesC64 = 6;
constexpr GemmTile kTileC128 = {32, 32, 2100, 2100};

inline int64_t CeilDiv(int64_t a, int64_t b) { return (a + b - 1) / b; }

// Clocks per k on the busiest SM of a launch over `z` products of M x N.
inline double TileClocks(const GemmTile &t, int64_t M, int64_t N, int64_t z)
{
    const int64_t per_sm = CeilDiv(CeilDiv(M, t.bm) * CeilDiv(N, t.bn) * z, SmCount());
    return std::max(t.alone, (double)per_sm * t.shared);
}

// Split-k factor of a batched product (fixed: the slices of a sliced network
// keep their bits whatever tile a launch gets): GemmSplits over tiles of 128
// (complex64) or 64 (complex128) rows, 32 when M <= 32, and 64 columns.
template <typename T> int64_t BatchedSplits(int64_t batch, int64_t M, int64_t N, int64_t K)
{
    const int64_t bm = M <= 32 ? 32 : (sizeof(T) == 4 ? 128 : 64);
    return GemmSplits(CeilDiv(M, bm) * CeilDiv(N, 64) * batch, batch, K,
                      batch * M * N * (int64_t)(2 * sizeof(T)));
}

// k ranges of one product (jetgpu_contract): products of few tiles leave SMs
// idle, so k is cut while the busiest SM then finishes sooner, adding the
// ranges' sums (a launch, and their bytes through L2) included. At least 64 k
// a range, and none below 256: steps of k <= 64 add in one order everywhere
// (grouped launches and skinny kernels give the same bits). At most 1,024 of
// complex64: past that a CTA's own start and end cost more than the fuller last
// wave saves (2 x 40 outputs, k = 2^18: 1,024 ranges 115 us, 4,096 149). Never fewer
// than a batch of one gets, whose sums would otherwise be the closer ones: an
// output of four ranges of 839 k was 1.5 times as far off as one of nine of 373.
constexpr int64_t kSingleMinK = 256, kSingleRanges = 1024;
constexpr double kReduceClocks = 6000.0; // a launch and its latency
constexpr double kReduceBytes = 2000.0;  // partial sums per clock

// The clocks are per k, so short products, which load and store more than they
// multiply, are picked apart. A slice of 16 k is mostly zeros for k = 2..8, and the
// 32-row tiles' two or three CTAs per SM keep too little in flight. us with the
// clocks' pick / with the pick here:
//   20 x 300,000 outputs   k = 2 47 / 23, 16 50 / 37, 32 79 / 65, 65 158 / 137,
//                          128 240 / 236
//   64 of 27 x 81          k = 3 3.4 / 2.6, 27 4.6 / 4.3 (81 8.8 / 8.1)
//   500 x 500              k = 2 3.1 / 2.6, 32 4.1 / 4.1 (64 6.0 / 6.4)
//   65,536 x 33            k <= 8 12.6 / 11.3, 16 16.8 / 16.8
//   4000 x 4096            k <= 8 37.5 / 37.8
// Launches of at most one 32 x 32 tile per SM have nothing to gain.
inline int PickTileC64(int64_t M, int64_t N, int64_t K, int64_t z)
{
    int best = 0;
    for (int i = 1; i < kLongTilesC64; ++i)
        if (TileClocks(kTilesC64[i], M, N, z) < TileClocks(kTilesC64[best], M, N, z))
            best = i;
    if (K <= 8 && best == 0)
        return 6;
    const int64_t tiles = CeilDiv(M, 32) * CeilDiv(N, 32) * z;
    if ((best == 4 || best == 5) && tiles > (int64_t)SmCount() &&
        K <= (tiles > 8 * (int64_t)SmCount() ? 96 : 32))
        return 7;
    return best;
}

template <typename T> int64_t SingleSplits(int64_t M, int64_t N, int64_t K)
{
    if (K < kSingleMinK || SmCount() < 1)
        return 1;
    const int64_t first = BatchedSplits<T>(1, M, N, K);
    int64_t best = 0;
    double least = 0;
    for (int64_t S = 1; K / S >= kSingleMinK / 4; S *= 2) {
        const double bytes = (double)S * M * N * 2 * sizeof(T);
        if (S > 1 && (bytes > (double)(32 << 20) || (sizeof(T) == 4 && S > kSingleRanges)))
            break;
        if (S < first)
            continue;
        const int64_t kchunk = CeilDiv(K, S);
        const GemmTile &t = sizeof(T) == 4 ? kTilesC64[PickTileC64(M, N, kchunk, S)] : kTileC128;
        const double clocks = TileClocks(t, M, N, S) * (double)kchunk +
                              (S > 1 ? kReduceClocks + bytes / kReduceBytes : 0.0);
        if (best == 0 || clocks < least) {
            best = S;
            least = clocks;
        }
    }
    return best > 0 ? best : first;
}

// Split-k factor for the vector kernels: enough CTAs to fill the GPU, with at
// least 1024 k per chunk.
int64_t SplitK(int64_t blocks_per_split, int64_t K)
{
    int64_t target = (int64_t)SmCount() * 4;
    int64_t s = blocks_per_split >= target ? 1 : target / blocks_per_split;
    int64_t max_s = (K + 1023) / 1024;
    if (s > max_s)
        s = max_s;
    return s < 1 ? 1 : s;
}

// Smallest power of two >= v, at most `cap`.
inline int Pow2AtLeast(int64_t v, int cap)
{
    int p = 1;
    while (p < v && p < cap)
        p <<= 1;
    return p;
}

// CTAs per batch element of the vector kernels, the rows (gemv_rows_kernel)
// or columns (gemv_cols_kernel) each CTA covers, and the vector length.
inline void VectorShape(int64_t m, int64_t n, int64_t &blocks, int &per_cta, int64_t &len)
{
    if (n == 1 && m > 1) {
        per_cta = Pow2AtLeast(m, 8);
        len = m;
    }
    else {
        per_cta = Pow2AtLeast(n, 256); // 1: the dot product
        len = n;
    }
    blocks = (len + per_cta - 1) / per_cta;
}

// Bytes of partial sums the split-k vector products of `batch` products use
// (0 for matrix products or when one split suffices).
template <typename T>
size_t VectorWorkspace(int64_t batch, int64_t m, int64_t n, int64_t k)
{
    using V = typename C2<T>::type;
    if (batch < 1)
        return 0;
    if (m > 1 && n > 1) {
        int mt, nt;
        SmallTile(m, n, k, mt, nt);
        if (mt) { // small output, long k: partial sums of its k ranges
            const int64_t S =
                SmallSplits(batch, k, batch * m * n * (int64_t)sizeof(V), sizeof(V));
            return S > 1 ? (size_t)(S * batch * m * n) * sizeof(V) : 0;
        }
        // Matrix products: partial sums of the k splits.
        const int64_t S = BatchedSplits<T>(batch, m, n, k);
        return S > 1 ? (size_t)(S * batch * m * n) * sizeof(V) : 0;
    }
    int64_t blocks, len;
    int per_cta;
    VectorShape(m, n, blocks, per_cta, len);
    const int64_t S = SplitK(blocks * batch, k);
    return S > 1 ? (size_t)(S * batch * len) * sizeof(V) : 0;
}

// GEMV (n == 1), GEMV^T (m == 1) and DOTU (both) of `batch` products, split
// over k into partial sums when the caller supplied room for them, reduced
// in a fixed order (deterministic).
template <typename T>
int MultiplyVectorT(const typename C2<T>::type *A, const typename C2<T>::type *B,
                    typename C2<T>::type *C, int64_t batch, int64_t sa, int64_t sb, int64_t M,
                    int64_t N, int64_t K, T scale, void *ws, size_t ws_bytes,
                    cudaStream_t stream)
{
    using V = typename C2<T>::type;
    JETGPU_REQUIRE(batch <= 65535, "batch too large for one launch");
    const size_t need = VectorWorkspace<T>(batch, M, N, K);
    const bool split = need > 0 && ws != nullptr && ws_bytes >= need;
    int64_t blocks, len;
    int per_cta;
    VectorShape(M, N, blocks, per_cta, len);
    const int64_t S = split ? SplitK(blocks * batch, K) : 1;
    const int64_t kchunk = (K + S - 1) / S;
    V *dst = S > 1 ? (V *)ws : C;
    const dim3 grid((unsigned)blocks, (unsigned)S, (unsigned)batch);
    const auto launch = [&](auto kernel) {
        kernel<<<grid, 256, 0, stream>>>(A, B, dst, N == 1 && M > 1 ? M : N, K, kchunk, scale,
                                         sa, sb, per_cta);
    };
    if (N == 1 && M > 1)
        launch(gemv_rows_kernel<T>);
    else if (sizeof(T) == 8 && per_cta == 1)
        launch(gemv_cols_kernel<T, 1>);
    else
        launch(gemv_cols_kernel<T, 2>);
    int rc = CheckLaunch(N == 1 && M > 1 ? "gemv_rows_kernel" : "gemv_cols_kernel");
    if (rc || S == 1)
        return rc;
    return ReducePartials<T>(dst, C, batch * len, S, stream);
}

// The plan of closing_kernel, false where it does not apply: extents that are
// not powers of 2, operands past 2^31 elements, outputs that SmallTile does not
// take. Operands as ContractForm's (A permuted to (free, common), B to (common,
// free)).
bool PlanClosing(int a_rank, const uint64_t *a_shape, const int32_t *a_perm, int b_rank,
                 const uint64_t *b_shape, const int32_t *b_perm, uint64_t m, uint64_t n, uint64_t k,
                 int klog, ClosingPlan &p)
{
    int mt, nt;
    const auto pow2 = [](uint64_t v) { return v > 0 && (v & (v - 1)) == 0; };
    if (!pow2(m) || !pow2(n) || !pow2(k) || m > 32 || n > 32 || k > (1ull << 31) ||
        m * k > (1ull << 31) || n * k > (1ull << 31))
        return false;
    SmallTile((int64_t)m, (int64_t)n, (int64_t)k, mt, nt);
    if (!mt)
        return false;
    const auto log2of = [](uint64_t v) {
        int l = 0;
        while (v >>= 1)
            ++l;
        return l;
    };
    const int nk = log2of(k), nm = log2of(m), nn = log2of(n);
    // Memory bit of every bit of the permuted index, lowest first.
    int a_bit[64], b_bit[64];
    const auto bits = [&](int rank, const uint64_t *shape, const int32_t *perm, int total,
                          int *out) {
        int place[64], at = 0, cnt = 0;
        if (rank > 64)
            return false;
        for (int i = rank - 1; i >= 0; --i) {
            if (!pow2(shape[i]))
                return false;
            place[i] = at;
            at += log2of(shape[i]);
        }
        if (at != total)
            return false;
        for (int j = rank - 1; j >= 0; --j)
            for (int u = 0; u < log2of(shape[perm[j]]); ++u)
                out[cnt++] = place[perm[j]] + u;
        return true;
    };
    if (!bits(a_rank, a_shape, a_perm, nm + nk, a_bit) ||
        !bits(b_rank, b_shape, b_perm, nk + nn, b_bit))
        return false;
    const int *ak = a_bit, *am = a_bit + nk, *bn = b_bit, *bk = b_bit + nn;
    // The tile's k bits: the lowest of A and of B in turn, the larger operand
    // first.
    bool in_tile[32] = {};
    int chosen[8], count = 0;
    for (int place = 0; place < 64 && count < klog; ++place)
        for (int side = 0; side < 2; ++side)
            for (int t = 0; t < nk && count < klog; ++t)
                if (!in_tile[t] && ((side == 0) == (nn >= nm) ? bk[t] : ak[t]) == place) {
                    in_tile[t] = true;
                    chosen[count++] = t;
                }
    std::sort(chosen, chosen + klog, [&](int x, int y) { return ak[x] < ak[y]; });
    int rest[32], nrest = 0;
    for (int t = 0; t < nk; ++t)
        if (!in_tile[t])
            rest[nrest++] = t;
    std::sort(rest, rest + nrest, [&](int x, int y) {
        const int u = ak[x] < bk[x] ? ak[x] : bk[x], v = ak[y] < bk[y] ? ak[y] : bk[y];
        return u != v ? u < v : x < y;
    });
    p = ClosingPlan{};
    p.tile_bits = nrest;
    const auto side = [&](ClosingSide &s, const int *kbit, const int *free_bit, int nfree,
                          int across) {
        std::vector<std::pair<int, int>> el; // memory bit, place in shared memory
        for (int i = 0; i < klog; ++i) // additive over bits, as ClosingRow is
            el.push_back({kbit[chosen[i]], klog == kClosingLog<float>
                                               ? ClosingRow<float2>(1 << i, across)
                                               : ClosingRow<double2>(1 << i, across)});
        for (int u = 0; u < nfree; ++u)
            el.push_back({free_bit[u], 1 << u});
        std::sort(el.begin(), el.end());
        for (size_t i = 0; i < el.size(); ++i) { // at most 6 + 5
            s.src[i] = 1u << el[i].first;
            s.dst[i] = (uint32_t)el[i].second;
        }
        uint32_t below = 0; // offsets that trailing ones leave
        for (int i = 0; i < nrest; ++i) {
            s.tile[i] = 1u << kbit[rest[i]];
            s.step[i] = s.tile[i] - below;
            below += s.tile[i];
        }
        s.step[nrest] = 0u - below; // past the last tile: not loaded
    };
    side(p.a, ak, am, nm, mt);
    side(p.b, bk, bn, nn, nt);
    return true;
}

template <typename T>
int ClosingT(const ClosingPlan &p, const typename C2<T>::type *A, const typename C2<T>::type *B,
             typename C2<T>::type *C, int64_t M, int64_t N, int64_t K, T scale, void *ws,
             size_t ws_bytes, cudaStream_t stream)
{
    using V = typename C2<T>::type;
    const int64_t tiles = K >> kClosingLog<T>;
    // One wave; four tiles a CTA at least, or one where a tile keeps the FP64
    // pipe busy for 20 us; the ranges' sums fit the workspace.
    int64_t S = std::min<int64_t>((int64_t)SmCount() * (sizeof(T) == 4 ? 3 : 1),
                                  sizeof(T) == 4 ? tiles / 4 : tiles);
    S = std::min<int64_t>(S, ws ? (int64_t)(ws_bytes / (size_t)(M * N * (int64_t)sizeof(V))) : 1);
    S = std::max<int64_t>(S, 1);
    const int64_t per_cta = CeilDiv(tiles, S);
    S = CeilDiv(tiles, per_cta);
    V *dst = S > 1 ? (V *)ws : C;
    int mt, nt;
    SmallTile(M, N, K, mt, nt);
    int rc = JETGPU_OK;
    const auto launch = [&](auto kernel, size_t shared) {
        // Enqueues nothing: a captured stream takes it too.
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)shared) != cudaSuccess)
            rc = SetError(JETGPU_ERR_CUDA, "closing_kernel: shared memory limit not set");
        else
            kernel<<<(unsigned)S, 256, shared, stream>>>(A, B, dst, (int)M, (int)N,
                                                         (uint32_t)tiles, (uint32_t)per_cta,
                                                         scale, p);
    };
    if (mt == 4)
        launch(closing_kernel<T, 4, 8>, ClosingShared<T, 4, 8>());
    else if (mt == 8)
        launch(closing_kernel<T, 8, 16>, ClosingShared<T, 8, 16>());
    else if (mt == 16 && nt == 16)
        launch(closing_kernel<T, 16, 16>, ClosingShared<T, 16, 16>());
    else if (mt == 16)
        launch(closing_kernel<T, 16, 32>, ClosingShared<T, 16, 32>());
    else
        launch(closing_kernel<T, 32, 16>, ClosingShared<T, 32, 16>());
    if (rc || (rc = CheckLaunch("closing_kernel")) || S == 1)
        return rc;
    return ReducePartials<T>(dst, C, M * N, S, stream);
}

// Matrix product of `batch` pairs (strides sa, sb; 0 = shared), split over k
// into the workspace when the tiles alone would leave SMs idle and the caller
// supplied room for the partial sums (reduced in a fixed order).
template <typename T>
int GemmT(const typename C2<T>::type *A, const typename C2<T>::type *B, typename C2<T>::type *C,
          int64_t batch, int64_t sa, int64_t sb, int64_t M, int64_t N, int64_t K, T scale,
          void *ws, size_t ws_bytes, cudaStream_t stream, int64_t single_splits = 0)
{
    using V = typename C2<T>::type;
    const size_t need = VectorWorkspace<T>(batch, M, N, K);
    int mt, nt;
    SmallTile(M, N, K, mt, nt);
    if (mt) {
        JETGPU_REQUIRE(batch <= 65535, "batch too large for one launch");
        const int64_t S = (need > 0 && ws != nullptr && ws_bytes >= need)
                              ? SmallSplits(batch, K, batch * M * N * (int64_t)sizeof(V),
                                            sizeof(V))
                              : 1;
        const int64_t kchunk = (K + S - 1) / S;
        V *dst = S > 1 ? (V *)ws : C;
        const dim3 grid((unsigned)S, 1u, (unsigned)batch);
        const auto launch = [&](auto kernel) {
            kernel<<<grid, 256, 0, stream>>>(A, B, dst, M, N, K, scale, sa, sb, kchunk);
        };
        if (mt == 4)
            launch(gemm_small_kernel<T, 4, 8>);
        else if (mt == 8)
            launch(gemm_small_kernel<T, 8, 16>);
        else if (mt == 16 && nt == 16)
            launch(gemm_small_kernel<T, 16, 16>);
        else if (mt == 16)
            launch(gemm_small_kernel<T, 16, 32>);
        else
            launch(gemm_small_kernel<T, 32, 16>);
        int rc = CheckLaunch("gemm_small_kernel");
        if (rc || S == 1)
            return rc;
        return ReducePartials<T>(dst, C, batch * M * N, S, stream);
    }
    const int64_t S = single_splits > 0 ? single_splits
                      : (need > 0 && ws != nullptr && ws_bytes >= need)
                          ? BatchedSplits<T>(batch, M, N, K)
                          : 1;
    const int64_t kchunk = (K + S - 1) / S;
    const int tile = sizeof(T) == 4 ? PickTileC64(M, N, kchunk, batch * S) : 0;
    const GemmTile t = sizeof(T) == 4 ? kTilesC64[tile] : kTileC128;
    const int64_t tiles = CeilDiv(M, t.bm) * CeilDiv(N, t.bn);
    JETGPU_REQUIRE(tiles <= 0x7fffffffLL && batch * S <= 65535, "product too large for one launch");
    const dim3 grid((unsigned)tiles, 1u, (unsigned)(batch * S));
    V *dst = S > 1 ? (V *)ws : C;
    const auto launch = [&](auto kernel, int threads) {
        kernel<<<grid, threads, 0, stream>>>(A, B, dst, M, N, K, scale, sa, sb, (int)S, kchunk);
    };
    if constexpr (std::is_same<T, double>::value) {
        launch(gemm_kernel<double, 2, 2, 16, 16, 8, 1>, 256);
    }
    else {
        switch (tile) {
        case 0:
            launch(gemm_kernel<float, 8, 4, 16, 8, 8, 3>, 128);
            break;
        case 1:
            launch(gemm_kernel<float, 4, 4, 16, 16, 16, 2>, 256);
            break;
        case 2:
            launch(gemm_kernel<float, 8, 4, 8, 8, 8, 6>, 64);
            break;
        case 3:
            launch(gemm_kernel<float, 4, 2, 16, 16, 16, 2>, 256);
            break;
        case 4:
            launch(gemm_kernel<float, 2, 4, 16, 16, 16, 2>, 256);
            break;
        case 5:
            launch(gemm_kernel<float, 2, 2, 16, 16, 16, 3>, 256);
            break;
        case 6:
            launch(gemm_kernel<float, 4, 4, 16, 16, 8, 3>, 256);
            break;
        default:
            launch(gemm_kernel<float, 4, 4, 16, 8, 8, 5>, 128);
        }
    }
    int rc = CheckLaunch("gemm_kernel");
    if (rc || S == 1)
        return rc;
    if (std::is_same<T, float>::value && single_splits > 0)
        return SumPartials(dst, C, (uint64_t)(M * N), (uint64_t)S, stream);
    return ReducePartials<T>(dst, C, batch * M * N, S, stream);
}

template <typename T>
int MultiplyT(const void *Av, const void *Bv, void *Cv, int64_t M, int64_t N,
              int64_t K, int scale_exp, void *ws, size_t ws_bytes,
              cudaStream_t stream)
{
    using V = typename C2<T>::type;
    const V *A = (const V *)Av;
    const V *B = (const V *)Bv;
    V *C = (V *)Cv;
    const T scale = (T)ldexp(1.0, scale_exp);
    if (M == 0 || N == 0)
        return JETGPU_OK;
    if (K == 0) {
        fill_zero<T><<<GridFor((M * N + 255) / 256, 4), 256, 0, stream>>>(
            C, M * N);
        return CheckLaunch("fill_zero");
    }
    if (M > 1 && N > 1)
        return GemmT<T>(A, B, C, 1, 0, 0, M, N, K, scale, ws, ws_bytes, stream);
    return MultiplyVectorT<T>(A, B, C, 1, 0, 0, M, N, K, scale, ws, ws_bytes, stream);
}

template <typename T>
int MultiplyBatchedT(const void *Av, const void *Bv, void *Cv, int64_t batch, int64_t sa,
                     int64_t sb, int64_t M, int64_t N, int64_t K, int scale_exp, void *ws,
                     size_t ws_bytes, cudaStream_t stream)
{
    using V = typename C2<T>::type;
    const V *A = (const V *)Av;
    const V *B = (const V *)Bv;
    V *C = (V *)Cv;
    const T scale = (T)ldexp(1.0, scale_exp);
    if (M == 0 || N == 0 || batch == 0)
        return JETGPU_OK;
    if (K == 0) {
        fill_zero<T><<<GridFor((batch * M * N + 255) / 256, 4), 256, 0, stream>>>(C, batch * M * N);
        return CheckLaunch("fill_zero");
    }
    if (M > 1 && N > 1)
        return GemmT<T>(A, B, C, batch, sa, sb, M, N, K, scale, ws, ws_bytes, stream);
    return MultiplyVectorT<T>(A, B, C, batch, sa, sb, M, N, K, scale, ws, ws_bytes, stream);
}

} // namespace

int MultiplyPlainBatched(const void *A, const void *B, void *C, uint64_t batch, uint64_t sa,
                         uint64_t sb, uint64_t m, uint64_t n, uint64_t k, int dtype,
                         int scale_exp, void *workspace, size_t ws_bytes, cudaStream_t stream)
{
    JETGPU_REQUIRE(dtype == JETGPU_C64 || dtype == JETGPU_C128, "bad dtype");
    if (dtype == JETGPU_C128)
        return MultiplyBatchedT<double>(A, B, C, (int64_t)batch, (int64_t)sa, (int64_t)sb,
                                        (int64_t)m, (int64_t)n, (int64_t)k, scale_exp, workspace,
                                        ws_bytes, stream);
    return MultiplyBatchedT<float>(A, B, C, (int64_t)batch, (int64_t)sa, (int64_t)sb, (int64_t)m,
                                   (int64_t)n, (int64_t)k, scale_exp, workspace, ws_bytes,
                                   stream);
}

int SumPartials(const void *part, void *out, uint64_t len, uint64_t splits, cudaStream_t stream)
{
    if (splits >= kManyRanges) {
        sum_many_kernel<<<GridFor((len + 31) / 32, 4), 32 * kManyWarps, 0, stream>>>(
            (const float2 *)part, (float2 *)out, (int64_t)len, (int64_t)splits);
        return CheckLaunch("sum_many_kernel");
    }
    sum_partials_kernel<<<GridFor((len + 255) / 256, 8), 256, 0, stream>>>(
        (const float2 *)part, (float2 *)out, (int64_t)len, (int64_t)splits);
    return CheckLaunch("sum_partials_kernel");
}

namespace {

// The k ranges jetgpu_contract cuts a matrix product into (1: its plain path).
int64_t SingleRanges(uint64_t m, uint64_t n, uint64_t k, int dtype)
{
    int mt, nt;
    SmallTile((int64_t)m, (int64_t)n, (int64_t)k, mt, nt);
    if (m < 2 || n < 2 || k == 0 || mt)
        return 1;
    return dtype == JETGPU_C128 ? SingleSplits<double>((int64_t)m, (int64_t)n, (int64_t)k)
                                : SingleSplits<float>((int64_t)m, (int64_t)n, (int64_t)k);
}

} // namespace

size_t MultiplySingleWorkspace(uint64_t m, uint64_t n, uint64_t k, int dtype)
{
    const int64_t S = SingleRanges(m, n, k, dtype);
    return std::max(MultiplyPlainWorkspace(m, n, k, dtype),
                    S > 1 ? (size_t)S * m * n * ElemBytes(dtype) : 0);
}

int MultiplySingle(const void *A, const void *B, void *C, uint64_t m, uint64_t n, uint64_t k,
                   int dtype, int scale_exp, void *workspace, size_t ws_bytes,
                   cudaStream_t stream)
{
    const int64_t S = SingleRanges(m, n, k, dtype);
    const size_t bytes = (size_t)S * m * n * ElemBytes(dtype);
    if (S < 2 || workspace == nullptr || ws_bytes < bytes)
        return MultiplyPlain(A, B, C, m, n, k, dtype, scale_exp, workspace, ws_bytes, stream);
    if (dtype == JETGPU_C128)
        return GemmT<double>((const double2 *)A, (const double2 *)B, (double2 *)C, 1, 0, 0,
                             (int64_t)m, (int64_t)n, (int64_t)k, ldexp(1.0, scale_exp), workspace,
                             bytes, stream, S);
    return GemmT<float>((const float2 *)A, (const float2 *)B, (float2 *)C, 1, 0, 0, (int64_t)m,
                        (int64_t)n, (int64_t)k, (float)ldexp(1.0, scale_exp), workspace, bytes,
                        stream, S);
}

int ClosingContract(const void *A, int a_rank, const uint64_t *a_shape, const int32_t *a_perm,
                    const void *B, int b_rank, const uint64_t *b_shape, const int32_t *b_perm,
                    void *C, uint64_t m, uint64_t n, uint64_t k, int dtype, int scale_exp,
                    void *workspace, size_t ws_bytes, cudaStream_t stream, bool &taken)
{
    ClosingPlan p;
    const int klog = dtype == JETGPU_C128 ? kClosingLog<double> : kClosingLog<float>;
    taken = PlanClosing(a_rank, a_shape, a_perm, b_rank, b_shape, b_perm, m, n, k, klog, p);
    if (!taken)
        return JETGPU_OK;
    if (dtype == JETGPU_C128)
        return ClosingT<double>(p, (const double2 *)A, (const double2 *)B, (double2 *)C,
                                (int64_t)m, (int64_t)n, (int64_t)k, ldexp(1.0, scale_exp),
                                workspace, ws_bytes, stream);
    return ClosingT<float>(p, (const float2 *)A, (const float2 *)B, (float2 *)C, (int64_t)m,
                           (int64_t)n, (int64_t)k, (float)ldexp(1.0, scale_exp), workspace,
                           ws_bytes, stream);
}

size_t MultiplyPlainWorkspace(uint64_t m, uint64_t n, uint64_t k, int dtype)
{
    return MultiplyPlainBatchedWorkspace(1, m, n, k, dtype);
}

size_t MultiplyPlainBatchedWorkspace(uint64_t batch, uint64_t m, uint64_t n, uint64_t k,
                                     int dtype)
{
    return dtype == JETGPU_C128 ? VectorWorkspace<double>(batch, m, n, k)
                                : VectorWorkspace<float>(batch, m, n, k);
}

int MultiplyPlain(const void *A, const void *B, void *C, uint64_t m,
                  uint64_t n, uint64_t k, int dtype, int scale_exp,
                  void *workspace, size_t ws_bytes, cudaStream_t stream)
{
    JETGPU_REQUIRE(dtype == JETGPU_C64 || dtype == JETGPU_C128, "bad dtype");
    if (m * n > 0)
        JETGPU_REQUIRE(C != nullptr, "null output");
    if (m * n * k > 0)
        JETGPU_REQUIRE(A != nullptr && B != nullptr, "null operand");
    if (dtype == JETGPU_C128)
        return MultiplyT<double>(A, B, C, (int64_t)m, (int64_t)n, (int64_t)k,
                                 scale_exp, workspace, ws_bytes, stream);
    return MultiplyT<float>(A, B, C, (int64_t)m, (int64_t)n, (int64_t)k,
                            scale_exp, workspace, ws_bytes, stream);
}

} // namespace jetgpu

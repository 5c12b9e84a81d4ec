// Tiled SIMT GEMM for sm_103a, used for Matrix * Matrix and for the trailing-matrix
// updates of the blocked factorisations:
//     C = alpha * op(A) * op(B) + beta * C,   row-major, op = identity or transpose.
// FP32 uses FFMA (74 TFLOP/s on GB300); FP64 uses DFMA (GB300's FP64 rate is the same
// ~1 TFLOP/s through DFMA and through DMMA) for small products and for what the tensor-core
// form (gemm_f64tc.cuh) leaves. Tiles are double-buffered through shared memory; every thread owns a
// TM x TN register tile split into 4x4 quadrants to keep shared-memory reads
// conflict-free.
#pragma once

#include <type_traits>

#include "common.cuh"
#include "gemm_f64tc.cuh"
#include "gemm_tc.cuh"

namespace rl {

template <class T>
struct GemmCfg;
template <>
struct GemmCfg<float> {
    static constexpr int BM = 128, BN = 128, BK = 8, TM = 8, TN = 8;
};
template <>
struct GemmCfg<double> {
    static constexpr int BM = 64, BN = 64, BK = 8, TM = 4, TN = 4;
};

template <class T>
__device__ __forceinline__ void lds4(const T *p, T (&o)[4]);
template <>
__device__ __forceinline__ void lds4<float>(const float *p, float (&o)[4]) {
    float4 v = *reinterpret_cast<const float4 *>(p);
    o[0] = v.x, o[1] = v.y, o[2] = v.z, o[3] = v.w;
}
template <>
__device__ __forceinline__ void lds4<double>(const double *p, double (&o)[4]) {
    double2 v0 = reinterpret_cast<const double2 *>(p)[0];
    double2 v1 = reinterpret_cast<const double2 *>(p)[1];
    o[0] = v0.x, o[1] = v0.y, o[2] = v1.x, o[3] = v1.y;
}

// op(A) is m x k: A[i * lda + p] (TA = false) or A[p * lda + i] (TA = true).
// op(B) is k x n: B[p * ldb + j] (TB = false) or B[j * ldb + p] (TB = true).
// LOWER = true computes only the tiles that touch the lower triangle (i >= j) and only
// writes elements with i >= j (the SYRK form used by Cholesky). stop (FP64 LOWER, may be null): a
// status word; if it is set C stays as it is.
template <class T, bool TA, bool TB, bool LOWER>
__global__ void __launch_bounds__((GemmCfg<T>::BM / GemmCfg<T>::TM) * (GemmCfg<T>::BN / GemmCfg<T>::TN))
    gemm_kernel(int m, int n, int k, T alpha, const T *__restrict__ A, long long lda, const T *__restrict__ B,
                long long ldb, T beta, T *__restrict__ C, long long ldc, int kslice, long long zstride, const int *stop) {
    constexpr int BM = GemmCfg<T>::BM, BN = GemmCfg<T>::BN, BK = GemmCfg<T>::BK;
    constexpr int TM = GemmCfg<T>::TM, TN = GemmCfg<T>::TN;
    constexpr int NTX = BN / TN, NTY = BM / TM, NT = NTX * NTY;
    constexpr int SM_ = TM / 4, SN_ = TN / 4;  // quadrants per thread
    constexpr int A_PER = BM * BK / NT, B_PER = BK * BN / NT;
    static_assert(A_PER >= 1 && B_PER >= 1, "tile too small for the block");

    __shared__ __align__(16) T As[2][BK][BM];
    __shared__ __align__(16) T Bs[2][BK][BN];

    if (gridDim.z > 1) {  // split K: slice z of the reduction into its own partial C
        const int kz = blockIdx.z * kslice;
        k = max(0, min(kslice, k - kz));
        A += TA ? (long long)kz * lda : kz;
        B += TB ? kz : (long long)kz * ldb;
        C += blockIdx.z * zstride;
    }
    const int tid = threadIdx.x;
    const int tx = tid % NTX, ty = tid / NTX;
    const int row0 = blockIdx.y * BM, col0 = blockIdx.x * BN;
    if (LOWER && col0 > row0 + BM - 1) return;  // tile strictly above the diagonal
    T acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; i++)
#pragma unroll
        for (int j = 0; j < TN; j++) acc[i][j] = T(0);

    T ra[A_PER], rb[B_PER];

    auto load_tile = [&](int k0) {
#pragma unroll
        for (int e = 0; e < A_PER; e++) {
            int idx = tid + e * NT;
            int i, p;
            if (TA) {  // consecutive threads along i (contiguous in memory)
                i = idx % BM;
                p = idx / BM;
            } else {  // consecutive threads along p
                p = idx % BK;
                i = idx / BK;
            }
            int gi = row0 + i, gp = k0 + p;
            T v = T(0);
            if (gi < m && gp < k) v = TA ? A[(long long)gp * lda + gi] : A[(long long)gi * lda + gp];
            ra[e] = v;
        }
#pragma unroll
        for (int e = 0; e < B_PER; e++) {
            int idx = tid + e * NT;
            int j, p;
            if (TB) {
                p = idx % BK;
                j = idx / BK;
            } else {
                j = idx % BN;
                p = idx / BN;
            }
            int gj = col0 + j, gp = k0 + p;
            T v = T(0);
            if (gj < n && gp < k) v = TB ? B[(long long)gj * ldb + gp] : B[(long long)gp * ldb + gj];
            rb[e] = v;
        }
    };
    auto store_tile = [&](int buf) {
#pragma unroll
        for (int e = 0; e < A_PER; e++) {
            int idx = tid + e * NT;
            int i, p;
            if (TA) {
                i = idx % BM;
                p = idx / BM;
            } else {
                p = idx % BK;
                i = idx / BK;
            }
            As[buf][p][i] = ra[e];
        }
#pragma unroll
        for (int e = 0; e < B_PER; e++) {
            int idx = tid + e * NT;
            int j, p;
            if (TB) {
                p = idx % BK;
                j = idx / BK;
            } else {
                j = idx % BN;
                p = idx / BN;
            }
            Bs[buf][p][j] = rb[e];
        }
    };

    const int ktiles = (k + BK - 1) / BK;
    if (ktiles > 0) {
        int stopped = 0;  // read with the first tile in flight
    if constexpr (LOWER && std::is_same<T, double>::value)
        if (stop) stopped = *stop;
    load_tile(0);
    if (stopped) return;
        store_tile(0);
    }
    __syncthreads();
    for (int kt = 0; kt < ktiles; kt++) {
        const int buf = kt & 1;
        if (kt + 1 < ktiles) load_tile((kt + 1) * BK);
#pragma unroll
        for (int p = 0; p < BK; p++) {
            T a[TM], b[TN];
#pragma unroll
            for (int s = 0; s < SM_; s++) {
                T q[4];
                lds4<T>(&As[buf][p][s * (BM / SM_) + ty * 4], q);
#pragma unroll
                for (int r = 0; r < 4; r++) a[s * 4 + r] = q[r];
            }
#pragma unroll
            for (int s = 0; s < SN_; s++) {
                T q[4];
                lds4<T>(&Bs[buf][p][s * (BN / SN_) + tx * 4], q);
#pragma unroll
                for (int r = 0; r < 4; r++) b[s * 4 + r] = q[r];
            }
#pragma unroll
            for (int i = 0; i < TM; i++)
#pragma unroll
                for (int j = 0; j < TN; j++) acc[i][j] = fma(a[i], b[j], acc[i][j]);
        }
        if (kt + 1 < ktiles) store_tile(buf ^ 1);
        __syncthreads();
    }

#pragma unroll
    for (int i = 0; i < TM; i++) {
        const int gi = row0 + (i / 4) * (BM / SM_) + ty * 4 + (i % 4);
        if (gi >= m) continue;
#pragma unroll
        for (int j = 0; j < TN; j++) {
            const int gj = col0 + (j / 4) * (BN / SN_) + tx * 4 + (j % 4);
            if (gj >= n) continue;
            if (LOWER && gj > gi) continue;
            T *cp = C + (long long)gi * ldc + gj;
            T v = alpha * acc[i][j];
            if (beta != T(0)) v = fma(beta, *cp, v);
            *cp = v;
        }
    }
}

// The same product for few outputs: 32 x 32 (FP32) or 16 x 16 (FP64) outputs per CTA of 128
// threads, K in chunks of 32 through shared memory, so that a product of a few 64 x 64 tiles
// (T^T W and W = V^T A of a Householder block, the solves' small updates) spreads over the
// SMs: on this part a 64 x 64 x 64 FP64 product is 70 us of one SM's FP64 unit. T^T W of a
// 1201 x 499 QR (64 x n2 x 64) went from ~270 to 8 us, in FP32 (2999 x 1501) from 17 to 4. Sums
// run over k in order, as in gemm_kernel.
template <class T>
constexpr int gemm_few_tile() {
    return sizeof(T) == 4 ? 32 : 16;
}
template <class T, bool TA, bool TB, bool LOWER>
__device__ __forceinline__ void gemm_few_product(int row0, int col0, int m, int n, int k, T alpha, const T *__restrict__ A,
                                                 long long lda, const T *__restrict__ B, long long ldb, T beta,
                                                 T *__restrict__ C, long long ldc) {
    constexpr int BT = gemm_few_tile<T>(), BK = 32, R = BT * BT / 128, RS = 128 / BT;  // outputs a thread: rows ty + RS i
    __shared__ T As[BK][BT + 1], Bs[BK][BT + 1];
    const int tid = threadIdx.x, tx = tid % BT, ty = tid / BT;
    constexpr int PER = BK * BT / 128;
    T ra[PER], rb[PER], acc[R];
#pragma unroll
    for (int i = 0; i < R; i++) acc[i] = T(0);
    auto load = [&](int k0) {
#pragma unroll
        for (int e = 0; e < PER; e++) {
            const int idx = tid + e * 128;
            const int ia = TA ? idx % BT : idx / BK, pa = TA ? idx / BT : idx % BK;
            ra[e] = (row0 + ia < m && k0 + pa < k)
                        ? (TA ? A[(long long)(k0 + pa) * lda + row0 + ia] : A[(long long)(row0 + ia) * lda + k0 + pa])
                        : T(0);
            const int jb = TB ? idx / BK : idx % BT, pb = TB ? idx % BK : idx / BT;
            rb[e] = (col0 + jb < n && k0 + pb < k)
                        ? (TB ? B[(long long)(col0 + jb) * ldb + k0 + pb] : B[(long long)(k0 + pb) * ldb + col0 + jb])
                        : T(0);
        }
    };
    load(0);
    for (int k0 = 0; k0 < k; k0 += BK) {
#pragma unroll
        for (int e = 0; e < PER; e++) {
            const int idx = tid + e * 128;
            if (TA)
                As[idx / BT][idx % BT] = ra[e];
            else
                As[idx % BK][idx / BK] = ra[e];
            if (TB)
                Bs[idx % BK][idx / BK] = rb[e];
            else
                Bs[idx / BT][idx % BT] = rb[e];
        }
        __syncthreads();
        if (k0 + BK < k) load(k0 + BK);
        const int lim = min(BK, k - k0);
#pragma unroll 8
        for (int p = 0; p < lim; p++) {
            const T b = Bs[p][tx];
#pragma unroll
            for (int i = 0; i < R; i++) acc[i] = fma(As[p][ty + RS * i], b, acc[i]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < R; i++) {
        const int gi = row0 + ty + RS * i, gj = col0 + tx;
        if (gi < m && gj < n && !(LOWER && gj > gi)) {
            T *cp = C + (long long)gi * ldc + gj;
            T v = alpha * acc[i];
            if (beta != T(0)) v = fma(beta, *cp, v);
            *cp = v;
        }
    }
}

template <class T, bool TA, bool TB>
static __global__ void __launch_bounds__(128)
    gemm_few_kernel(int m, int n, int k, T alpha, const T *__restrict__ A, long long lda, const T *__restrict__ B, long long ldb,
                    T beta, T *__restrict__ C, long long ldc) {
    constexpr int BT = gemm_few_tile<T>();
    gemm_few_product<T, TA, TB, false>(blockIdx.y * BT, blockIdx.x * BT, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc);
}

// The tiles of a product that the tensor-core form left (gemm_f64tc.cuh): usually none, and then
// this is a launch of CTAs that read one word. kLeftCtas CTAs per SM go over the 16 x 16 tiles, each
// inside one tile of the flags, so that a few flagged tiles still spread over the SMs (LOWER: the
// elements i >= j). Sums run over k in order, as in gemm_kernel, whose 64 x 64 tiles took them before
// (us, and the whole product on gemm_kernel without the tensor-core form): identity times dense
// 192^3 49 (230, 204), 512^3 269 (568, 532), 1024^3 1,861 (2,112, 2,070), 2048^3 14,205 (14,407,
// 14,303); lower triangle times dense 256^3 94 (336, 270), 2048^3 1,575 (2,753, 14,303). Nothing left:
// 2048^3 648 (654).
constexpr int kLeftCtas = 8;
template <bool TA, bool TB, bool LOWER>
static __global__ void __launch_bounds__(128)
    gemm_left_kernel(int m, int n, int k, double alpha, const double *__restrict__ A, long long lda, const double *__restrict__ B,
                     long long ldb, double beta, double *__restrict__ C, long long ldc, int kslice, long long zstride,
                     DgemmTcTiles only) {
    constexpr int BT = gemm_few_tile<double>();
    static_assert(tc64::BM % BT == 0 && 64 % BT == 0 && 80 % BT == 0, "inside one tile of the flags");
    if (*only.nfail == 0) return;
    if (gridDim.z > 1) {  // split K, as in gemm_kernel
        const int kz = blockIdx.z * kslice;
        k = max(0, min(kslice, k - kz));
        A += TA ? (long long)kz * lda : kz;
        B += TB ? kz : (long long)kz * ldb;
        C += blockIdx.z * zstride;
    }
    const int tn = (n + BT - 1) / BT;
    const long long total = (long long)tn * ((m + BT - 1) / BT);
    for (long long t = blockIdx.x; t < total; t += gridDim.x) {
        const int row0 = (int)(t / tn) * BT, col0 = (int)(t % tn) * BT;
        if (LOWER && col0 > row0 + BT - 1) continue;
        if (only.flags[(row0 / tc64::BM) * only.gx + col0 / only.bn])
            gemm_few_product<double, TA, TB, LOWER>(row0, col0, m, n, k, alpha, A, lda, B, ldb, beta, C, ldc);
    }
}

// Launches C = alpha * op(A) op(B) + beta * C on `stream`. FP32 products with at least
// a 128 x 128 tile's worth of C and K >= 256 go to the tcgen05 kernel (gemm_tc.cuh).
// A product with fewer tiles than SMs and a long K (the V^T A2 and V^T V products of a
// Householder block, K = the panel height) is split along K into partial tiles that
// run at once, then added in slice order. The tensor-core forms wait (bounded): *err, a device
// status word of the caller's (0 or its first error; null: none is kept), receives
// RL_ERR_TIMEOUT when a wait runs out, and the tile of C NaN. The FP64 SYRK form (LOWER) leaves C
// as it is when *err is set already: a Cholesky that has failed does not run on.
template <class T, bool TA, bool TB, bool LOWER = false>
rl_status gemm(int m, int n, int k, T alpha, const T *A, long long lda, const T *B, long long ldb, T beta, T *C,
               long long ldc, cudaStream_t stream, int *err) {
    if (m <= 0 || n <= 0) return RL_OK;
    constexpr int BM = GemmCfg<T>::BM, BN = GemmCfg<T>::BN, BK = GemmCfg<T>::BK;
    constexpr int NT = (BM / GemmCfg<T>::TM) * (BN / GemmCfg<T>::TN);
    dim3 grid((n + BN - 1) / BN, (m + BM - 1) / BM);
    const int tiles = (int)(grid.x * grid.y), sms = num_sms();
    if constexpr (std::is_same<T, float>::value) {  // FP32 with enough work: tensor cores (3xTF32)
        if (sgemm_tc_eligible(m, n, k)) {
            const int tc_tiles = ceil_div(n, tc::BN) * ceil_div(m, tc::BM);
            int ks = 1;
            if (!LOWER && tc_tiles < sms / 2 && k >= 1024) ks = std::min({16, ceil_div(sms, tc_tiles), k / 256});
            return sgemm_tc<TA, TB>(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, LOWER, stream, err, ks);
        }
    }
    if constexpr (!LOWER) {
        // Few outputs, short K: small tiles over the SMs. gemm_kernel's tiles take BM BN K
        // multiply-adds of one SM each; here every SM takes a share.
        constexpr int BT = gemm_few_tile<T>();
        const bool tc = std::is_same<T, double>::value && dgemm_tc_eligible(m, n, k);
        if (tiles * 4 <= sms && k <= 512 && !tc) {
            RL_LAUNCH((gemm_few_kernel<T, TA, TB>), dim3(ceil_div(n, BT), ceil_div(m, BT)), 128, 0, stream, m, n, k, alpha, A, lda,
                      B, ldb, beta, C, ldc);
            return RL_OK;
        }
    }
    DevBuf<unsigned char> ws;
    DgemmTcTiles left;
    if constexpr (std::is_same<T, double>::value) {  // FP64 with enough work: exact slices on the tensor cores
        bool taken = false;
        const int max_k = dgemm_tc_eligible(m, n, k) ? dgemm_tc_max_k(m, n, LOWER) : k;
        if (k > max_k) {  // equal parts of K, added into C in order
            const int part = ceil_div(ceil_div(k, ceil_div(k, max_k)), tc64::BK) * tc64::BK;
            for (int p = 0; p < k; p += part)
                RL_TRY((gemm<T, TA, TB, LOWER>(m, n, std::min(part, k - p), alpha, A + (TA ? p * lda : (long long)p), lda,
                                               B + (TB ? (long long)p : p * ldb), ldb, p ? T(1) : beta, C, ldc, stream, err)));
            return RL_OK;
        }
        if (dgemm_tc_eligible(m, n, k))
            RL_TRY((dgemm_tc<TA, TB>(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, LOWER, stream, err, ws, left, taken)));
        // what follows computes the tiles that were left (usually none), or all of C
    }
    auto launch = [&](int nz, T al, T be, T *out, long long ldo, int kslice, long long zstride) -> rl_status {
        if constexpr (std::is_same<T, double>::value)
            if (left.flags) {
                constexpr int BT = gemm_few_tile<T>();
                const long long small = (long long)ceil_div(n, BT) * ceil_div(m, BT);
                RL_LAUNCH((gemm_left_kernel<TA, TB, LOWER>), dim3((int)std::min<long long>(small, kLeftCtas * sms), 1, nz), 128, 0,
                          stream, m, n, k, al, A, lda, B, ldb, be, out, ldo, kslice, zstride, left);
                return RL_OK;
            }
        grid.z = nz;
        RL_LAUNCH((gemm_kernel<T, TA, TB, LOWER>), grid, NT, 0, stream, m, n, k, al, A, lda, B, ldb, be, out, ldo, kslice, zstride,
                  LOWER ? (const int *)err : nullptr);
        return RL_OK;
    };
    int ksplit = 1;
    if (!LOWER && tiles < sms && k >= 1024) ksplit = std::min({16, ceil_div(2 * sms, tiles), k / 256});
    if (ksplit > 1) {
        const int kslice = ceil_div(ceil_div(k, ksplit), BK) * BK;
        ksplit = ceil_div(k, kslice);
        const long long zstride = (long long)m * n;
        DevBuf<T> part;
        const rl_status mem = part.alloc((size_t)ksplit * zstride, stream);
        if (mem != RL_OK && left.flags) {  // usually nothing is left: not a reason to fail
            cudaGetLastError();
            return launch(1, alpha, beta, C, ldc, k, 0ll);
        }
        RL_TRY(mem);
        RL_TRY(launch(ksplit, T(1), T(0), part.p, (long long)n, kslice, zstride));
        const int rg = std::min(4 * sms, ceil_div(zstride, 256));
        if constexpr (std::is_same<T, double>::value)
            if (left.flags) {
                RL_LAUNCH(dgemm_tc_reduce_kernel, rg, 256, 0, stream, m, n, ksplit, alpha, part.p, beta, C, ldc, left.flags,
                          left.nfail, left.bn, left.gx, 1);
                return RL_OK;
            }
        RL_LAUNCH(splitk_reduce_kernel<T>, rg, 256, 0, stream, m, n, ksplit, alpha, part.p, beta, C, ldc);
        return RL_OK;
    }
    return launch(1, alpha, beta, C, ldc, k, 0ll);
}

}  // namespace rl

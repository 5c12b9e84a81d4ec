// Device-side orchestration shared by the host entry points: blocked factorisations
// (LU, Cholesky, Householder QR), Q formation, triangular solves and factor solves on
// buffers already on the GPU. Every function launches on the given stream; the ones
// that return a numerical status synchronise to read it.
#pragma once

#include <algorithm>
#include <type_traits>
#include <vector>

#include "batch.cuh"
#include "dense.cuh"
#include "gemm.cuh"
#include "mixed.cuh"
#include "small.cuh"

namespace rl {


template <class T>
inline rl_status read_status(const int *dstatus, cudaStream_t s) {
    int h = 0;
    RL_TRY_CUDA(cudaMemcpyAsync(&h, dstatus, sizeof(int), cudaMemcpyDeviceToHost, s));
    RL_TRY_CUDA(cudaStreamSynchronize(s));
    return h;
}

template <class K>
inline rl_status set_smem(K kern, size_t bytes) {
    static_assert(std::is_pointer<K>::value, "kernel pointer");
    if (bytes > 48 * 1024)
        RL_TRY_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
    return RL_OK;
}

// Sizes up to which one CTA factors a single matrix (the batched kernels keep CTA_NMAX). A
// panel of a cluster costs ~1.5 us a column whatever its height; one CTA's FP64 unit makes
// 2 multiply-adds a cycle, so FP64 leaves it beyond the 64 rows of small_lu_kernel (LU, host
// call, one CTA against blocked: n = 64 416 and 196 us, 128 951 and 400, 512 16,016 and
// 1,798). FP32 LU crosses at n = 256 (536 and 515; 512: 1,827 and 1,083), FP32 Cholesky
// between 384 and 512 (547 and 636; 919 and 793), FP64 Cholesky at once with its diagonal
// blocks on small_chol_kernel.
template <class T>
constexpr int one_cta_lu() {
    return sizeof(T) == 8 ? kSmallN : 240;
}
template <class T>
constexpr int one_cta_chol() {
    return sizeof(T) == 8 ? kSmallN : 448;
}

// One CTA factors a matrix with n <= CTA_NMAX; kind 0 LU (ipiv out), 1 Cholesky. The status
// word is set, not read; host_st and host_mark as small_chol_kernel takes them.
template <class T>
rl_status factor_small_async(T *A, long long lda, int n, int kind, int *ipiv, int *st, cudaStream_t s, T tiny,
                             int *host_st = nullptr, int host_mark = 0) {
    if (n <= kSmallN) {
        if (kind)
            RL_LAUNCH(small_chol_kernel<T>, 1, 256, 0, s, A, (int)lda, n, st, tiny, host_st, host_mark);
        else
            RL_LAUNCH(small_lu_kernel<T>, 1, 256, 0, s, A, (int)lda, n, ipiv, (T *)nullptr, st, tiny);
        return RL_OK;
    }
    const size_t smem = cta_smem_bytes<T>();
    RL_TRY(set_smem(factor_one_kernel<T>, smem));
    RL_LAUNCH(factor_one_kernel<T>, 1, CTA_THREADS, smem, s, A, (int)lda, n, kind, ipiv, st, tiny);
    return RL_OK;
}
template <class T>
rl_status factor_small(T *A, long long lda, int n, int kind, int *ipiv, cudaStream_t s, T tiny = Eps<T>::value) {
    DevBuf<int> st;
    RL_TRY(st.alloc(1, s));
    RL_TRY_CUDA(cudaMemsetAsync(st.p, 0, sizeof(int), s));
    RL_TRY(factor_small_async<T>(A, lda, n, kind, ipiv, st.p, s, tiny));
    return read_status<T>(st.p, s);
}

// A calling thread's view of a factorisation in progress: a page-locked status word that kernels set
// to this call's mark (a kernel that an earlier call left behind sets an older one) and an event behind
// the kernel to look at, kept until the thread ends; a second word is the status of host calls
// (dense.cu). Without them (no memory) the host reads a status in device memory at the end.
struct StatusWatch {
    int *word = nullptr, mark = 0;
    cudaEvent_t ev = nullptr;
    int *call_word() const { return word + 8; }
    ~StatusWatch() {
        if (word) cudaFreeHost(word);
        if (ev) cudaEventDestroy(ev);
    }
    bool begin() {
        if (!word && cudaHostAlloc(reinterpret_cast<void **>(&word), 64, cudaHostAllocDefault) != cudaSuccess) word = nullptr;
        if (!ev && cudaEventCreateWithFlags(&ev, cudaEventDisableTiming) != cudaSuccess) ev = nullptr;
        if (!word || !ev) {
            cudaGetLastError();
            return false;
        }
        *(volatile int *)word = *(volatile int *)call_word() = 0;
        mark = mark % INT_MAX + 1;
        return true;
    }
    bool failed() const { return *(volatile int *)word == mark; }
};
inline StatusWatch &status_watch() {
    static thread_local StatusWatch w;
    return w;
}

// Cooperative panel geometry: G CTAs of rows_per rows each.
template <class T>
void panel_geometry(int mrows, int &G, int &rows_per) {
    const int target = std::is_same<T, double>::value ? 64 : 128;
    G = std::max(1, std::min(num_sms(), (mrows + target - 1) / target));
    rows_per = (mrows + G - 1) / G;
}

template <class T>
rl_status launch_coop(void *kern, int G, size_t smem, void **args, cudaStream_t s) {
    RL_TRY_CUDA(cudaLaunchCooperativeKernel(kern, dim3(G), dim3(256), args, smem, s));
    count_launch();
    return RL_OK;
}

// Largest thread-block cluster (16 or 8 CTAs, 0: none) on which `kern` can run with
// `smem` bytes of dynamic shared memory per CTA; sets the kernel's attributes.
template <class K>
int probe_cluster(K kern, size_t smem) {
    int found = 0;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) == cudaSuccess) {
        for (int c : {16, 8}) {
            cudaLaunchConfig_t cfg = {};
            cudaLaunchAttribute at[1];
            at[0].id = cudaLaunchAttributeClusterDimension;
            at[0].val.clusterDim.x = c;
            at[0].val.clusterDim.y = 1;
            at[0].val.clusterDim.z = 1;
            cfg.gridDim = dim3(c);
            cfg.blockDim = dim3(256);
            cfg.dynamicSmemBytes = smem;
            cfg.attrs = at;
            cfg.numAttrs = 1;
            int nclusters = 0;
            if (cudaOccupancyMaxActiveClusters(&nclusters, kern, &cfg) == cudaSuccess && nclusters >= 1) {
                found = c;
                break;
            }
        }
    }
    cudaGetLastError();  // a refused query is not an error of the factorisation
    return found;
}

// Cluster size and rows per CTA for a panel of mrows rows of row_bytes each plus `extra`
// bytes per CTA: about `target_rows` rows per CTA, clamped to [2, cmax] and to at least
// the CTAs that the shared memory needs; 0 when even cmax CTAs would need more than
// kClusterSmem bytes each. FP64 panels take 64 rows per CTA (their row updates run at
// the SM's FP64 rate, so every SM added shortens a column); FP32 panels take 256 (their
// updates are cheap: up to 16 CTAs measured the same), which leaves the SMs of a GPC to
// other streams' kernels where fewer will do.
template <class T>
constexpr int panel_target_rows() {
    return sizeof(T) == 8 ? 64 : 256;
}
constexpr size_t kClusterSmem = 224 * 1024;
// dynamic shared memory of lu_panel_cluster_kernel beside its static tables, for 1024 rows a
// CTA at most (FP32; FP64 holds fewer by size)
template <class T>
constexpr size_t kPanelSmem = kClusterSmem - sizeof(PanelTables<T>);
inline int cluster_shape(int mrows, size_t row_bytes, size_t extra, int cmax, int target_rows, int &rows_per) {
    const int cmin = (int)(((size_t)mrows * row_bytes + (kClusterSmem - extra) - 1) / (kClusterSmem - extra));
    if (cmin > cmax || cmax == 0) return 0;
    int C = std::max(cmin, std::min(cmax, ceil_div(mrows, target_rows)));
    C = std::max(C, 2);
    while (C < cmax && ceil_div(mrows, C) * row_bytes > kClusterSmem - extra) C++;  // whole rows round up
    rows_per = ceil_div(mrows, C);
    return rows_per * row_bytes > kClusterSmem - extra ? 0 : C;
}

template <class K, class... Args>
rl_status launch_cluster(K kern, int C, size_t smem, cudaStream_t s, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = C;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(C);
    cfg.blockDim = dim3(256);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    RL_TRY_CUDA(cudaLaunchKernelEx(&cfg, kern, args...));
    count_launch();
    return RL_OK;
}

// The LU panel on one cluster when it fits (launched = true), else nothing: the cooperative panel
// takes it. Threads per row and rows per thread follow the rows a CTA holds (256 threads); each
// instance says for itself how large a cluster it can have.
template <class T, int TPR, int RPT>
static rl_status lu_panel_cluster_launch(T *P, long long lda, int mrows, int kb, int k0, int C, int rows_per, int *ipiv, int *err,
                                         T tiny, cudaStream_t s, bool &launched) {
    static const int cmax = probe_cluster(lu_panel_cluster_kernel<T, TPR, RPT>, kPanelSmem<T>);
    if (C > cmax) return RL_OK;
    RL_TRY(launch_cluster(lu_panel_cluster_kernel<T, TPR, RPT>, C, (size_t)rows_per * (PanelNB<T>::value + 1) * sizeof(T), s, P,
                          lda, mrows, kb, k0, rows_per, ipiv, err, tiny, wait_ns()));
    launched = true;
    return RL_OK;
}

template <class T>
static rl_status lu_panel_cluster(T *P, long long lda, int mrows, int kb, int k0, int *ipiv, int *err, T tiny, cudaStream_t s,
                           bool &launched) {
    constexpr int NB = PanelNB<T>::value;
    launched = false;
    const size_t row_bytes = (NB + 1) * sizeof(T);
    int rows_per = 0;
    if (tune(RL_TUNE_PANEL_LOOKAHEAD) != 0) {  // look-ahead form: three table slots
        auto kern = lu_panel_cluster_la_kernel<T>;
        static const int cmax_hw = probe_cluster(kern, kClusterSmem);
        const size_t extra = (3 * 16 * NB + 3 * NB) * sizeof(T);
        const int C = cluster_shape(mrows, row_bytes, extra, std::min<int>(cmax_hw, (int)tune(RL_TUNE_PANEL_CLUSTER_MAX)),
                                    panel_target_rows<T>(), rows_per);
        if (C == 0) return RL_OK;
        int tpr = 1;  // threads per row: every thread busy when the CTA holds few rows
        while (tpr < 8 && rows_per * tpr * 2 <= 256) tpr *= 2;
        RL_TRY(launch_cluster(kern, C, (size_t)rows_per * row_bytes + extra, s, P, lda, mrows, kb, k0, rows_per, tpr, ipiv,
                              err, tiny));
        launched = true;
        return RL_OK;
    }
    static const int cmax_hw = probe_cluster(lu_panel_cluster_kernel<T, 1, 1>, kPanelSmem<T>);
    const int C = cluster_shape(mrows, row_bytes, kClusterSmem - kPanelSmem<T>,
                                std::min<int>(cmax_hw, (int)tune(RL_TUNE_PANEL_CLUSTER_MAX)), panel_target_rows<T>(), rows_per);
    if (C == 0) return RL_OK;
    if (rows_per <= 64)
        return lu_panel_cluster_launch<T, 4, 1>(P, lda, mrows, kb, k0, C, rows_per, ipiv, err, tiny, s, launched);
    if (rows_per <= 128)
        return lu_panel_cluster_launch<T, 2, 1>(P, lda, mrows, kb, k0, C, rows_per, ipiv, err, tiny, s, launched);
    if (rows_per <= 256)
        return lu_panel_cluster_launch<T, 1, 1>(P, lda, mrows, kb, k0, C, rows_per, ipiv, err, tiny, s, launched);
    if (rows_per <= 512)
        return lu_panel_cluster_launch<T, 1, 2>(P, lda, mrows, kb, k0, C, rows_per, ipiv, err, tiny, s, launched);
    if constexpr (sizeof(T) == 4)  // FP64 rows of 520 bytes end at 407
        return lu_panel_cluster_launch<T, 1, 4>(P, lda, mrows, kb, k0, C, rows_per, ipiv, err, tiny, s, launched);
    return RL_OK;
}

// The Householder panel on one cluster when it fits (launched = true), else nothing.
template <class T>
static rl_status qr_panel_cluster(T *P, long long lda, int mrows, int kb, T *tau, int *err, cudaStream_t s, bool &launched) {
    constexpr int NB = PanelNB<T>::value;
    constexpr size_t cap = kClusterSmem - sizeof(QrTables<T>);
    launched = false;
    auto kern = qr_panel_cluster_kernel<T>;
    static const int cmax_hw = probe_cluster(kern, cap);
    const int cmax = std::min<int>(cmax_hw, (int)tune(RL_TUNE_PANEL_CLUSTER_MAX));
    const size_t row_bytes = (NB + 1) * sizeof(T);
    int rows_per = 0;
    const int C = cluster_shape(mrows, row_bytes, kClusterSmem - cap, cmax, panel_target_rows<T>(), rows_per);
    if (C == 0) return RL_OK;
    int tpr = 1;  // threads per row: every thread busy when the CTA holds few rows
    while (tpr < 8 && rows_per * tpr * 2 <= 256) tpr *= 2;
    RL_TRY(launch_cluster(kern, C, (size_t)rows_per * row_bytes, s, P, lda, mrows, kb, rows_per, tpr, tau, err, wait_ns()));
    launched = true;
    return RL_OK;
}

// op(A) Y = Y' in place (triangular solve; modes and paths at the definition below).
template <class T, class TA = T>
rl_status tri_solve_dev(const TA *A, long long lda, int n, T *Y, long long ldy, int nrhs, int mode, int *dstatus,
                        cudaStream_t s, T tiny = Eps<T>::value);

// Outer block width of the blocked Cholesky. FP32 (the mixed-precision factor and
// Matrix<f32>): 256-column blocks, each factored with the 64-column panels confined to
// the block, then ONE trailing update of K = 256 on the tensor cores (tcgen05, 3xTF32;
// the K = 64 updates of the inner panels measured slower there and stay on the SIMT
// kernel). FP64: 0, one block spanning the matrix (K = 64 updates). The LU has its own
// widths (lu_factor_dev).
template <class T>
constexpr int outer_nb() {
    return std::is_same<T, float>::value ? 256 : 0;
}

// Blocked right-looking LU for any n: panel (one cluster, or a cooperative grid for
// panels too tall for a cluster), row swaps, U12 solve, GEMM. Within an outer block the
// swaps, U12 solves and updates of each 64-column panel cover the block's columns only;
// the block's swaps reach the other columns afterwards (LAPACK's getrf order), then
// U12 = L11^-1 A12 and A22 -= L21 U12 with K = the block width. The pivots are those of
// partial pivoting over the whole column either way.
template <class T>
rl_status lu_factor_dev(T *A, long long lda, int n, int *ipiv, cudaStream_t s, T tiny = Eps<T>::value) {
    NvtxRange nvtx_("rl.lu.factor");
    if (n <= 0) return RL_OK;
    if (n <= one_cta_lu<T>()) return factor_small<T>(A, lda, n, 0, ipiv, s, tiny);
    constexpr int NB = PanelNB<T>::value;
    int Gmax, rp;
    panel_geometry<T>(n, Gmax, rp);
    if ((size_t)rp * (NB + 1) * sizeof(T) > 200 * 1024) return RL_ERR_INVALID_ARG;  // n beyond ~50k
    DevBuf<T> cand, rowj;
    DevBuf<PanelSync> sync;
    RL_TRY(cand.alloc((size_t)2 * Gmax * (2 + NB), s));
    RL_TRY(rowj.alloc(2 * NB, s));
    RL_TRY(sync.alloc(1, s));
    auto pk = lu_panel_kernel<T>;
    RL_TRY(set_smem(pk, 200 * 1024));
    // The error word is sticky across panels (only the barrier counter is reset per
    // launch) and read once at the end: a failed panel leaves identity pivots, the work
    // after it runs on in-range indices, and every later panel stops at its first barrier.
    RL_TRY_CUDA(cudaMemsetAsync(sync.p, 0, sizeof(PanelSync), s));
    unsigned long long wns = wait_ns();
    int NBO = n;  // outer block width (FP32: RL_TUNE_LU_OUTER_NB, a multiple of NB)
    if constexpr (std::is_same<T, float>::value) {
        // automatic: at n = 2048 / 4096 one level measured 9.4 / 20.5 ms against 10.5 / 24.2
        // with 256-column blocks; at 8192 / 16384 1024-column blocks 58.2 / 171 ms against
        // 59.1 / 179 with 512, 62.4 / 206 with 256 and 62.0 / 229 with one level (mixed
        // solves, nrhs 1)
        const long long v = tune(RL_TUNE_LU_OUTER_NB);
        const int w = v < 0 ? (n < 6144 ? 0 : 1024) : (int)(v / NB) * NB;
        if (w >= NB) NBO = w;
    } else if (n >= 3072) {
        // FP64: the trailing products run on the tensor cores, where K = 64 is dominated by C's
        // traffic and a tile's fixed cost. FP64 solves with one level / 256 / 512 / 1024-column
        // blocks: n = 2048 8.6 / 9.6 / 9.8 / 9.6 ms, 4096 28.9 / 26.6 / 26.3 / 26.5, 8192 139 /
        // 94.6 / 88.5 / 89.2.
        NBO = 512;
    }
    for (int K0 = 0; K0 < n; K0 += NBO) {
        const int K1 = std::min(n, K0 + NBO), KB = K1 - K0;
        for (int k0 = K0; k0 < K1; k0 += NB) {
            const int kb = std::min(NB, K1 - k0), mrows = n - k0;
            int G, rows_per;
            panel_geometry<T>(mrows, G, rows_per);
            const size_t smem = ((size_t)rows_per * (NB + 1) + NB) * sizeof(T);
            T *P = A + (long long)k0 * lda + k0;
            int *ip = ipiv + k0;
            bool clustered = false;
            RL_TRY(lu_panel_cluster<T>(P, lda, mrows, kb, k0, ip, &sync.p->err, tiny, s, clustered));
            if (!clustered) {
                if (k0 > 0) RL_TRY_CUDA(cudaMemsetAsync(&sync.p->ctr, 0, sizeof(unsigned), s));
                void *args[] = {&P,       &lda,   (void *)&mrows, (void *)&kb, &k0,  &rows_per,
                                &ip,      &cand.p, &rowj.p,       &sync.p,     &tiny, &wns};
                RL_TRY(launch_coop<T>((void *)pk, G, smem, args, s));
            }
            // the swaps in the block's other columns (every other column for one block)
            RL_TRY(laswp<T>(A + K0, lda, KB, k0 - K0, k0 - K0 + kb, ipiv, k0, k0 + kb, s));
            const int n2 = K1 - k0 - kb, m2 = mrows - kb;
            if (n2 > 0) {
                // mode 0 (unit lower triangle) has no pivot to check: no status word
                RL_LAUNCH(trsm_diag_kernel<T>, ceil_div(n2, kTrsmCols), 128, 0, s, P, lda, kb, P + kb, lda, n2, 0,
                          (int *)nullptr, tiny);
                RL_TRY((gemm<T, false, false>(m2, n2, kb, T(-1), P + (long long)kb * lda, lda, P + kb, lda, T(1),
                                             P + (long long)kb * lda + kb, lda, s, &sync.p->err)));
            }
        }
        if (K1 < n) {
            // the block's swaps in the columns left and right of it, then U12 and the
            // K = KB trailing update (tensor cores for FP32)
            RL_TRY(laswp<T>(A, lda, n, K0, K1, ipiv, K0, K1, s));
            const int N2 = n - K1;
            T *L11 = A + (long long)K0 * lda + K0;
            RL_TRY(tri_solve_dev<T>(L11, lda, KB, L11 + KB, lda, N2, 0, &sync.p->err, s, tiny));
            RL_TRY((gemm<T, false, false>(N2, N2, KB, T(-1), L11 + (long long)KB * lda, lda, L11 + KB, lda, T(1),
                                         L11 + (long long)KB * lda + KB, lda, s, &sync.p->err)));
        } else if (K0 > 0) {
            RL_TRY(laswp<T>(A, lda, K0, 0, 0, ipiv, K0, K1, s));  // the last block's swaps on the left
        }
    }
    int err = 0;
    RL_TRY_CUDA(cudaMemcpyAsync(&err, &sync.p->err, sizeof(int), cudaMemcpyDeviceToHost, s));
    RL_TRY_CUDA(cudaStreamSynchronize(s));
    return err;
}

// Blocked right-looking Cholesky: diagonal block by one CTA, L21 = A21 L11^-T, SYRK.
// FP32: 256-column blocks (outer_nb); L11^-1 comes from a triangular solve with the
// identity, L21 = A21 (L11^-1)^T and the lower-triangle SYRK A22 -= L21 L21^T (K = 256)
// run on the tensor cores. FP64: 64-column blocks, L21 by substitution, the SYRK as gemm()
// takes it. The strict upper triangle is never written either way.
template <class T>
rl_status chol_factor_dev(T *A, long long lda, int n, cudaStream_t s, T tiny = Eps<T>::value) {
    NvtxRange nvtx_("rl.cholesky.factor");
    if (n <= 0) return RL_OK;
    if (n <= one_cta_chol<T>()) return factor_small<T>(A, lda, n, 1, nullptr, s, tiny);
    if constexpr (outer_nb<T>() > 0) {
        constexpr int NBO = outer_nb<T>();
        DevBuf<T> Linv, T21;
        DevBuf<int> st;
        RL_TRY(Linv.alloc((size_t)NBO * NBO, s));
        RL_TRY(T21.alloc((size_t)(n - std::min(n, NBO)) * NBO, s));
        RL_TRY(st.alloc(1, s));
        RL_TRY_CUDA(cudaMemsetAsync(st.p, 0, sizeof(int), s));
        for (int K0 = 0; K0 < n; K0 += NBO) {
            const int KB = std::min(NBO, n - K0), m2 = n - K0 - KB;
            T *P = A + (long long)K0 * lda + K0;
            RL_TRY(factor_small<T>(P, lda, KB, 1, nullptr, s, tiny));
            if (m2 <= 0) continue;
            const long long kk = (long long)KB * KB;
            RL_LAUNCH(eye_kernel<T>, (int)((kk + 255) / 256), 256, 0, s, Linv.p, (long long)KB, KB, KB);
            RL_TRY(tri_solve_dev<T>(P, lda, KB, Linv.p, KB, KB, 1, st.p, s, tiny));
            T *A21 = P + (long long)KB * lda;
            RL_TRY((gemm<T, false, true>(m2, KB, KB, T(1), A21, lda, Linv.p, KB, T(0), T21.p, KB, s, st.p)));
            RL_TRY_CUDA(cudaMemcpy2DAsync(A21, lda * sizeof(T), T21.p, KB * sizeof(T), KB * sizeof(T), m2,
                                          cudaMemcpyDeviceToDevice, s));
            RL_TRY((gemm<T, false, true, true>(m2, m2, KB, T(-1), A21, lda, A21, lda, T(1), A21 + KB, lda, s, st.p)));
        }
        return read_status<T>(st.p, s);
    }
    constexpr int NB = PanelNB<T>::value;
    // One sticky status word, read at the end. A matrix that is not positive definite stops at the
    // block that says so: the kernels already queued behind it leave A alone, and the host looks at
    // the block's outcome while the GPU runs that block's L21 and SYRK, so that neither waits for
    // the other. A failure in the first block, n = 512 / 4096 / 8192: 78 / 222 / 650 us (50 / 180 / 579
    // with a read after every block, 775 / 11,129 / 58,573 with one read at the end).
    StatusWatch &watch = status_watch();
    const bool watched = watch.begin();
    DevBuf<int> st;
    RL_TRY(st.alloc(1, s));
    RL_TRY_CUDA(cudaMemsetAsync(st.p, 0, sizeof(int), s));
    for (int k0 = 0; k0 < n; k0 += NB) {
        const int kb = std::min(NB, n - k0), mrows = n - k0;
        if (k0 && watched) {  // the block before
            RL_TRY_CUDA(cudaEventSynchronize(watch.ev));
            if (watch.failed()) break;
        }
        T *P = A + (long long)k0 * lda + k0;
        RL_TRY(factor_small_async<T>(P, lda, kb, 1, nullptr, st.p, s, tiny, watched ? watch.word : nullptr, watch.mark));
        const int m2 = mrows - kb;
        if (m2 > 0) {
            if (watched) RL_TRY_CUDA(cudaEventRecord(watch.ev, s));
            RL_LAUNCH(trsm_right_lt_kernel<T>, ceil_div(m2, kTrsmCols), 128, 0, s, P, lda, kb, P + (long long)kb * lda, lda,
                      m2, (const int *)st.p);
            T *L21 = P + (long long)kb * lda;
            RL_TRY((gemm<T, false, true, true>(m2, m2, kb, T(-1), L21, lda, L21, lda, T(1), L21 + kb, lda, s, st.p)));
        }
    }
    return read_status<T>(st.p, s);
}

// Tm of a reflector block V (mrows x kb): partial Gram matrices, then the T recursion.
template <class T>
rl_status block_t_factor(const T *V, int mrows, int kb, const T *tau, T *part, int max_parts, T *Tm,
                         cudaStream_t s) {
    const int nparts = ceil_div(mrows, kGramRows);
    if (nparts > max_parts) return RL_ERR_INVALID_ARG;
    RL_LAUNCH(gram_partial_kernel<T>, dim3(nparts, 10), 128, 0, s, V, mrows, kb, part);
    const size_t smem = 2 * 64 * 65 * sizeof(T);
    RL_TRY(set_smem(larft_kernel<T>, smem));
    RL_LAUNCH(larft_kernel<T>, 1, 256, smem, s, part, nparts, tau, kb, Tm);
    return RL_OK;
}

// X (mrows x q) -= V W with V the mrows x kb reflectors of a panel, W kb x q. FP64: the
// unit-triangular rows of V apart, whose few entries would send the first row of tiles of the
// tensor-core product to the FP64 unit (its accuracy check is per tile, gemm_f64tc.cuh).
template <class T>
rl_status block_update(const T *V, int mrows, int kb, const T *W, T *X, long long ldx, int q, cudaStream_t s,
                       int *err) {
    const int head = sizeof(T) == 8 && mrows > kb ? kb : 0;
    if (head)
        RL_TRY((gemm<T, false, false>(head, q, kb, T(-1), V, kb, W, q, T(1), X, ldx, s, err)));
    return gemm<T, false, false>(mrows - head, q, kb, T(-1), V + (long long)head * kb, kb, W, q, T(1), X + (long long)head * ldx,
                                 ldx, s, err);
}

// Blocked Householder QR with compact-WY trailing updates; nrefl reflectors
// (min(m, n) for a plain QR; n for the augmented least-squares matrix).
template <class T>
rl_status qr_factor_dev(T *A, long long lda, int m, int n, int nrefl, T *tau, cudaStream_t s) {
    NvtxRange nvtx_("rl.qr.factor");
    if (nrefl <= 0) return RL_OK;
    constexpr int NB = PanelNB<T>::value;
    int Gmax, rp;
    panel_geometry<T>(m, Gmax, rp);
    if ((size_t)rp * (NB + 1) * sizeof(T) > 200 * 1024) return RL_ERR_INVALID_ARG;
    DevBuf<T> part, x0buf, V, Gp, Tm, W1, W2;
    DevBuf<PanelSync> sync;
    RL_TRY(part.alloc((size_t)2 * Gmax * (1 + NB), s));
    RL_TRY(x0buf.alloc(2, s));
    RL_TRY(sync.alloc(1, s));
    RL_TRY(V.alloc((size_t)m * NB, s));
    const int max_parts = ceil_div(m, kGramRows);
    RL_TRY(Gp.alloc((size_t)max_parts * 64 * 64, s));
    RL_TRY(Tm.alloc(NB * NB, s));
    RL_TRY(W1.alloc((size_t)NB * std::max(1, n), s));
    RL_TRY(W2.alloc((size_t)NB * std::max(1, n), s));
    auto pk = qr_panel_kernel<T>;
    RL_TRY(set_smem(pk, 200 * 1024));
    // Sticky error word, read once at the end (see lu_factor_dev).
    RL_TRY_CUDA(cudaMemsetAsync(sync.p, 0, sizeof(PanelSync), s));
    unsigned long long wns = wait_ns();
    for (int k0 = 0; k0 < nrefl; k0 += NB) {
        const int kb = std::min(NB, nrefl - k0), mrows = m - k0;
        int G, rows_per;
        panel_geometry<T>(mrows, G, rows_per);
        const size_t smem = ((size_t)rows_per * (NB + 1) + NB) * sizeof(T);
        T *P = A + (long long)k0 * lda + k0;
        T *tk = tau + k0;
        bool clustered = false;
        RL_TRY(qr_panel_cluster<T>(P, lda, mrows, kb, tk, &sync.p->err, s, clustered));
        if (!clustered) {
            if (k0 > 0) RL_TRY_CUDA(cudaMemsetAsync(&sync.p->ctr, 0, sizeof(unsigned), s));
            void *args[] = {&P, &lda, (void *)&mrows, (void *)&kb, &rows_per, &tk, &part.p, &x0buf.p, &sync.p, &wns};
            RL_TRY(launch_coop<T>((void *)pk, G, smem, args, s));
        }
        const int n2 = n - k0 - kb;
        if (n2 <= 0) continue;
        const long long mk = (long long)mrows * kb;
        RL_LAUNCH(extract_v_kernel<T>, (int)((mk + 255) / 256), 256, 0, s, P, lda, mrows, kb, V.p);
        RL_TRY(block_t_factor<T>(V.p, mrows, kb, tk, Gp.p, max_parts, Tm.p, s));
        T *A2 = P + kb;
        RL_TRY((gemm<T, true, false>(kb, n2, mrows, T(1), V.p, kb, A2, lda, T(0), W1.p, n2, s, &sync.p->err)));
        RL_TRY((gemm<T, true, false>(kb, n2, kb, T(1), Tm.p, kb, W1.p, n2, T(0), W2.p, n2, s, &sync.p->err)));
        RL_TRY(block_update<T>(V.p, mrows, kb, W2.p, A2, lda, n2, s, &sync.p->err));
    }
    int err = 0;
    RL_TRY_CUDA(cudaMemcpyAsync(&err, &sync.p->err, sizeof(int), cudaMemcpyDeviceToHost, s));
    RL_TRY_CUDA(cudaStreamSynchronize(s));
    return err;
}

// Q[:, 0:k] of a compact QR (HouseholderComposition::first_k_columns): reflector panels
// applied in reverse order to I[:, 0:k], each as Q2 -= V (T (V^T Q2)). The rows and columns of
// a panel's own reflectors are still those of the identity, Q2 = [I 0; 0 Q3] (Q3 an identity
// too for the first panel applied), so V^T Q2 = [V1^T, V2^T Q3] takes a product for the
// columns of Q3 only. *err: a status word for the products' waits (gemm()), read by the caller.
template <class T>
rl_status qr_first_k_dev(const T *QR, long long lda, int m, int n, const T *tau, int k, T *Q, long long ldq,
                         cudaStream_t s, int *err) {
    if (m <= 0 || k <= 0) return RL_OK;
    constexpr int NB = PanelNB<T>::value;
    const long long mk = (long long)m * k;
    RL_LAUNCH(eye_kernel<T>, (int)((mk + 255) / 256), 256, 0, s, Q, ldq, m, k);
    const int jmax = std::min(std::min(m, n), k);
    if (jmax <= 0) return RL_OK;
    DevBuf<T> V, Gp, Tm, W1, W2;
    RL_TRY(V.alloc((size_t)m * NB, s));
    const int max_parts = ceil_div(m, kGramRows);
    RL_TRY(Gp.alloc((size_t)max_parts * 64 * 64, s));
    RL_TRY(Tm.alloc(NB * NB, s));
    RL_TRY(W1.alloc((size_t)NB * k, s));
    RL_TRY(W2.alloc((size_t)NB * k, s));
    for (int k0 = ((jmax - 1) / NB) * NB; k0 >= 0; k0 -= NB) {
        const int kb = std::min(NB, jmax - k0), mrows = m - k0, nc = k - k0;
        const T *P = QR + (long long)k0 * lda + k0;
        const long long mkb = (long long)mrows * kb;
        RL_LAUNCH(extract_v_kernel<T>, (int)((mkb + 255) / 256), 256, 0, s, P, lda, mrows, kb, V.p);
        RL_TRY(block_t_factor<T>(V.p, mrows, kb, tau + k0, Gp.p, max_parts, Tm.p, s));
        T *Q2 = Q + (long long)k0 * ldq + k0;
        const int copied = k0 + kb == jmax ? nc : kb;  // columns of V^T Q2 that are columns of V^T
        RL_LAUNCH(v_transpose_kernel<T>, ceil_div((long long)kb * copied, 256), 256, 0, s, V.p, kb, copied, W1.p, (long long)nc);
        if (copied < nc)
            RL_TRY((gemm<T, true, false>(kb, nc - kb, mrows - kb, T(1), V.p + (long long)kb * kb, kb,
                                         Q2 + (long long)kb * ldq + kb, ldq, T(0), W1.p + kb, nc, s, err)));
        RL_TRY((gemm<T, false, false>(kb, nc, kb, T(1), Tm.p, kb, W1.p, nc, T(0), W2.p, nc, s, err)));
        RL_TRY(block_update<T>(V.p, mrows, kb, W2.p, Q2, ldq, nc, s, err));
    }
    return RL_OK;
}

// X <- Q X (trans = false) or X <- Q^T X (trans = true) for the m x q matrix X (row
// stride ldx), Q = H_0 H_1 ... H_{p-1} from the compact QR (m x n, p = min(m, n)):
// HouseholderComposition::left_multiply_into (householder.rs:203-227) applies the
// reflectors from the last to the first, Q^T takes them from the first to the last.
// Per 64-reflector panel (compact WY, Q_i = I - V T V^T): X[k0:, :] -= V (op(T) (V^T X[k0:, :]))
// with op(T) = T for Q, T^T for Q^T. *err as in qr_first_k_dev.
template <class T>
rl_status qr_apply_q_dev(const T *QR, long long lda, int m, int n, const T *tau, int q, T *X, long long ldx, bool trans,
                         cudaStream_t s, int *err) {
    const int p = std::min(m, n);
    if (m <= 0 || q <= 0 || p <= 0) return RL_OK;
    constexpr int NB = PanelNB<T>::value;
    DevBuf<T> V, Gp, Tm, W1, W2;
    RL_TRY(V.alloc((size_t)m * NB, s));
    const int max_parts = ceil_div(m, kGramRows);
    RL_TRY(Gp.alloc((size_t)max_parts * 64 * 64, s));
    RL_TRY(Tm.alloc(NB * NB, s));
    RL_TRY(W1.alloc((size_t)NB * q, s));
    RL_TRY(W2.alloc((size_t)NB * q, s));
    const int last = ((p - 1) / NB) * NB;
    for (int i = 0; i <= last / NB; i++) {
        const int k0 = trans ? i * NB : last - i * NB;
        const int kb = std::min(NB, p - k0), mrows = m - k0;
        const T *P = QR + (long long)k0 * lda + k0;
        const long long mkb = (long long)mrows * kb;
        RL_LAUNCH(extract_v_kernel<T>, (int)((mkb + 255) / 256), 256, 0, s, P, lda, mrows, kb, V.p);
        RL_TRY(block_t_factor<T>(V.p, mrows, kb, tau + k0, Gp.p, max_parts, Tm.p, s));
        T *X2 = X + (long long)k0 * ldx;
        RL_TRY((gemm<T, true, false>(kb, q, mrows, T(1), V.p, kb, X2, ldx, T(0), W1.p, q, s, err)));
        if (trans)
            RL_TRY((gemm<T, true, false>(kb, q, kb, T(1), Tm.p, kb, W1.p, q, T(0), W2.p, q, s, err)));
        else
            RL_TRY((gemm<T, false, false>(kb, q, kb, T(1), Tm.p, kb, W1.p, q, T(0), W2.p, q, s, err)));
        RL_TRY(block_update<T>(V.p, mrows, kb, W2.p, X2, ldx, q, s, err));
    }
    return RL_OK;
}

// One launch of the triangular sweep by substitution, or (FP64, one right-hand side) with the
// inverted diagonal blocks Dinv: the 1-wide instance for one right-hand side (the 8-wide one would
// issue 8 FMAs per element, 7 of them predicated off, each a full issue of the FP64 pipe for T =
// double). ws as trsv_sweep_kernel takes it.
template <class T, class TA, int RW, int ROWS = sweep_rows<T>()>
static rl_status sweep_launch_w(const TA *A, long long lda, int n, const T *Dinv, T *Y, long long ldy, int nrhs, int mode,
                                int *dstatus, cudaStream_t s, T tiny, void *ws) {
    using cfg = SweepCfg<T, RW, ROWS>;
    auto kern = trsv_sweep_kernel<T, TA, RW, ROWS>;
    static int per_sm = 0;
    static const cudaError_t attr = [&] {
        const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cfg::SMEM_LT);
        return e != cudaSuccess ? e : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, cfg::THREADS, cfg::SMEM_LT);
    }();
    RL_TRY_CUDA(attr);
    const int groups = sweep_groups(nrhs), nb = ceil_div(n, cfg::BR);
    T *x = static_cast<T *>(ws);
    int *tickets = reinterpret_cast<int *>(x + (size_t)groups * n * RW);
    const dim3 grid(std::min(nb, std::max(1, per_sm) * num_sms()), groups);
    RL_LAUNCH(kern, grid, cfg::THREADS, mode == 3 ? cfg::SMEM_LT : cfg::SMEM, s, A, lda, n, Y, ldy, nrhs, mode, x, tickets, dstatus, tiny, wait_ns(),
              (int)tune(RL_TUNE_TEST_WITHHOLD_SWEEP_BLOCK), Dinv);
    return RL_OK;
}
template <class T, class TA>
static rl_status sweep_launch(const TA *A, long long lda, int n, const T *Dinv, T *Y, long long ldy, int nrhs, int mode,
                              int *dstatus, cudaStream_t s, T tiny, void *ws) {
    if constexpr (sweep_rows<T>() > 64)
        if (n <= 64)  // one block either way: half the threads and shared memory
            return sweep_width(nrhs) == 1
                       ? sweep_launch_w<T, TA, 1, 64>(A, lda, n, Dinv, Y, ldy, nrhs, mode, dstatus, s, tiny, ws)
                       : sweep_launch_w<T, TA, kSweepRhs, 64>(A, lda, n, Dinv, Y, ldy, nrhs, mode, dstatus, s, tiny, ws);
    return sweep_width(nrhs) == 1 ? sweep_launch_w<T, TA, 1>(A, lda, n, Dinv, Y, ldy, nrhs, mode, dstatus, s, tiny, ws)
                                  : sweep_launch_w<T, TA, kSweepRhs>(A, lda, n, Dinv, Y, ldy, nrhs, mode, dstatus, s, tiny, ws);
}

// One launch of trsv_inv_kernel (FP32, inverted diagonal blocks); ws as above.
template <int RW>
static rl_status sweep_inv_launch(const float *A, long long lda, int n, const float *Dinv, float *Y, long long ldy, int nrhs,
                                  int mode, int *dstatus, cudaStream_t s, void *ws) {
    static int per_sm = 0;
    static const cudaError_t q = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, trsv_inv_kernel<RW>, 256, 0);
    RL_TRY_CUDA(q);
    const int groups = sweep_groups(nrhs), nb = ceil_div(n, kInvRows);
    float *x = static_cast<float *>(ws);
    int *tickets = reinterpret_cast<int *>(x + (size_t)groups * n * RW);
    // every group's chain runs from the start: the CTAs that fit are shared out over the groups
    const dim3 grid(std::min(nb, std::max(1, std::max(1, per_sm) * num_sms() / groups)), groups);
    RL_LAUNCH(trsv_inv_kernel<RW>, grid, 256, 0, s, A, lda, n, Y, ldy, nrhs, mode, x, tickets, dstatus, wait_ns(),
              (int)tune(RL_TUNE_TEST_WITHHOLD_SWEEP_BLOCK), Dinv);
    return RL_OK;
}

// Blocked triangular solve op(A) X = Y in place (A n x n, Y n x nrhs).
// mode 0: unit lower, 1: lower, 2: upper, 3: L^T with L lower. |d_ii| < eps is
// recorded as RL_ERR_DIV_BY_ZERO in *dstatus. A may be stored in a narrower type TA than
// the arithmetic type T for at most kSweepGroups x kSweepRhs right-hand sides (an FP32
// factor applied in FP64), kSweepRhs on a GPU shared with other workers.
template <class T, class TA>
rl_status tri_solve_dev(const TA *A, long long lda, int n, T *Y, long long ldy, int nrhs, int mode, int *dstatus,
                        cudaStream_t s, T tiny) {
    if (n <= 0 || nrhs <= 0) return RL_OK;
    constexpr int NB = 64;
    if (nrhs <= kSweepRhs && g_shared_gpu) {
        // Few right-hand sides on a shared GPU: per 64-row block a one-CTA diagonal solve
        // (warp per column) and a warp-per-row GEMV update, all short launches.
        const int wpb = 8, gridr = std::max(1, std::min(4 * num_sms(), ceil_div(n, wpb)));
        if (mode == 0 || mode == 1) {
            for (int b0 = 0; b0 < n; b0 += NB) {
                const int bs = std::min(NB, n - b0), rest = n - b0 - bs;
                T *Yb = Y + (long long)b0 * ldy;
                RL_LAUNCH((trsv_diag_kernel<T, TA>), 1, 256, 0, s, A + (long long)b0 * lda + b0, lda, bs, Yb, ldy, nrhs, mode,
                          dstatus, tiny);
                if (rest > 0)
                    RL_LAUNCH((gemv_update_kernel<T, TA>), std::min(gridr, ceil_div(rest, wpb)), 32 * wpb, 0, s,
                              A + (long long)(b0 + bs) * lda + b0, lda, rest, bs, Yb, ldy, Yb + (long long)bs * ldy,
                              nrhs, false);
            }
        } else {
            for (int b1 = n; b1 > 0; b1 -= NB) {
                const int b0 = std::max(0, b1 - NB), bs = b1 - b0;
                T *Yb = Y + (long long)b0 * ldy;
                RL_LAUNCH((trsv_diag_kernel<T, TA>), 1, 256, 0, s, A + (long long)b0 * lda + b0, lda, bs, Yb, ldy, nrhs, mode,
                          dstatus, tiny);
                if (b0 > 0) {
                    if (mode == 2)
                        RL_LAUNCH((gemv_update_kernel<T, TA>), std::min(gridr, ceil_div(b0, wpb)), 32 * wpb, 0, s, A + b0, lda,
                                  b0, bs, Yb, ldy, Y, nrhs, false);
                    else
                        RL_LAUNCH((gemv_update_kernel<T, TA>), ceil_div(b0, 256), 256, 0, s, A + (long long)b0 * lda, lda, b0,
                                  bs, Yb, ldy, Y, nrhs, true);
                }
            }
        }
        return RL_OK;
    }
    if (sweep_groups(nrhs) > 0 && !g_shared_gpu) {
        // Up to kSweepGroups x kSweepRhs right-hand sides: the whole solve in one launch
        // (trsv_sweep_kernel, groups of kSweepRhs columns side by side). The blocked form
        // below costs two launches per 64-row block, a 64-step chain on a few CTAs and a
        // GEMM whose tiles would be mostly empty.
        DevBuf<unsigned char> ws;
        RL_TRY(ws.alloc(sweep_ws_bytes<T>(n, nrhs), s));
        RL_TRY_CUDA(cudaMemsetAsync(ws.p, 0xff, sweep_ws_bytes<T>(n, nrhs), s));
        return sweep_launch<T, TA>(A, lda, n, nullptr, Y, ldy, nrhs, mode, dstatus, s, tiny, ws.p);
    }
    if constexpr (!std::is_same<T, TA>::value) {
        return RL_ERR_INVALID_ARG;  // mixed storage: few right-hand sides only
    } else {
        const int gr = ceil_div(nrhs, kTrsmCols);
        if (mode == 0 || mode == 1) {
            for (int b0 = 0; b0 < n; b0 += NB) {
                const int bs = std::min(NB, n - b0);
                const T *D = A + (long long)b0 * lda + b0;
                T *Yb = Y + (long long)b0 * ldy;
                RL_LAUNCH(trsm_diag_kernel<T>, gr, 128, 0, s, D, lda, bs, Yb, ldy, nrhs, mode, dstatus, tiny);
                const int rest = n - b0 - bs;
                if (rest > 0)
                    RL_TRY((gemm<T, false, false>(rest, nrhs, bs, T(-1), A + (long long)(b0 + bs) * lda + b0, lda, Yb, ldy,
                                                  T(1), Yb + (long long)bs * ldy, ldy, s, dstatus)));
            }
        } else {
            for (int b1 = n; b1 > 0; b1 -= NB) {
                const int b0 = std::max(0, b1 - NB), bs = b1 - b0;
                const T *D = A + (long long)b0 * lda + b0;
                T *Yb = Y + (long long)b0 * ldy;
                RL_LAUNCH(trsm_diag_kernel<T>, gr, 128, 0, s, D, lda, bs, Yb, ldy, nrhs, mode, dstatus, tiny);
                if (b0 > 0) {
                    if (mode == 2)
                        RL_TRY((gemm<T, false, false>(b0, nrhs, bs, T(-1), A + b0, lda, Yb, ldy, T(1), Y, ldy, s, dstatus)));
                    else
                        RL_TRY((gemm<T, true, false>(b0, nrhs, bs, T(-1), A + (long long)b0 * lda, lda, Yb, ldy, T(1), Y,
                                                     ldy, s, dstatus)));
                }
            }
        }
        return RL_OK;
    }
}

// Inverses of op(A)'s 64 x 64 diagonal blocks, formed in T (ceil(n / 64) row-major blocks in Dinv,
// zero beyond a partial last one; diag_inverse_kernel).
inline size_t diag_inverse_elems(int n) { return (size_t)ceil_div(n, kInvRows) * kInvRows * kInvRows; }
template <class T, class TA>
rl_status diag_inverse(const TA *A, long long lda, int n, int mode, T *Dinv, int *dstatus, cudaStream_t s, T tiny) {
    if (n <= 0) return RL_OK;
    RL_LAUNCH((diag_inverse_kernel<T, TA>), ceil_div(n, kInvRows), 64, 0, s, A, lda, n, mode, Dinv, dstatus, tiny);
    return RL_OK;
}

// op(A) Y = Y' in one sweep launch whose block solves are products with the diagonal blocks'
// inverses Dinv (diag_inverse): FP32 with at most kSweepGroups x kSweepRhs right-hand sides, or FP64
// with one. ws: sweep_ws_bytes<T>(n, nrhs) bytes with all bits set. More right-hand sides, or a GPU
// shared with other streams of this library (the serving workers, see tri_solve_dev), take
// tri_solve_dev's substitution paths instead.
template <class T, class TA>
rl_status tri_solve_inv_dev(const TA *A, long long lda, int n, const T *Dinv, T *Y, long long ldy, int nrhs, int mode,
                            int *dstatus, cudaStream_t s, T tiny, void *ws) {
    if (sweep_groups(nrhs) == 0 || g_shared_gpu)
        return tri_solve_dev<T, TA>(A, lda, n, Y, ldy, nrhs, mode, dstatus, s, tiny);
    if (n <= 0 || nrhs <= 0) return RL_OK;
    if constexpr (std::is_same<T, double>::value)
        return sweep_launch_w<T, TA, 1>(A, lda, n, Dinv, Y, ldy, nrhs, mode, dstatus, s, tiny, ws);
    else
        return nrhs == 1 ? sweep_inv_launch<1>(A, lda, n, Dinv, Y, ldy, nrhs, mode, dstatus, s, ws)
                         : sweep_inv_launch<kSweepRhs>(A, lda, n, Dinv, Y, ldy, nrhs, mode, dstatus, s, ws);
}

// Solve with factors already on the device. kind 0 = LU (dperm: stored permutation),
// 1 = Cholesky. B (n x nrhs, stride ldb) is overwritten.
template <class T>
rl_status factor_solve_dev(const T *F, long long lda, int n, int kind, const uint64_t *dperm, T *B, long long ldb,
                           int nrhs, cudaStream_t s) {
    if (n <= 0 || nrhs <= 0) return RL_OK;
    DevBuf<int> st;
    RL_TRY(st.alloc(1, s));
    RL_TRY_CUDA(cudaMemsetAsync(st.p, 0, sizeof(int), s));
    // Up to CTA_NMAX rows a CTA per right-hand side, or one sweep for a single one from the
    // size where its chain of blocks is shorter (host calls, FP64 n = 96 128 and 113 us, 512
    // 602 and 226; FP32 n = 256 122 and 120, 512 191 and 147). Many right-hand sides stay a
    // CTA each (inverse, FP64 n = 512: 1,470 and 1,667 us).
    const bool sweep = nrhs == 1 && !g_shared_gpu && n > (sizeof(T) == 8 ? 88 : 256);
    if (n <= CTA_NMAX && !sweep) {
        const size_t smem = cta_smem_bytes<T>();
        RL_TRY(set_smem(solve_one_kernel<T>, smem));
        RL_LAUNCH(solve_one_kernel<T>, nrhs, CTA_THREADS, smem, s, F, (int)lda, n, kind, kind ? nullptr : dperm, B, ldb,
                  st.p, Eps<T>::value);
        return read_status<T>(st.p, s);
    }
    if (kind == 1) {
        RL_TRY(tri_solve_dev<T>(F, lda, n, B, ldb, nrhs, 1, st.p, s));
        RL_TRY(tri_solve_dev<T>(F, lda, n, B, ldb, nrhs, 3, st.p, s));
        return read_status<T>(st.p, s);
    }
    DevBuf<T> Y;
    RL_TRY(Y.alloc((size_t)n * nrhs, s));
    const long long tot = (long long)n * nrhs;
    RL_LAUNCH(permute_rows_kernel<T>, (int)((tot + 255) / 256), 256, 0, s, B, ldb, Y.p, (long long)nrhs, n, nrhs,
              dperm);
    RL_TRY(tri_solve_dev<T>(F, lda, n, Y.p, nrhs, nrhs, 0, st.p, s));
    RL_TRY(tri_solve_dev<T>(F, lda, n, Y.p, nrhs, nrhs, 2, st.p, s));
    RL_TRY_CUDA(cudaMemcpy2DAsync(B, ldb * sizeof(T), Y.p, nrhs * sizeof(T), nrhs * sizeof(T), n,
                                  cudaMemcpyDeviceToDevice, s));
    return read_status<T>(st.p, s);
}

inline rl_status check_perm(size_t n, const uint64_t *perm) {
    std::vector<unsigned char> seen(n, 0);
    for (size_t i = 0; i < n; i++) {
        if (perm[i] >= n || seen[perm[i]]) return RL_ERR_INVALID_PERMUTATION;
        seen[perm[i]] = 1;
    }
    return RL_OK;
}

inline bool fits_int(size_t v) { return v <= (size_t)INT32_MAX; }

}  // namespace rl

// Kernels of the blocked (multi-CTA) factorisations used above one_cta_lu / one_cta_chol rows
// (dense_ops.cuh) and for every HouseholderQr: cooperative panel kernels with a bounded grid barrier, row swaps,
// diagonal-block triangular solves and the compact-WY T factor. Trailing updates are
// GEMMs (gemm.cuh).
#pragma once

#include <algorithm>
#include <climits>

#include <cooperative_groups.h>

#include "factor_cta.cuh"

namespace rl {

// a / p from r = 1 / p: the rounded product corrected by its exact remainder (Markstein, IBM
// J. Res. Dev. 34, 1990).
template <class T>
__device__ __forceinline__ T quotient(T a, T p, T r) {
    const T q = a * r;
    const T e = fma(-q, p, a);
    const T c = fma(e, r, q);
    return e == e ? c : q;  // an infinite product has no remainder
}

// The biased exponent of x (0: zero or subnormal), and whether x times a value of exponent es could
// leave the normal range: overflow, or lose bits that x has. On integers: a comparison of doubles takes
// the FP64 unit.
__device__ __forceinline__ int exponent_of(float x) { return (int)(__float_as_uint(x) >> 23) & 0xff; }
__device__ __forceinline__ int exponent_of(double x) { return (__double2hiint(x) >> 20) & 0x7ff; }
__device__ __forceinline__ bool scaling_wide(float x, int es) {
    const int e = exponent_of(x) + es - 127;  // of the product, or one below it
    return (e < 3 || e > 252) && (__float_as_uint(x) << 1) != 0u;
}
__device__ __forceinline__ bool scaling_wide(double x, int es) {
    const int e = exponent_of(x) + es - 1023;
    return (e < 3 || e > 2044) && (__double_as_longlong(x) << 1) != 0;
}

// Largest panel width of the blocked paths.
template <class T>
struct PanelNB {
    static constexpr int value = 64;
};

// ------------------------------------------------------------------ grid barrier --
// All CTAs of a cooperative launch arrive on `ctr`; thread 0 spins (bounded by
// `limit` ns of wall time, RL_TUNE_WAIT_TIMEOUT_NS) until the count reaches `target`.
// On timeout the error word is set and every CTA leaves the kernel at its next barrier.

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ unsigned ld_acquire_u32(const unsigned *p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ int ld_acquire(const int *p) { return (int)ld_acquire_u32(reinterpret_cast<const unsigned *>(p)); }
__device__ __forceinline__ void st_release(int *p, int v) {
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

static __device__ bool grid_barrier(unsigned *ctr, unsigned target, int *err, unsigned long long limit) {
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(ctr, 1u);
        const unsigned long long t0 = global_ns();
        int ok = 1;
        for (;;) {
            if (ld_acquire_u32(ctr) >= target) break;
            if (*(volatile int *)err != 0) {
                ok = 0;
                break;
            }
            if (global_ns() - t0 > limit) {
                atomicCAS(err, 0, RL_ERR_TIMEOUT);
                ok = 0;
                break;
            }
            __nanosleep(64);
        }
        __threadfence();
        s_ok = ok && (*(volatile int *)err == 0);
    }
    __syncthreads();
    return s_ok != 0;
}

// Shared state of one cooperative panel launch (global memory, zeroed per launch).
struct PanelSync {
    unsigned ctr;
    int err;     // RL_ERR_TIMEOUT or a numerical status, first writer wins
    int pad[2];
};

// ------------------------------------------------------------------- LU panel --
// Factors the panel rows [0, mrows) x cols [0, kb) of `P` (row stride lda; P points at
// A[k0][k0]) with partial pivoting. CTA g owns rows [g*rows_per, ...) staged in shared
// memory row-major (stride NB + 1). Per column: local argmax -> publish candidate row
// -> one grid barrier -> every CTA picks the same winner (largest |v|, smallest row on
// ties), swaps, scales and updates its rows. ipiv receives k0-based global pivots.
// cand: 2 slots x G x (2 + NB) values, rowj: 2 slots x NB values.
template <class T>
static __global__ void __launch_bounds__(256) lu_panel_kernel(T *P, long long lda, int mrows, int kb, int k0, int rows_per,
                                                       int *ipiv, T *cand, T *rowj, PanelSync *sync, T tiny,
                                                       unsigned long long wait_ns) {
    constexpr int NB = PanelNB<T>::value;
    constexpr int LDR = NB + 1;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T *R = reinterpret_cast<T *>(smem_raw);  // rows_per x LDR
    T *prow = R + (size_t)rows_per * LDR;    // pivot row copy (NB)
    __shared__ T s_v[8];
    __shared__ int s_i[8];
    const int G = gridDim.x, g = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int r0 = g * rows_per, r1 = min(mrows, r0 + rows_per), nr = max(0, r1 - r0);
    const int CS = 2 + NB;  // candidate record: |v|, row, then the row's values

    // Identity pivots first: a launch that stops early (error or timeout) still leaves
    // in-range pivots for the row swaps that follow it on the stream.
    if (g == 0)
        for (int j = tid; j < kb; j += blockDim.x) ipiv[j] = k0 + j;
    for (int idx = tid; idx < nr * kb; idx += blockDim.x) {
        const int r = idx / kb, c = idx - r * kb;
        R[r * LDR + c] = P[(long long)(r0 + r) * lda + c];
    }
    __syncthreads();
    __shared__ int s_q[8];
    for (int j = 0; j < kb; j++) {
        const int slot = j & 1;
        T bv = T(-1);
        int bi = INT_MAX;
        for (int r = max(j - r0, 0) + tid; r < nr; r += blockDim.x) {
            const T v = absT(R[r * LDR + j]);
            if (v > bv) {
                bv = v;
                bi = r0 + r;
            }
        }
        warp_amax(bv, bi);
        if (lane == 0) {
            s_v[warp] = bv;
            s_i[warp] = bi;
        }
        __syncthreads();
        bv = s_v[0];
        bi = s_i[0];
        for (int w = 1; w < (int)(blockDim.x >> 5); w++) amax_combine(bv, bi, s_v[w], s_i[w]);
        T *mine = cand + ((size_t)slot * G + g) * CS;
        if (tid == 0) {
            mine[0] = bv;
            mine[1] = (T)(bi == INT_MAX ? -1 : bi);
        }
        if (bi != INT_MAX && tid < kb) mine[2 + tid] = R[(bi - r0) * LDR + tid];
        if (j >= r0 && j < r1 && tid < kb) rowj[slot * NB + tid] = R[(j - r0) * LDR + tid];
        if (!grid_barrier(&sync->ctr, (unsigned)(G * (j + 1)), &sync->err, wait_ns)) return;
        // Winner over all CTAs, identical in every CTA: thread q reads CTA q's candidate,
        // then a block argmax (largest |v|, smallest row on ties).
        T wv = T(-1);
        int wi = INT_MAX, wg = -1;
        for (int q = tid; q < G; q += blockDim.x) {
            const volatile T *c = cand + ((size_t)slot * G + q) * CS;
            const T v = c[0];
            const int i = (int)c[1];
            if (i >= 0 && (v > wv || (v == wv && i < wi))) {
                wv = v;
                wi = i;
                wg = q;
            }
        }
        warp_amax3(wv, wi, wg);
        __syncthreads();  // s_v / s_i of the local argmax are read no more
        if (lane == 0) {
            s_v[warp] = wv;
            s_i[warp] = wi;
            s_q[warp] = wg;
        }
        __syncthreads();
        wv = s_v[0];
        wi = s_i[0];
        wg = s_q[0];
        for (int w = 1; w < (int)(blockDim.x >> 5); w++)
            if (s_v[w] > wv || (s_v[w] == wv && s_i[w] < wi)) {
                wv = s_v[w];
                wi = s_i[w];
                wg = s_q[w];
            }
        if (wi == INT_MAX) {  // no finite candidate (NaN column): keep the diagonal
            wi = j;
            wg = -1;
        }
        if (wg >= 0 && wv < tiny) {
            if (g == 0 && tid == 0) atomicCAS(&sync->err, 0, RL_ERR_DIV_BY_ZERO);
            return;
        }
        if (tid < kb) {
            T v;
            if (wg >= 0)
                v = ((volatile T *)(cand + ((size_t)slot * G + wg) * CS))[2 + tid];
            else
                v = ((volatile T *)rowj)[slot * NB + tid];
            prow[tid] = v;
        }
        __syncthreads();
        if (wi != j) {
            if (j >= r0 && j < r1 && tid < kb) R[(j - r0) * LDR + tid] = prow[tid];
            if (wi >= r0 && wi < r1 && tid < kb) R[(wi - r0) * LDR + tid] = ((volatile T *)rowj)[slot * NB + tid];
        }
        if (g == 0 && tid == 0) ipiv[j] = k0 + wi;
        __syncthreads();
        const T inv_p = T(1) / prow[j];  // multipliers by the reciprocal: one division per column
        for (int r = max(j + 1 - r0, 0) + tid; r < nr; r += blockDim.x) {
            T *row = R + r * LDR;
            const T l = row[j] * inv_p;
            row[j] = l;
            for (int c = j + 1; c < kb; c++) row[c] = fma(-l, prow[c], row[c]);
        }
        __syncthreads();
    }
    for (int idx = tid; idx < nr * kb; idx += blockDim.x) {
        const int r = idx / kb, c = idx - r * kb;
        P[(long long)(r0 + r) * lda + c] = R[r * LDR + c];
    }
}

// |v| as an unsigned key that orders like |v| (non-negative IEEE values order like
// their bits), 0 for NaN, which never wins: the pivot search compares keys on the
// integer pipe. On GB300 an FP64 comparison issues on the FP64 pipe, which a warp
// occupies for tens of cycles; the integer form also keeps FP32 and FP64 alike.
__device__ __forceinline__ unsigned long long amax_key(float v) {
    const unsigned u = __float_as_uint(v) & 0x7fffffffu;
    return u > 0x7f800000u ? 0ull : (unsigned long long)u + 1ull;
}
__device__ __forceinline__ unsigned long long amax_key(double v) {
    const unsigned long long u = (unsigned long long)__double_as_longlong(v) & 0x7fffffffffffffffull;
    return u > 0x7ff0000000000000ull ? 0ull : u + 1ull;
}

// Largest key over the warp and the smallest index among the lanes holding it, in every
// lane, on the redux instructions (keys of FP32 values fit in 32 bits; FP64 keys are
// reduced high word first). Lanes without a candidate hold key 0 and index INT_MAX.
template <class T>
__device__ __forceinline__ void warp_amax_key(unsigned long long &k, int &i) {
    bool top;
    if (sizeof(T) == 4) {
        const unsigned k32 = (unsigned)k;
        const unsigned kmax = __reduce_max_sync(0xffffffffu, k32);
        top = k32 == kmax;
        k = kmax;
    } else {
        const unsigned hi = (unsigned)(k >> 32), lo = (unsigned)k;
        const unsigned hmax = __reduce_max_sync(0xffffffffu, hi);
        const unsigned lmax = __reduce_max_sync(0xffffffffu, hi == hmax ? lo : 0u);
        top = hi == hmax && lo == lmax;
        k = ((unsigned long long)hmax << 32) | lmax;
    }
    i = (int)__reduce_min_sync(0xffffffffu, top ? (unsigned)i : 0xffffffffu);
}

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// Cluster primitives of the panel kernels: a 16-byte store into another CTA's shared memory
// that counts its bytes on that CTA's mbarrier, and the (bounded) wait for them.
__device__ __forceinline__ uint32_t smem_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint32_t cluster_addr(uint32_t a, int rank) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
__device__ __forceinline__ void st_async16(uint32_t dst, uint4 v, uint32_t bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(dst),
                 "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void cl_mbar_init(uint64_t *bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void cl_mbar_expect(uint64_t *bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool cl_mbar_wait(uint64_t *bar, unsigned parity, unsigned long long limit) {
    const uint32_t a = smem_addr(bar);
    unsigned long long t0 = 0;
    for (unsigned spin = 0;; spin++) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(a), "r"(parity)
            : "memory");
        if (done) return true;
        if ((spin & 63u) == 63u) {  // the timer is read once per 64 polls
            if (t0 == 0)
                t0 = global_ns();
            else if (global_ns() - t0 > limit)
                return false;
        }
    }
}

// After a wait that ran out: st.async stores of other CTAs into this one may still be under way, which
// neither the mbarrier (given up) nor a cluster barrier waits for. They take about a microsecond; a CTA
// stays for 100 before it gives up its shared memory.
__device__ __forceinline__ void cl_settle() {
    const unsigned long long t0 = global_ns();
    while (global_ns() - t0 < 100000) __nanosleep(1000);
}

// LU panel on one thread-block cluster (up to 16 CTAs): the same algorithm as
// lu_panel_kernel with the cross-CTA exchange on chip. CTA g owns the rows
// [g * rows_per, ...), staged in shared memory. The panel is factored 16 columns at a time
// in registers: TPR consecutive threads share a row (TPR > 1 when a CTA holds few rows, so
// that the FP64 updates use every scheduler), thread q of them owning the columns
// c = q (mod TPR) of the 16, and a thread group holds RPT rows. Per column:
//   1. the threads search the column of their rows, the warps reduce on integer keys, each
//      warp's best row goes to shared memory; one CTA barrier;
//   2. the CTA pushes its candidate (16 columns), row j if it holds it, and its record (key,
//      row, 1 / pivot) into every CTA's tables with st.async, which counts the bytes on the
//      receiver's mbarrier: one one-way trip, no cluster barrier;
//   3. every CTA waits for its own table to be complete; every warp picks the same winner;
//   4. swap and update in registers.
// After the 16 columns the row swaps reach the panel's other columns: their composition (at
// most 32 rows) is formed from the pivots, the moved rows and the 16 pivot rows are read from
// the CTAs that hold them, one cluster barrier, then U12 = L11^-1 A12 (in every
// CTA) and the update of the columns to the right, each row adding its 16 products in
// column order: every element sees the operations of the unblocked elimination, in the same
// order. Tables and barriers are double-buffered by column parity: a CTA pushes column
// j + 2 only after it has received every CTA's column j + 1, which those push after their
// last read of column j's tables.
// Bound by a column's chain of dependent steps (FP32: ~2,500 cycles, of which the exchange
// is ~500) or by the FP64 unit of the cluster's SMs. The form before pushed all 64 columns
// and passed a cluster barrier per column, with the panel in shared memory: 172 us per FP32
// panel averaged over n = 4096, 89 now; 16 CTAs of 512 rows 250 and 119 us; FP64 234 and
// 201 us.
// A failing pivot is seen by all CTAs at the same column and acted on after the next CTA
// barrier (the flag is kept per column parity, so a thread ahead by a column does not show
// its finding to one that still has to read the last column's). Every wait is bounded
// (RL_ERR_TIMEOUT); a CTA whose wait ran out tells the others before it leaves.
constexpr int kPanelSub = 16;
template <class T>
struct PanelTables {
    static constexpr int RECW = sizeof(T) == 4 ? 1 : 2;  // 16-byte words of a record
    uint4 rec[2][16][RECW];                             // {key lo, key hi | 1 / pivot, row, -}, {1 / pivot}
    T tab[2][16][kPanelSub];                            // every CTA's candidate row
    T rowj[2][kPanelSub];                               // row j
    T cand[2][8][kPanelSub];                            // the warps' candidates
    T candj[2][kPanelSub];                              // row j, in the CTA that holds it
    T L11t[kPanelSub][kPanelSub];                       // L11t[k][i] = l_ik of the pivot rows
    T U[64 - kPanelSub][kPanelSub];                     // U12 by columns
    unsigned long long s_k[2][8];
    int s_i[2][8];
    int piv[kPanelSub];
    int dst[32];        // moved rows of this CTA: where to (-1: none) ...
    uint32_t src[32];   // ... and where every moved row is (cluster shared address)
    uint64_t full[2];
    int fail[2];  // by column parity: 1 = a wait ran out, 2 = a failing pivot
    int dead;     // another CTA's wait ran out
};

__device__ __forceinline__ float ld_cluster(uint32_t a, float) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ double ld_cluster(uint32_t a, double) {
    double v;
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
    return v;
}
// N consecutive values (16-byte aligned) from / to shared memory, 16 bytes at a time.
template <int N, class T>
__device__ __forceinline__ void ldv(const T *p, T (&v)[N]) {
    constexpr int W = 16 / (int)sizeof(T);
#pragma unroll
    for (int i = 0; i < N; i += W) {
        const uint4 x = *reinterpret_cast<const uint4 *>(p + i);
        const T *e = reinterpret_cast<const T *>(&x);
#pragma unroll
        for (int u = 0; u < W; u++) v[i + u] = e[u];
    }
}
template <int N, class T>
__device__ __forceinline__ void stv(T *p, const T (&v)[N]) {
    constexpr int W = 16 / (int)sizeof(T);
#pragma unroll
    for (int i = 0; i < N; i += W) {
        uint4 x;
        T *e = reinterpret_cast<T *>(&x);
#pragma unroll
        for (int u = 0; u < W; u++) e[u] = v[i + u];
        *reinterpret_cast<uint4 *>(p + i) = x;
    }
}

// Rows in the tables and in registers are kept rotated: at local column step jo the entry
// q L + i of a row is its column ((jo + i) mod L) TPR + q.
template <class T, int TPR, int RPT>
static __global__ void __launch_bounds__(256) lu_panel_cluster_kernel(T *P, long long lda, int mrows, int kb, int k0,
                                                              int rows_per, int *ipiv, int *err, T tiny,
                                                              unsigned long long wait_ns) {
    namespace cg = cooperative_groups;
    constexpr int NB = PanelNB<T>::value, LDR = NB + 1, SW = kPanelSub, L = SW / TPR, G = 256 / TPR;
    constexpr int RECW = PanelTables<T>::RECW, CH = SW * (int)sizeof(T) / 16;  // 16-byte words of a record, a row
    static_assert(16 * CH <= 224, "one candidate word per thread of warps 1 .. 7");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T *R = reinterpret_cast<T *>(smem_raw);  // rows_per x LDR
    __shared__ __align__(16) PanelTables<T> S;
    cg::cluster_group cluster = cg::this_cluster();
    const int C = (int)cluster.num_blocks(), g = (int)cluster.block_rank();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int r0 = g * rows_per, r1 = min(mrows, r0 + rows_per), nr = max(0, r1 - r0);
    const int q = tid & (TPR - 1), grp = tid / TPR;
    const unsigned long long ktiny = amax_key(tiny);
    const unsigned bytes = (unsigned)(16 * (C * (RECW + CH) + CH));
    if (g == 0)
        for (int j = tid; j < kb; j += 256) ipiv[j] = k0 + j;
    for (int idx = tid; idx < nr * kb; idx += 256) {
        const int r = idx / kb, c = idx - r * kb;
        R[r * LDR + c] = P[(long long)(r0 + r) * lda + c];
    }
    if (tid == 0) {
        S.fail[0] = S.fail[1] = S.dead = 0;
        cl_mbar_init(&S.full[0], 1);
        cl_mbar_init(&S.full[1], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    cluster.sync();
    cluster_arrive();  // waited for before the first read of other CTAs' rows
    bool arrived = true, stop = false;
    // what this thread pushes per column: warp 0 lane d the record to CTA d, thread 32 + e
    // word e % CH of the candidate (and of row j) to CTA e / CH
    const int pe = tid - 32, pto = warp == 0 ? lane : pe / CH, pch = pe & (CH - 1);
    const bool pusher = warp == 0 ? lane < C : pe < C * CH;
    const int peer = min(pto, C - 1);
    const uint32_t bar_to = cluster_addr(smem_addr(&S.full[0]), peer);
    const uint32_t tab_to = cluster_addr(warp == 0 ? smem_addr(&S.rec[0][g][0]) : smem_addr(S.tab[0][g]) + 16 * pch, peer);
    const uint32_t rowj_to = cluster_addr(smem_addr(S.rowj[0]) + 16 * (pch & (CH - 1)), peer);
    for (int c0 = 0; c0 < kb && !stop; c0 += SW) {
        const int w = min(SW, kb - c0);
        T a[RPT][L];
#pragma unroll
        for (int k = 0; k < RPT; k++) {
            const int r = grp + k * G;
#pragma unroll
            for (int i = 0; i < L; i++) {
                const int c = c0 + i * TPR + q;
                a[k][i] = (r < nr && c < kb) ? R[r * LDR + c] : T(0);
            }
        }
        // The column loop is rolled over jl / TPR, the body unrolled over the TPR owners.
        for (int jo = 0; jo < L && !stop; jo++) {
#pragma unroll
            for (int qj = 0; qj < TPR; qj++) {
                const int jl = jo * TPR + qj, j = c0 + jl, slot = j & 1;
                if (jl >= w || stop) break;
                // 1. local candidate
                unsigned long long bk = 0ull;
                int bi = INT_MAX;
                if (q == qj)
#pragma unroll
                    for (int k = 0; k < RPT; k++) {
                        const int r = grp + k * G;
                        if (r < nr && r0 + r >= j) {
                            const unsigned long long key = amax_key(a[k][0]);
                            if (key > bk) {
                                bk = key;
                                bi = r0 + r;
                            }
                        }
                    }
                warp_amax_key<T>(bk, bi);
#pragma unroll
                for (int k = 0; k < RPT; k++) {
                    const int gr = r0 + grp + k * G;
                    if (gr == bi && bk != 0ull) stv<L>(&S.cand[slot][warp][q * L], a[k]);
                    if (gr == j && j < r1) stv<L>(&S.candj[slot][q * L], a[k]);
                }
                if (lane == 0) {
                    S.s_k[slot][warp] = bk;
                    S.s_i[slot][warp] = bi;
                }
                __syncthreads();
                if (*(volatile int *)&S.fail[slot ^ 1]) {
                    stop = true;
                    break;
                }
                bk = lane < 8 ? S.s_k[slot][lane] : 0ull;
                bi = lane < 8 ? S.s_i[slot][lane] : INT_MAX;
                const unsigned long long mk = bk;
                const int mi = bi;
                warp_amax_key<T>(bk, bi);
                const int bw = bk != 0ull ? __ffs(__ballot_sync(0xffffffffu, mk == bk && mi == bi)) - 1 : 0;
                // 2. push
                const uint32_t bar = bar_to + 8 * slot;
                if (warp == 0) {
                    if (lane == 0) cl_mbar_expect(&S.full[slot], bytes);
                    // the candidate's entry in column j: owner qj, rotated index 0
                    const T inv = bk != 0ull ? T(1) / S.cand[slot][bw][qj * L] : T(0);
                    if (pusher) {
                        const uint32_t d = tab_to + slot * (unsigned)sizeof(S.rec[0]);
                        const unsigned row = bk != 0ull ? (unsigned)bi : (unsigned)INT_MAX;
                        if (sizeof(T) == 4) {
                            st_async16(d, make_uint4((unsigned)bk, __float_as_uint((float)inv), row, 0u), bar);
                        } else {
                            st_async16(d, make_uint4((unsigned)bk, (unsigned)(bk >> 32), row, 0u), bar);
                            const unsigned long long ib = (unsigned long long)__double_as_longlong((double)inv);
                            st_async16(d + 16, make_uint4((unsigned)ib, (unsigned)(ib >> 32), 0u, 0u), bar);
                        }
                    }
                } else if (pusher) {
                    st_async16(tab_to + slot * (unsigned)sizeof(S.tab[0]),
                               reinterpret_cast<const uint4 *>(S.cand[slot][bw])[pch], bar);
                    if (j >= r0 && j < r1)
                        st_async16(rowj_to + slot * (unsigned)sizeof(S.rowj[0]),
                                   reinterpret_cast<const uint4 *>(S.candj[slot])[pch], bar);
                }
                // 3. the winner, the same in every warp of every CTA
                if (!cl_mbar_wait(&S.full[slot], (j >> 1) & 1, wait_ns)) S.fail[slot] = 1;
                unsigned long long wk = 0ull;
                int wi = INT_MAX;
                if (lane < C) {
                    const uint4 v = S.rec[slot][lane][0];
                    wk = sizeof(T) == 4 ? (unsigned long long)v.x : ((unsigned long long)v.y << 32) | v.x;
                    wi = (int)v.z;
                }
                const unsigned long long rk = wk;
                const int ri = wi;
                warp_amax_key<T>(wk, wi);
                int wg = -1;
                if (wk != 0ull) {
                    wg = __ffs(__ballot_sync(0xffffffffu, rk == wk && ri == wi)) - 1;
                    wi = min(max(wi, j), mrows - 1);  // in range even after a wait that ran out
                    if (wk < ktiny) {                 // the same decision in every CTA
                        if (g == 0 && tid == 0) atomicCAS(err, 0, RL_ERR_DIV_BY_ZERO);
                        S.fail[slot] = 2;
                    }
                } else {  // no finite candidate (NaN column): keep the diagonal
                    wi = j;
                }
                const T *oldj = S.rowj[slot];
                const T *prow = wg >= 0 ? S.tab[slot][wg] : oldj;
                T inv_p;
                if (wg < 0) {
                    inv_p = T(1) / oldj[qj * L];
                } else if (sizeof(T) == 4) {
                    inv_p = (T)__uint_as_float(S.rec[slot][wg][0].y);
                } else {
                    const uint4 v = S.rec[slot][wg][RECW - 1];
                    inv_p = (T)__longlong_as_double((long long)(((unsigned long long)v.y << 32) | v.x));
                }
                // 4. swap and update
                T pr[L];
                ldv<L>(prow + q * L, pr);
#pragma unroll
                for (int k = 0; k < RPT; k++) {
                    const int r = grp + k * G, gr = r0 + r;
                    const bool live = r < nr && gr > j;
                    if (wi != j && r < nr && (gr == j || gr == wi)) ldv<L>((gr == j ? prow : oldj) + q * L, a[k]);
                    T l = a[k][0] * inv_p;  // the thread that owns column j
                    if (TPR > 1) l = __shfl_sync(0xffffffffu, l, qj, TPR);
                    if (qj < TPR - 1) {
                        if (live) {
                            if (q == qj)
                                a[k][0] = l;
                            else if (q > qj)
                                a[k][0] = fma(-l, pr[0], a[k][0]);
#pragma unroll
                            for (int i = 1; i < L; i++)
                                if (jo + i < L) a[k][i] = fma(-l, pr[i], a[k][i]);
                        }
                    } else {  // the last owner: update and rotate at once
                        T first = a[k][0];
                        if (live) {
                            if (q == qj) first = l;
#pragma unroll
                            for (int i = 1; i < L; i++) a[k][i - 1] = jo + i < L ? fma(-l, pr[i], a[k][i]) : a[k][i];
                        } else {
#pragma unroll
                            for (int i = 1; i < L; i++) a[k][i - 1] = a[k][i];
                        }
                        a[k][L - 1] = first;
                    }
                }
                if (warp == 7) {  // for the block's end: the pivot and row jl of L11
                    if (lane == 0) {
                        S.piv[jl] = wi;
                        if (g == 0) ipiv[j] = k0 + wi;
                    }
                    if (lane < SW) S.L11t[lane][jl] = prow[(lane & (TPR - 1)) * L + ((lane / TPR - jo) & (L - 1))];
                }
            }
            if (jo * TPR + TPR > w && !stop) {  // a short last block skipped the rotating step
#pragma unroll
                for (int k = 0; k < RPT; k++) {
                    const T first = a[k][0];
#pragma unroll
                    for (int i = 1; i < L; i++) a[k][i - 1] = a[k][i];
                    a[k][L - 1] = first;
                }
            }
        }
        if (stop) break;
        // registers back to the staged rows (after L rotations the columns are in order)
#pragma unroll
        for (int k = 0; k < RPT; k++) {
            const int r = grp + k * G;
#pragma unroll
            for (int i = 0; i < L; i++) {
                const int c = c0 + i * TPR + q;
                if (r < nr && c < kb) R[r * LDR + c] = a[k][i];
            }
        }
        if (kb <= SW) break;
        // The swaps in the panel's other columns. Lane l < 16 of warp 0 takes position c0 + l,
        // lane 16 + t the outside position first swapped in at column t, and follows the
        // swaps backwards to the row that ends there.
        const int nright = kb - c0 - w, nother = c0 + nright;
        cluster_wait();  // every CTA's last update of these columns is visible
        arrived = false;
        __syncthreads();
        if (*(volatile int *)&S.fail[(c0 + w - 1) & 1]) break;
        if (warp == 0) {
            const int t0 = lane & 15;
            int pos = lane < 16 ? c0 + lane : (t0 < w ? S.piv[t0] : -1);
            if (lane >= 16 && pos < c0 + SW) pos = -1;
            for (int t = 0; t < t0; t++)
                if (lane >= 16 && S.piv[t] == pos) pos = -1;
            int at = pos;
            for (int t = w - 1; t >= 0; t--) {
                const int x = S.piv[t], y = c0 + t;
                at = at == x ? y : (at == y ? x : at);
            }
            const int sg = max(at, 0) / rows_per;
            S.dst[lane] = pos >= 0 && at != pos && pos >= r0 && pos < r1 ? pos - r0 : -1;
            S.src[lane] = cluster_addr(smem_addr(R + (max(at, 0) - sg * rows_per) * LDR), min(sg, C - 1));
        }
        __syncthreads();
        constexpr int MV = 32 * (NB - SW) / 256, UV = SW * (NB - SW) / 256;
        T mv[MV], uv[UV];
#pragma unroll
        for (int i = 0; i < MV; i++) {
            const int e = tid + i * 256, m = e / (NB - SW), cc = e % (NB - SW), c = cc < c0 ? cc : cc + w;
            if (cc < nother && S.dst[m] >= 0) mv[i] = ld_cluster(S.src[m] + c * (unsigned)sizeof(T), T(0));
        }
        if (nright > 0)
#pragma unroll
            for (int i = 0; i < UV; i++) {
                const int e = tid + i * 256, m = e / (NB - SW), cc = e % (NB - SW);
                if (cc < nright) uv[i] = ld_cluster(S.src[m] + (c0 + SW + cc) * (unsigned)sizeof(T), T(0));
            }
        if (nright > 0)
#pragma unroll
            for (int i = 0; i < UV; i++) {
                const int e = tid + i * 256, m = e / (NB - SW), cc = e % (NB - SW);
                if (cc < nright) S.U[cc][m] = uv[i];
            }
        cluster.sync();  // every read of the old rows is done
        if (*(volatile int *)&S.dead) break;
#pragma unroll
        for (int i = 0; i < MV; i++) {
            const int e = tid + i * 256, m = e / (NB - SW), cc = e % (NB - SW), c = cc < c0 ? cc : cc + w;
            if (cc < nother && S.dst[m] >= 0) R[S.dst[m] * LDR + c] = mv[i];
        }
        if (nright <= 0) break;
        // w = 16 here: U12 = L11^-1 A12, a thread per column, rows in order
        if (tid < nright) {
            T x[SW];
            ldv<SW>(S.U[tid], x);
#pragma unroll
            for (int k = 0; k < SW - 1; k++) {
                T l[SW];
                ldv<SW>(S.L11t[k], l);
#pragma unroll
                for (int i = k + 1; i < SW; i++) x[i] = fma(-l[i], x[k], x[i]);
            }
            stv<SW>(S.U[tid], x);
        }
        __syncthreads();
        // the rows below the pivots: A22 -= L21 U12; the pivot rows: U12 itself
        for (int k = 0; k < RPT; k++) {
            const int r = grp + k * G, gr = r0 + r;
            if (r >= nr || gr < c0) continue;
            T *row = R + (size_t)r * LDR + c0;
            if (gr < c0 + SW) {
                for (int c = q; c < nright; c += TPR) row[SW + c] = S.U[c][gr - c0];
                continue;
            }
            T l[SW];
#pragma unroll
            for (int i = 0; i < SW; i++) l[i] = row[i];
#pragma unroll 2
            for (int c = q; c < nright; c += TPR) {
                T v = row[SW + c], u[SW];
                ldv<SW>(S.U[c], u);
#pragma unroll
                for (int i = 0; i < SW; i++) v = fma(-l[i], u[i], v);
                row[SW + c] = v;
            }
        }
        __syncthreads();
        cluster_arrive();
        arrived = true;
    }
    __syncthreads();
    if (S.fail[0] == 1 || S.fail[1] == 1) {
        if (tid == 0) atomicCAS(err, 0, RL_ERR_TIMEOUT);
        if (tid < C) *cluster.map_shared_rank(&S.dead, tid) = 1;
    }
    if (arrived) cluster_wait();
    __syncthreads();
    for (int idx = tid; idx < nr * kb; idx += 256) {
        const int r = idx / kb, c = idx - r * kb;
        P[(long long)(r0 + r) * lda + c] = R[r * LDR + c];
    }
    cluster.sync();  // no CTA leaves while another may still use its shared memory
    if (*(volatile int *)&S.dead) cl_settle();
}

// The same panel with look-ahead across columns. After column j's winner is known a CTA
// updates only column j + 1 of its rows, finds its candidate for column j + 1, completes
// that candidate row (and row j + 1, if it holds it), pushes them and ARRIVES at the
// cluster barrier; the rest of column j's elimination (columns j + 2 .. kb - 1 of its
// other rows) runs while the barrier completes, and the CTA WAITS only before reading
// column j + 1's records. Every element gets the same fma(-l, u, a) as in
// lu_panel_cluster_kernel, so the factors and pivots are identical. The tables have three
// slots: a CTA may push column j + 1 while another still eliminates with column j - 1's
// pivot row.
template <class T>
static __global__ void __launch_bounds__(256) lu_panel_cluster_la_kernel(T *P, long long lda, int mrows, int kb, int k0,
                                                                  int rows_per, int tpr, int *ipiv, int *err, T tiny) {
    namespace cg = cooperative_groups;
    constexpr int NB = PanelNB<T>::value;
    constexpr int LDR = NB + 1;
    constexpr int CMAX = 16, NS = 3;
    constexpr int VW = 16 / (int)sizeof(T);
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T *tab = reinterpret_cast<T *>(smem_raw);  // NS x CMAX x NB: every CTA's candidate row
    T *rowj = tab + NS * CMAX * NB;            // NS x NB: row j (pushed by the CTA holding it)
    T *R = rowj + NS * NB;                     // rows_per x LDR
    __shared__ unsigned long long s_k[8], rec_k[NS * CMAX];
    __shared__ int s_i[8], rec_i[NS * CMAX];
    __shared__ T rec_inv[NS * CMAX];
    cg::cluster_group cluster = cg::this_cluster();
    const int C = (int)cluster.num_blocks(), g = (int)cluster.block_rank();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int r0 = g * rows_per, r1 = min(mrows, r0 + rows_per), nr = max(0, r1 - r0);
    const int q = tid & (tpr - 1), grp = tid / tpr, G = (int)blockDim.x / tpr;
    const int rpt = (rows_per + G - 1) / G;
    const unsigned long long ktiny = amax_key(tiny);
    const int nch = (kb + VW - 1) / VW;
    if (g == 0)
        for (int j = tid; j < kb; j += blockDim.x) ipiv[j] = k0 + j;
    for (int idx = tid; idx < nr * kb; idx += blockDim.x) {
        const int r = idx / kb, c = idx - r * kb;
        R[r * LDR + c] = P[(long long)(r0 + r) * lda + c];
    }
    __syncthreads();
    // candidate of this CTA for column c (rows >= c; thread group q == c mod tpr scans)
    auto candidate = [&](int c, unsigned long long &bk, int &bi) {
        bk = 0ull;
        bi = INT_MAX;
        if (q == (c & (tpr - 1)))
            for (int k = 0; k < rpt; k++) {
                const int r = grp + k * G;
                if (r < nr && r0 + r >= c) {
                    const unsigned long long key = amax_key(R[r * LDR + c]);
                    if (key > bk) {
                        bk = key;
                        bi = r0 + r;
                    }
                }
            }
        warp_amax_key<T>(bk, bi);
        if (lane == 0) {
            s_k[warp] = bk;
            s_i[warp] = bi;
        }
        __syncthreads();
        bk = s_k[0];
        bi = s_i[0];
        for (int w = 1; w < (int)(blockDim.x >> 5); w++) {
            const unsigned long long k2 = s_k[w];
            const int i2 = s_i[w];
            if (k2 > bk || (k2 == bk && i2 < bi)) {
                bk = k2;
                bi = i2;
            }
        }
    };
    // push the candidate row bi (complete) and row c (if held) into every CTA's slot for
    // column c, with the record; then arrive
    auto push = [&](int c, unsigned long long bk, int bi) {
        const int slot = c % NS;
        if (bk != 0ull)
            for (int idx = tid; idx < C * nch; idx += blockDim.x) {
                const int dst = idx / nch, ch = idx - dst * nch;
                const T *src = R + (size_t)(bi - r0) * LDR + ch * VW;
                uint4 v;
                T *vt = reinterpret_cast<T *>(&v);
#pragma unroll
                for (int e = 0; e < VW; e++) vt[e] = src[e];
                *reinterpret_cast<uint4 *>(cluster.map_shared_rank(tab + (slot * CMAX + g) * NB + ch * VW, dst)) = v;
            }
        if (c >= r0 && c < r1)
            for (int idx = tid; idx < C * nch; idx += blockDim.x) {
                const int dst = idx / nch, ch = idx - dst * nch;
                const T *src = R + (size_t)(c - r0) * LDR + ch * VW;
                uint4 v;
                T *vt = reinterpret_cast<T *>(&v);
#pragma unroll
                for (int e = 0; e < VW; e++) vt[e] = src[e];
                *reinterpret_cast<uint4 *>(cluster.map_shared_rank(rowj + slot * NB + ch * VW, dst)) = v;
            }
        if (warp == 0) {
            const T inv = bk != 0ull ? T(1) / R[(bi - r0) * LDR + c] : T(0);
            if (lane < C) {
                const int e = slot * CMAX + g;
                *cluster.map_shared_rank(rec_k + e, lane) = bk;
                *cluster.map_shared_rank(rec_i + e, lane) = bk != 0ull ? bi : INT_MAX;
                *cluster.map_shared_rank(rec_inv + e, lane) = inv;
            }
        }
        cluster_arrive();
    };
    {
        unsigned long long bk;
        int bi;
        candidate(0, bk, bi);
        push(0, bk, bi);
    }
    int skip0 = -1, skip1 = -1;  // rows completed before their push (not eliminated again)
    for (int j = 0; j < kb; j++) {
        const int slot = j % NS, qj = j & (tpr - 1);
        cluster_wait();  // column j's records and rows are in every CTA's tables
        unsigned long long wk = lane < C ? rec_k[slot * CMAX + lane] : 0ull;
        int wi = lane < C ? rec_i[slot * CMAX + lane] : INT_MAX;
        warp_amax_key<T>(wk, wi);
        int wg = -1;
        if (wk != 0ull) {
            if (wk < ktiny) {
                if (g == 0 && tid == 0) atomicCAS(err, 0, RL_ERR_DIV_BY_ZERO);
                break;
            }
            wg = wi / rows_per;
        } else {
            wi = j;
        }
        const T *oldj = rowj + slot * NB;
        const T *prow = wg >= 0 ? tab + (slot * CMAX + wg) * NB : oldj;
        if (g == 0 && tid == 0) ipiv[j] = k0 + wi;
        const T inv_p = wg >= 0 ? rec_inv[slot * CMAX + wg] : T(1) / oldj[j];
        if (wi != j && tid < kb) {
            if (j >= r0 && j < r1) R[(j - r0) * LDR + tid] = prow[tid];
            if (wi >= r0 && wi < r1 && tid < j) R[(wi - r0) * LDR + tid] = oldj[tid];
        }
        // (a) multipliers and column j + 1 of every row below j
        const int q1 = (j + 1) & (tpr - 1);
        for (int k = 0; k < rpt; k++) {
            const int r = grp + k * G, gr = r0 + r;
            const bool valid = r < nr && gr > j;
            T *row = R + (size_t)(valid ? r : 0) * LDR;
            const T *src = gr == wi ? oldj : row;
            T l = T(0);
            if (valid && q == qj) l = src[j] * inv_p;
            if (tpr > 1) l = __shfl_sync(0xffffffffu, l, qj, tpr);
            if (valid) {
                if (q == qj) row[j] = l;
                if (j + 1 < kb && q == q1) row[j + 1] = fma(-l, prow[j + 1], src[j + 1]);
            }
        }
        if (j + 1 >= kb) break;
        // (b) the candidate for column j + 1 (the barrier inside also orders (a))
        unsigned long long bk;
        int bi;
        candidate(j + 1, bk, bi);
        // (c) complete the rows pushed for column j + 1: the candidate and row j + 1
        skip0 = bk != 0ull ? bi : -1;
        skip1 = (j + 1 >= r0 && j + 1 < r1) ? j + 1 : -1;
        for (int t = 0; t < 2; t++) {
            const int gr = t == 0 ? skip0 : skip1;
            if (gr < 0 || (t == 1 && gr == skip0)) continue;
            T *row = R + (size_t)(gr - r0) * LDR;
            const T *src = gr == wi ? oldj : row;
            const T l = row[j];
            for (int c = j + 2 + tid; c < kb; c += blockDim.x) row[c] = fma(-l, prow[c], src[c]);
        }
        __syncthreads();
        push(j + 1, bk, bi);
        // (d) the rest of column j's elimination, while the barrier completes
        const int cfirst = j + 2 + ((q - j - 2) & (tpr - 1));
        for (int k = 0; k < rpt; k++) {
            const int r = grp + k * G, gr = r0 + r;
            if (r >= nr || gr <= j || gr == skip0 || gr == skip1) continue;
            T *row = R + (size_t)r * LDR;
            const T *src = gr == wi ? oldj : row;
            const T l = row[j];
#pragma unroll 4
            for (int c = cfirst; c < kb; c += tpr) row[c] = fma(-l, prow[c], src[c]);
        }
    }
    __syncthreads();
    for (int idx = tid; idx < nr * kb; idx += blockDim.x) {
        const int r = idx / kb, c = idx - r * kb;
        P[(long long)(r0 + r) * lda + c] = R[r * LDR + c];
    }
    cluster.sync();  // no CTA leaves while another may still read its shared memory
}

// ------------------------------------------------------------ Householder panel --
// Unblocked Householder QR of the panel rows [0, mrows) x cols [0, kb) (P points at
// A[k0][k0]), reflector by reflector exactly as HouseholderReflection::compute and
// buffered_left_multiply_into (householder.rs:32-130) but with the reductions split
// over CTAs: sigma = dot(x[1..], x[1..]) and u = A^T v are summed from per-CTA partials
// in CTA order after a grid barrier. Two barriers per column. tau receives kb values.
// part: 2 slots x G x (1 + NB) partial sums; x0buf: 2 slots.
template <class T>
static __global__ void __launch_bounds__(256) qr_panel_kernel(T *P, long long lda, int mrows, int kb, int rows_per, T *tau,
                                                       T *part, T *x0buf, PanelSync *sync,
                                                       unsigned long long wait_ns) {
    constexpr int NB = PanelNB<T>::value;
    constexpr int LDR = NB + 1;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T *R = reinterpret_cast<T *>(smem_raw);  // rows_per x LDR
    T *u = R + (size_t)rows_per * LDR;       // NB
    __shared__ T s_red[8][NB + 1];
    const int G = gridDim.x, g = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nw = blockDim.x >> 5;
    const int r0 = g * rows_per, r1 = min(mrows, r0 + rows_per), nr = max(0, r1 - r0);
    const int PS = 1 + NB;
    for (int idx = tid; idx < nr * kb; idx += blockDim.x) {
        const int r = idx / kb, c = idx - r * kb;
        R[r * LDR + c] = P[(long long)(r0 + r) * lda + c];
    }
    __syncthreads();
    unsigned phase = 0;
    for (int j = 0; j < kb; j++) {
        const int slot = j & 1;
        // (1) sigma partial over rows > j, in row order per thread then tree order.
        T s = T(0);
        for (int r = max(j + 1 - r0, 0) + tid; r < nr; r += blockDim.x) {
            const T v = R[r * LDR + j];
            s = fma(v, v, s);
        }
        s = warp_sum(s);
        if (lane == 0) s_red[warp][0] = s;
        __syncthreads();
        if (tid == 0) {
            T t = T(0);
            for (int w = 0; w < nw; w++) t += s_red[w][0];
            part[((size_t)slot * G + g) * PS] = t;
            if (j >= r0 && j < r1) x0buf[slot] = R[(j - r0) * LDR + j];
        }
        if (!grid_barrier(&sync->ctr, (unsigned)(G * (++phase)), &sync->err, wait_ns)) return;
        // sigma = sum of the CTAs' partials, a fixed tree over q (thread q, then warps)
        T sigma = T(0);
        for (int q = tid; q < G; q += blockDim.x) sigma += ((volatile T *)part)[((size_t)slot * G + q) * PS];
        sigma = warp_sum(sigma);
        __syncthreads();  // s_red from step (1) is read no more
        if (lane == 0) s_red[warp][0] = sigma;
        __syncthreads();
        sigma = T(0);
        for (int w = 0; w < nw; w++) sigma += s_red[w][0];
        const T x0 = ((volatile T *)x0buf)[slot];
        if (sigma == T(0)) {  // already a multiple of e1: tau = 0, nothing changes
            if (g == 0 && tid == 0) tau[j] = T(0);
            if (!grid_barrier(&sync->ctr, (unsigned)(G * (++phase)), &sync->err, wait_ns)) return;
            continue;
        }
        const T x_norm = sqrt(x0 * x0 + sigma);
        const T v0 = x0 > T(0) ? x0 + x_norm : x0 - x_norm;
        const T two = T(2);
        const T t = two * v0 * v0 / (v0 * v0 + sigma);
        if (g == 0 && tid == 0) tau[j] = t;
        // (2) u_c = sum_r v_r a[r][c] for c >= j over owned rows r >= j, with
        // v_r = x_r / v0 (v_j = 1) formed on the fly so that column j still holds x.
        for (int c = j + warp; c < kb; c += nw) {
            T acc = T(0);
            for (int r = max(j - r0, 0) + lane; r < nr; r += 32) {
                const T vr = (r0 + r == j) ? T(1) : R[r * LDR + j] / v0;
                acc = fma(vr, R[r * LDR + c], acc);
            }
            acc = warp_sum(acc);
            if (lane == 0) part[((size_t)slot * G + g) * PS + 1 + c] = acc;
        }
        if (!grid_barrier(&sync->ctr, (unsigned)(G * (++phase)), &sync->err, wait_ns)) return;
        // u_c = sum over CTAs of the partials: warp per column, lanes over CTAs
        for (int c = j + warp; c < kb; c += nw) {
            T a = T(0);
            for (int q = lane; q < G; q += 32) a += ((volatile T *)part)[((size_t)slot * G + q) * PS + 1 + c];
            a = warp_sum(a);
            if (lane == 0) u[c] = a;
        }
        __syncthreads();
        // (3) a[r][c] += (-tau v_r) u_c for c > j (ger, internal_utils.rs:67-83); the
        // diagonal becomes x0 - tau u_j and v[1..] is stored below it (store_in_col).
        for (int r = max(j - r0, 0) + tid; r < nr; r += blockDim.x) {
            T *row = R + r * LDR;
            const bool diag = (r0 + r == j);
            const T vr = diag ? T(1) : row[j] / v0;
            const T sc = -t * vr;
            for (int c = j + 1; c < kb; c++) row[c] = fma(sc, u[c], row[c]);
            row[j] = diag ? x0 - t * u[j] : vr;
        }
        __syncthreads();
    }
    for (int idx = tid; idx < nr * kb; idx += blockDim.x) {
        const int r = idx / kb, c = idx - r * kb;
        P[(long long)(r0 + r) * lda + c] = R[r * LDR + c];
    }
}

// Householder panel on one thread-block cluster (up to 16 CTAs), one exchange per column. With
// x the column below row j, the sums s_c = sum_r x_r a_rc for c >= j give everything at once:
// sigma = s_j and, as v = (1, x / v0), u_c = a_jc + s_c / v0. Per column:
//   1. the warps take up to 8 columns each, a lane the rows lane + 32 i, and reduce them
//      together (warp_reduce_scatter: 9 additions for 8 columns; in FP64 an addition is 64
//      cycles of a scheduler's unit, like a multiply-add);
//   2. every partial sum, and row j from the CTA that holds it, goes to all CTAs by st.async,
//      counted on their mbarriers (no cluster barrier, no CTA barrier);
//   3. each CTA adds the partials in rank order, one warp forms tau and 1 / v0, and w_c =
//      tau u_c is shared;
//   4. a_rc -= v_r w_c, `tpr` threads per row; v takes the column's place.
// Tables are double-buffered by column parity: a CTA pushes column j + 2 only after it has all
// partials of column j + 1, which the others push after their last read of column j's tables.
// Two exchanges behind cluster barriers (sigma, then u) and a butterfly per column sum took
// 302 us per 64-column panel of a 2999 x 1501 FP32 QR, this 163; the whole 1201 x 499 FP64 QR
// with its thin Q (8 panels) went from 11.05 to 9.0 ms. Bound by a column's chain: two CTA
// barriers, the exchange, and tau's square root and divisions in one thread.
template <class T>
struct QrTables {
    T tab[2][16][64];  // partial sums of column c from CTA g
    T rowj[2][64];
    T w[64];
    T tau, v0, inv_v0, diag;
    int zero;
    uint64_t full[2];
    int fail[2];  // a wait ran out, by column parity
};

__device__ __forceinline__ void st_async(uint32_t dst, float v, uint32_t bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(dst), "r"(__float_as_uint(v)),
                 "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void st_async(uint32_t dst, double v, uint32_t bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(dst),
                 "l"(__double_as_longlong(v)), "r"(bar)
                 : "memory");
}

// Sums of N columns c = first, first + 8, ... of a warp, pushed to every CTA's tables.
template <class T, int N>
__device__ __forceinline__ void qr_dots(const T *R, int LDR, int rbeg, int nr, int j, int first, int kb, const T *rowj, int C, int g,
                                        uint32_t tab_a, uint32_t row_a, uint32_t bar_a) {
    const int lane = threadIdx.x & 31;
    T acc[N];
#pragma unroll
    for (int k = 0; k < N; k++) acc[k] = T(0);
    for (int r = rbeg + lane; r < nr; r += 32) {
        const T *row = R + (size_t)r * LDR;
        const T x = row[j];
#pragma unroll
        for (int k = 0; k < N; k++)
            if (first + 8 * k < kb) acc[k] = fma(x, row[first + 8 * k], acc[k]);
    }
    int k;
    const T sum = warp_reduce_scatter<N>(acc, lane, k);
    constexpr int PER = 32 / N;  // lanes that hold a column's sum
    const int c = first + 8 * k;
    if (c >= kb) return;
    for (int to = lane % PER; to < C; to += PER) {
        const uint32_t bar = cluster_addr(bar_a, to);
        st_async(cluster_addr(tab_a + (unsigned)((g * 64 + c) * sizeof(T)), to), sum, bar);
        if (rowj) st_async(cluster_addr(row_a + (unsigned)(c * sizeof(T)), to), rowj[c], bar);
    }
}

template <class T>
static __global__ void __launch_bounds__(256) qr_panel_cluster_kernel(T *P, long long lda, int mrows, int kb,
                                                              int rows_per, int tpr, T *tau, int *err,
                                                              unsigned long long wait_ns) {
    namespace cg = cooperative_groups;
    constexpr int NB = PanelNB<T>::value, LDR = NB + 1;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T *R = reinterpret_cast<T *>(smem_raw);  // rows_per x LDR
    __shared__ __align__(16) QrTables<T> S;
    cg::cluster_group cluster = cg::this_cluster();
    const int C = (int)cluster.num_blocks(), g = (int)cluster.block_rank();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int r0 = g * rows_per, r1 = min(mrows, r0 + rows_per), nr = max(0, r1 - r0);
    const int q = tid & (tpr - 1), grp = tid / tpr, G = 256 / tpr, rpt = (rows_per + G - 1) / G;
    for (int idx = tid; idx < nr * kb; idx += 256) {
        const int r = idx / kb, c = idx - r * kb;
        R[r * LDR + c] = P[(long long)(r0 + r) * lda + c];
    }
    if (tid == 0) {
        S.fail[0] = S.fail[1] = 0;
        cl_mbar_init(&S.full[0], 1);
        cl_mbar_init(&S.full[1], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    cluster.sync();
    bool bad = false;
    for (int j = 0; j < kb; j++) {
        const int slot = j & 1, ncol = (kb - j + 7) / 8, rbeg = max(j + 1 - r0, 0);
        const bool hold = j >= r0 && j < r1;
        if (tid == 0) cl_mbar_expect(&S.full[slot], (unsigned)((kb - j) * (C + 1) * sizeof(T)));
        // 1, 2. partial sums of columns j + warp, j + warp + 8, ...
        {
            const T *rj = hold ? R + (size_t)(j - r0) * LDR : nullptr;
            const uint32_t ta = smem_addr(&S.tab[slot][0][0]), ra = smem_addr(&S.rowj[slot][0]), ba = smem_addr(&S.full[slot]);
            const int first = j + warp;
            if (ncol > 4)
                qr_dots<T, 8>(R, LDR, rbeg, nr, j, first, kb, rj, C, g, ta, ra, ba);
            else if (ncol > 2)
                qr_dots<T, 4>(R, LDR, rbeg, nr, j, first, kb, rj, C, g, ta, ra, ba);
            else
                qr_dots<T, 2>(R, LDR, rbeg, nr, j, first, kb, rj, C, g, ta, ra, ba);
        }
        if (!cl_mbar_wait(&S.full[slot], (j >> 1) & 1, wait_ns)) S.fail[slot] = 1;
        // 3. warp 0: sigma, tau, 1 / v0
        const int c = j + tid;
        T sc = T(0);
        if (c < kb)
            for (int k = 0; k < C; k++) sc += S.tab[slot][k][c];  // CTAs in rank order
        if (tid == 0) {
            const T sigma = sc, x0 = S.rowj[slot][j];
            S.zero = sigma == T(0);  // already a multiple of e1: tau = 0, nothing changes
            T t = T(0), inv = T(0), d = x0, v0 = T(1);
            if (!S.zero) {
                const T x_norm = sqrt(x0 * x0 + sigma);
                v0 = x0 > T(0) ? x0 + x_norm : x0 - x_norm;
                t = T(2) * v0 * v0 / (v0 * v0 + sigma);
                inv = T(1) / v0;
                d = x0 - t * (x0 + sigma * inv);
            }
            S.tau = t;
            S.v0 = v0;
            S.inv_v0 = inv;
            S.diag = d;
            if (g == 0) tau[j] = t;
        }
        __syncthreads();
        if (*(volatile int *)&S.fail[slot]) {
            bad = true;
            break;
        }
        if (!S.zero) {
            const T inv = S.inv_v0;
            if (c < kb) S.w[c] = S.tau * (S.rowj[slot][c] + sc * inv);
            __syncthreads();
            // 4. a_rc -= v_r w_c for c > j (v_j = 1); the diagonal, and v below it
            for (int k = 0; k < rpt; k++) {  // the same count in every thread
                const int r = grp + k * G;
                const bool mine = r < nr && r0 + r >= j, diag = r0 + r == j;
                T *row = R + (size_t)(mine ? r : 0) * LDR;
                const T v = mine ? (diag ? T(1) : quotient(row[j], S.v0, inv)) : T(0);
                __syncwarp();
                if (mine) {
                    const int first = j + 1 + ((q - j - 1) & (tpr - 1));
#pragma unroll 4
                    for (int cc = first; cc < kb; cc += tpr) row[cc] = fma(-v, S.w[cc], row[cc]);
                    if (q == 0) row[j] = diag ? S.diag : v;
                }
            }
        }
        __syncthreads();
    }
    if (bad) {
        if (tid == 0) atomicCAS(err, 0, RL_ERR_TIMEOUT);
    }
    for (int idx = tid; idx < nr * kb; idx += 256) {
        const int r = idx / kb, c = idx - r * kb;
        P[(long long)(r0 + r) * lda + c] = R[r * LDR + c];
    }
    cluster.sync();  // no CTA leaves while another may still store into its shared memory
    if (*(volatile int *)&S.fail[0] | *(volatile int *)&S.fail[1]) cl_settle();
}

// ------------------------------------------------------------------- row swaps --
// Applies ipiv[j0..j1) (global rows; step j swaps rows j and ipiv[j]) to the columns
// [0, c_skip0) and [c_skip1, ncols) of A, 64 columns per CTA, in blocks of 64 pivots:
// the rows a block touches (its own 64 rows and the pivot rows outside them, at most
// 128) are staged in shared memory with all loads in flight at once, the block's swaps
// run there in order (thread per column), and the rows are written back. A swap chain
// applied straight to global memory would wait one memory round trip per pivot.
constexpr int kSwapCols = 64, kSwapBlock = 64;
template <class T>
static __global__ void __launch_bounds__(256) laswp_kernel(T *A, long long lda, int ncols, int c_skip0, int c_skip1,
                                                    const int *ipiv, int j0, int j1) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T *S = reinterpret_cast<T *>(smem_raw);  // 2 * kSwapBlock slots x kSwapCols columns
    __shared__ int s_piv[kSwapBlock], s_slot[kSwapBlock], s_row[2 * kSwapBlock];
    const int tid = threadIdx.x, t = tid & (kSwapCols - 1), quarter = tid / kSwapCols;
    const int nother = ncols - (c_skip1 - c_skip0);
    const int c = blockIdx.x * kSwapCols + t;
    const bool act = c < nother;
    const int gc = c < c_skip0 ? c : c + (c_skip1 - c_skip0);
    for (int b = j0; b < j1; b += kSwapBlock) {
        const int kb = min(kSwapBlock, j1 - b);
        if (tid < kb) s_piv[tid] = ipiv[b + tid];
        __syncthreads();
        // slot of each pivot row: its place in [b, b + kb), else an outside slot named
        // by the first step that swaps it in (the slot that stages it)
        if (tid < kb) {
            const int p = s_piv[tid];
            int sl;
            if (p >= b && p < b + kb) {
                sl = p - b;
            } else {
                int first = tid;
                for (int u = 0; u < tid; u++)
                    if (s_piv[u] == p) {
                        first = u;
                        break;
                    }
                sl = kSwapBlock + first;
            }
            s_slot[tid] = sl;
            s_row[tid] = b + tid;
            s_row[kSwapBlock + tid] = sl == kSwapBlock + tid ? p : -1;
        } else if (tid < kSwapBlock) {
            s_row[tid] = -1;
            s_row[kSwapBlock + tid] = -1;
        }
        __syncthreads();
        if (act) {
            T v[2 * kSwapBlock / 4];
#pragma unroll
            for (int i = 0; i < 2 * kSwapBlock / 4; i++) {
                const int r = s_row[quarter + 4 * i];
                v[i] = r >= 0 ? A[(long long)r * lda + gc] : T(0);
            }
#pragma unroll
            for (int i = 0; i < 2 * kSwapBlock / 4; i++) S[(quarter + 4 * i) * kSwapCols + t] = v[i];
        }
        __syncthreads();
        if (act && quarter == 0)
            for (int u = 0; u < kb; u++) {
                const int sl = s_slot[u];
                if (sl != u) {
                    const T x = S[u * kSwapCols + t];
                    S[u * kSwapCols + t] = S[sl * kSwapCols + t];
                    S[sl * kSwapCols + t] = x;
                }
            }
        __syncthreads();
        if (act)
#pragma unroll 4
            for (int i = 0; i < 2 * kSwapBlock / 4; i++) {
                const int sl = quarter + 4 * i, r = s_row[sl];
                if (r >= 0) A[(long long)r * lda + gc] = S[sl * kSwapCols + t];
            }
        __syncthreads();  // the staging area and slot map are reused by the next block
    }
}

// Launch of laswp_kernel over the columns outside [c_skip0, c_skip1).
template <class T>
static rl_status laswp(T *A, long long lda, int ncols, int c_skip0, int c_skip1, const int *ipiv, int j0, int j1,
                cudaStream_t s) {
    const int nother = ncols - (c_skip1 - c_skip0);
    if (nother <= 0 || j1 <= j0) return RL_OK;
    const size_t smem = sizeof(T) * 2 * kSwapBlock * kSwapCols;
    static const cudaError_t attr =
        cudaFuncSetAttribute(laswp_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    RL_TRY_CUDA(attr);
    RL_LAUNCH(laswp_kernel<T>, ceil_div(nother, kSwapCols), 256, smem, s, A, lda, ncols, c_skip0, c_skip1, ipiv, j0, j1);
    return RL_OK;
}

// ------------------------------------------------------------ pivots as a row map --
// rows[i] = the original row at position i after the swaps ipiv[0..n) (step j swaps rows
// j and ipiv[j] >= j), so that P b is one gather instead of a chain of swaps; stored, if
// given, receives the inverse map (the reference's stored form). One CTA:
//   1. every 64-pivot block's swaps, composed by one warp over the block's at most 128
//      slots (64 dependent shared-memory swaps; the blocks do not depend on one another),
//      written as (destination row, source row) pairs to `moves`;
//   2. the blocks applied to the map in order, 128 entries at once.
// The chain is n / 64 block steps of two barriers, not n swaps. Applying the swaps to one
// column block after block took 365 us per application at n = 3000, one thread over the
// swaps 178 us at n = 1024; with the map a re-solve at n = 3000 went from 2917 to 1455 us
// and a mixed solve at n = 4096 with 7 refinement steps from 23.85 to 19.99 ms. The map
// lives in shared memory up to kRowMapSmem rows, in `rows` itself beyond.
constexpr int kRowMapThreads = 512, kRowMapSmem = 40000;
static __global__ void __launch_bounds__(kRowMapThreads) pivots_to_rows_kernel(const int *__restrict__ ipiv, int n,
                                                                        int2 *__restrict__ moves, int *rows,
                                                                        uint64_t *stored) {
    constexpr int B = kSwapBlock, NW = kRowMapThreads / 32;
    extern __shared__ __align__(16) int map_smem[];
    __shared__ int s_piv[NW][B], s_row[NW][2 * B];
    __shared__ unsigned char s_slot[NW][B], s_at[NW][2 * B];
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int nb = (n + B - 1) / B;
    for (int blk = w; blk < nb; blk += NW) {
        const int b = blk * B, kb = min(B, n - b);
        for (int u = lane; u < 2 * B; u += 32) {
            if (u < kb) s_piv[w][u] = ipiv[b + u];
            s_row[w][u] = u < kb ? b + u : -1;
            s_at[w][u] = (unsigned char)u;
        }
        __syncwarp();
        for (int u = lane; u < kb; u += 32) {  // the slot of each pivot row (see laswp_kernel)
            const int p = s_piv[w][u];
            int sl = p - b;
            if (p >= b + kb) {
                int first = 0;
                while (s_piv[w][first] != p) first++;
                sl = B + first;
                if (first == u) s_row[w][sl] = p;
            }
            s_slot[w][u] = (unsigned char)sl;
        }
        __syncwarp();
        if (lane == 0)
            for (int u = 0; u < kb; u++) {
                const int sl = s_slot[w][u];
                const unsigned char x = s_at[w][u];
                s_at[w][u] = s_at[w][sl];
                s_at[w][sl] = x;
            }
        __syncwarp();
        for (int u = lane; u < 2 * B; u += 32) {
            const int dst = s_row[w][u];
            moves[(size_t)blk * 2 * B + u] = make_int2(dst, dst < 0 ? -1 : s_row[w][s_at[w][u]]);
        }
        __syncwarp();
    }
    int *map = n <= kRowMapSmem ? map_smem : rows;
    for (int i = tid; i < n; i += kRowMapThreads) map[i] = i;
    __syncthreads();
    for (int blk = 0; blk < nb; blk++) {
        int2 mv = make_int2(-1, -1);
        int v = 0;
        if (tid < 2 * B) {
            mv = moves[(size_t)blk * 2 * B + tid];
            if (mv.x >= 0) v = map[mv.y];
        }
        __syncthreads();
        if (mv.x >= 0) map[mv.x] = v;
        __syncthreads();
    }
    for (int i = tid; i < n; i += kRowMapThreads) {
        const int r = map[i];
        if (map != rows) rows[i] = r;
        if (stored) stored[r] = i;
    }
}

static inline rl_status pivots_to_rows(const int *ipiv, int n, int *rows, uint64_t *stored, cudaStream_t s) {
    DevBuf<int2> moves;
    RL_TRY(moves.alloc((size_t)ceil_div(n, kSwapBlock) * 2 * kSwapBlock, s));
    const size_t smem = n <= kRowMapSmem ? sizeof(int) * n : 0;
    static const cudaError_t attr = cudaFuncSetAttribute(
        pivots_to_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(sizeof(int) * kRowMapSmem));
    RL_TRY_CUDA(attr);
    RL_LAUNCH(pivots_to_rows_kernel, 1, kRowMapThreads, smem, s, ipiv, n, moves.p, rows, stored);
    return RL_OK;
}

// Y[i][:] = B[rows[i]][:] (n x nrhs; Y does not overlap B).
template <class T>
static __global__ void gather_rows_kernel(const T *__restrict__ B, long long ldb, T *__restrict__ Y, long long ldy, int n,
                                   int nrhs, const int *__restrict__ rows) {
    const long long total = (long long)n * nrhs;
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(e / nrhs), c = (int)(e - (long long)i * nrhs);
        Y[(long long)i * ldy + c] = B[(long long)rows[i] * ldb + c];
    }
}

template <class T>
rl_status gather_rows(const T *B, long long ldb, T *Y, long long ldy, int n, int nrhs, const int *rows, cudaStream_t s) {
    const long long tot = (long long)n * nrhs;
    RL_LAUNCH(gather_rows_kernel<T>, (int)std::min<long long>(8LL * num_sms(), (tot + 255) / 256), 256, 0, s, B, ldb, Y, ldy,
              n, nrhs, rows);
    return RL_OK;
}

// ------------------------------------------------------- diagonal-block solves --
// Solves op(D) X = Y in place for the bs x bs diagonal block D (bs <= 64, row stride
// ldd) and Y = bs x nrhs (row stride ldy). mode 0: D unit lower; 1: D lower; 2: D upper;
// 3: D^T with D lower (L^T). |d_ii| < tiny (modes 1-3) records RL_ERR_DIV_BY_ZERO in
// status and leaves Y unchanged. CTA per 8 columns, warp per 2 columns, 16 lanes per
// column each holding 4 of its rows in registers: step j broadcasts x_j within the
// column's lanes by a shuffle and every lane updates its rows, y_i -= d_ij x_j in
// increasing j (the order of the reference's substitution). The FP64 work of a U12
// solve is spread over every scheduler of every SM instead of a few CTAs' threads. The block is
// loaded with all 32 loads of a thread in flight: an element at a time, with a division by bs
// for its place, it was half of the kernel's time (FP32 20 -> 10.6 us a launch, FP64 33 -> 24).
constexpr int kTrsmCols = 8;
template <class T>
static __global__ void __launch_bounds__(128) trsm_diag_kernel(const T *D, long long ldd, int bs, T *Y, long long ldy,
                                                        int nrhs, int mode, int *status, T tiny) {
    __shared__ T Ds[64][65];
    __shared__ T Ys[64][kTrsmCols];
    __shared__ int s_bad;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int c0 = blockIdx.x * kTrsmCols;
    if (tid == 0) s_bad = 0;
    {  // the block and the columns, every load in flight before the first store
        T d[32], yv[64 * kTrsmCols / 128];
#pragma unroll
        for (int e = 0; e < 32; e++) {
            const int i = 2 * e + (tid >> 6), j = tid & 63;
            d[e] = (i < bs && j < bs) ? D[(long long)i * ldd + j] : T(0);
        }
#pragma unroll
        for (int e = 0; e < 64 * kTrsmCols / 128; e++) {
            const int i = (tid + 128 * e) / kTrsmCols, cc = tid % kTrsmCols;
            yv[e] = (i < bs && c0 + cc < nrhs) ? Y[(long long)i * ldy + c0 + cc] : T(0);
        }
#pragma unroll
        for (int e = 0; e < 32; e++) Ds[2 * e + (tid >> 6)][tid & 63] = d[e];
#pragma unroll
        for (int e = 0; e < 64 * kTrsmCols / 128; e++) Ys[(tid + 128 * e) / kTrsmCols][tid % kTrsmCols] = yv[e];
    }
    __syncthreads();
    if (mode != 0 && tid < bs && absT(Ds[tid][tid]) < tiny) s_bad = 1;
    __syncthreads();
    if (s_bad) {
        if (tid == 0) atomicCAS(status, 0, RL_ERR_DIV_BY_ZERO);
        return;
    }
    const int col = 2 * warp + (lane >> 4), r16 = lane & 15;
    T y[4];
#pragma unroll
    for (int sl = 0; sl < 4; sl++) y[sl] = Ys[16 * sl + r16][col];
    if (mode <= 1) {
#pragma unroll
        for (int j = 0; j < 64; j++) {
            if (j < bs) {
                if (mode == 1 && r16 == (j & 15)) y[j >> 4] = y[j >> 4] / Ds[j][j];
                const T xj = __shfl_sync(0xffffffffu, y[j >> 4], j & 15, 16);
#pragma unroll
                for (int sl = j >> 4; sl < 4; sl++) {
                    const int i = 16 * sl + r16;
                    if (i > j && i < bs) y[sl] = fma(-Ds[i][j], xj, y[sl]);
                }
            }
        }
    } else {
#pragma unroll
        for (int j = 63; j >= 0; j--) {
            if (j < bs) {
                if (r16 == (j & 15)) y[j >> 4] = y[j >> 4] / Ds[j][j];
                const T xj = __shfl_sync(0xffffffffu, y[j >> 4], j & 15, 16);
#pragma unroll
                for (int sl = 0; sl <= (j >> 4); sl++) {
                    const int i = 16 * sl + r16;
                    if (i < j) y[sl] = fma(-(mode == 2 ? Ds[i][j] : Ds[j][i]), xj, y[sl]);
                }
            }
        }
    }
    __syncthreads();
#pragma unroll
    for (int sl = 0; sl < 4; sl++) Ys[16 * sl + r16][col] = y[sl];
    __syncthreads();
    for (int idx = tid; idx < bs * kTrsmCols; idx += blockDim.x) {
        const int i = idx / kTrsmCols, cc = idx - i * kTrsmCols;
        if (c0 + cc < nrhs) Y[(long long)i * ldy + c0 + cc] = Ys[i][cc];
    }
}

// ------------------------------------------- few-right-hand-side triangular sweep --
// op(A) X = Y in place for up to 8 right-hand sides in ONE launch: each CTA takes BR-row
// blocks of the solution in solve order by an atomic ticket (forward for modes 0 / 1,
// backward for modes 2 / 3; the modes are those of tri_solve_dev). A block folds in every
// block solved before it as it is published, solves its diagonal block and publishes its
// rows. The sweep is a chain of n / BR blocks, so the kernel is built around the time from
// one block's solution to the next one's:
//   * solutions travel through a separate buffer preset to a NaN pattern that no result has
//     (all bits set): a reader polls the values themselves, so publishing needs neither a
//     flag nor a fence, one trip to L2 instead of three;
//   * the tile of A that meets the awaited block is in registers before the wait, a warp
//     holding 8 rows and a lane the columns lane + 32 u; the products stay per lane over all
//     blocks and are reduced once, after the last one;
//   * the diagonal block is in shared memory from the start: as its inverse (Dinv, FP64 and one
//     right-hand side: the solve is one more BR x BR product) or scaled by its reciprocal
//     diagonal, so that a substitution step is one shuffle and one multiply-add (a block whose
//     scaled entries leave the normal range is substituted unscaled).
// BR = 128 for FP32 (64 up to 64 rows); 64 for FP64, where the products of a tile are bound by the FP64 unit.
// The form before (64-row blocks, a flag per block behind a fence, the folded sums through
// shared memory) against this one, per sweep: FP64 by substitution n = 4096 992 and 461 us.
// A CTA waits only on tickets taken before its own, by CTAs that are running, so the sweep
// always progresses; every wait is bounded by wait_ns (RL_TUNE_WAIT_TIMEOUT_NS,
// RL_ERR_TIMEOUT), after which the CTA goes on with zeros and publishes, so no later block
// waits in turn. withhold >= 0 is a test setting (RL_TUNE_TEST_WITHHOLD_SWEEP_BLOCK): that
// block is solved but never published.
// More than kSweepRhs right-hand sides run as groups of kSweepRhs columns side by side:
// blockIdx.y is the group, with its own ticket and solutions.
// ws: sweep_ws_bytes, all bits set: per group the solutions (n x RW), then the tickets.
constexpr int kSweepRhs = 8, kSweepGroups = 16;
template <class T>
constexpr int sweep_rows() {
    return sizeof(T) == 4 ? 128 : 64;
}

// Right-hand-side groups of a sweep over nrhs columns, 0 when the sweep does not take
// them (more than kSweepGroups groups); columns a group holds; bytes of the workspace.
inline int sweep_groups(int nrhs) {
    const int g = (nrhs + kSweepRhs - 1) / kSweepRhs;
    return g <= kSweepGroups ? g : 0;
}
inline int sweep_width(int nrhs) { return nrhs == 1 ? 1 : kSweepRhs; }
template <class T>
inline size_t sweep_ws_bytes(int n, int nrhs) {
    const size_t b = (size_t)sweep_groups(nrhs) * ((size_t)n * sweep_width(nrhs) * sizeof(T) + 16);
    return (b + 15) & ~(size_t)15;  // a second workspace behind this one is aligned as well
}

__device__ __forceinline__ float sweep_peek(const float *p) {
    unsigned v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return __uint_as_float(v);
}
__device__ __forceinline__ double sweep_peek(const double *p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return __longlong_as_double((long long)v);
}
__device__ __forceinline__ bool sweep_unset(float v) { return __float_as_uint(v) == 0xffffffffu; }
__device__ __forceinline__ bool sweep_unset(double v) { return (unsigned long long)__double_as_longlong(v) == ~0ull; }
// The published value at p, waiting for it (bounded; 0 and *fail set when the wait runs out).
template <class T>
__device__ __forceinline__ T sweep_get(const T *p, volatile int *fail, unsigned long long limit) {
    T v = sweep_peek(p);
    unsigned long long t0 = 0;
    for (unsigned spin = 0; sweep_unset(v); spin++) {
        if ((spin & 63u) == 63u) {
            if (*fail) return T(0);
            const unsigned long long t = global_ns();
            if (t0 == 0)
                t0 = t;
            else if (t - t0 > limit) {
                *fail = 1;
                return T(0);
            }
        }
        v = sweep_peek(p);
    }
    return v;
}
// The published values at p and p + 1 (8-byte aligned) with one load a poll; of the two the
// first `have` are awaited, the others are 0.
__device__ __forceinline__ float2 sweep_get2(const float *p, int have, volatile int *fail, unsigned long long limit) {
    if (have <= 0) return make_float2(0.f, 0.f);
    unsigned long long t0 = 0;
    for (unsigned spin = 0;; spin++) {
        unsigned a, b;
        asm volatile("ld.relaxed.gpu.global.v2.u32 {%0, %1}, [%2];" : "=r"(a), "=r"(b) : "l"(p) : "memory");
        if (have < 2) b = 0u;
        if (a != 0xffffffffu && b != 0xffffffffu) return make_float2(__uint_as_float(a), __uint_as_float(b));
        if ((spin & 63u) == 63u) {
            const unsigned long long t = global_ns();
            if (t0 == 0) t0 = t;
            if (*fail || t - t0 > limit) {
                *fail = 1;
                return make_float2(0.f, 0.f);
            }
        }
    }
}
__device__ __forceinline__ void sweep_put(float *p, float v) {
    const unsigned u = __float_as_uint(v);
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(u == 0xffffffffu ? 0x7fffffffu : u) : "memory");
}
__device__ __forceinline__ void sweep_put(double *p, double v) {
    const unsigned long long u = (unsigned long long)__double_as_longlong(v);
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(u == ~0ull ? 0x7fffffffffffffffull : u) : "memory");
}

template <class T, int RW, int ROWS>
struct SweepCfg {
    static constexpr int BR = ROWS, WARPS = BR / 8, THREADS = 32 * WARPS, CPL = BR / 32, LDD = BR + 1;
    // the diagonal block, v and the awaited solution; behind them the warps' column sums (L^T only)
    static constexpr size_t SMEM = sizeof(T) * (BR * LDD + 2 * BR * RW), SMEM_LT = SMEM + sizeof(T) * WARPS * BR * RW;
};

template <class T, class TA, int RW, int ROWS>
static __global__ void __launch_bounds__(SweepCfg<T, RW, ROWS>::THREADS) trsv_sweep_kernel(const TA *__restrict__ A, long long lda,
                                                             int n, T *__restrict__ Y, long long ldy, int nrhs, int mode,
                                                             T *ws, int *tickets, int *status, T tiny,
                                                             unsigned long long wait_ns, int withhold,
                                                             const T *__restrict__ Dinv) {
    using cfg = SweepCfg<T, RW, ROWS>;
    constexpr int BR = cfg::BR, CPL = cfg::CPL, LDD = cfg::LDD, THREADS = cfg::THREADS, WARPS = cfg::WARPS;
    constexpr bool INV = sizeof(T) == 8 && RW == 1;  // the instance that is called with Dinv
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T *Ds = reinterpret_cast<T *>(smem_raw);  // BR x LDD: the inverse, or the scaled diagonal block
    T *v = Ds + BR * LDD;                     // BR x RW: right-hand side minus the folded sums
    T *xs = v + BR * RW;                      // BR x RW: the awaited block's solution (RW > 1)
    T *red = xs + BR * RW;                    // WARPS x BR x RW: column sums of the warps (L^T)
    __shared__ T inv[BR];
    __shared__ int s_t, s_fail;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nb = (n + BR - 1) / BR;
    const bool fwd = mode <= 1, trans = mode == 3;
    Y += (long long)blockIdx.y * kSweepRhs;
    nrhs = min(kSweepRhs, nrhs - (int)blockIdx.y * kSweepRhs);
    ws += (size_t)blockIdx.y * n * RW;
    if (tid == 0) s_fail = 0;
    for (;;) {
        __syncthreads();  // the previous block's shared state is no longer read
        if (tid == 0) s_t = atomicAdd(tickets + blockIdx.y, 1) + 1;  // preset to -1
        __syncthreads();
        if (s_t >= nb) break;
        const int b = fwd ? s_t : nb - 1 - s_t, r0 = b * BR, bs = min(BR, n - r0);
        // The row whose sum this lane ends with (8 rows of the warp, 4 lanes a row) and its
        // right-hand side; L^T: thread t ends with element t of the block.
        const int mrow = warp * 8 + (lane >> 2);
        T y[RW];
        if (!trans)
#pragma unroll
            for (int c = 0; c < RW; c++) y[c] = (mrow < bs && c < nrhs) ? Y[(long long)(r0 + mrow) * ldy + c] : T(0);
        // The diagonal block, every load in flight before the first store (element by element the
        // staging alone was ~20 us of a sweep).
        constexpr int DP = BR * BR / THREADS;
        T dv[DP];
#pragma unroll
        for (int q = 0; q < DP; q++) {
            const int e = tid + q * THREADS, i = e / BR, j = e % BR;
            if (INV && Dinv)
                dv[q] = Dinv[(long long)b * BR * BR + e];
            else
                dv[q] = (i < bs && j < bs) ? T(A[(long long)(r0 + i) * lda + r0 + j]) : T(0);
        }
#pragma unroll
        for (int q = 0; q < DP; q++) {
            const int e = tid + q * THREADS, i = e / BR, j = e % BR;
            Ds[!(INV && Dinv) && trans ? j * LDD + i : i * LDD + j] = dv[q];
        }
        bool scaled = true;
        if (!(INV && Dinv)) {
            __syncthreads();
            if (tid < BR) {
                const T d = tid < bs ? Ds[tid * LDD + tid] : T(1);
                if (mode != 0 && absT(d) < tiny) atomicCAS(status, 0, RL_ERR_DIV_BY_ZERO);
                inv[tid] = mode == 0 ? T(1) : T(1) / d;
            }
            __syncthreads();
            if (mode != 0) {
                bool wide = false;
                for (int e = tid; e < bs * BR; e += THREADS) {
                    const int i = e / BR, j = e % BR;
                    const T d = Ds[i * LDD + j], f = inv[i];
                    wide |= (fwd ? j < i : j > i) && scaling_wide(d, exponent_of(f));
                    Ds[i * LDD + j] = d * f;
                }
                if (__syncthreads_or(wide)) {  // the entries as they are, again
                    scaled = false;
                    for (int e = tid; e < BR * BR; e += THREADS) {
                        const int i = e / BR, j = e % BR;
                        Ds[trans ? j * LDD + i : i * LDD + j] =
                            (i < bs && j < bs) ? T(A[(long long)(r0 + i) * lda + r0 + j]) : T(0);
                    }
                }
            }
        }
        // the fold: acc[i][c] of row warp 8 + i over this lane's columns; L^T: acc[u][c] of
        // column lane + 32 u of the block over this warp's 8 rows of the earlier block
        constexpr int NA = 8;  // rows a warp holds of a tile
        T acc[(CPL > NA ? CPL : NA)][RW];
#pragma unroll
        for (int i = 0; i < (CPL > NA ? CPL : NA); i++)
#pragma unroll
            for (int c = 0; c < RW; c++) acc[i][c] = T(0);
        const int nk = fwd ? b : nb - 1 - b;  // blocks solved before this one
        TA cur[NA][CPL], nxt[NA][CPL];
        auto load = [&](int kk, TA (&t)[NA][CPL]) {
            const int k = fwd ? kk : nb - 1 - kk, c0 = k * BR, ks = min(BR, n - c0);
#pragma unroll
            for (int i = 0; i < NA; i++)
#pragma unroll
                for (int u = 0; u < CPL; u++) {
                    const int wr = warp * 8 + i, lc = lane + 32 * u;
                    if (trans)
                        t[i][u] = (wr < ks && lc < bs) ? A[(long long)(c0 + wr) * lda + r0 + lc] : TA(0);
                    else
                        t[i][u] = (wr < bs && lc < ks) ? A[(long long)(r0 + wr) * lda + c0 + lc] : TA(0);
                }
        };
        if (nk > 0) load(0, cur);
        for (int kk = 0; kk < nk; kk++) {
            // One right-hand side: the next tile is under way while this one waits. With 8
            // the sums take those registers.
            if (RW == 1 && kk + 1 < nk) load(kk + 1, nxt);
            const int k = fwd ? kk : nb - 1 - kk, c0 = k * BR, ks = min(BR, n - c0);
            if (RW == 1) {
                if (!trans) {
#pragma unroll
                    for (int u = 0; u < CPL; u++) {
                        const int lc = lane + 32 * u;
                        const T x = lc < ks ? sweep_get(ws + c0 + lc, &s_fail, wait_ns) : T(0);
#pragma unroll
                        for (int i = 0; i < NA; i++) acc[i][0] = fma(T(cur[i][u]), x, acc[i][0]);
                    }
                } else {
                    const int wr = warp * 8 + (lane & 7);
                    const T xl = wr < ks ? sweep_get(ws + c0 + wr, &s_fail, wait_ns) : T(0);
#pragma unroll
                    for (int i = 0; i < NA; i++) {
                        const T x = __shfl_sync(0xffffffffu, xl, i);
#pragma unroll
                        for (int u = 0; u < CPL; u++) acc[u][0] = fma(T(cur[i][u]), x, acc[u][0]);
                    }
                }
            } else {
                __syncthreads();  // the last block's solution is no longer read
                for (int e = tid; e < BR * RW; e += THREADS)
                    xs[e] = e < ks * RW && e % RW < nrhs ? sweep_get(ws + (size_t)c0 * RW + e, &s_fail, wait_ns) : T(0);
                __syncthreads();
#pragma unroll
                for (int w0 = 0; w0 < (trans ? NA : CPL); w0++) {
                    T x[RW];
                    ldv<RW>(xs + (trans ? warp * 8 + w0 : lane + 32 * w0) * RW, x);
                    if (trans) {
#pragma unroll
                        for (int u = 0; u < CPL; u++)
#pragma unroll
                            for (int c = 0; c < RW; c++) acc[u][c] = fma(T(cur[w0][u]), x[c], acc[u][c]);
                    } else {
#pragma unroll
                        for (int i = 0; i < NA; i++)
#pragma unroll
                            for (int c = 0; c < RW; c++) acc[i][c] = fma(T(cur[i][w0 & (CPL - 1)]), x[c], acc[i][c]);
                    }
                }
                if (kk + 1 < nk) load(kk + 1, cur);
            }
            if (RW == 1)
#pragma unroll
                for (int i = 0; i < NA; i++)
#pragma unroll
                    for (int u = 0; u < CPL; u++) cur[i][u] = nxt[i][u];
        }
        // v = y - sums
        if (!trans) {
#pragma unroll
            for (int c = 0; c < RW; c++) {
                T s8[8];
#pragma unroll
                for (int i = 0; i < 8; i++) s8[i] = acc[i][c];
                int row;
                const T sum = warp_reduce_scatter<8>(s8, lane, row);
                if ((lane & 3) == 0) v[mrow * RW + c] = y[c] - sum;
            }
        } else {
#pragma unroll
            for (int u = 0; u < CPL; u++)
#pragma unroll
                for (int c = 0; c < RW; c++) red[((size_t)warp * BR + lane + 32 * u) * RW + c] = acc[u][c];
            __syncthreads();
            for (int e = tid; e < BR * RW; e += THREADS) {
                T sum = T(0);
#pragma unroll
                for (int wq = 0; wq < WARPS; wq++) sum += red[(size_t)wq * BR * RW + e];
                const int i = e / RW, c = e % RW;
                v[e] = (i < bs && c < nrhs ? Y[(long long)(r0 + i) * ldy + c] : T(0)) - sum;
            }
        }
        __syncthreads();
        auto publish = [&](int i, int c, T x) {
            if (i < bs && c < nrhs) {
                if (b != withhold) sweep_put(ws + (size_t)(r0 + i) * RW + c, x);
                Y[(long long)(r0 + i) * ldy + c] = x;
            }
        };
        if (INV && Dinv) {
            T o[8][RW];
#pragma unroll
            for (int i = 0; i < 8; i++)
#pragma unroll
                for (int c = 0; c < RW; c++) o[i][c] = T(0);
#pragma unroll
            for (int u = 0; u < CPL; u++) {
                T x[RW];
                if constexpr (RW == 1)
                    x[0] = v[lane + 32 * u];
                else
                    ldv<RW>(v + (lane + 32 * u) * RW, x);
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    const T d = Ds[(warp * 8 + i) * LDD + lane + 32 * u];
#pragma unroll
                    for (int c = 0; c < RW; c++) o[i][c] = fma(d, x[c], o[i][c]);
                }
            }
#pragma unroll
            for (int c = 0; c < RW; c++) {
                T s8[8];
#pragma unroll
                for (int i = 0; i < 8; i++) s8[i] = o[i][c];
                int row;
                const T x = warp_reduce_scatter<8>(s8, lane, row);
                if ((lane & 3) == 0) publish(mrow, c, x);
            }
        } else if (warp < RW) {
            // substitution with the scaled rows: warp c solves right-hand side c, lane l
            // holds the rows l + 32 h
            const int c = warp;
            // The products with each other group of 32 unknowns are summed apart (t) and subtracted
            // once: fewer roundings at the size of z.
            T z[CPL], t[CPL];
#pragma unroll
            for (int h = 0; h < CPL; h++) {
                z[h] = v[(lane + 32 * h) * RW + c] * (scaled ? inv[lane + 32 * h] : T(1));
                t[h] = T(0);
            }
            if (!scaled) {
                for (int k = 0; k < bs; k++) {
                    const int kk = fwd ? k : bs - 1 - k, q = kk & 31;
#pragma unroll
                    for (int hb = 0; hb < CPL; hb++) {
                        if (kk / 32 != hb) continue;
                        const T xk = __shfl_sync(0xffffffffu, z[hb], q) * inv[kk];
#pragma unroll
                        for (int h = 0; h < CPL; h++)
                            if (fwd ? h > hb || (h == hb && lane > q) : h < hb || (h == hb && lane < q))
                                z[h] = fma(-Ds[(lane + 32 * h) * LDD + kk], xk, z[h]);
                    }
                }
#pragma unroll
                for (int h = 0; h < CPL; h++) z[h] *= inv[lane + 32 * h];
            } else if (fwd) {
#pragma unroll
                for (int hb = 0; hb < CPL; hb++) {  // the 32 unknowns being eliminated
                    const int lim = min(32, bs - hb * 32);  // a short block's steps only
#pragma unroll 4
                    for (int q = 0; q < lim; q++) {
                        const T xk = __shfl_sync(0xffffffffu, z[hb], q);
                        if (lane > q) z[hb] = fma(-Ds[(lane + 32 * hb) * LDD + hb * 32 + q], xk, z[hb]);
#pragma unroll
                        for (int h = hb + 1; h < CPL; h++) t[h] = fma(Ds[(lane + 32 * h) * LDD + hb * 32 + q], xk, t[h]);
                    }
#pragma unroll
                    for (int h = hb + 1; h < CPL; h++) z[h] -= t[h], t[h] = T(0);
                }
            } else {
#pragma unroll
                for (int hb = CPL - 1; hb >= 0; hb--) {
#pragma unroll 4
                    for (int q = min(32, bs - hb * 32) - 1; q >= 0; q--) {
                        const T xk = __shfl_sync(0xffffffffu, z[hb], q);
                        if (lane < q) z[hb] = fma(-Ds[(lane + 32 * hb) * LDD + hb * 32 + q], xk, z[hb]);
#pragma unroll
                        for (int h = 0; h < hb; h++) t[h] = fma(Ds[(lane + 32 * h) * LDD + hb * 32 + q], xk, t[h]);
                    }
#pragma unroll
                    for (int h = 0; h < hb; h++) z[h] -= t[h], t[h] = T(0);
                }
            }
#pragma unroll
            for (int h = 0; h < CPL; h++) publish(lane + 32 * h, c, z[h]);
        }
        if (tid == 0 && *(volatile int *)&s_fail) atomicCAS(status, 0, RL_ERR_TIMEOUT);
    }
}

// The FP32 sweep with inverted 64 x 64 diagonal blocks (Dinv, from diag_inverse_kernel): the
// refinement of the mixed single-system solvers, RW = 1 or 8 right-hand sides a group. Which
// step of a refinement passes its test hangs on the last bits of every correction at the edge
// of the test, and whether it converges on how far the inverses are from the triangle's, so the
// block size and the order of the sums are part of the results and are fixed here: thread (row,
// quarter) of a block adds the products with its 16 columns of every block solved before, in
// solve order; the quarters are added as (0 + 1) + (2 + 3), in the L^T mode as
// ((0 + 1) + 2) + 3; v = y - sums; x_b = Dinv_b v in the same quarters. (With 128-row blocks and
// the sums spread over the lanes 2 of 8 systems of kappa = 1e6, n = 4096, ended a step sooner,
// with an error of 5e-9 in place of 5e-10, and systems made of Hadamard factors, which converge
// here in 10 to 16 steps, went to the FP64 fallback.)
// The chain from one block's solutions to the next one's is what it takes: the solutions are
// polled in place (ws as in trsv_sweep_kernel), two values a lane in one load, by each warp for
// itself without a CTA barrier (RW = 1) or once per CTA; the tiles of A are in registers
// kInvDepth blocks ahead; a thread's share of Dinv and of the right-hand side is loaded before
// the fold.
// Per sweep, with the 128-row form before: n = 3000 47 us (45), 4096 64 (61.5), 16384 333 (296);
// n = 2048 with 8 right-hand sides 62 (65), n = 8192 with 64 508 (665; the CTAs of all 8 groups
// resident from the start, with the grid in group order 970). Tiles 4 blocks ahead: the same for
// one right-hand side, 658 for 64 (registers).
constexpr int kInvRows = 64, kInvDepth = 2;
template <int RW>
static __global__ void __launch_bounds__(256) trsv_inv_kernel(const float *__restrict__ A, long long lda, int n,
                                                              float *__restrict__ Y, long long ldy, int nrhs, int mode,
                                                              float *ws, int *tickets, int *status,
                                                              unsigned long long wait_ns, int withhold,
                                                              const float *__restrict__ Dinv) {
    constexpr int BR = kInvRows, DEPTH = kInvDepth, OWN = RW == 1 ? 1 : 2;  // OWN: columns a thread ends with
    // A quarter's 16 x RW values, 16 bytes further for each quarter: the four quarters of a warp
    // read from different banks.
    constexpr int QS = 16 * RW + 4;
    __shared__ __align__(16) float xs[RW == 1 ? 8 : 1][2][4 * QS];  // the awaited solutions (RW = 1: a warp's copy)
    __shared__ __align__(16) float v[4 * QS];
    __shared__ float red[4][BR][RW];  // the quarters' sums (L^T)
    __shared__ int s_t, s_fail;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nb = (n + BR - 1) / BR;
    const bool fwd = mode <= 1, trans = mode == 3;
    const bool vec = !trans && (lda & 3) == 0 && (reinterpret_cast<uintptr_t>(A) & 15) == 0;
    const int rr = tid >> 2, qq = tid & 3;                                 // row and quarter of the block's product
    const int r = trans ? tid & (BR - 1) : rr, q = trans ? tid >> 6 : qq;  // and of the fold
    Y += (long long)blockIdx.y * RW;
    nrhs = min(RW, nrhs - (int)blockIdx.y * RW);
    ws += (size_t)blockIdx.y * n * RW;
    const int c0y = RW == 1 ? 0 : 2 * qq, own = RW == 1 ? (qq == 0 ? 1 : 0) : min(2, nrhs - c0y);
    if (tid == 0) s_fail = 0;
    for (;;) {
        __syncthreads();  // the previous block's shared state is no longer read
        if (tid == 0) s_t = atomicAdd(tickets + blockIdx.y, 1) + 1;  // preset to -1
        __syncthreads();
        if (s_t >= nb) break;
        const int b = fwd ? s_t : nb - 1 - s_t, r0 = b * BR, bs = min(BR, n - r0);
        const int nk = fwd ? b : nb - 1 - b;  // blocks solved before this one
        float d[16], t[DEPTH][16], acc[RW], y[OWN];
        ldv<16>(Dinv + ((long long)b * BR + rr) * BR + qq * 16, d);
#pragma unroll
        for (int c = 0; c < OWN; c++) y[c] = c < own && rr < bs ? Y[(long long)(r0 + rr) * ldy + c0y + c] : 0.f;
        auto load = [&](int kk, float (&o)[16]) {
            const int c0 = (fwd ? kk : nb - 1 - kk) * BR, ks = min(BR, n - c0);
            if (vec && ks == BR) {
                if (r < bs) {
                    ldv<16>(A + (long long)(r0 + r) * lda + c0 + q * 16, o);
                } else {
#pragma unroll
                    for (int jj = 0; jj < 16; jj++) o[jj] = 0.f;
                }
                return;
            }
#pragma unroll
            for (int jj = 0; jj < 16; jj++) {
                const int j = q * 16 + jj;
                o[jj] = (r < bs && j < ks) ? (trans ? A[(long long)(c0 + j) * lda + r0 + r] : A[(long long)(r0 + r) * lda + c0 + j])
                                           : 0.f;
            }
        };
        // 16 terms of every column's sum: a times the quarter's values at p
        auto dot16 = [&](const float (&a)[16], const float *p, float (&o)[RW]) {
            if constexpr (RW == 1) {
                float x[16];
                ldv<16>(p, x);
#pragma unroll
                for (int jj = 0; jj < 16; jj++) o[0] = fmaf(a[jj], x[jj], o[0]);
            } else {
#pragma unroll
                for (int jj = 0; jj < 16; jj++) {
                    float x[RW];
                    ldv<RW>(p + jj * RW, x);
#pragma unroll
                    for (int c = 0; c < RW; c++) o[c] = fmaf(a[jj], x[c], o[c]);
                }
            }
        };
#pragma unroll
        for (int u = 0; u < DEPTH; u++)
            if (u < nk) load(u, t[u]);
#pragma unroll
        for (int c = 0; c < RW; c++) acc[c] = 0.f;
        for (int k0 = 0; k0 < nk; k0 += DEPTH) {
#pragma unroll
            for (int u = 0; u < DEPTH; u++) {
                const int kk = k0 + u;
                if (kk >= nk) break;
                const int c0 = (fwd ? kk : nb - 1 - kk) * BR, ks = min(BR, n - c0);
                // A buffer of the two is written again only after the barrier that follows the
                // reads of the other.
                float *w = xs[RW == 1 ? warp : 0][u & 1];
                if constexpr (RW == 1) {
                    const int p = 2 * lane + (trans ? 16 * q : 0);  // L^T: the quarter's 16 are enough
                    if (!trans || lane < 8)
                        *reinterpret_cast<float2 *>(w + (p >> 4) * QS + (p & 15)) =
                            sweep_get2(ws + c0 + p, ks - p, &s_fail, wait_ns);
                    __syncwarp();
                } else {
                    *reinterpret_cast<float2 *>(w + (rr >> 4) * QS + (rr & 15) * RW + c0y) =
                        sweep_get2(ws + (size_t)(c0 + rr) * RW + c0y, rr < ks ? own : 0, &s_fail, wait_ns);
                    __syncthreads();
                }
                dot16(t[u], w + q * QS, acc);
                if (kk + DEPTH < nk) load(kk + DEPTH, t[u]);
            }
        }
        // the quarters' sums of this thread's columns: (0 + 1) + (2 + 3)
        auto quarters = [&](float (&o)[RW], float (&out)[OWN]) {
            if constexpr (RW == 1) {
                o[0] += __shfl_xor_sync(0xffffffffu, o[0], 1);
                out[0] = o[0] + __shfl_xor_sync(0xffffffffu, o[0], 2);
            } else {  // lane q keeps the columns 2 q, 2 q + 1 and gives the others away
                const bool odd = qq & 1, high = qq & 2;
                float h[4];
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const int e = (i & 1) + 4 * (i >> 1);  // columns 0 1 4 5, and 2 3 6 7 of an odd lane
                    const float keep = odd ? o[e + 2] : o[e], give = odd ? o[e] : o[e + 2];
                    h[i] = keep + __shfl_xor_sync(0xffffffffu, give, 1);
                }
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    const float keep = high ? h[i + 2] : h[i], give = high ? h[i] : h[i + 2];
                    out[i] = keep + __shfl_xor_sync(0xffffffffu, give, 2);
                }
            }
        };
        float *vo = v + (rr >> 4) * QS + (rr & 15) * RW + c0y, sum[OWN];
        if (!trans) {
            quarters(acc, sum);
        } else {
#pragma unroll
            for (int c = 0; c < RW; c++) red[q][r][c] = acc[c];
            __syncthreads();
#pragma unroll
            for (int c = 0; c < OWN; c++)
                sum[c] = (((0.f + red[0][rr][c0y + c]) + red[1][rr][c0y + c]) + red[2][rr][c0y + c]) + red[3][rr][c0y + c];
        }
        if (RW > 1 || qq == 0)
#pragma unroll
            for (int c = 0; c < OWN; c++) vo[c] = y[c] - sum[c];
        __syncthreads();
        float x[RW], xo[OWN];
#pragma unroll
        for (int c = 0; c < RW; c++) x[c] = 0.f;
        dot16(d, v + qq * QS, x);
        quarters(x, xo);
        if (rr < bs)
#pragma unroll
            for (int c = 0; c < OWN; c++)
                if (c < own) {
                    if (b != withhold) sweep_put(ws + (size_t)(r0 + rr) * RW + c0y + c, xo[c]);
                    Y[(long long)(r0 + rr) * ldy + c0y + c] = xo[c];
                }
        if (tid == 0 && *(volatile int *)&s_fail) atomicCAS(status, 0, RL_ERR_TIMEOUT);
    }
}

// Dinv_b = op(D_b)^-1 for every 64 x 64 diagonal block D_b of A (n x n, stored as TA),
// formed in T, one CTA per block: 64 threads, thread j solving op(D_b) x = e_j by
// substitution (op and the unit diagonal as in trsv_sweep_kernel's modes). Written
// row-major 64 x 64 per block, zero beyond a partial last block. |d_ii| < tiny records
// RL_ERR_DIV_BY_ZERO.
template <class T, class TA>
static __global__ void __launch_bounds__(64) diag_inverse_kernel(const TA *__restrict__ A, long long lda, int n, int mode,
                                                             T *__restrict__ Dinv, int *status, T tiny) {
    constexpr int BR = 64;
    __shared__ T M[BR][BR + 1];  // op(D_b)
    __shared__ T X[BR][BR + 1];  // column j: thread j's solution
    const int b = blockIdx.x, r0 = b * BR, bs = min(BR, n - r0), j = threadIdx.x;
    for (int idx = j; idx < BR * BR; idx += blockDim.x) {
        const int r = idx / BR, c = idx - r * BR;
        T v = T(0);
        if (r < bs && c < bs)
            v = T(mode == 3 ? A[(long long)(r0 + c) * lda + r0 + r] : A[(long long)(r0 + r) * lda + r0 + c]);
        M[r][c] = v;
        X[r][c] = T(0);
    }
    __syncthreads();
    const bool unit = mode == 0, lower = mode <= 1;
    if (j < bs) {
        if (!unit && absT(M[j][j]) < tiny) atomicCAS(status, 0, RL_ERR_DIV_BY_ZERO);
        if (lower) {
            for (int i = j; i < bs; i++) {
                T v = i == j ? T(1) : T(0);
                for (int k = j; k < i; k++) v = fma(-M[i][k], X[k][j], v);
                X[i][j] = unit ? v : v / M[i][i];
            }
        } else {
            for (int i = j; i >= 0; i--) {
                T v = i == j ? T(1) : T(0);
                for (int k = i + 1; k <= j; k++) v = fma(-M[i][k], X[k][j], v);
                X[i][j] = v / M[i][i];
            }
        }
    }
    __syncthreads();
    T *out = Dinv + (long long)b * BR * BR;
    for (int idx = j; idx < BR * BR; idx += blockDim.x) out[idx] = X[idx / BR][idx % BR];
}

// Row-wise solve X D^T = Y for the rows of Y (m x bs, stride ldy), D lower bs x bs: the
// Cholesky panel L21 = A21 L11^-T. As trsm_diag_kernel: CTA per 8 rows, 16 lanes per row each
// holding 4 of its entries, so that the FP64 work is on every SM (a thread per row put the
// 64-step chain of 2,016 multiply-adds on 11 SMs at m = 1,400: 129 us). With *status set (D's
// factorisation, or an earlier one, has failed) nothing is done.
template <class T>
static __global__ void __launch_bounds__(128) trsm_right_lt_kernel(const T *D, long long ldd, int bs, T *Y, long long ldy,
                                                            int m, const int *status) {
    __shared__ T Ds[64][65];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int failed = *status;  // read with D in flight
    {
        T d[32];
#pragma unroll
        for (int e = 0; e < 32; e++) {
            const int i = 2 * e + (tid >> 6), j = tid & 63;
            d[e] = (i < bs && j < bs) ? D[(long long)i * ldd + j] : T(0);
        }
        if (failed) return;
#pragma unroll
        for (int e = 0; e < 32; e++) Ds[2 * e + (tid >> 6)][tid & 63] = d[e];
    }
    __syncthreads();
    const int row = blockIdx.x * kTrsmCols + 2 * warp + (lane >> 4), r16 = lane & 15;
    T *yp = Y + (long long)row * ldy;
    T y[4];
#pragma unroll
    for (int sl = 0; sl < 4; sl++) y[sl] = (row < m && 16 * sl + r16 < bs) ? yp[16 * sl + r16] : T(0);
#pragma unroll
    for (int j = 0; j < 64; j++) {
        if (j < bs) {
            if (r16 == (j & 15)) y[j >> 4] = y[j >> 4] / Ds[j][j];
            const T xj = __shfl_sync(0xffffffffu, y[j >> 4], j & 15, 16);
#pragma unroll
            for (int sl = j >> 4; sl < 4; sl++) {
                const int i = 16 * sl + r16;
                if (i > j && i < bs) y[sl] = fma(-Ds[i][j], xj, y[sl]);
            }
        }
    }
#pragma unroll
    for (int sl = 0; sl < 4; sl++)
        if (row < m && 16 * sl + r16 < bs) yp[16 * sl + r16] = y[sl];
}

// ------------------------------------------------------------- compact WY helpers --
// V (mrows x kb, row stride kb) = the panel's reflectors with the implicit unit diagonal
// and zeros above it.
template <class T>
static __global__ void extract_v_kernel(const T *P, long long lda, int mrows, int kb, T *V) {
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (long long)mrows * kb) return;
    const int r = (int)(idx / kb), c = (int)(idx - (long long)r * kb);
    V[idx] = r > c ? P[(long long)r * lda + c] : (r == c ? T(1) : T(0));
}

// W[i][j] = V[j][i] for i < kb, j < cols (V with row stride kb).
template <class T>
static __global__ void v_transpose_kernel(const T *V, int kb, int cols, T *W, long long ldw) {
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (long long)kb * cols) return;
    const int i = (int)(idx / cols), j = (int)(idx - (long long)i * cols);
    W[(long long)i * ldw + j] = V[(long long)j * kb + i];
}

// Partial Gram matrices of the reflector block V (mrows x kb, row stride kb, kb <= 64): CTA
// (c, t) sums V[r]^T V[r] over chunk c of the rows for tile t of the 10 16 x 16 tiles on or
// above the diagonal, into part[c] (64 x 64; the tiles below are not written). FP64 is bound
// by the SMs' FP64 units, so the product is cut into enough CTAs for all of them: 256-row
// chunks with whole 64 x 64 products took 267 us at m = 1201.
constexpr int kGramRows = 128;  // rows per chunk
template <class T>
static __global__ void __launch_bounds__(128) gram_partial_kernel(const T *__restrict__ V, int mrows, int kb,
                                                                  T *__restrict__ part) {
    __shared__ T Va[64][17], Vb[64][17];
    int t = blockIdx.y, ti = 0;  // tile row ti, column tj >= ti
    while (t >= 4 - ti) t -= 4 - ti++;
    const int tj = ti + t, tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    if (tj * 16 >= kb) return;
    const int rbeg = blockIdx.x * kGramRows, rend = min(mrows, rbeg + kGramRows);
    T acc0 = T(0), acc1 = T(0);
    for (int r0 = rbeg; r0 < rend; r0 += 64) {
#pragma unroll
        for (int e = tid; e < 64 * 16; e += 128) {
            const int r = e >> 4, c = e & 15;
            Va[r][c] = (r0 + r < rend && ti * 16 + c < kb) ? V[(long long)(r0 + r) * kb + ti * 16 + c] : T(0);
            Vb[r][c] = (r0 + r < rend && tj * 16 + c < kb) ? V[(long long)(r0 + r) * kb + tj * 16 + c] : T(0);
        }
        __syncthreads();
        const int lim = min(64, rend - r0);
#pragma unroll 8
        for (int r = 0; r < lim; r++) {
            const T b = Vb[r][tx];
            acc0 = fma(Va[r][ty], b, acc0);
            acc1 = fma(Va[r][ty + 8], b, acc1);
        }
        __syncthreads();
    }
    T *out = part + (size_t)blockIdx.x * 64 * 64 + (ti * 16) * 64 + tj * 16 + tx;
    out[ty * 64] = acc0;
    out[(ty + 8) * 64] = acc1;
}

// T factor of H_0 ... H_{kb-1} = I - V T V^T (upper triangular, kb x kb): the Gram matrix
// Gm = V^T V is the sum of the partial Gram matrices (added in part order). The four 16 x 16
// diagonal blocks of T follow from T[j][j] = tau_j, T[0:j, j] = -tau_j T[0:j, 0:j] Gm[0:j, j],
// a warp each; two diagonal blocks join by T12 = -T1 (Gm12 T2), 16 and 16 columns, then 32 and
// 32. The recursion over all 64 columns at once was a chain of 64 dot products of up to 63
// terms in one thread each: 121 us in FP64 and 46 us in FP32, this 49 and 29.
template <class T>
static __global__ void __launch_bounds__(256) larft_kernel(const T *part, int nparts, const T *tau, int kb, T *Tm) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T (*G)[65] = reinterpret_cast<T (*)[65]>(smem_raw);  // 64 x 65 each
    T (*Ts)[65] = G + 64;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    for (int idx = t; idx < 64 * 64; idx += 256) {
        const int i = idx >> 6, j = idx & 63;
        T sum = T(0);
        if (i < j && j < kb)
            for (int c = 0; c < nparts; c++) sum += part[(size_t)c * 64 * 64 + idx];
        G[i][j] = sum;
        Ts[i][j] = T(0);
    }
    __syncthreads();
    if (warp < 4) {
        const int o = warp * 16;
        for (int j = 0; j < 16 && o + j < kb; j++) {
            const T tj = tau[o + j];
            if (lane < j) {
                T s = T(0);
                for (int q = lane; q < j; q++) s = fma(Ts[o + lane][o + q], G[o + q][o + j], s);
                Ts[o + lane][o + j] = -tj * s;
            }
            if (lane == j) Ts[o + j][o + j] = tj;
            __syncwarp();
        }
    }
    __syncthreads();
    for (int h = 16; h <= 32; h *= 2) {  // T12 of the pairs of h x h blocks
        const int pairs = 32 / h, total = pairs * h * h;
        T p[4];
#pragma unroll
        for (int e = 0; e < 4; e++) {  // P = Gm12 T2 (T2 upper triangular)
            const int idx = t + e * 256;
            p[e] = T(0);
            if (idx < total) {
                const int o = idx / (h * h) * 2 * h, i = idx / h % h, j = idx % h;
                for (int q = 0; q <= j; q++) p[e] = fma(G[o + i][o + h + q], Ts[o + h + q][o + h + j], p[e]);
            }
        }
        __syncthreads();
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const int idx = t + e * 256;
            if (idx < total) G[idx / (h * h) * 2 * h + idx / h % h][idx / (h * h) * 2 * h + h + idx % h] = p[e];
        }
        __syncthreads();
#pragma unroll
        for (int e = 0; e < 4; e++) {  // T12 = -T1 P (T1 upper triangular)
            const int idx = t + e * 256;
            if (idx < total) {
                const int o = idx / (h * h) * 2 * h, i = idx / h % h, j = idx % h;
                T s = T(0);
                for (int q = i; q < h; q++) s = fma(Ts[o + i][o + q], G[o + q][o + h + j], s);
                Ts[o + i][o + h + j] = -s;
            }
        }
        __syncthreads();
    }
    for (int idx = t; idx < kb * kb; idx += 256) Tm[idx] = Ts[idx / kb][idx % kb];
}

// Identity-like start for first_k_columns: Q (m x k) = I[:, 0:k].
template <class T>
static __global__ void eye_kernel(T *Q, long long ldq, int m, int k) {
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (long long)m * k) return;
    const int r = (int)(idx / k), c = (int)(idx - (long long)r * k);
    Q[(long long)r * ldq + c] = r == c ? T(1) : T(0);
}

// Gathers rows: Y[perm[i]][:] = B[i][:] (the reference's P * b, applied to nrhs columns).
template <class T>
static __global__ void permute_rows_kernel(const T *B, long long ldb, T *Y, long long ldy, int n, int nrhs,
                                    const uint64_t *perm) {
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (long long)n * nrhs) return;
    const int i = (int)(idx / nrhs), c = (int)(idx - (long long)i * nrhs);
    Y[(long long)perm[i] * ldy + c] = B[(long long)i * ldb + c];
}

// det helpers: sequential fold of the diagonal in row order (the reference's fold), and
// the parity of a stored permutation by cycle resolution (permutation_matrix.rs:479-509).
template <class T>
static __global__ void det_kernel(const T *A, long long lda, int n, const uint64_t *perm, uint64_t *scratch, int square,
                           T *out) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    T d = T(1);
    for (int i = 0; i < n; i++) d = d * A[(long long)i * lda + i];
    if (square) {
        out[0] = d * d;
        return;
    }
    int odd = 0;
    if (perm) {
        for (int i = 0; i < n; i++) scratch[i] = perm[i];
        for (int i = 0; i < n; i++) {
            uint64_t target = scratch[i];
            while ((uint64_t)i != target) {
                const uint64_t nt = scratch[target];
                odd ^= 1;
                scratch[target] = target;
                target = nt;
            }
            scratch[i] = i;
        }
    }
    const T p_det = odd ? T(0) - T(1) : T(1);
    out[0] = p_det * d;
}

}  // namespace rl

// One matrix with n <= 64 on one CTA of 256 threads: LU with partial pivoting (and the solve
// of one right-hand side in the same launch) and Cholesky, in registers. Four consecutive
// threads share a row, thread q of them owning the columns c = q (mod 4), so that the row
// updates use all four schedulers: FP64 work issues at 2 multiply-adds per cycle and SM here,
// and the one-CTA factorisation of factor_cta.cuh, with a row per thread, took 229 us for
// n = 47 in FP64 and its solve another 37 (two thirds of a warp's lanes idle, a division per
// thread); this takes 84 us with the solve (n = 16: 60 + 18, 27 now). A column's reciprocal (and square root) is formed by one warp and shared, two CTA
// barriers per column; multipliers are corrected to the quotient a / p by its remainder
// (Markstein, IBM J. Res. Dev. 34, 1990), so they are the reference's (lu.rs:609,
// cholesky.rs:160-171) in all but rare last-bit cases.
#pragma once

#include "dense.cuh"

namespace rl {

constexpr int kSmallN = 64;

// The next local column to a[0], the finished one to the end.
template <class T>
__device__ __forceinline__ void rotate4(T (&a)[16]) {
    const T first = a[0];
#pragma unroll
    for (int i = 1; i < 16; i++) a[i - 1] = a[i];
    a[15] = first;
}

// a + b in a call: under a predicate the addition would take the FP64 unit of warps that do not need it.
template <class T>
__device__ __noinline__ T add_apart(T a, T b) {
    return a + b;
}

template <class T>
struct SmallLuSmem {
    T row[2][8][kSmallN];  // the warps' candidate rows by column parity (entry q 16 + i, rotated)
    T rowj[2][kSmallN];    // the row at position j
    T rhs[2][8], rhs0[2][8], rhsj[2];
    T M[kSmallN][kSmallN + 1];
    T y[kSmallN];
    T piv, inv;
    unsigned long long k[2][8];
    int i[2][8];
    int bad;
};

// PA = LU in place (row-major, stride lda), ipiv (may be null) 0-based; with b, also
// b <- A^-1 b. A pivot with |p| < tiny sets *status = RL_ERR_DIV_BY_ZERO (A and b are then
// left as they came).
template <class T>
static __global__ void __launch_bounds__(256) small_lu_kernel(T *A, int lda, int n, int *ipiv, T *b, int *status, T tiny) {
    constexpr int L = 16;
    __shared__ __align__(16) SmallLuSmem<T> S;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, q = tid & 3, r = tid >> 2;
    // The right-hand side's products with the first 32 unknowns are summed apart from it in the rows
    // from 32 on (warps 4 to 7: y the sum, y0 the right-hand side, until column 32): fewer roundings at
    // its size (n = 64, diagonally weighted: forward error 1.01 of blocked substitution's, 1.22 without).
    T a[L], y = (b && r < n) ? b[r] : T(0), y0 = T(0);
    if (warp >= 4) y0 = y, y = T(0);
#pragma unroll
    for (int i = 0; i < L; i++) {
        const int c = 4 * i + q;
        a[i] = (r < n && c < n) ? A[(long long)r * lda + c] : T(0);
    }
    if (tid == 0) S.bad = 0;
    const unsigned long long ktiny = amax_key(tiny);
    int my_piv = 0;   // thread j: the pivot of column j
    int my_inv = 0;   // the exponent of 1 / U's diagonal in row r
    for (int jo = 0; 4 * jo < n; jo++) {
#pragma unroll
        for (int qj = 0; qj < 4; qj++) {
            const int j = 4 * jo + qj, slot = j & 1;
            if (j >= n) break;
            unsigned long long bk = 0ull;
            int bi = INT_MAX;
            if (q == qj && r >= j && r < n) {
                bk = amax_key(a[0]);
                bi = r;
            }
            warp_amax_key<T>(bk, bi);
            if (bk != 0ull && r == bi) {
                stv<L>(&S.row[slot][warp][q * L], a);
                if (q == 0) S.rhs[slot][warp] = y, S.rhs0[slot][warp] = y0;
            }
            if (r == j) {
                stv<L>(&S.rowj[slot][q * L], a);
                if (q == 0) S.rhsj[slot] = y;
            }
            if (lane == 0) {
                S.k[slot][warp] = bk;
                S.i[slot][warp] = bi;
            }
            __syncthreads();
            bk = lane < 8 ? S.k[slot][lane] : 0ull;
            bi = lane < 8 ? S.i[slot][lane] : INT_MAX;
            warp_amax_key<T>(bk, bi);
            const bool none = bk == 0ull;  // a NaN column: the diagonal stays
            const int wi = none ? j : bi, bw = wi >> 3;
            const T *prow = none ? S.rowj[slot] : S.row[slot][bw];
            if (warp == (j & 7)) {  // a different warp each column
                if (lane == 0) {
                    const T p = prow[qj * L];
                    S.piv = p;
                    S.inv = T(1) / p;
                    if (!none && bk < ktiny) S.bad = 1;
                }
            }
            T pr[L];
            ldv<L>(prow + q * L, pr);
            T yj = none ? S.rhsj[slot] : S.rhs[slot][bw];
            if (!none && bw >= 4 && j < 32) yj = add_apart(yj, S.rhs0[slot][bw]);
            if (wi != j && (r == j || r == wi)) {
                ldv<L>((r == j ? prow : S.rowj[slot]) + q * L, a);
                const T old = S.rhsj[slot];
                const bool apart = warp >= 4 && j < 32;  // row wi, there
                y = r == j ? yj : (apart ? T(0) : old);
                y0 = old;
            }
            if (tid == j) my_piv = wi;
            __syncthreads();
            if (r == j) my_inv = exponent_of(S.inv);
            if (S.bad) {
                if (tid == 0) atomicCAS(status, 0, RL_ERR_DIV_BY_ZERO);
                return;
            }
            const T p = S.piv, inv = S.inv;
            const bool live = r > j && r < n;
            T l = T(0);
            if (live && q == qj) l = quotient(a[0], p, inv);
            l = __shfl_sync(0xffffffffu, l, qj, 4);
            if (live) {
                if (q == qj)
                    a[0] = l;
                else if (q > qj)
                    a[0] = fma(-l, pr[0], a[0]);
                if (q == 0) y = fma(-l, yj, y);
#pragma unroll
                for (int i = 1; i < L; i++) {
                    if (4 * (jo + i) >= n) break;  // the same for all threads: no multiply-add past n
                    a[i] = fma(-l, pr[i], a[i]);
                }
            }
        }
        if (4 * jo + 4 <= n) rotate4(a);
        if (jo == 7 && warp >= 4) y = add_apart(y, y0);
    }
    // full rotations so far; a[i] is the local column (done + i) mod 16
    const int done = n / 4;
    if (ipiv && tid < n) ipiv[tid] = my_piv;
    bool wide = false;  // an entry of U too far from its row's diagonal to be scaled by it
#pragma unroll
    for (int i = 0; i < L; i++) {
        const int c = 4 * ((done + i) & (L - 1)) + q;
        if (r < n && c < n) {
            wide |= c > r && scaling_wide(a[i], my_inv);
            A[(long long)r * lda + c] = a[i];
            S.M[r][c] = a[i];
        }
    }
    if (!b) return;
    if (q == 0) S.y[r] = y;
    const bool lost = __syncthreads_or(wide) != 0;
    // U x = y by one warp, lane l the rows l and l + 32; rows scaled by the reciprocal
    // diagonal, so a step is one shuffle and one multiply-add; with the entries as they are if a
    // scaled one could leave the normal range.
    if (warp == 0) {
        T z[2], d[2];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int i = lane + 32 * h;
            d[h] = i < n ? T(1) / S.M[i][i] : T(0);
            z[h] = i < n ? quotient(S.y[i], S.M[i][i], d[h]) : T(0);
        }
        T t = T(0);  // the products with the unknowns from 32 on, summed apart
        for (int k = n - 1; k >= 32; k--) {
            const T x = __shfl_sync(0xffffffffu, z[1], k - 32);
            t = fma(S.M[lane][k] * d[0], x, t);
            if (lane + 32 < k) z[1] = fma(-(S.M[lane + 32][k] * d[1]), x, z[1]);
        }
        z[0] -= t;
        for (int k = min(n, 32) - 1; k > 0; k--) {
            const T x = __shfl_sync(0xffffffffu, z[0], k);
            if (lane < k) z[0] = fma(-(S.M[lane][k] * d[0]), x, z[0]);
        }
        if (lost) {
#pragma unroll
            for (int h = 0; h < 2; h++) z[h] = lane + 32 * h < n ? S.y[lane + 32 * h] : T(0);
            for (int k = n - 1; k >= 0; k--) {
                const T x = __shfl_sync(0xffffffffu, k < 32 ? z[0] : z[1], k & 31) / S.M[k][k];
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int i = lane + 32 * h;
                    if (i == k) z[h] = x;
                    if (i < k) z[h] = fma(-S.M[i][k], x, z[h]);
                }
            }
        }
#pragma unroll
        for (int h = 0; h < 2; h++)
            if (lane + 32 * h < n) b[lane + 32 * h] = z[h];
    }
}

template <class T>
struct SmallCholSmem {
    T col[2][kSmallN];  // column j by parity
    T lc[2][kSmallN];   // column j times 1 / l_jj, the update's factors
    T s, inv;
    int bad;
};

// Lower Cholesky in place; only the lower triangle is read or written. A diagonal with
// |d| < tiny or d < 0 sets *status = RL_ERR_DECOMP_FAILURE and leaves A as it came, as does a
// status that is set already (an earlier block's); a failure also sets *host_word (page-locked memory,
// may be null) to host_mark. The diagonal is stored as
// d / sqrt(d) (cholesky.rs:160-163).
template <class T>
static __global__ void __launch_bounds__(256) small_chol_kernel(T *A, int lda, int n, int *status, T tiny, int *host_word,
                                                                int host_mark) {
    constexpr int L = 16;
    __shared__ SmallCholSmem<T> S;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, q = tid & 3, r = tid >> 2;
    const int failed = *status;  // read with A in flight
    T a[L];
#pragma unroll
    for (int i = 0; i < L; i++) {
        const int c = 4 * i + q;
        a[i] = (r < n && c <= r) ? A[(long long)r * lda + c] : T(0);
    }
    if (failed) return;
    if (tid == 0) S.bad = 0;
    for (int jo = 0; 4 * jo < n; jo++) {
#pragma unroll
        for (int qj = 0; qj < 4; qj++) {
            const int j = 4 * jo + qj, slot = j & 1;
            if (j >= n) break;
            if (q == qj) S.col[slot][r] = a[0];
            __syncthreads();
            if (warp == (j & 7) && lane == 0) {
                const T d = S.col[slot][j];
                if (absT(d) < tiny || d < T(0)) S.bad = 1;
                const T s = sqrt(d);
                S.s = s;
                S.inv = T(1) / s;
            }
            __syncthreads();
            if (S.bad) {
                if (tid == 0) {
                    atomicCAS(status, 0, RL_ERR_DECOMP_FAILURE);
                    if (host_word) *(volatile int *)host_word = host_mark;
                }
                return;
            }
            const T s = S.s, inv = S.inv, own = S.col[slot][r];
            const bool live = r >= j && r < n;
            const T li = own * inv;  // update factors by the reciprocal; the stored entry is the quotient
            if (q == qj) S.lc[slot][r] = li;
            __syncthreads();
            if (live) {
                if (q == qj)
                    a[0] = quotient(own, s, inv);
                else if (q > qj && 4 * jo + q <= r)
                    a[0] = fma(-li, S.lc[slot][4 * jo + q], a[0]);
#pragma unroll
                for (int i = 1; i < L; i++) {
                    if (4 * (jo + i) > 8 * warp + 7) break;  // past the warp's last row
                    const int c = 4 * (jo + i) + q;
                    if (c <= r) a[i] = fma(-li, S.lc[slot][c], a[i]);
                }
            }
        }
        if (4 * jo + 4 <= n) rotate4(a);
    }
    const int done = n / 4;
#pragma unroll
    for (int i = 0; i < L; i++) {
        const int c = 4 * ((done + i) & (L - 1)) + q;
        if (r < n && c <= r) A[(long long)r * lda + c] = a[i];
    }
}

}  // namespace rl

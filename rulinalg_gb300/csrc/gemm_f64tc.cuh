// FP64 GEMM on the 5th-generation tensor cores, C = alpha op(A) op(B) + beta C, with at
// least the accuracy of the FP64 unit's dot products. GB300 runs 1.25 TFLOP/s of FP64; its
// BF16 tensor rate is 1500 times that, so a product of exact integer slices wins although it
// takes 28 BF16 products (the error-free splitting of Ozaki, Ogita, Oishi and Rump, Numer.
// Algorithms 59, 2012).
//
// Slices. Row i of op(A) is scaled by a power of two, |a_ip| < 2^E_i, and rounded to the
// fixed point Y = round(a_ip 2^(63 - E_i)), cut into 8 balanced base-256 digits
// Y = sum_t d_t 256^(7 - t), |d_t| <= 128; likewise the columns of op(B). A digit is an
// integer of at most 8 bits, exact in BF16, stored as d_t 2^(-8t). Of the digit products
// those of i + j <= 6 are kept, 28 of them (the 7 leading digits: 55 bits), or those of
// i + j <= 7, 36 of them (63 bits); group g = i + j carries the weight 2^(-14 - 8g).
// Groups 0 .. 4 are sums of integers below 2^24 in magnitude as long as a tensor-memory
// accumulator covers K <= 192 (5 pairs x 192 x 2^14 < 2^24), so FP32 accumulation is exact;
// after each 192 they are read back and added exactly into 64-bit integers, which hold the
// 2^46 sum of a 2^-E b 2^-F over 65,536 columns (MAX_K, half of their range); a longer K is cut
// into products of at most that many columns per CTA, added into C one after another. The groups
// after them share one accumulator, read back with them and summed in FP32: the tensor
// core's truncation leaves about 2^-55 2^(E_i + F_j) per 192 columns of K there, a seventh of
// that with the 36 products' read-back after every 64.
//
// Accuracy. With 28 products the rounding to 55 bits and the dropped groups leave an error
// of about sqrt(k) 2^-56 (at most 4 k 2^-56) times 2^(E_i + F_j), with 36 products 2^8
// less. With S = sum_p |a_ip b_pj| an FP64 dot product's bound is k 2^-53 S_ij; the 28 or 36
// products are used where S_ij >= 2^(E_i + F_j + 1) or 2^(E_i + F_j - 8).
// Every tile finds the smallest S_ij 2^(-E_i - F_j) of its elements first, from a ninth slice that holds |a| 2^-E and
// |b| 2^-F truncated to BF16 (a lower bound), and takes 28 or 36 products by it. A tile
// with an element below both (rows and columns whose large entries do not meet, as after
// grading or in sparse operands), with an infinity or NaN, or with a row whose largest
// entry is outside 2^(+-400), is left to the FP64 unit (gemm_left_kernel over the
// flagged tiles). Measured rms error in units of 2^-53 |A||B|, against the FP64 unit's kernel:
// N(0,1) entries, 512^2 x 256 0.18 (0.47), 2048^3 0.08 (0.47); n on the diagonal 2.0 (8.2)
// at n = 2048; lognormal entries 1.3 (11.3).
//
// Kernel: one CTA per 128 x BN tile of C; five exact accumulators and the rounded one take
// 6 BN <= 480 of the 512 tensor-memory columns, which is what limits BN to 80. K runs in
// chunks of 32 through two stages of shared memory, each holding the slice tiles of both
// operands (64-byte swizzle). A producer lane, an MMA lane (56 or 72 MMAs per chunk, all
// from one load of the 14 or 16 tiles) and 8 warps that drain the accumulators. Every
// wait is bounded (RL_ERR_TIMEOUT in the caller's status word, NaN over the tile).
#pragma once

#include <cuda_bf16.h>

#include "gemm_tc.cuh"

namespace rl {
namespace tc64 {

constexpr int BM = 128, BK = 32, STAGES = 2, NS = 8, NG = 5;  // NS digits, NG exact groups
constexpr int PLANES = NS + 1;                                // the digits and the magnitudes
constexpr int SUPER7 = 6, SUPER8 = 2;                         // K chunks per drain: 192 / 64
constexpr int A_TILE = BM * BK * 2;                           // one slice tile: 8 KB
constexpr int DRAIN_WARPS = 8, THREADS = 32 * (DRAIN_WARPS + 2);
constexpr int MAX_K = 65536;                                  // columns a 64-bit accumulator covers
constexpr int EXP_LIM = 400;
constexpr float GUARD7 = 0x1p1f, GUARD8 = 0x1p-8f;  // least S_ij 2^(-E_i - F_j) for 7 / 8 digits
template <int BN>
struct Cfg {
    static constexpr int B_TILE = BN * BK * 2;
    static constexpr int STAGE = NS * (A_TILE + B_TILE);
    static constexpr int LDS = BN + 1;  // row stride of the staged tile of C
    static constexpr int SMEM = STAGES * STAGE + 1024 + 256;
    static_assert(BM * LDS * 8 <= STAGES * STAGE, "C tile staging");
    static_assert((NG + 1) * BN <= 512, "tensor memory");
};

// largest |x| of a row as the high word of its bits (1 for a value with an empty high word)
__device__ __forceinline__ unsigned mag_key(double x) {
    const unsigned hi = (unsigned)__double2hiint(x) & 0x7fffffffu;
    return hi ? hi : (__double2loint(x) != 0 ? 1u : 0u);
}
// exponent E with |x| < 2^E for every x of the row; false: the row is not sliced
__device__ __forceinline__ bool row_exp(unsigned key, int &E) {
    E = key ? (int)(key >> 20) - 1022 : 0;
    return key == 0 || (E >= -EXP_LIM && E <= EXP_LIM);
}

// The 8 digits of x and |x| 2^-E truncated (slot 8) as BF16 bits.
__device__ __forceinline__ void digits(double x, int E, bool ok, unsigned short (&o)[PLANES]) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(x);
    int ef = (int)(b >> 52) & 0x7ff;
    unsigned long long m = b & 0xfffffffffffffull;
    const int fe = ef - E - 1023 + 127;  // BF16 exponent field of |x| 2^-E, at most 126
    o[NS] = ok && ef && fe > 0 ? (unsigned short)((fe << 7) | (int)(m >> 45)) : (unsigned short)0;
    if (ef)
        m |= 1ull << 52;
    else
        ef = 1;
    const int sh = ef - 1012 - E;  // Y = |x| 2^(63 - E) = m 2^sh, sh <= 10
    unsigned long long Y;
    if (sh >= 0)
        Y = m << (sh & 15);
    else
        Y = -sh <= 54 ? (m + (1ull << (-sh - 1))) >> -sh : 0ull;
    if (!ok) Y = 0ull;
    auto bf = [](int d, int t) {  // d 2^(-8t), exact
        const float f = __int_as_float(0x4B400000 + d) - 12582912.f;
        return (unsigned short)(__float_as_uint(f * __int_as_float((127 - 8 * t) << 23)) >> 16);
    };
    long long s = (b >> 63) ? -(long long)Y : (long long)Y;
#pragma unroll
    for (int t = NS - 1; t > 0; t--) {
        const int d = (int)((s + 128) & 255) - 128;
        o[t] = bf(d, t);
        s = (s - d) >> 8;
    }
    o[0] = bf((int)s, 0);
}

__device__ __forceinline__ uint64_t desc_sw64(uint32_t addr) {
    uint64_t d = 0;
    d |= (uint64_t)((addr >> 4) & 0x3FFFu);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(512 >> 4) << 32;  // stride byte offset: 8 rows x 64 bytes
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)4 << 61;  // layout: 64-byte swizzle
    return d;
}
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}
__device__ __forceinline__ void mma_bf16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                         uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void tma_load_3d(void *dst, const CUtensorMap *map, int x, int y, int z, uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(
            tc::smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(tc::smem_u32(bar))
        : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc::smem_u32(bar)) : "memory");
}
// 8 accumulator columns of this warp's 32 lanes; the caller waits (tmem_wait_ld).
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float (&v)[8]) {
    uint32_t r[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr));
#pragma unroll
    for (int i = 0; i < 8; i++) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// One operand as rows x k (rows of op(A), columns of op(B)): element (r, p) at
// X[r ld + p], or X[p ld + r] with `trans`.
struct Operand {
    const double *X;
    long long ld;
    int rows, trans;
    unsigned *key;       // rows: mag_key of the row's largest entry, zeroed before the pass
    __nv_bfloat16 *S;    // PLANES slices of rows x kp
    int blocks;          // of the launch's grid
};

}  // namespace tc64

// Row maxima of both operands. trans = 0: a warp per row; trans = 1: a thread per row over
// 64 values of p (consecutive threads read consecutive addresses either way).
static __global__ void __launch_bounds__(256) f64_row_max_kernel(tc64::Operand a, tc64::Operand b, int k) {
    using namespace tc64;
    const bool second = (int)blockIdx.x >= a.blocks;
    const Operand o = second ? b : a;
    const int blk = (int)blockIdx.x - (second ? a.blocks : 0);
    if (!o.trans) {
        const int lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
        for (int r = blk * wpb + (threadIdx.x >> 5); r < o.rows; r += o.blocks * wpb) {
            const double *row = o.X + (long long)r * o.ld;
            unsigned m = 0;
#pragma unroll 8
            for (int p = lane; p < k; p += 32) m = max(m, mag_key(row[p]));
            m = __reduce_max_sync(0xffffffffu, m);
            if (lane == 0) o.key[r] = m;
        }
        return;
    }
    const int cb = (o.rows + 255) / 256, kb = (k + 63) / 64;
    for (int t = blk; t < cb * kb; t += o.blocks) {
        const int r = (t % cb) * 256 + threadIdx.x, p0 = (t / cb) * 64, p1 = min(k, p0 + 64);
        if (r >= o.rows) continue;
        unsigned m = 0;
#pragma unroll 8
        for (int p = p0; p < p1; p++) m = max(m, mag_key(o.X[(long long)p * o.ld + r]));
        if (m) atomicMax(o.key + r, m);
    }
}

// The slices of both operands, K-major, zero beyond k. trans = 0: a thread takes 8
// consecutive p of a row (one 16-byte store per slice); trans = 1: 32 x 32 tiles through
// shared memory, then 4 consecutive p per thread. Bound by memory: 8 bytes in, 18 out per
// element.
static __global__ void __launch_bounds__(256) f64_slice_kernel(tc64::Operand a, tc64::Operand b, int k, int kp) {
    using namespace tc64;
    __shared__ double tile[32][33];
    const bool second = (int)blockIdx.x >= a.blocks;
    const Operand o = second ? b : a;
    const int blk = (int)blockIdx.x - (second ? a.blocks : 0), tid = threadIdx.x;
    const long long plane = (long long)o.rows * kp;
    unsigned short *S = reinterpret_cast<unsigned short *>(o.S);
    if (!o.trans) {
        const int per = kp / 8;
        const long long total = (long long)o.rows * per;
        for (long long e = (long long)blk * 256 + tid; e < total; e += (long long)o.blocks * 256) {
            const int r = (int)(e / per), p0 = (int)(e - (long long)r * per) * 8;
            const double *row = o.X + (long long)r * o.ld;
            double x[8];
#pragma unroll
            for (int u = 0; u < 8; u++) x[u] = p0 + u < k ? row[p0 + u] : 0.0;
            int E;
            const bool ok = row_exp(o.key[r], E);
            uint4 q[PLANES];
            unsigned short *qs = reinterpret_cast<unsigned short *>(q);
#pragma unroll
            for (int u = 0; u < 8; u++) {
                unsigned short d[PLANES];
                digits(x[u], E, ok, d);
#pragma unroll
                for (int t = 0; t < PLANES; t++) qs[t * 8 + u] = d[t];
            }
#pragma unroll
            for (int t = 0; t < PLANES; t++) *reinterpret_cast<uint4 *>(S + t * plane + (long long)r * kp + p0) = q[t];
        }
        return;
    }
    const int rb = (o.rows + 31) / 32, kb = kp / 32;
    for (long long t0 = blk; t0 < (long long)rb * kb; t0 += o.blocks) {
        const int r0 = (int)(t0 % rb) * 32, p0 = (int)(t0 / rb) * 32;
        __syncthreads();
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int p = p0 + (tid >> 5) + 8 * j, r = r0 + (tid & 31);
            tile[(tid >> 5) + 8 * j][tid & 31] = (p < k && r < o.rows) ? o.X[(long long)p * o.ld + r] : 0.0;
        }
        __syncthreads();
        const int r = tid >> 3, pq = (tid & 7) * 4;
        if (r0 + r < o.rows) {
            int E;
            const bool ok = row_exp(o.key[r0 + r], E);
            uint2 q[PLANES];
            unsigned short *qs = reinterpret_cast<unsigned short *>(q);
#pragma unroll
            for (int u = 0; u < 4; u++) {
                unsigned short d[PLANES];
                digits(tile[pq + u][r], E, ok, d);
#pragma unroll
                for (int t = 0; t < PLANES; t++) qs[t * 4 + u] = d[t];
            }
#pragma unroll
            for (int t = 0; t < PLANES; t++)
                *reinterpret_cast<uint2 *>(S + t * plane + (long long)(r0 + r) * kp + p0 + pq) = q[t];
        }
    }
}

// ok[tile] = 0 and *nfail for a tile left to the FP64 unit. zstride != 0: K is split over
// blockIdx.z, slice z writes its partial sums (alpha = 1, beta = 0) to C + z zstride; the
// check always covers the whole K, so all slices of a tile decide alike.
template <int BN>
static __global__ void __launch_bounds__(tc64::THREADS, 1)
    dgemm_tc_kernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB, int m, int n, int nkc, const unsigned *__restrict__ keyA, const unsigned *__restrict__ keyB, double alpha,
                    double beta, double *C, long long ldc, int lower, int *flags, int *nfail, int kc_per,
                    long long zstride, int *err, const int *stop, unsigned long long wait_ns, int withhold) {
    using namespace tc64;
    using tc::mbar_expect_tx;
    using tc::mbar_wait;
    using tc::mma_commit;
    using tc::smem_u32;
    using cfg = Cfg<BN>;
    constexpr int HC = BN / 2;  // columns per drain warp
    const int row0 = blockIdx.y * BM, col0 = blockIdx.x * BN;
    if (lower && col0 >= row0 + BM) return;
    extern __shared__ unsigned char smem_raw[];
    unsigned char *smem =
        reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + STAGES * cfg::STAGE);
    uint64_t *empty = full + STAGES;
    uint64_t *tfull = empty + STAGES;
    uint64_t *tempty = tfull + 1;
    uint64_t *drained = tempty + 1;  // after a wait that ran out: every MMA issued has completed
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(drained + 1);
    __shared__ int s_fail, s_stop;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 32) s_stop = stop ? *stop : 0;  // read while the tensor memory is allocated
    const int c_begin = blockIdx.z * kc_per;
    const int nk = max(0, min(nkc, c_begin + kc_per) - c_begin);
    C += blockIdx.z * zstride;

    if (warp == DRAIN_WARPS) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(512)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        s_fail = 0;
        for (int s = 0; s < STAGES; s++) {
            tc::mbar_init(&full[s], 1);
            tc::mbar_init(&empty[s], 1);
        }
        tc::mbar_init(tfull, 1);
        tc::mbar_init(tempty, DRAIN_WARPS);
        tc::mbar_init(drained, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;
    constexpr uint32_t idesc = idesc_bf16(BM, BN);
    if (s_stop) {  // the factorisation this product belongs to has failed
        if (warp == DRAIN_WARPS)
            asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
        return;
    }

    // Phase 1: the magnitudes' product over the whole K, a stage holding up to 8 chunks of
    // the one slice.
    const int gst = (nkc + NS - 1) / NS;  // stages it takes
    int use = 0;                          // stages filled (producer) / consumed (MMA) so far
    if (warp == DRAIN_WARPS && lane == 0) {
        for (; use < gst; use++) {
            const int s = use % STAGES, c0 = use * NS, cnt = min(NS, nkc - c0);
            if (use >= STAGES && !mbar_wait(&empty[s], (use / STAGES - 1) & 1, wait_ns)) {
                s_fail = 1;
                break;
            }
            unsigned char *st = smem + s * cfg::STAGE;
            mbar_expect_tx(&full[s], cnt * (A_TILE + cfg::B_TILE));
            for (int u = 0; u < cnt; u++) {
                tma_load_3d(st + u * A_TILE, &mapA, (c0 + u) * BK, row0, NS, &full[s]);
                tma_load_3d(st + NS * A_TILE + u * cfg::B_TILE, &mapB, (c0 + u) * BK, col0, NS, &full[s]);
            }
        }
    } else if (warp == DRAIN_WARPS + 1 && lane == 0) {
        for (; use < gst; use++) {
            const int s = use % STAGES, c0 = use * NS, cnt = min(NS, nkc - c0);
            if (!mbar_wait(&full[s], (use / STAGES) & 1, wait_ns)) {
                s_fail = 1;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t base = smem_u32(smem + s * cfg::STAGE);
            for (int u = 0; u < cnt; u++)
#pragma unroll
                for (int ks = 0; ks < BK / 16; ks++)
                    mma_bf16(tmem, desc_sw64(base + u * A_TILE + ks * 32),
                             desc_sw64(base + NS * A_TILE + u * cfg::B_TILE + ks * 32), idesc,
                             (use > 0 || u > 0 || ks > 0) ? 1u : 0u);
            mma_commit(&empty[s]);
        }
        // withhold: a test setting, this tile's first accumulators are never announced
        if ((int)(blockIdx.y * gridDim.x + blockIdx.x) != withhold) mma_commit(tfull);
    }
    __syncwarp();
    bool ok = true, seven = true;
    const int quad = warp & 3, half = warp >> 2;  // drain warps: tensor-memory lanes, column half
    const int r = row0 + quad * 32 + lane;
    const uint32_t tbase = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(half * HC);
    unsigned ka = 0;
    if (warp < DRAIN_WARPS) {
        ok = mbar_wait(tfull, 0, wait_ns);
        if (!ok) s_fail = 1;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        int E;
        ka = r < m ? keyA[r] : 0u;
        bool good = row_exp(ka, E);
        float least = INFINITY;
#pragma unroll
        for (int c = 0; c < HC; c += 8) {
            float v[8];
            tmem_ld8(tbase + c, v);
            tmem_wait_ld();
#pragma unroll
            for (int j = 0; j < 8; j++) {
                const int cc = col0 + half * HC + c + j;
                const unsigned kb = cc < n ? keyB[cc] : 0u;
                good &= row_exp(kb, E);
                if (ka != 0u && kb != 0u && !(lower && cc > r)) least = fminf(least, v[j]);
            }
        }
        ok &= good && least >= GUARD8;
        seven = least >= GUARD7;
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    }
    const bool take = __syncthreads_and(ok) != 0;
    const int ns = __syncthreads_and(seven) ? NS - 1 : NS;  // digits this tile takes
    const bool timed_out = s_fail != 0;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");

    // Phase 2: the product.
    const int super = ns == NS ? SUPER8 : SUPER7;
    int issued = use;
    if (take) {
        if (warp == DRAIN_WARPS && lane == 0) {
            for (int c = 0; c < nk; c++, use++) {
                const int s = use % STAGES;
                if (use >= STAGES && !mbar_wait(&empty[s], (use / STAGES - 1) & 1, wait_ns)) {
                    s_fail = 1;
                    break;
                }
                unsigned char *st = smem + s * cfg::STAGE;
                mbar_expect_tx(&full[s], ns * (A_TILE + cfg::B_TILE));
                const int x = (c_begin + c) * BK;
                for (int t = 0; t < ns; t++) {
                    tma_load_3d(st + t * A_TILE, &mapA, x, row0, t, &full[s]);
                    tma_load_3d(st + NS * A_TILE + t * cfg::B_TILE, &mapB, x, col0, t, &full[s]);
                }
                issued = use + 1;
            }
        } else if (warp == DRAIN_WARPS + 1 && lane == 0) {
            for (int c = 0; c < nk; c++, use++) {
                const int s = use % STAGES, in = c % super;
                // the accumulators of the chunks before have been read
                if (in == 0 && c > 0 && !mbar_wait(tempty, (c / super - 1) & 1, wait_ns)) {
                    s_fail = 1;
                    break;
                }
                if (!mbar_wait(&full[s], (use / STAGES) & 1, wait_ns)) {
                    s_fail = 1;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t base = smem_u32(smem + s * cfg::STAGE);
                // accumulator 0 .. NG - 1: the exact groups; NG: the groups after them. ks
                // outermost: a descriptor's 16 columns of K, then every pair of digits.
                for (int ks = 0; ks < BK / 16; ks++) {
                    auto pair = [&](int g, int i, uint32_t accumulate) {
                        mma_bf16(tmem + (uint32_t)((g < NG ? g : NG) * BN), desc_sw64(base + i * A_TILE + ks * 32),
                                 desc_sw64(base + NS * A_TILE + (g - i) * cfg::B_TILE + ks * 32), idesc, accumulate);
                    };
                    const uint32_t more = in > 0 || ks > 0 ? 1u : 0u;
#pragma unroll
                    for (int g = 0; g < NS - 1; g++)
#pragma unroll
                        for (int i = 0; i <= g; i++) pair(g, i, (i > 0 || g > NG) ? 1u : more);
                    if (ns == NS)
#pragma unroll
                        for (int i = 0; i < NS; i++) pair(NS - 1, i, 1u);
                }
                mma_commit(&empty[s]);
                if (in == super - 1 || c + 1 == nk) mma_commit(tfull);
            }
            if (s_fail) mma_commit(tfull);
        }
        __syncwarp();
    }
    double *stage = reinterpret_cast<double *>(smem);
    if (take && warp < DRAIN_WARPS) {
        long long acc[HC];
        float low[HC];
#pragma unroll
        for (int j = 0; j < HC; j++) acc[j] = 0, low[j] = 0.f;
        const int ndrain = (nk + super - 1) / super;
        for (int d = 0; d < ndrain; d++) {
            if (!mbar_wait(tfull, (d + 1) & 1, wait_ns)) {
                s_fail = 1;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
            for (int c = 0; c < HC; c += 8) {
                float v[NG + 1][8];
#pragma unroll
                for (int g = 0; g <= NG; g++) tmem_ld8(tbase + (uint32_t)(g * BN + c), v[g]);
                tmem_wait_ld();
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    long long t = (long long)__float2int_rn(v[0][j]) << 32;
#pragma unroll
                    for (int g = 1; g < NG; g++)
                        t += (long long)__float2int_rn(v[g][j] * (float)(1ull << (8 * g))) * (1ll << (32 - 8 * g));
                    acc[c + j] += t;
                    low[c + j] += v[NG][j];
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(tempty);
        }
        // the operand stages are no longer read (every MMA has completed): stage the tile
        int E, F;
        row_exp(ka, E);
        asm volatile("bar.sync 1, %0;" ::"r"(32 * DRAIN_WARPS) : "memory");
        const unsigned long long abits = (unsigned long long)__double_as_longlong(alpha);
#pragma unroll
        for (int j = 0; j < HC; j++) {
            const int cc = col0 + half * HC + j;
            row_exp(cc < n ? keyB[cc] : 0u, F);
            // (acc + low 2^32) alpha 2^(E + F - 46): the power of two joins alpha exactly
            const double w = fma((double)low[j], 4294967296.0, (double)acc[j]);
            const double sc =
                __longlong_as_double((long long)(abits + ((unsigned long long)(long long)(E + F - 46) << 52)));
            stage[(quad * 32 + lane) * cfg::LDS + half * HC + j] = w * sc;
        }
    }
    if (!take && !timed_out && blockIdx.z == 0 && tid == 0) {
        flags[blockIdx.y * gridDim.x + blockIdx.x] = 1;
        atomicAdd(nfail, 1);
    }
    __syncthreads();
    const bool dead = s_fail != 0;
    // no copy may land and no MMA may run after the CTA has given up its memory
    if (dead && warp == DRAIN_WARPS + 1 && lane == 0) {
        mma_commit(drained);
        mbar_wait(drained, 0, wait_ns);
    }
    if (dead && warp == DRAIN_WARPS && lane == 0)
        for (int c = max(0, issued - STAGES); c < issued; c++) mbar_wait(&full[c % STAGES], (c / STAGES) & 1, wait_ns);
    if (take || dead) {
        for (int e = tid; e < BM * BN; e += THREADS) {
            const int i = e / BN, j = e - i * BN, gi = row0 + i, gj = col0 + j;
            if (gi < m && gj < n && !(lower && gj > gi)) {
                double v = dead ? __longlong_as_double(0x7ff8000000000000ll) : stage[i * cfg::LDS + j];
                double *cp = C + (long long)gi * ldc + gj;
                if (!dead && beta != 0.0) v = fma(beta, *cp, v);
                *cp = v;
            }
        }
    }
    if (dead && tid == 0 && err) atomicCAS(err, 0, RL_ERR_TIMEOUT);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == DRAIN_WARPS)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
}

// splitk_reduce_kernel over the tiles (BM x bn, gx a row) whose flag is `want`: the ones
// the tensor cores took (0) or left (1).
static __global__ void dgemm_tc_reduce_kernel(int m, int n, int nz, double alpha, const double *__restrict__ P, double beta,
                                              double *C, long long ldc, const int *__restrict__ flags,
                                              const int *__restrict__ nfail, int bn, int gx, int want) {
    if (want && *nfail == 0) return;
    const long long total = (long long)m * n;
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(e / n), j = (int)(e - (long long)i * n);
        if (flags[(i / tc64::BM) * gx + j / bn] != want) continue;
        double sum = 0.0;
        for (int z = 0; z < nz; z++) sum += P[z * total + e];
        double *cp = C + (long long)i * ldc + j;
        double v = alpha * sum;
        if (beta != 0.0) v = fma(beta, *cp, v);
        *cp = v;
    }
}

// rows x kp slices as PLANES planes; boxes of box_rows x 32 of one plane, 64-byte swizzle.
inline rl_status make_slice_map(CUtensorMap &map, const __nv_bfloat16 *S, int rows, int kp, int box_rows) {
    auto enc = tensor_map_encoder();
    if (!enc) return RL_ERR_CUDA;
    const cuuint64_t dims[3] = {(cuuint64_t)kp, (cuuint64_t)rows, (cuuint64_t)tc64::PLANES};
    const cuuint64_t strides[2] = {(cuuint64_t)kp * 2, (cuuint64_t)kp * 2 * rows};
    const cuuint32_t box[3] = {(cuuint32_t)tc64::BK, (cuuint32_t)box_rows, 1};
    const cuuint32_t estr[3] = {1, 1, 1};
    const CUresult r = enc(&map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<__nv_bfloat16 *>(S), dims, strides, box, estr,
                           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? RL_OK : RL_ERR_CUDA;
}

// Shapes worth the tensor cores: the slicing passes (34 bytes an element of A and B), five
// launches and a tile's fixed cost against m n k on the FP64 unit. 256 x 256 with K = 64
// measured 67-83 us against 92 on the FP64 unit, 512 x 512 with K = 256 87 against 289,
// 2048^3 0.66 ms against 14.3 (26 TFLOP/s); below 6e6 multiply-adds the FP64 unit stays, or
// below 1e6 for a long K, where it has few outputs to spread (V^T A of a panel, 64 x 50 with
// K = 800: ~120 us and ~40).
inline bool dgemm_tc_eligible(int m, int n, int k) {
    return m >= 64 && n >= 32 && k >= 32 && (double)m * n * k >= (k > 512 ? 1e6 : 6e6);
}

// One CTA per tile, 1 per SM: the tile width with the smaller cost in waves of tiles.
inline int dgemm_tc_bn(int m, int n) {
    const int sms = num_sms(), rows = ceil_div(m, tc64::BM);
    const long long w80 = ceil_div((long long)rows * ceil_div(n, 80), sms) * 80LL;
    const long long w64 = ceil_div((long long)rows * ceil_div(n, 64), sms) * 72LL;  // 64-wide tiles run at 8/9 of the rate
    return w64 < w80 ? 64 : 80;
}

// Slices of K that run at once (few tiles and a long K: at least one drain each, to fill the
// SMs), and the longest K of one product, each slice within its accumulators' MAX_K columns.
inline int dgemm_tc_ksplit(int m, int n, int nkc, bool lower) {
    const int tiles = ceil_div(n, dgemm_tc_bn(m, n)) * ceil_div(m, tc64::BM);
    return lower ? 1 : std::max(1, std::min({16, num_sms() / tiles, nkc / tc64::SUPER7}));
}
inline int dgemm_tc_max_k(int m, int n, bool lower) {
    return tc64::MAX_K * dgemm_tc_ksplit(m, n, tc64::MAX_K, lower);
}

struct DgemmTcTiles {  // the tiles left to the FP64 unit
    const int *flags = nullptr, *nfail = nullptr;
    int bn = 0, gx = 0;
};

// C = alpha op(A) op(B) + beta C. `taken` = false: nothing was done (no memory for the
// slices, a stream being captured, an alpha the exponent arithmetic does not cover). `left`
// names the tiles that the caller still has to compute, on the same stream, with buffers that
// live in `ws`.
template <int BN>
static rl_status dgemm_tc_launch(int m, int n, int nkc, const CUtensorMap &mA, const __nv_bfloat16 *Sb, int kp,
                          const unsigned *keyA, const unsigned *keyB, double alpha, double beta, double *C, long long ldc,
                          bool lower, int *flags, double *part, int ks, cudaStream_t s, int *err) {
    using namespace tc64;
    static const cudaError_t attr =
        cudaFuncSetAttribute(dgemm_tc_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg<BN>::SMEM);
    RL_TRY_CUDA(attr);
    CUtensorMap mB;
    RL_TRY(make_slice_map(mB, Sb, n, kp, BN));
    dim3 grid(ceil_div(n, BN), ceil_div(m, BM), ks);
    const bool split = ks > 1;
    RL_LAUNCH(dgemm_tc_kernel<BN>, grid, THREADS, Cfg<BN>::SMEM, s, mA, mB, m, n, nkc, keyA, keyB, split ? 1.0 : alpha,
              split ? 0.0 : beta, split ? part : C, split ? (long long)n : ldc, lower ? 1 : 0, flags + 1, flags,
              ceil_div(nkc, ks), split ? (long long)m * n : 0ll, err, lower ? err : nullptr, wait_ns(),
              (int)tune(RL_TUNE_TEST_WITHHOLD_PRODUCT_TILE));
    return RL_OK;
}

template <bool TA, bool TB>
rl_status dgemm_tc(int m, int n, int k, double alpha, const double *A, long long lda, const double *B, long long ldb, double beta,
                   double *C, long long ldc, bool lower, cudaStream_t s, int *err, DevBuf<unsigned char> &ws,
                   DgemmTcTiles &left, bool &taken) {
    using namespace tc64;
    taken = false;
    const double aa = alpha < 0 ? -alpha : alpha;
    if (!(aa >= 0x1p-100 && aa <= 0x1p100)) return RL_OK;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    RL_TRY_CUDA(cudaStreamIsCapturing(s, &cap));
    if (cap != cudaStreamCaptureStatusNone) return RL_OK;
    const int sms = num_sms(), kp = ceil_div(k, BK) * BK, nkc = kp / BK;
    const int bn = dgemm_tc_bn(m, n), gx = ceil_div(n, bn), tiles = gx * ceil_div(m, BM);
    const int ks = dgemm_tc_ksplit(m, n, nkc, lower);
    if (ceil_div(nkc, ks) * BK > MAX_K) return RL_ERR_INVALID_ARG;  // the caller cuts K (dgemm_tc_max_k)
    const bool same = (const void *)A == (const void *)B && lda == ldb && m == n && TA != TB;
    auto round = [](size_t v) { return (v + 255) & ~(size_t)255; };
    const size_t key_b = round(((size_t)m + n) * 4), flag_b = round(((size_t)tiles + 1) * 4);
    const size_t a_b = round((size_t)m * kp * 2 * PLANES), b_b = same ? 0 : round((size_t)n * kp * 2 * PLANES);
    const size_t p_b = ks > 1 ? (size_t)ks * m * n * 8 : 0;
    if (ws.alloc(key_b + flag_b + a_b + b_b + p_b, s) != RL_OK) {
        cudaGetLastError();
        return RL_OK;
    }
    unsigned *key = reinterpret_cast<unsigned *>(ws.p);
    int *flags = reinterpret_cast<int *>(ws.p + key_b);
    auto *Sa = reinterpret_cast<__nv_bfloat16 *>(ws.p + key_b + flag_b);
    auto *Sb = same ? Sa : reinterpret_cast<__nv_bfloat16 *>(ws.p + key_b + flag_b + a_b);
    double *part = reinterpret_cast<double *>(ws.p + key_b + flag_b + a_b + b_b);
    RL_TRY_CUDA(cudaMemsetAsync(ws.p, 0, key_b + flag_b, s));
    auto blocks_max = [&](int rows, int trans) {
        return (int)std::min<long long>(8LL * sms, trans ? (long long)ceil_div(rows, 256) * ceil_div(k, 64) : ceil_div(rows, 8));
    };
    auto blocks_slice = [&](int rows, int trans) {
        return (int)std::min<long long>(8LL * sms, trans ? (long long)ceil_div(rows, 32) * nkc : ceil_div((long long)rows * (kp / 8), 256));
    };
    Operand a{A, lda, m, TA ? 1 : 0, key, Sa, 0}, b{B, ldb, n, TB ? 0 : 1, same ? key : key + m, Sb, 0};
    a.blocks = blocks_max(m, a.trans), b.blocks = same ? 0 : blocks_max(n, b.trans);
    RL_LAUNCH(f64_row_max_kernel, a.blocks + b.blocks, 256, 0, s, a, b, k);
    a.blocks = blocks_slice(m, a.trans), b.blocks = same ? 0 : blocks_slice(n, b.trans);
    RL_LAUNCH(f64_slice_kernel, a.blocks + b.blocks, 256, 0, s, a, b, k, kp);
    CUtensorMap mA;
    RL_TRY(make_slice_map(mA, Sa, m, kp, BM));
    RL_TRY(bn == 64 ? dgemm_tc_launch<64>(m, n, nkc, mA, Sb, kp, a.key, b.key, alpha, beta, C, ldc, lower, flags, part, ks, s,
                                               err)
                    : dgemm_tc_launch<80>(m, n, nkc, mA, Sb, kp, a.key, b.key, alpha, beta, C, ldc, lower, flags, part, ks, s,
                                               err));
    if (ks > 1)
        RL_LAUNCH(dgemm_tc_reduce_kernel, (int)std::min<long long>(4LL * sms, ((long long)m * n + 255) / 256), 256, 0, s, m, n, ks,
                  alpha, part, beta, C, ldc, flags + 1, flags, bn, gx, 0);
    left = DgemmTcTiles{flags + 1, flags, bn, gx};
    taken = true;
    return RL_OK;
}

}  // namespace rl

// FP64 superblock product on the tensor cores.
//
// GB300's FP64 pipe does 1.0-1.2 TFLOP/s, its bf16 tensor cores 1 900.  The
// dense part of the direct product (src/DMRG_SUPERBLOCK_SETUP.f90:767-796),
//     D_k = H_L(k) W_k + W_k H_R(k)^T ,   W_k = psi_k as row-major [Dl x Dr],
// is formed here from exact integer products (the error-free splitting of
// Ozaki, Ogita, Oishi and Rump, "Error-free transformations of matrix
// multiplication by using fast routines of matrix multiplication", Numer.
// Algorithms 59 (2012)):
//   * Every row of an operand gets a power of two 2^e above its largest element,
//     and each element becomes the integer nearest x 2^(61-e), written as seven
//     digits of nine bits, -256 .. 255 (the first below 128), each exact in bf16.
//   * The products of digits i and j (0 .. 6) with i + j = d <= 6 (28 pairs) are
//     accumulated in FP32 tensor memory, one accumulator per d.  They are
//     integers, exact below 2^24: over K = 64 columns (one slab) that holds for
//     d = 3 and 4, over two slabs for d = 2, over four for d = 0 and 1, whatever
//     the digits are; d = 5 and 6 (unit 2^-59 of the largest product) are read
//     every four slabs as one FP32 sum.
//   * The epilogue warps collect the weighted sums in 96 bits per output; the
//     last kernel rounds them once to FP64.
// So a product's error is one rounding plus about 2^-61 sqrt(K) (largest H in the
// row) (largest W in the column): relative to the largest elements, where a
// chain of FP64 FMAs errs relative to the products it adds.  With elements of
// one size that is less than the chain's error (against sums in FP64 pairs
// 1.3-4.9e-16 where the chains had 1.7-8.7e-16); with a graded row, or where
// large elements meet small ones only, it is more.  The solvers need no more:
// a Krylov vector is accurate relative to its norm.  A product that goes to the
// caller (nss_hv) has every element checked against sum |H||W| (k_split_size,
// k_split_terms<true>), and k_hv_fp64 sums the tiles that do not pass.
//
// What bounds it: a slab of a 128 x 64 tile is 40 MMAs (digit i of A against
// digits 0 .. 6-i of B, which lie one after the other in shared memory and land
// in the accumulators i .. 6, N <= 256), measured at ~130 cycles each for N
// from 64 to 256.  Draining the accumulators of every slab took 7 700 cycles
// (conversions), longer than the MMAs: hence the periods above.  In digit order
// the accumulator d is complete after digit d, so it is drained while the next
// digits run.
//
// Kernel: persistent, one CTA per SM, 10 warps: one lane issues the TMA copies
// (seven A digit boxes, released one by one as their MMAs finish; the seven B
// boxes double buffered), one lane the MMAs, eight warps drain.  Every wait is
// bounded as in k_sector_mma.cu.
#include "func_limits.hpp"
#include "sector_split.cuh"
#include "tc_common.cuh"

#include <algorithm>
#include <cmath>
#include <cstring>

namespace nss {

namespace {

constexpr int SP_THREADS = 320;            // producer, MMA, 8 epilogue warps
constexpr int SP_EPI0 = 2, SP_NEPI = 8;

// instruction descriptor, kind::f16: D FP32, A and B bf16, both K-major
__device__ __forceinline__ constexpr uint32_t idesc_bf16(int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(SP_M >> 4) << 24);
}

__device__ __forceinline__ void mma_bf16(uint32_t tmem, uint64_t ad, uint64_t bd, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem),
        "l"(ad), "l"(bd), "r"(idesc), "r"(acc));
}

// x as an integer multiple of 2^(e - 61), rounded to nearest (|x| < 2^e), plus
// the offset that makes all seven base-512 digits non-negative
__device__ __forceinline__ uint64_t to_fixed(double x, int e) {
    const uint64_t b = (uint64_t)__double_as_longlong(x);
    const int ex = (int)(b >> 52) & 0x7ff;
    const uint64_t man = (b & 0xfffffffffffffull) | ((uint64_t)(ex ? 1 : 0) << 52);
    // x = man 2^(max(ex,1) - 1075); shift by max(ex,1) - 1075 + 61 - e <= 8
    const int sh = (ex ? ex : 1) - 1014 - e;
    uint64_t m;
    if (sh >= 0) {
        m = man << sh;
    } else {
        const int r = -sh;
        m = r > 54 ? 0 : ((man + ((uint64_t)1 << (r - 1))) >> r);
    }
    const int64_t v = (b >> 63) ? -(int64_t)m : (int64_t)m;
    constexpr uint64_t OFFSET = 256ull * (1ull + (1ull << 9) + (1ull << 18) + (1ull << 27) + (1ull << 36) +
                                          (1ull << 45) + (1ull << 54));
    return (uint64_t)(v + (int64_t)OFFSET);
}

// digit q (0: the most significant) as bf16 bits
__device__ __forceinline__ uint32_t digit_bf16(uint64_t u, int q) {
    const uint32_t f = q == 0 ? (uint32_t)(u >> 54) : ((uint32_t)(u >> (9 * (SP_D - 1 - q))) & 511u);
    return __float_as_uint(__uint_as_float(0x4B000000u | f) - 8388864.0f) >> 16;
}

// |x| 2^-e as bf16 bits, towards zero (0 from 2^-126 on, and for subnormals)
__device__ __forceinline__ uint32_t size_bf16(double x, int e) {
    const uint32_t hi = (uint32_t)__double2hiint(x) & 0x7fffffffu;
    const int ex = (int)(hi >> 20) - 896 - e;
    return ex <= 0 || hi < 0x100000u ? 0u : ((uint32_t)ex << 7) | ((hi >> 13) & 0x7fu);
}

// high word of |x| -> scale exponent e with |x| < 2^e for the largest such word of a row
__device__ __forceinline__ int scale_exp(uint32_t hiabs) {
    const int ex = (int)(hiabs >> 20);
    if (ex >= 0x7ff) return SP_BADEXP;
    return (ex ? ex : 1) - 1022;
}

// FP32 value of x 2^-e by its bits (conversions run at the FP64 pipe's rate),
// truncated; for products that are far below FP64 rounding
__device__ __forceinline__ float trunc32(double x, int e) {
    const uint64_t b = (uint64_t)__double_as_longlong(x);
    const int ex = ((int)(b >> 52) & 0x7ff) - 896 - e;
    if (ex <= 0) return 0.f;
    const uint32_t s = (uint32_t)(b >> 32) & 0x80000000u;
    return __uint_as_float(s | ((uint32_t)min(ex, 254) << 23) | ((uint32_t)(b >> 29) & 0x7fffffu));
}

}  // namespace

// Digits of SP_ROWS rows of one operand per CTA, one warp a row.  The strip
// (rows of a row-major matrix, or its columns: kind 1) is read once into shared
// memory with all loads in flight; the row's largest high word gives the scale;
// then chunk by chunk a lane turns two elements into 2 x 7 digits, whole
// 128-byte rows per store.  Integer arithmetic only: 45 operations an element,
// and 14 bytes written.  A strip beyond SP_STRIP columns is read twice, chunk by
// chunk.
constexpr int SP_STRIP = 768;
__global__ void __launch_bounds__(32 * SP_ROWS) k_split_pack(const double *__restrict__ x, const SplitJob *__restrict__ jobs,
                                                             uint32_t *__restrict__ pool, int *__restrict__ exps,
                                                             int *__restrict__ nnzs, float *__restrict__ x32, bool sizes,
                                                             int *clear, const int *stop) {
    if (stop && *stop) return;
    if (clear && blockIdx.x == 0 && threadIdx.x < SP_REDO_LIST) clear[threadIdx.x] = 0;
    extern __shared__ double strip[];
    const SplitJob J = jobs[blockIdx.x];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const double *X = x + J.src;
    const int r = J.r0 + warp;                       // the warp's row
    const bool on = r < J.rows;
    const int nch = (J.k + SP_KC - 1) / SP_KC;
    const int part = J.k <= SP_STRIP ? J.k : SP_KC;  // columns staged at once
    const int ld = part | 1;
    const double *mine = strip + warp * ld;
    auto load = [&](int k0, int kn) {
        if (J.kind == 0) {
            if (on)
#pragma unroll 8
                for (int k = lane; k < kn; k += 32) strip[warp * ld + k] = X[(int64_t)r * J.ld + k0 + k];
        } else {
            const int c = threadIdx.x % SP_ROWS;
            const bool in = J.r0 + c < J.rows;
#pragma unroll 8
            for (int k = threadIdx.x / SP_ROWS; k < kn; k += 32)
                strip[c * ld + k] = in ? X[(int64_t)(k0 + k) * J.ld + J.r0 + c] : 0.0;
        }
    };
    uint32_t m = 0;
    int cnt = 0;                                     // the row's nonzero elements
    for (int k0 = 0; k0 < J.k; k0 += part) {
        const int kn = min(part, J.k - k0);
        if (k0) __syncthreads();
        load(k0, kn);
        __syncthreads();
        if (on)
            for (int k = lane; k < kn; k += 32) {
                const uint32_t hi = (uint32_t)__double2hiint(mine[k]) & 0x7fffffffu;
                m = max(m, hi);
                cnt += (hi | (uint32_t)__double2loint(mine[k])) != 0;
            }
    }
    m = __reduce_max_sync(0xffffffffu, m);
    cnt = __reduce_add_sync(0xffffffffu, cnt);
    const int e = cnt ? scale_exp(m) : SP_ZEROEXP;
    const bool live = e < SP_BADEXP && e > SP_ZEROEXP;   // else the digits are zeros
    if (on && lane == 0) {
        exps[J.exp + r] = e;
        nnzs[J.exp + r] = cnt;
    }
    for (int c = 0; c < nch; ++c) {
        int k0 = c * SP_KC, kn = min(SP_KC, J.k - k0), at = k0;
        if (J.k > SP_STRIP) {
            __syncthreads();
            load(k0, kn);
            __syncthreads();
            at = 0;
        }
        if (!on) continue;
        const double a = 2 * lane < kn ? mine[at + 2 * lane] : 0.0, b = 2 * lane + 1 < kn ? mine[at + 2 * lane + 1] : 0.0;
        uint64_t ua = 0, ub = 0;
        if (live) {
            ua = to_fixed(a, e);
            ub = to_fixed(b, e);
        }
        if (sizes)
            pool[((int64_t)J.abs + (int64_t)c * J.rows + r) * (SP_KC / 2) + lane] =
                live ? (size_bf16(a, e) | (size_bf16(b, e) << 16)) : 0u;
        if (x32 && J.kind == 0) {
            float *o = x32 + J.src + (int64_t)r * J.ld + k0 + 2 * lane;
            if (2 * lane < kn) o[0] = live ? trunc32(a, e) : 0.f;
            if (2 * lane + 1 < kn) o[1] = live ? trunc32(b, e) : 0.f;
        }
#pragma unroll
        for (int q = 0; q < SP_D; ++q)
            pool[((int64_t)J.row + (int64_t)(c * SP_D + q) * J.rows + r) * (SP_KC / 2) + lane] =
                live ? (digit_bf16(ua, q) | (digit_bf16(ub, q) << 16)) : 0u;
    }
}

namespace {

template <int BN>
struct SplitCfg {
    static constexpr int A_BYTES = SP_M * 128, B_BYTES = BN * 128;      // one digit box
    static constexpr int SMEM = SP_D * A_BYTES + 2 * SP_D * B_BYTES + 1024;
    static constexpr int HALF = BN / 2;
    static constexpr uint32_t TCOLS = BN == 64 ? 512 : 256;
    static_assert(SMEM <= 232448 - 256, "shared memory plan");
};

__device__ __forceinline__ void tmem_ld16(uint32_t addr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(addr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

}  // namespace

template <int BN>
__global__ void __launch_bounds__(SP_THREADS, 1) k_sector_split(const __grid_constant__ CUtensorMap map_a,
                                                                 const __grid_constant__ CUtensorMap map_b,
                                                                 const SplitItem *__restrict__ items,
                                                                 const int2 *__restrict__ ranges,
                                                                 int64_t *__restrict__ out, int *__restrict__ out0,
                                                                 int64_t plane, uint32_t spin, int *err, const int *stop) {
    using C = SplitCfg<BN>;
    if (stop && *stop) return;   // before any TMEM allocation: uniform exit
    extern __shared__ uint8_t sp_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)sp_raw + 1023) & ~(uintptr_t)1023);
    uint8_t *sa = smem, *sbuf = smem + SP_D * C::A_BYTES;
    __shared__ __align__(8) uint64_t fulla[SP_D], emptya[SP_D], fullb[2], emptyb[2], tfull[SP_D], tempty, drain;
    __shared__ uint32_t tmem_base;
    __shared__ int abort_s;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int2 rg = ranges[blockIdx.x];
    if (threadIdx.x == 0) {
        for (int q = 0; q < SP_D; ++q) {
            mbar_init(smem_u32(&fulla[q]), 1);
            mbar_init(smem_u32(&emptya[q]), 1);
            mbar_init(smem_u32(&tfull[q]), 1);
        }
        for (int q = 0; q < 2; ++q) {
            mbar_init(smem_u32(&fullb[q]), 1);
            mbar_init(smem_u32(&emptyb[q]), 1);
        }
        mbar_init(smem_u32(&tempty), SP_NEPI);
        mbar_init(smem_u32(&drain), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"((uint64_t)&map_a) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"((uint64_t)&map_b) : "memory");
        abort_s = 0;
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base)),
                     "r"(C::TCOLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_base;
    volatile int *abort = &abort_s;
    const uint32_t drain_spin = spin > (1u << 22) ? spin : (1u << 22);
    auto give_up = [&]() {
        *abort = 1;
        atomicExch(err, 1);
    };
    auto slabs = [](int k) { return (k + SP_KC - 1) / SP_KC; };
    // slab c of nk: is accumulator d read after it? (see the periods above)
    auto due = [](int d, int c, int nk) {
        return c == nk - 1 || d == 3 || d == 4 || (d == 2 ? (c & 1) == 1 : (c & 3) == 3);
    };

    if (warp == 0 && lane == 0) {
        // ---- TMA producer
        int it = 0;                   // slabs issued
        int na = 0, nb = 0;           // A boxes and B buffers issued
        bool ok = true;
        for (int i = rg.x; i < rg.y && ok && !*abort; ++i) {
            const SplitItem m = items[i];
            const int nk = slabs(m.k);
            for (int c = 0; c < nk && ok; ++c, ++it) {
                const int bs = it & 1;
                if (!mbar_wait(smem_u32(&emptyb[bs]), ((uint32_t)(it >> 1) & 1u) ^ 1u, spin, abort)) { give_up(); ok = false; break; }
                const uint32_t fb = smem_u32(&fullb[bs]);
                mbar_expect_tx(fb, (uint32_t)(SP_D * C::B_BYTES));
                for (int q = 0; q < SP_D; ++q)
                    tma_load_2d(smem_u32(sbuf + (size_t)(bs * SP_D + q) * C::B_BYTES), &map_b, 0,
                                m.b_row + (c * SP_D + q) * m.b_rows + m.n0, fb);
                ++nb;
                for (int q = 0; q < SP_D; ++q) {
                    if (!mbar_wait(smem_u32(&emptya[q]), ((uint32_t)it & 1u) ^ 1u, spin, abort)) { give_up(); ok = false; break; }
                    const uint32_t fa = smem_u32(&fulla[q]);
                    mbar_expect_tx(fa, (uint32_t)C::A_BYTES);
                    tma_load_2d(smem_u32(sa + (size_t)q * C::A_BYTES), &map_a, 0, m.a_row + (c * SP_D + q) * m.a_rows + m.m0, fa);
                    ++na;
                }
            }
        }
        // no copy of this CTA may still be landing when it leaves (bounded, by a
        // limit of its own, and not cut short by the abort flag)
        volatile int never = 0;
        for (int q = 0; q < SP_D; ++q) {
            const int fills = na / SP_D + (q < na % SP_D ? 1 : 0);
            if (fills && !mbar_wait(smem_u32(&fulla[q]), (uint32_t)(fills - 1) & 1u, drain_spin, &never)) atomicExch(err, 1);
        }
        for (int q = 0; q < 2; ++q) {
            const int fills = (nb + 1 - q) / 2;
            if (fills && !mbar_wait(smem_u32(&fullb[q]), (uint32_t)(fills - 1) & 1u, drain_spin, &never)) atomicExch(err, 1);
        }
    } else if (warp == 1 && lane == 0) {
        // ---- MMA issuer
        int it = 0;
        bool issued = false, ok = true;
        for (int i = rg.x; i < rg.y && ok && !*abort; ++i) {
            const int k = items[i].k, nk = slabs(k);
            for (int c = 0; c < nk && ok; ++c, ++it) {
                const int bs = it & 1;
                const int ks = min(SP_KC / 16, (k - c * SP_KC + 15) / 16);   // K steps with anything in them
                if (!mbar_wait(smem_u32(&tempty), ((uint32_t)it & 1u) ^ 1u, spin, abort) ||
                    !mbar_wait(smem_u32(&fullb[bs]), (uint32_t)(it >> 1) & 1u, spin, abort)) {
                    give_up();
                    ok = false;
                    break;
                }
                const uint32_t b0 = smem_u32(sbuf + (size_t)bs * SP_D * C::B_BYTES);
#pragma unroll
                for (int q = 0; q < SP_D; ++q) {
                    if (!mbar_wait(smem_u32(&fulla[q]), (uint32_t)it & 1u, spin, abort)) {
                        give_up();
                        ok = false;
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t a0 = smem_u32(sa + (size_t)q * C::A_BYTES);
                    // digit q of A against digits 0 .. 6-q of B: accumulators
                    // q .. 6, n0 columns on from there
                    auto mma = [&](int kk, int n0, int n, uint32_t acc) {
                        mma_bf16(tmem + (uint32_t)(q * BN + n0), desc_sw128(a0 + kk * 32),
                                 desc_sw128(b0 + (uint32_t)n0 * 128 + kk * 32), idesc_bf16(n), acc);
                    };
                    const int n = (SP_D - q) * BN;
                    for (int kk = 0; kk < ks; ++kk) {
                        if (q == 0 && kk == 0 && (c & 3) != 0) {
                            // accumulators that go on (d = 0, 1, 5, 6, and 2 in odd
                            // slabs) beside those that start over
                            const int d0 = (c & 1) ? 3 : 2;
                            mma(0, 0, d0 * BN, 1u);
                            mma(0, d0 * BN, (5 - d0) * BN, 0u);
                            mma(0, 5 * BN, 2 * BN, 1u);
                            continue;
                        }
                        const uint32_t acc = (q > 0 || kk > 0) ? 1u : 0u;
#pragma unroll
                        for (int n0 = 0; n0 < n; n0 += 256) mma(kk, n0, min(256, n - n0), acc);
                    }
                    issued = true;
                    mma_commit(smem_u32(&emptya[q]));   // this A box may be refilled
                    if (due(q, c, nk)) mma_commit(smem_u32(&tfull[q]));   // ... and accumulator q is complete
                }
                if (ok) mma_commit(smem_u32(&emptyb[bs]));
            }
        }
        if (issued) {   // every MMA of this lane done before the CTA frees its TMEM
            mma_commit(smem_u32(&drain));
            volatile int never = 0;
            if (!mbar_wait(smem_u32(&drain), 0u, drain_spin, &never)) atomicExch(err, 1);
        }
    } else if (warp >= SP_EPI0) {
        // ---- epilogue: warp w owns TMEM lanes 32 (w % 4) .. +31 (its rows) and
        // half of the columns
        const int qr = warp & 3, h = (warp - SP_EPI0) >> 2;
        const uint32_t tq = tmem + ((uint32_t)(32 * qr) << 16) + (uint32_t)(h * C::HALF);
        uint32_t par[SP_D];           // parities of the next completion of each accumulator
#pragma unroll
        for (int d = 0; d < SP_D; ++d) par[d] = 0u;
        for (int i = rg.x; i < rg.y && !*abort; ++i) {
            const SplitItem m = items[i];
            const int nk = slabs(m.k);
            // the output is (s0 2^42 + sum) 2^-6 units of d = 4
            int s0[C::HALF];
            int64_t sum[C::HALF];
#pragma unroll
            for (int j = 0; j < C::HALF; ++j) sum[j] = s0[j] = 0;
            bool ok = true;
            for (int c = 0; c < nk && ok; ++c) {
                auto ready = [&](int d) -> bool {
                    bool got = true;
                    if (lane == 0) got = mbar_wait(smem_u32(&tfull[d]), par[d], spin, abort);
                    par[d] ^= 1u;
                    if (__shfl_sync(0xffffffffu, got ? 1 : 0, 0) == 0) {
                        if (lane == 0) give_up();
                        return false;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    return true;
                };
#pragma unroll
                for (int d = 0; d < 5; ++d) {
                    if (!ok || !due(d, c, nk)) continue;
                    if (!(ok = ready(d))) continue;
#pragma unroll
                    for (int c0 = 0; c0 < C::HALF; c0 += 16) {
                        uint32_t r[16];
                        tmem_ld16(tq + (uint32_t)(d * BN + c0), r);
#pragma unroll
                        for (int j = 0; j < 16; ++j) {
                            const int x = __float2int_rn(__uint_as_float(r[j]));
                            if (d == 0) s0[c0 + j] += x;
                            else sum[c0 + j] += (int64_t)x * (int64_t)(1ll << (42 - 9 * d));
                        }
                    }
                }
                if (ok && due(5, c, nk)) {
                    ok = ready(5) && ready(6);
                    if (ok)
#pragma unroll
                        for (int c0 = 0; c0 < C::HALF; c0 += 16) {
                            uint32_t r5[16], r6[16];
                            tmem_ld16(tq + (uint32_t)(5 * BN + c0), r5);
                            tmem_ld16(tq + (uint32_t)(6 * BN + c0), r6);
#pragma unroll
                            for (int j = 0; j < 16; ++j)
                                sum[c0 + j] += __float2int_rn(fmaf(__uint_as_float(r6[j]), 0x1p-12f, __uint_as_float(r5[j]) * 0x1p-3f));
                        }
                }
                if (!ok) break;
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&tempty));
            }
            if (!ok) break;
            const int il = m.m0 + 32 * qr + lane, ir0 = m.n0 + h * C::HALF;
            if (il < m.dl) {
                // the planes are column-major: a warp's 32 rows of a column are
                // one run (row-major, a lane writing its own row, took 16 000
                // cycles an item)
                const int64_t o = (int64_t)m.plane * plane + m.off + (int64_t)ir0 * m.dl + il;
#pragma unroll
                for (int j = 0; j < C::HALF; ++j)
                    if (ir0 + j < m.dr) {
                        out[o + (int64_t)j * m.dl] = sum[j];
                        out0[o + (int64_t)j * m.dl] = s0[j];
                    }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(C::TCOLS));
}

// sum |H||W| of every output, in units of the operands' scales and a little
// below (bf16 towards zero, FP32 sums): the products of the absolute values, 128
// x sn outputs a tile (an MMA takes ~130 cycles whatever its width).  One lane
// issues the copies (four slabs of A and B in flight), one the MMAs, four warps
// store.  Waits are bounded as in k_sector_split.
namespace {
constexpr int SZ_THREADS = 192, SZ_STAGES = 4;
struct SizeCfg {
    static constexpr int A_BYTES = SP_M * 128, B_BYTES = SP_SN * 128;
    static constexpr int SMEM = SZ_STAGES * (A_BYTES + B_BYTES) + 1024;
    static_assert(SMEM <= 232448 - 256, "shared memory plan");
};
}  // namespace

__global__ void __launch_bounds__(SZ_THREADS, 1) k_split_size(const __grid_constant__ CUtensorMap map_a,
                                                               const __grid_constant__ CUtensorMap map_b,
                                                               const SplitItem *__restrict__ items,
                                                               const int2 *__restrict__ ranges, float *__restrict__ out,
                                                               int64_t plane, int sn, uint32_t spin, int *err, const int *stop) {
    using C = SizeCfg;
    if (stop && *stop) return;   // before any TMEM allocation: uniform exit
    extern __shared__ uint8_t sp_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)sp_raw + 1023) & ~(uintptr_t)1023);
    __shared__ __align__(8) uint64_t full[SZ_STAGES], empty[SZ_STAGES], tfull, tempty, drain;
    __shared__ uint32_t tmem_base;
    __shared__ int abort_s;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int2 rg = ranges[blockIdx.x];
    if (threadIdx.x == 0) {
        for (int q = 0; q < SZ_STAGES; ++q) {
            mbar_init(smem_u32(&full[q]), 1);
            mbar_init(smem_u32(&empty[q]), 1);
        }
        mbar_init(smem_u32(&tfull), 1);
        mbar_init(smem_u32(&tempty), 4);
        mbar_init(smem_u32(&drain), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        abort_s = 0;
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base)),
                     "r"((uint32_t)SP_SN));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_base;
    volatile int *abort = &abort_s;
    const uint32_t drain_spin = spin > (1u << 22) ? spin : (1u << 22);
    auto give_up = [&]() {
        *abort = 1;
        atomicExch(err, 1);
    };
    auto slabs = [](int k) { return (k + SP_KC - 1) / SP_KC; };
    auto abox = [&](int st) { return smem_u32(smem + (size_t)st * (C::A_BYTES + C::B_BYTES)); };
    // columns of an item's tile, a multiple of 16
    auto width = [&](const SplitItem &m) { return min(sn, (m.dr - m.n0 + 15) & ~15); };

    if (warp == 0 && lane == 0) {
        // ---- TMA producer
        int it = 0, issued = 0;
        bool ok = true;
        for (int i = rg.x; i < rg.y && ok && !*abort; ++i) {
            const SplitItem m = items[i];
            for (int c = 0; c < slabs(m.k); ++c, ++it) {
                const int st = it % SZ_STAGES;
                if (!mbar_wait(smem_u32(&empty[st]), ((uint32_t)(it / SZ_STAGES) & 1u) ^ 1u, spin, abort)) { give_up(); ok = false; break; }
                const uint32_t fb = smem_u32(&full[st]);
                mbar_expect_tx(fb, (uint32_t)(C::A_BYTES + sn * 128));
                tma_load_2d(abox(st), &map_a, 0, m.a_row + c * m.a_rows + m.m0, fb);
                tma_load_2d(abox(st) + C::A_BYTES, &map_b, 0, m.b_row + c * m.b_rows + m.n0, fb);
                ++issued;
            }
        }
        // no copy of this CTA may still be landing when it leaves
        volatile int never = 0;
        for (int q = 0; q < SZ_STAGES; ++q) {
            const int fills = (issued + SZ_STAGES - 1 - q) / SZ_STAGES;
            if (fills && !mbar_wait(smem_u32(&full[q]), (uint32_t)(fills - 1) & 1u, drain_spin, &never)) atomicExch(err, 1);
        }
    } else if (warp == 1 && lane == 0) {
        // ---- MMA issuer
        int it = 0;
        bool issued = false, ok = true;
        for (int i = rg.x; i < rg.y && ok && !*abort; ++i) {
            const SplitItem m = items[i];
            const int nk = slabs(m.k);
            if (!mbar_wait(smem_u32(&tempty), ((uint32_t)(i - rg.x) & 1u) ^ 1u, spin, abort)) { give_up(); break; }
            for (int c = 0; c < nk; ++c, ++it) {
                const int st = it % SZ_STAGES;
                if (!mbar_wait(smem_u32(&full[st]), (uint32_t)(it / SZ_STAGES) & 1u, spin, abort)) { give_up(); ok = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const int ks = min(SP_KC / 16, (m.k - c * SP_KC + 15) / 16);   // K steps with anything in them
                for (int kk = 0; kk < ks; ++kk)
                    mma_bf16(tmem, desc_sw128(abox(st) + kk * 32), desc_sw128(abox(st) + C::A_BYTES + kk * 32),
                             idesc_bf16(width(m)), c > 0 || kk > 0 ? 1u : 0u);
                issued = true;
                mma_commit(smem_u32(&empty[st]));
            }
            if (ok) mma_commit(smem_u32(&tfull));
        }
        if (issued) {   // every MMA of this lane done before the CTA frees its TMEM
            mma_commit(smem_u32(&drain));
            volatile int never = 0;
            if (!mbar_wait(smem_u32(&drain), 0u, drain_spin, &never)) atomicExch(err, 1);
        }
    } else if (warp >= 2) {
        // ---- warp w stores the rows of TMEM lanes 32 (w % 4) .. +31
        const int qr = warp & 3;
        for (int i = rg.x; i < rg.y && !*abort; ++i) {
            const SplitItem m = items[i];
            bool got = true;
            if (lane == 0) got = mbar_wait(smem_u32(&tfull), (uint32_t)(i - rg.x) & 1u, spin, abort);
            if (__shfl_sync(0xffffffffu, got ? 1 : 0, 0) == 0) {
                if (lane == 0) give_up();
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int il = m.m0 + 32 * qr + lane;
            float *o = out + (int64_t)m.plane * plane + m.off + (int64_t)m.n0 * m.dl + il;
            for (int c0 = 0; c0 < width(m); c0 += 16) {
                uint32_t r[16];
                tmem_ld16(tmem + ((uint32_t)(32 * qr) << 16) + (uint32_t)c0, r);
                if (il < m.dl)
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        if (m.n0 + c0 + j < m.dr) o[(int64_t)(c0 + j) * m.dl] = __uint_as_float(r[j]);
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&tempty));
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)SP_SN));
}

// hv = plane 0 + plane 1 (rounded to FP64) + sum_t A W_q B^T, one CTA per 8 x
// 32 outputs of a sector, a warp a row.  Per term A's row and B's columns give
// their dominant (column, value).  The entries of A's row beside it (below 2^-40
// of A's largest: rounding left by the renormalisation, up to a block sector's
// width of them) are summed in FP32 against the FP32 copy of W, which is scaled
// by its rows' powers of two: an error of 2^-61 of A's largest times W's.  A lane holds one
// such entry, its gather is broadcast, eight gathers in flight.  Two FP64
// operations a term and output, spread over all SMs (in the GEMM's epilogue
// they would hold one SM's FP64 pipe for 8 us a tile); the chain of dependent
// loads bounds it, hence the tile and term records.
//
// GUARD (a product for the caller): a side of an element passes when the error
// that the digits leave in it, 2^-61.3 sqrt(nonzero products) 2^e for a row and a
// column of scale 2^e (the six digit products of i + j = 7 that are dropped, 148
// rms a digit), is below 2^-53 of the element's sum |H||W| over both sides, one
// rounding of a sum of that size.  The small entries of A pass when what FP32
// leaves of them is below 2^-53 of the dominant products' sizes and the dense
// part.  Elements that rows with an Inf or NaN enter do not pass.  Tiles of 4 x 8
// that hold one that does not go to the list of k_hv_fp64, which sums the terms
// and the sides that failed.
constexpr float SP_PASS = 0.0032f;               // 2^(53 - 61.3)
constexpr int SP_LOWEXP = -960;                  // 2^-61 of it is FP64's smallest normal number
struct SplitTerms {
    const SplitTerm *terms;
    const int *tcol, *dptr, *dcol, *exps, *nnzs;
    const float *size;
    int *redo;
    const double *tval;
    const float *dval;
    const DevTerm *csr;
    const int *ab_rp, *ab_col;
    const double *ab_val;
};

template <bool GUARD>
__global__ void __launch_bounds__(256, 4) k_split_terms(const double *__restrict__ v, const float *__restrict__ v32,
                                                     const int64_t *__restrict__ planes,
                                                     const int *__restrict__ planes0, int64_t n, double *__restrict__ hv,
                                                     const SplitTile *__restrict__ tiles, SplitTerms T, const int *stop) {
    if (stop && *stop) return;
    __shared__ double dense[8][33];
    __shared__ unsigned failed;                      // tiles of k_hv_fp64 with something that does not pass (left, right << 8, terms << 16)
    if (GUARD && threadIdx.x == 0) failed = 0;
    if (GUARD) __syncthreads();
    const SplitTile t = tiles[blockIdx.x];
    {   // the two planes (column-major), eight rows of four columns a warp
        const int r = threadIdx.x & 7, c = threadIdx.x >> 3, il = t.row0 + r, ir = t.col0 + c;
        const bool in = il < t.dl && ir < t.dr;
        double x = 0.0;
        if (in) {
            const int64_t e = t.off + (int64_t)ir * t.dl + il;
            const int64_t p0 = planes[e], p1 = planes[n + e];
            const int q0 = planes0[e], q1 = planes0[n + e];
            // H_L row, W column; W row, H_R row
            const int i0 = t.exp + il, i1 = t.exp + 2 * t.dl + t.dr + ir, i2 = t.exp + t.dl + t.dr + il, i3 = t.exp + t.dl + ir;
            const int x0 = T.exps[i0], x1 = T.exps[i1], y0 = T.exps[i2], y1 = T.exps[i3];
            const bool bad = x0 >= SP_BADEXP || x1 >= SP_BADEXP || y0 >= SP_BADEXP || y1 >= SP_BADEXP;
            x = bad ? __longlong_as_double(0x7ff8000000000000ll)
                    : fixed_to_double(q0, p0, x0 + x1 - 56) + fixed_to_double(q1, p1, y0 + y1 - 56);
            if constexpr (GUARD) {
                // both sides in units of the larger scale (a row of zeros: nothing)
                const bool zl = min(x0, x1) == SP_ZEROEXP, zr = min(y0, y1) == SP_ZEROEXP;
                const int el = zl ? SP_ZEROEXP : x0 + x1, er = zr ? SP_ZEROEXP : y0 + y1, em = max(el, er);
                auto unit = [&](bool z, int d) { return z || d < -126 ? 0.f : __int_as_float((127 + d) << 23); };
                const float fl = unit(zl, el - em), fr = unit(zr, er - em);
                const float sum = fl * T.size[e] + fr * T.size[n + e];
                // planes of this scale may round to a subnormal, which fixed_to_double
                // does not give; above it what it drops is below the digits' error
                const bool low = (!zl && el < SP_LOWEXP) || (!zr && er < SP_LOWEXP);
                const bool left = bad || low || sum < SP_PASS * fl * sqrtf((float)min(T.nnzs[i0], T.nnzs[i1]));
                const bool right = bad || low || sum < SP_PASS * fr * sqrtf((float)min(T.nnzs[i2], T.nnzs[i3]));
                if (left || right) atomicOr(&failed, (left ? 1u : 0u) << ((r / 4) * 4 + c / 8) | (right ? 0x100u : 0u) << ((r / 4) * 4 + c / 8));
            }
        }
        dense[r][c] = x;
    }
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const int il = t.row0 + (threadIdx.x >> 5), ir = t.col0 + lane;
    if (il < t.dl) {                                 // whole warps
        const bool in = ir < t.dr;
        const int64_t e0 = t.off + (int64_t)il * t.dr + ir;
        double acc = 0.0;
        double rest = 0.0, sizes = 0.0;              // error of the small entries' sums; |dominant products|
        bool dusty = false;
        // the dominant entries, four terms' loads in flight
        for (int tb = t.t0; tb < t.t1; tb += 4) {
            SplitTerm tm[4];
            int aj[4], bj[4];
            double c[4], w[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) tm[q] = T.terms[min(tb + q, t.t1 - 1)];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const bool on = tb + q < t.t1 && !tm[q].general;
                dusty = dusty || tm[q].general || tm[q].dust >= 0;
                aj[q] = on ? T.tcol[tm[q].a + il] : -1;
                bj[q] = on && in ? T.tcol[tm[q].b + ir] : -1;
                c[q] = (on ? T.tval[tm[q].a + il] : 0.0) * (on && in ? T.tval[tm[q].b + ir] : 0.0);
            }
#pragma unroll
            for (int q = 0; q < 4; ++q)
                w[q] = aj[q] >= 0 && bj[q] >= 0 ? v[tm[q].off + (int64_t)aj[q] * tm[q].drq + bj[q]] : 0.0;
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (aj[q] >= 0 && bj[q] >= 0) acc = fma(c[q], w[q], acc);
        }
        if (dusty)
            for (int ti = t.t0; ti < t.t1; ++ti) {
                const SplitTerm tm = T.terms[ti];
                if (tm.general) {                        // several sizeable entries in a row: the CSR loop
                    if (!in) continue;
                    const DevTerm c = T.csr[tm.term];
                    const double *W = v + tm.off;
                    for (int ja = T.ab_rp[c.a_rp + il]; ja < T.ab_rp[c.a_rp + il + 1]; ++ja) {
                        const int64_t row = (int64_t)T.ab_col[ja] * tm.drq;
                        double cb = 0.0;
                        for (int jb = T.ab_rp[c.b_rp + ir]; jb < T.ab_rp[c.b_rp + ir + 1]; ++jb)
                            cb = fma(T.ab_val[jb], W[row + T.ab_col[jb]], cb);
                        acc = fma(T.ab_val[ja], cb, acc);
                    }
                    continue;
                }
                const int bj = in ? T.tcol[tm.b + ir] : -1;
                if (GUARD && bj >= 0 && T.tcol[tm.a + il] >= 0)
                    sizes = fma(fabs(T.tval[tm.a + il] * T.tval[tm.b + ir]), fabs(v[tm.off + (int64_t)T.tcol[tm.a + il] * tm.drq + bj]), sizes);
                if (tm.dust < 0) continue;
                const int p0 = T.dptr[tm.dust + il], p1 = T.dptr[tm.dust + il + 1];   // uniform over the warp
                const float *W32 = v32 + tm.off + max(bj, 0);
                for (int p = p0; p < p1; p += 32) {
                    const int cnt = min(32, p1 - p);
                    const int dc = lane < cnt ? T.dcol[p + lane] : 0;
                    const int ex = lane < cnt ? T.exps[tm.ew + dc] : SP_ZEROEXP;
                    // powers of two of the input rows relative to the largest of them
                    const int top = __reduce_max_sync(0xffffffffu, ex);
                    const float dx = lane < cnt ? T.dval[p + lane] : 0.f;
                    float dv = 0.f;
                    if (ex - top > -120) dv = dx * __int_as_float((127 + ex - top) << 23);
                    const int at = dc * tm.drq;
                    float s = 0.f, size = 0.f;
                    for (int u = 0; u < cnt; u += 8) {
                        float g[8];
#pragma unroll
                        for (int q = 0; q < 8; ++q) g[q] = W32[__shfl_sync(0xffffffffu, at, u + q)];
#pragma unroll
                        for (int q = 0; q < 8; ++q) {
                            const float a = __shfl_sync(0xffffffffu, dv, u + q);
                            s = fmaf(a, g[q], s);
                            if (GUARD) size = fmaf(fabsf(a), fabsf(g[q]), size);
                        }
                    }
                    if (top >= SP_BADEXP) {              // a row with an Inf or NaN
                        if (bj >= 0) acc = rest = __longlong_as_double(0x7ff8000000000000ll);
                        continue;
                    }
                    if constexpr (GUARD) {
                        // FP32 sums of 32 truncated elements: 2^-20 of their size; what
                        // lies 2^-120 below the largest row is left out, and a sum
                        // below FP32's normal range
                        const float most = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(fabsf(dx))));
                        const float lost = fmaf(0x1p-114f, most, 0x1p-126f);
                        const double unit = __hiloint2double(min(max(top + 1023, 1), 2046) << 20, 0);
                        if (bj >= 0 && top > SP_ZEROEXP) rest = fma((double)fmaf(size, 0x1p-20f, lost) * unit, fabs(T.tval[tm.b + ir]), rest);
                    }
                    if (bj >= 0 && s != 0.f) {
                        // s 2^top as a double by its bits (s is normal or negligible)
                        const uint32_t b = __float_as_uint(s);
                        const int e = (int)((b >> 23) & 0xff) - 127 + top + 1023;
                        if (e > 0 && e < 2047 && ((b >> 23) & 0xff))
                            acc = fma(__hiloint2double((int)((b & 0x80000000u) | ((uint32_t)e << 20) | ((b & 0x7fffffu) >> 3)),
                                                       (int)(b << 29)),
                                      T.tval[tm.b + ir], acc);
                        else if (GUARD && e <= 0)
                            rest += 0x1p-1022;
                    }
                }
            }
        if (GUARD && dusty && in && !(rest <= 0x1p-53 * (sizes + fabs(dense[threadIdx.x >> 5][lane]))))
            atomicOr(&failed, 0x10000u << ((threadIdx.x >> 7) * 4 + lane / 8));
        if (in) hv[e0] = dense[threadIdx.x >> 5][lane] + acc;
    }
    if constexpr (GUARD) {
        __syncthreads();
        if (threadIdx.x < 8) {
            const unsigned f = failed >> threadIdx.x;
            if (f & 0x10101u)
                T.redo[SP_REDO_LIST + atomicAdd(T.redo + SP_REDO_COUNT, 1)] =
                    (blockIdx.x * 8 + threadIdx.x) * 4 + (f & 1) + (f >> 7 & 2);
        }
    }
}

// ---------------------------------------------------------------------------
// Host side

bool split_wanted(const DevSb &s) {
    for (int k = 0; k < s.nsb; ++k)
        if (s.dls[k] > SP_KMAX || s.drs[k] > SP_KMAX) return false;
    const char *e = std::getenv("NSS_SPLIT64");
    return e ? std::atoi(e) != 0 : s.flops_dense >= 4e7;
}

void split_layout(const DevSb &s, const std::vector<int> &rowptr, const std::vector<int> &col,
                  const std::vector<double> &val, const std::vector<int> &csr, int nsm, SplitPlan &p) {
    p = SplitPlan{};
    auto slabs = [](int d) { return (d + SP_KC - 1) / SP_KC; };
    // pool rows and scale exponents of the four operands of every sector
    int64_t row = 0;
    struct Rows {
        int hl, hr, w, wt, ehl, ehr, ew, ewt, ahl, ahr, aw, awt;
    };
    std::vector<Rows> rs(s.nsb);
    auto jobs = [](std::vector<SplitJob> &v, int64_t src, int ld, int rows, int k, int kind, int row0, int exp0, int abs0) {
        for (int r = 0; r < rows; r += SP_ROWS) v.push_back(SplitJob{src, ld, rows, k, r, kind, row0, exp0, abs0});
    };
    int64_t tiles32 = 0;
    for (int k = 0; k < s.nsb; ++k) {
        const int dl = s.dls[k], dr = s.drs[k];
        Rows &R = rs[k];
        auto take = [&](int rows, int kk, int boxes = SP_D) {
            const int r0 = (int)row;
            row += (int64_t)boxes * slabs(kk) * rows;
            return r0;
        };
        R.hl = take(dl, dl);
        R.hr = take(dr, dr);
        R.w = take(dl, dr);
        R.wt = take(dr, dl);
        R.ahl = take(dl, dl, 1);
        R.ahr = take(dr, dr, 1);
        R.aw = take(dl, dr, 1);
        R.awt = take(dr, dl, 1);
        R.ehl = p.nexp;
        R.ehr = R.ehl + dl;
        R.ew = R.ehr + dr;
        R.ewt = R.ew + dl;
        p.nexp = R.ewt + dr;
        jobs(p.jobs_hl, s.hl_off[k], dl, dl, dl, 0, R.hl, R.ehl, R.ahl);
        jobs(p.jobs_hr, s.hr_off[k], dr, dr, dr, 0, R.hr, R.ehr, R.ahr);
        jobs(p.jobs_w, s.off[k], dr, dl, dr, 0, R.w, R.ew, R.aw);
        jobs(p.jobs_w, s.off[k], dr, dr, dl, 1, R.wt, R.ewt, R.awt);
        tiles32 += 2 * (int64_t)((dl + SP_M - 1) / SP_M) * ((dr + 31) / 32);
        for (int a = 0; a < dl; a += 8)
            for (int b = 0; b < dr; b += 32)
                p.tiles.push_back(SplitTile{a, b, dl, dr, s.term_ptr[k], s.term_ptr[k + 1], R.ehl, csr[k], s.off[k],
                                            s.hl_off[k], s.hr_off[k]});
        p.kmax = std::max({p.kmax, dl, dr});
    }
    row += std::max(SP_M, SP_SN);   // a box that starts near the end of the pool stays inside it
    p.pool_rows = row;
    // the longest packing jobs first
    std::stable_sort(p.jobs_w.begin(), p.jobs_w.end(), [](const SplitJob &a, const SplitJob &b) { return a.k > b.k; });
    // a slab of 32 columns takes nearly as long as one of 64 (7 MMAs a K step
    // against 10, 4 500 against 5 200 cycles): the narrow tile only where the
    // narrow items still go one to a CTA and its shorter epilogue shows
    p.bn = tiles32 <= nsm ? 32 : 64;
    for (int k = 0; k < s.nsb; ++k) {
        const int dl = s.dls[k], dr = s.drs[k];
        const Rows &R = rs[k];
        for (int m0 = 0; m0 < dl; m0 += SP_M)
            for (int n0 = 0; n0 < dr; n0 += p.bn) {
                p.items.push_back(SplitItem{R.hl, R.wt, dl, dr, dl, dl, dr, m0, n0, 0, s.off[k]});
                p.items.push_back(SplitItem{R.w, R.hr, dl, dr, dr, dl, dr, m0, n0, 1, s.off[k]});
            }
    }
    // the narrowest tiles of which every CTA gets one at most: what counts is
    // the time of a tile (loads and stores shrink with it)
    for (p.sn = 64; p.sn < SP_SN; p.sn *= 2) {
        int64_t tiles = 0;
        for (int k = 0; k < s.nsb; ++k) tiles += 2 * (int64_t)((s.dls[k] + SP_M - 1) / SP_M) * ((s.drs[k] + p.sn - 1) / p.sn);
        if (tiles <= nsm) break;
    }
    for (int k = 0; k < s.nsb; ++k) {
        const int dl = s.dls[k], dr = s.drs[k];
        const Rows &R = rs[k];
        for (int m0 = 0; m0 < dl; m0 += SP_M)
            for (int n0 = 0; n0 < dr; n0 += p.sn) {
                p.sitems.push_back(SplitItem{R.ahl, R.awt, dl, dr, dl, dl, dr, m0, n0, 0, s.off[k]});
                p.sitems.push_back(SplitItem{R.aw, R.ahr, dl, dr, dr, dl, dr, m0, n0, 1, s.off[k]});
            }
    }
    // longest first onto the least loaded CTA (an item costs its slabs plus
    // about one of epilogue)
    auto deal = [&](std::vector<SplitItem> &items, std::vector<int2> &rng) {
        std::stable_sort(items.begin(), items.end(),
                         [&](const SplitItem &a, const SplitItem &b) { return slabs(a.k) > slabs(b.k); });
        const int G = (int)std::min<size_t>(items.size(), (size_t)std::max(1, nsm));
        std::vector<int64_t> load(G, 0);
        std::vector<std::vector<int>> own(G);
        for (size_t e = 0; e < items.size(); ++e) {
            const int b = (int)(std::min_element(load.begin(), load.end()) - load.begin());
            load[b] += slabs(items[e].k) + 1;
            own[b].push_back((int)e);
        }
        std::vector<SplitItem> ordered;
        ordered.reserve(items.size());
        for (int g = 0; g < G; ++g) {
            const int start = (int)ordered.size();
            for (int e : own[g]) ordered.push_back(items[e]);
            rng.push_back(make_int2(start, (int)ordered.size()));
        }
        items.swap(ordered);
        return G;
    };
    p.grid = deal(p.items, p.rng);
    p.sgrid = deal(p.sitems, p.srng);
    // A x B terms: the dominant entry of every row, and the small rest of A's
    constexpr double SMALL = 0x1p-40;
    for (size_t ti = 0; ti < s.terms.size(); ++ti) {
        const DevTerm &tm = s.terms[ti];
        SplitTerm t{0, 0, 0, -1, (int)ti, s.drs[tm.in_sec], rs[tm.in_sec].ew, 0, s.off[tm.in_sec]};
        for (int side = 0; side < 2; ++side) {
            const int64_t rp = side == 0 ? tm.a_rp : tm.b_rp;
            const int nrow = side == 0 ? tm.a_nrow : tm.b_nrow;
            double mx = 0.0;
            bool multi = false;
            for (int i = 0; i < nrow; ++i) multi = multi || rowptr[rp + i + 1] - rowptr[rp + i] > 1;
            if (multi)
                for (int j = rowptr[rp]; j < rowptr[rp + nrow]; ++j) mx = std::max(mx, std::fabs(val[j]));
            (side == 0 ? t.a : t.b) = (int)p.tcol.size();
            const bool dusty = multi && side == 0;
            if (multi && side == 1) t.general = 1;
            if (dusty) {
                t.dust = (int)p.dptr.size();
                p.dptr.push_back((int)p.dcol.size());
            }
            for (int i = 0; i < nrow; ++i) {
                const int p0 = rowptr[rp + i], p1 = rowptr[rp + i + 1];
                int top = -1;
                for (int j = p0; j < p1; ++j)
                    if (top < 0 || std::fabs(val[j]) > std::fabs(val[top])) top = j;
                p.tcol.push_back(top < 0 ? -1 : col[top]);
                p.tval.push_back(top < 0 ? 0.0 : val[top]);
                if (!dusty) continue;
                for (int j = p0; j < p1; ++j) {
                    if (j == top || val[j] == 0.0) continue;
                    if (std::fabs(val[j]) > SMALL * mx || mx > 0x1p60 || mx < 0x1p-60) t.general = 1;
                    p.dcol.push_back(col[j]);
                    p.dval.push_back((float)val[j]);
                }
                p.dptr.push_back((int)p.dcol.size());
            }
        }
        p.terms.push_back(t);
    }
}

int split_finish(Ctx &c, const SplitPlan &p) {
    DevSb &s = c.sb;
    if (p.items.empty()) return NSS_OK;
    s.sp_ntiles = (int)p.tiles.size();
    // the sections that the device fills, at 256-byte boundaries
    const std::pair<void **, size_t> want[] = {
        {(void **)&s.d_sp_redo, sizeof(int) * (SP_REDO_LIST + 8 * p.tiles.size())},
        {(void **)&s.d_sp_exp, sizeof(int) * 2 * (size_t)p.nexp},
        {(void **)&s.d_sp_size, sizeof(float) * 2 * (size_t)s.n},
        {(void **)&s.d_sp_x32, sizeof(float) * (size_t)s.n},
        {(void **)&s.d_sp_out, sizeof(int64_t) * 2 * (size_t)s.n},
        {(void **)&s.d_sp_out0, sizeof(int) * 2 * (size_t)s.n},
        {(void **)&s.d_sp_pool, 2 * SP_KC * (size_t)p.pool_rows}};
    size_t need = 0;
    for (const auto &w : want) need += (w.second + 255) & ~(size_t)255;
    if (need > c.sp_cap) {
        ctx_free(c, c.sp_mem);
        c.sp_mem = nullptr;
        c.sp_cap = 0;
        // headroom: the size varies from step to step
        for (size_t cap : {need + need / 4, need}) {
            if (ctx_alloc(c, &c.sp_mem, cap, true) == cudaSuccess) {
                c.sp_cap = cap;
                break;
            }
            cudaGetLastError();
            c.sp_mem = nullptr;
        }
        if (!c.sp_mem) return NSS_OK;                // the products stay on the CUDA cores
    }
    size_t at = 0;
    for (const auto &w : want) {
        *w.first = c.sp_mem + at;
        at += (w.second + 255) & ~(size_t)255;
    }
    const int part = p.kmax <= SP_STRIP ? p.kmax : SP_STRIP;   // widest strip of a job
    const size_t smem = (size_t)SP_ROWS * (part | 1) * sizeof(double);
    s.sp_pack_smem = smem;
    NSS_CUDA_TRY(c, allow_smem((const void *)k_split_pack, smem));
    c.launches += 2;
    k_split_pack<<<(unsigned)p.jobs_hl.size(), 32 * SP_ROWS, smem, c.stream>>>(s.d_hl, s.d_sp_jobs_hl, s.d_sp_pool, s.d_sp_exp,
                                                                            s.d_sp_exp + p.nexp, nullptr, true, nullptr, nullptr);
    k_split_pack<<<(unsigned)p.jobs_hr.size(), 32 * SP_ROWS, smem, c.stream>>>(s.d_hr, s.d_sp_jobs_hr, s.d_sp_pool, s.d_sp_exp,
                                                                            s.d_sp_exp + p.nexp, nullptr, true, nullptr, nullptr);
    NSS_CUDA_TRY(c, cudaGetLastError());
    s.sp_nexp = p.nexp;
    s.sp_nitems = (int)p.items.size();
    s.sp_njobs = (int)p.jobs_w.size();
    s.sp_bn = p.bn;
    s.sp_grid = p.grid;
    s.sp_sgrid = p.sgrid;
    s.sp_sn = p.sn;
    const std::pair<unsigned char *, int> maps[3] = {{s.sp_map_a, SP_M}, {s.sp_map_b, p.bn}, {s.sp_map_s, p.sn}};
    for (const auto &m : maps)
        if (int rc = tc_tensor_map(c, m.first, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, s.d_sp_pool, SP_KC, p.pool_rows, m.second))
            return rc;
    return NSS_OK;
}

namespace {

template <int BN>
int launch_split(Ctx &c, int *err, const int *stop) {
    NSS_CUDA_TRY(c, allow_smem((const void *)k_sector_split<BN>, SplitCfg<BN>::SMEM));
    DevSb &s = c.sb;
    alignas(64) CUtensorMap ma, mb;
    std::memcpy(&ma, s.sp_map_a, sizeof(ma));
    std::memcpy(&mb, s.sp_map_b, sizeof(mb));
    k_sector_split<BN><<<s.sp_grid, SP_THREADS, SplitCfg<BN>::SMEM, c.stream>>>(ma, mb, s.d_sp_items, s.d_sp_rng, s.d_sp_out, s.d_sp_out0, s.n,
                                                                               wait_limit(), err, stop);
    return NSS_OK;
}

int launch_size(Ctx &c, int *err, const int *stop) {
    NSS_CUDA_TRY(c, allow_smem((const void *)k_split_size, SizeCfg::SMEM));
    DevSb &s = c.sb;
    alignas(64) CUtensorMap ma, mb;
    std::memcpy(&ma, s.sp_map_a, sizeof(ma));
    std::memcpy(&mb, s.sp_map_s, sizeof(mb));
    c.launches += 1;
    k_split_size<<<s.sp_sgrid, SZ_THREADS, SizeCfg::SMEM, c.stream>>>(ma, mb, s.d_sp_sitems, s.d_sp_srng, s.d_sp_size, s.n,
                                                                     s.sp_sn, wait_limit(), err, stop);
    return NSS_OK;
}

}  // namespace

int hv_device_split(Ctx &c, const double *d_v, double *d_hv, const int *stop, bool standalone) {
    DevSb &s = c.sb;
    int *err = standalone ? s.d_sp_redo + SP_REDO_ERR : s.d_tc_err, *nnzs = s.d_sp_exp + s.sp_nexp;
    c.launches += 3;
    k_split_pack<<<(unsigned)s.sp_njobs, 32 * SP_ROWS, s.sp_pack_smem, c.stream>>>(
        d_v, s.d_sp_jobs_w, s.d_sp_pool, s.d_sp_exp, nnzs, s.d_sp_x32, standalone, standalone ? s.d_sp_redo : nullptr, stop);
    if (standalone)
        if (int rc = launch_size(c, err, stop)) return rc;
    if (int rc = s.sp_bn == 64 ? launch_split<64>(c, err, stop) : launch_split<32>(c, err, stop)) return rc;
    SplitTerms T{s.d_sp_terms, s.d_sp_tcol, s.d_sp_dptr, s.d_sp_dcol, s.d_sp_exp, nnzs, s.d_sp_size, s.d_sp_redo, s.d_sp_tval,
                 s.d_sp_dval, s.d_terms, s.d_ab_rowptr, s.d_ab_col, s.d_ab_val};
    auto terms = standalone ? k_split_terms<true> : k_split_terms<false>;
    terms<<<(unsigned)s.sp_ntiles, 256, 0, c.stream>>>(d_v, s.d_sp_x32, s.d_sp_out, s.d_sp_out0, s.n, d_hv, s.d_sp_tiles, T, stop);
    NSS_CUDA_TRY(c, cudaGetLastError());
    return NSS_OK;
}

}  // namespace nss

// Lanczos eigensolver for the lowest eigenpairs of H_sb, on the GPU with the
// small tridiagonal problem on the host.
//
// Replaces SciFortran sp_eigh (ARPACK, called at src/DMRG_SUPERBLOCK.f90:
// 394-425) for the direct mode.  Algorithm: Lanczos with partial
// reorthogonalisation, the whole Krylov basis kept resident in HBM (no
// restarts), and a convergence test every CHECK steps on the tridiagonal matrix T_m:
// residual beta_m |s_m| <= tol |theta| for each wanted Ritz pair, the ARPACK
// criterion.  Breakdown (beta ~ 0, invariant subspace) restarts with a fresh
// random vector orthogonal to the basis.  Eigenvectors are gauge-dependent,
// so parity with the reference is on eigenvalues and on what the RDM derives
// from them.
//
// Orthogonality is kept by partial reorthogonalisation (H. D. Simon, "The
// Lanczos algorithm with partial reorthogonalization", Math. Comp. 42
// (1984)): a recurrence on the inner products omega_{j,k} = v_j . v_k, driven
// by alpha, beta and rounding terms, estimates the loss, and the projection
// against the whole basis (classical Gram-Schmidt, repeated when it removes
// more than half of the residual) runs only at a step where an estimate
// exceeds a threshold, and at the step after it.  A basis orthogonal to
// sqrt(eps) gives a tridiagonal matrix within eps ||H|| of the projection of
// H on its span, so Ritz values are as accurate as with a projection at every
// step; the threshold lies lower (struct Pro) so that the vectors are too.  On
// the measured superblocks 4 to 12 of 50 to 100 steps project.  A projection
// reads the basis twice (2 N m sizeof(T) bytes) and costs two more grid-wide
// exchanges.  Against projecting at every step, solves went from 5.6 to 3.3 ms
// (FP64, N = 3 958), 13.1 to 10.1 ms (FP64, 66 600), 2.72 to 2.52 ms (mixed,
// 66 600), 13.9 to 10.8 ms (mixed, 398 000), and 16 batched solves of up to
// 9 500 states from 10.9 to 10.1 ms.
//
// Per iteration j (m = j+1 basis vectors) two kinds of launch:
//   sector H*psi   w = H v_j                      (k_hv_* kernels)
//   k_orth         one cooperative launch, one CTA per SM, each CTA owning a
//                  contiguous slice of the rows; exchanges of sums separate
//                    alpha = v_j . w
//                    w -= alpha v_j + beta_{j-1} v_{j-1};  beta^2 = w.w
//                    (at a projecting step: h = V_m^T w; w -= V_m h, beta^2 =
//                    w.w, again if it fell by more than half)
//                    v_{j+1} = w / beta, or the breakdown flag
// Every grid-level sum is formed in one fixed order, by one CTA in k_orth
// (xchg_totals) and by every CTA alike in the persistent kernels, so all CTAs
// hold bitwise identical scalars and take the same branches.
//
// The tridiagonal problem (m <= a few hundred) is a chain of dependent FP64
// operations, which GB300's narrow FP64 pipe runs slowly on one SM; it is
// solved on the host (host_tridiag.cpp) from alpha/beta that k_orth writes
// into host-mapped memory, while the GPU already runs the next CHECK
// iterations.  On convergence the host raises a stop request in host-mapped
// memory; the next k_orth publishes it as the device stop flag, and every
// kernel still queued returns at once.  The decision depends only on the
// checked chunk, so results do not depend on that timing.
//
// Precision modes.  The kernels are templates over the type T of the Krylov
// vectors.  T = double is the plain method: FP64 everywhere.  T = float is
// the mixed method: H*psi in FP32 (k_hv_fp32 on CUDA cores, and the
// split-TF32 tensor-core sector GEMM k_sector_mma where the plan routes
// large sectors to it), the basis and the
// projections in FP32 with FP64 block partial sums, while alpha/beta, the
// tridiagonal eigensolve and the Ritz vector stay FP64; it runs to a relative
// residual of MIXED_TOL, and the energy is then refined in FP64 as the
// Rayleigh quotient psi.H.psi of the FP64 Ritz vector with the FP64 H*psi
// (error quadratic in the vector error: |dE|/|E| ~ 1e-13 at MIXED_TOL =
// 1e-7), whose FP64 residual ||H psi - E psi|| is reported.  On GB300 the
// FP64 pipe runs at about 1/70 of the FP32 one (1.06 against 78 TFLOP/s
// measured), which is what the mixed method buys.
#include "batch_words.hpp"
#include "device.cuh"
#include "func_limits.hpp"
#include "host_tridiag.hpp"
#include "hv_tile.cuh"

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <vector>

namespace nss {

namespace {

constexpr int NBLK = 304;         // grid of the restart-path reductions
constexpr int CHECK = 4;          // convergence test period (iterations)
constexpr int SUB = 1024;         // rows staged per shared-memory sub-chunk
constexpr double MIXED_TOL = 1e-7;

// residual target of the FP32 phase (env NSS_MIXED_TOL overrides, clamped to
// [1e-9, 1e-2]); the anchored FP64 phase then takes the vector to `tol`
double mixed_tol() {
    static const double v = [] {
        const char *e = std::getenv("NSS_MIXED_TOL");
        if (!e) return MIXED_TOL;
        const double x = std::atof(e);
        return x < 1e-9 ? 1e-9 : (x > 1e-2 ? 1e-2 : x);
    }();
    return v;
}
constexpr int ORTH_THREADS = 512;
constexpr int ORTH_WARPS = ORTH_THREADS / 32;

// device scalar slots (Ctx::lz.scal)
enum { S_WW = 0, S_BB = 1, S_ALPHA = 2, S_NRM = 3, S_NSCAL = 4 };
// device flag slots (Ctx::lz.flags); the host-mapped mirror uses the same
// indices and one more word, F_NFLAGS, for the host's stop request
enum { F_STOP = 0, F_PASS2 = 1, F_M = 2, F_CONV = 3, F_BREAK = 4, F_HOST = 5, F_ERR = 6, F_NFLAGS = 8 };

template <class T>
__device__ __forceinline__ T warp_sum(T x) {
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}

__device__ __forceinline__ uint64_t splitmix64(uint64_t x) {
    x += 0x9E3779B97F4A7C15ull;
    x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
    x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
    return x ^ (x >> 31);
}

// uniform(-1,1) start vector from a counter-based hash of (seed, stream, i)
__global__ void k_seti(int *p, int v) { *p = v; }

template <class T>
__global__ void k_random(T *x, int64_t n, uint64_t seed, uint64_t stream) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        uint64_t r = splitmix64(seed ^ splitmix64(stream * 0x632BE59BD9B4E019ull + (uint64_t)i));
        x[i] = (T)(2.0 * ((double)(r >> 11) * (1.0 / 9007199254740992.0)) - 1.0);
    }
}

// Last-CTA-done grid reduction helper: every CTA writes its partials, the
// last one to arrive sees all of them.
__device__ __forceinline__ bool last_block(unsigned *counter) {
    __shared__ unsigned last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = (atomicAdd(counter, 1u) == gridDim.x - 1);
    __syncthreads();
    if (last) __threadfence();
    return last != 0;
}

// Sum of the G per-CTA partials, by every thread of the last CTA (256
// threads): a serial loop over ~300 FP64 adds would cost ~20k cycles of
// dependent 64-cycle latency on this GPU.
__device__ __forceinline__ double lastblock_sum(const double *part, int G) {
    __shared__ double red_lb[8];
    double p = 0.0;
    for (int b = threadIdx.x; b < G; b += blockDim.x) p += part[b];
    p = warp_sum<double>(p);
    if ((threadIdx.x & 31) == 0) red_lb[threadIdx.x >> 5] = p;
    __syncthreads();
    double t = 0.0;
    for (int q = 0; q < (int)(blockDim.x >> 5); ++q) t += red_lb[q];
    __syncthreads();
    return t;
}

// Restart path only (a fresh start vector orthogonalised against the basis):
// h[l] = V[l] . w for l < m, and scal[S_WW] = w . w.  With threeterm != 0
// the recurrence step w -= alpha v_{m-1} + beta v_{m-2} (alpha from
// scal[S_ALPHA], beta = betas[m-2]) is applied to w first and the updated w
// is written back.  Per-thread sums in T, block and grid sums in FP64.
template <class T>
__global__ void __launch_bounds__(256) k_dots(const T *__restrict__ V, int m, T *__restrict__ w, int64_t n,
                                              double *__restrict__ part, double *__restrict__ h,
                                              double *__restrict__ scal, unsigned *counter, const int *flags,
                                              int pass2, int threeterm, const double *__restrict__ betas) {
    if (flags[F_STOP] || (pass2 && !flags[F_PASS2])) return;
    extern __shared__ double sm[];
    double *acc = sm;                      // [m+1]
    T *ws = (T *)(sm + (m + 2));           // [SUB]
    const T a3 = threeterm ? (T)scal[S_ALPHA] : (T)0;
    const T b3 = (threeterm && m >= 2) ? (T)betas[m - 2] : (T)0;
    const T *vj = V + (int64_t)(m - 1) * n;
    const T *vjm = (m >= 2) ? V + (int64_t)(m - 2) * n : V;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int l = tid; l <= m; l += 256) acc[l] = 0.0;
    const int64_t chunk = (n + gridDim.x - 1) / gridDim.x;
    const int64_t i0 = blockIdx.x * chunk, i1 = min(n, i0 + chunk);
    for (int64_t s0 = i0; s0 < i1; s0 += SUB) {
        const int len = (int)min((int64_t)SUB, i1 - s0);
        __syncthreads();
        if (threeterm) {
            for (int e = tid; e < len; e += 256) {
                T x = w[s0 + e] - a3 * vj[s0 + e];
                if (m >= 2) x -= b3 * vjm[s0 + e];
                ws[e] = x;
                w[s0 + e] = x;
            }
        } else {
            for (int e = tid; e < len; e += 256) ws[e] = w[s0 + e];
        }
        __syncthreads();
        for (int l = warp; l <= m; l += 8) {
            T p = (T)0;
            if (l < m) {
                const T *vl = V + (int64_t)l * n + s0;
                for (int e = lane; e < len; e += 32) p += vl[e] * ws[e];
            } else {
                for (int e = lane; e < len; e += 32) p += ws[e] * ws[e];
            }
            const double pd = warp_sum<double>((double)p);
            if (lane == 0) acc[l] += pd;
        }
    }
    __syncthreads();
    for (int l = tid; l <= m; l += 256) part[(int64_t)l * gridDim.x + blockIdx.x] = acc[l];
    if (!last_block(counter)) return;
    for (int l = warp; l <= m; l += 8) {
        double p = 0.0;
        for (int b = lane; b < (int)gridDim.x; b += 32) p += part[(int64_t)l * gridDim.x + b];
        p = warp_sum<double>(p);
        if (lane == 0) {
            if (l < m) h[l] = p;
            else scal[S_WW] = p;
        }
    }
    if (tid == 0) *counter = 0u;
}

// w -= V_m h ; beta^2 = w.w ; the last CTA records alpha_j and beta_j.
template <class T>
__global__ void __launch_bounds__(256) k_update(const T *__restrict__ V, int m, T *__restrict__ w, int64_t n,
                                                const double *__restrict__ h, double *__restrict__ part,
                                                double *__restrict__ scal, unsigned *counter, int *flags,
                                                double *alpha, double *beta, int pass2) {
    if (flags[F_STOP] || (pass2 && !flags[F_PASS2])) return;
    extern __shared__ double hsd[];
    T *hs = (T *)hsd;
    const int tid = threadIdx.x;
    for (int l = tid; l < m; l += 256) hs[l] = (T)h[l];
    __syncthreads();
    T ss = (T)0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + tid; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        T x = w[i];
        for (int l = 0; l < m; ++l) x -= V[(int64_t)l * n + i] * hs[l];
        w[i] = x;
        ss += x * x;
    }
    const double sd = warp_sum<double>((double)ss);
    __shared__ double red[8];
    if ((tid & 31) == 0) red[tid >> 5] = sd;
    __syncthreads();
    if (tid == 0) {
        double t = 0.0;
        for (int q = 0; q < 8; ++q) t += red[q];
        part[blockIdx.x] = t;
    }
    if (!last_block(counter)) return;
    const double bb = lastblock_sum(part, gridDim.x);
    if (tid != 0) return;
    const int j = m - 1;
    if (!pass2) {
        alpha[j] = scal[S_ALPHA] + h[j];
        flags[F_PASS2] = (bb < 0.5 * scal[S_WW]) ? 1 : 0;
    } else {
        alpha[j] += h[j];
    }
    scal[S_BB] = bb;
    beta[j] = sqrt(bb);
    *counter = 0u;
}

// x <- x / ||x|| over the whole GPU: k_sumsq (FP64 partial sums, the last
// CTA writes 1 / ||x||), then k_scale.
template <class T>
__global__ void __launch_bounds__(256) k_sumsq(const T *__restrict__ x, int64_t n, double *__restrict__ part,
                                               double *__restrict__ inv, unsigned *counter) {
    const int tid = threadIdx.x;
    double a = 0.0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + tid; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const double v = (double)x[i];
        a = fma(v, v, a);
    }
    a = warp_sum<double>(a);
    __shared__ double red[8];
    if ((tid & 31) == 0) red[tid >> 5] = a;
    __syncthreads();
    if (tid == 0) {
        double t = 0.0;
        for (int q = 0; q < 8; ++q) t += red[q];
        part[blockIdx.x] = t;
    }
    if (!last_block(counter)) return;
    const double t = lastblock_sum(part, gridDim.x);
    if (tid != 0) return;
    *inv = 1.0 / sqrt(t);
    *counter = 0u;
}

template <class T>
__global__ void __launch_bounds__(256) k_scale(T *__restrict__ x, int64_t n, const double *__restrict__ inv) {
    const double f = *inv;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        x[i] = (T)((double)x[i] * f);
}

// ---------------------------------------------------------------------------
// Fused orthogonalisation step (cooperative launch).
//
// Reductions are carried out in the basis type T: FP32 for the mixed
// method, FP64 for the plain one.  On GB300 an FP64 add or FMA occupies a
// warp's share of the FP64 pipe for 64 cycles (a division ~650), so FP64
// reduction trees inside the FP32 method would cost more than the FP32
// vector work they sum; FP32 sums are as accurate as the FP32 vectors and
// the FP32 products they add up.

struct OrthArgs {
    void *V, *w;                 // T*: basis [cap+1][n], work vector [n]
    int64_t n;
    int j, mmax, pstride;        // step, iteration cap, column stride of partials
    double *alpha, *beta;        // device tridiagonal coefficients
    void *part;                  // T*: per-CTA partials (five regions)
    unsigned *bar;               // grid barrier: arrival count, generation
    int *flags;                  // device flags
    double *h_alpha, *h_beta;    // host-mapped mirrors of alpha, beta
    int *h_flags;                // host-mapped flag mirror + stop request
    // anchored refinement (anc_u == nullptr: plain Lanczos), T* vectors: the
    // Krylov vectors are kept orthogonal to the anchor u and to ndefl
    // vectors defl[k*n..]; m_j = r . v_j (r = H u - theta0 u) goes to h_m[j]
    const void *anc_u, *anc_r, *defl;
    int ndefl;
    double *h_m;
    uint32_t spin;               // poll limit of the grid barriers (wait_limit)
    // replayed chunks (CUDA graph): the step is read from *jdev and advanced
    // by the kernel, and the new Lanczos vector is also written to vcur, the
    // fixed input of the next H*psi (null: step a.j, no copy)
    int *jdev;
    void *vcur;
    // omega estimates: [pstride] of v_j, [pstride] of v_{j-1}, then one int
    // (the next step projects whatever its estimates say) and, anchored, the
    // products of u and y_k with v_j and with v_{j-1}
    float *pro;
    // tagged exchange (see xchg_totals): the last epoch of the previous
    // launch, the words of the totals, of the columns' partials and of the
    // columns' totals
    unsigned *xep;
    uint64_t *xtot, *xpart, *xcol;
    // H v_j's tensor-core part, still to be added to w: tcn planes of n (FP32
    // only; null: w is complete)
    const float *tc = nullptr;
    int tcn = 0;
    // k_orth: an estimate above this makes the step project; every: all steps do
    float delta = 0.f;
    int every = 0;
};

// The omega recurrence's constants per basis type: level after a projection,
// rounding term per (beta_k + beta_j + |alpha_j|: H v_j is rounded at the size
// of its largest part), and the threshold.  sqrt(eps) would do
// for Ritz values; what a projection takes off a vector (up to beta times the
// threshold, mostly along a converged Ritz vector) is not in the tridiagonal
// matrix, though, and enters a wanted vector that has not converged yet.  At
// 5e-13 that stays below the solver's default tolerance (at 1e-8 a 96-state
// superblock's residual was 1e-10 |theta|); it costs two to four more
// projecting steps a solve.  For a tolerance below 1e-12 the threshold is half
// of it, and a threshold within PRO_EVERY levels of a projection (the tolerance
// of 1e-15 that a caller gets with 0) means a projection at every step: the third
// of three states had a residual of 4e-15 |E| by estimates of 5e-13 and has
// 7e-16.  The FP32 phase's vector is refined afterwards.
template <class T>
struct Pro;
template <>
struct Pro<double> {
    static constexpr float EPS1 = 4.4e-16f, NOISE = 2.2e-16f, DELTA = 5e-13f;
};
template <>
struct Pro<float> {
    static constexpr float EPS1 = 2.4e-7f, NOISE = 1.2e-7f, DELTA = 5e-5f;
};

constexpr float PRO_EVERY = 8.f;

constexpr int PRO_TAIL = 16;     // floats after the estimates: the int, then two rows of ANC_MAX products

// The start of a Lanczos run (or of a restart from a vector orthogonal to
// the basis): every estimate at the level of a projection
__global__ void k_pro_reset(float *pro, int ps, float eps1) {
    for (int k = threadIdx.x; k < 2 * ps; k += blockDim.x) pro[k] = eps1;
    if (threadIdx.x < PRO_TAIL) pro[2 * ps + threadIdx.x] = 0.f;
}

// The estimates of v_{j+1} from those of v_j (so) and v_{j-1} (sp) into sn,
// for the tridiagonal coefficients sa, sb (sa[j], sb[j] included); returns
// whether one exceeds the threshold (same value in every thread and CTA).
// Called by all threads; m = j + 1.  FP32 is enough for estimates, and an
// FP64 chain would take as long as the rest of a small step.
template <class T>
__device__ __forceinline__ bool pro_step(const float *so, const float *sp, const float *sa, const float *sb, float *sn,
                                         int j, float delta = Pro<T>::DELTA) {
    const float bj = sb[j], aj = sa[j], bp = j > 0 ? sb[j - 1] : 0.f, ib = 1.f / bj;
    int over = 0;
    for (int k = threadIdx.x; k <= j; k += blockDim.x) {
        float t;
        if (k < j) {
            const float bk = sb[k];
            const float up = k + 1 == j ? 1.f : so[k + 1];
            const float old = k + 1 == j ? 1.f : sp[k];
            t = bk * up + (sa[k] - aj) * so[k] - bp * old;
            if (k > 0) t += sb[k - 1] * so[k - 1];
            t += copysignf(Pro<T>::NOISE * (bk + bj + fabsf(aj)), t);
            t *= ib;
        } else {
            t = fmaxf(Pro<T>::EPS1, Pro<T>::NOISE * fabsf(aj) * ib);
        }
        sn[k] = t;
        if (!(fabsf(t) <= delta)) over = 1;
    }
    return __syncthreads_or(over) != 0;
}

constexpr int PA_COLS = 8;       // per-CTA values of the first phase (alpha, u.w, r.v, y_k.w)

// Grid-wide barrier for a cooperative launch (all CTAs resident).  The
// arrival counter only grows during a launch: barrier e of the launch waits
// for e*G arrivals (`epoch`, kept by each CTA), so there is no reset on the
// critical path; grid_exit zeroes the counter when the last CTA leaves.
// Bounded: a wait that runs out sets flags[F_ERR] and every later barrier
// returns false at once, so the kernel always ends.
// orders the writes that this thread has seen before its later stores (the
// lighter fence: __threadfence is sequentially consistent)
__device__ __forceinline__ void fence_acq_rel() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }
__device__ __forceinline__ unsigned ld_acquire_u32(const unsigned *p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ bool grid_sync(unsigned *bar, unsigned &epoch, int *err, uint32_t spin) {
    __shared__ int ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        int good = 1;
        epoch += gridDim.x;
        fence_acq_rel();
        atomicAdd(bar, 1u);
        uint32_t it = 0;
        while (ld_acquire_u32(bar) < epoch) {
            if (++it > spin) { atomicExch(err, 1); good = 0; break; }
            if ((it & 255u) == 0 && *(volatile int *)err) { good = 0; break; }
        }
        ok = good;
    }
    __syncthreads();
    return ok != 0;
}

// every CTA calls this once when it leaves a launch that may use grid_sync
__device__ __forceinline__ void grid_exit(unsigned *bar) {
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(bar + 1, 1u) == gridDim.x - 1) {
            atomicExch(bar, 0u);
            atomicExch(bar + 1, 0u);
        }
    }
}

// CTA sums of NV values at once, valid in thread 0; only the first nw warps
// hold values (uniform over the CTA).  An FP64 add takes a warp's share of the
// FP64 pipe for 64 cycles, so a small superblock's CTA, whose few rows fill
// one or two warps, must not run the tree on all sixteen.
template <class R, int NV>
__device__ __forceinline__ void block_sums(R (&v)[NV], R *scr, int nw = ORTH_WARPS) {
    const int warp = threadIdx.x >> 5;
    if (warp < nw) {
#pragma unroll
        for (int q = 0; q < NV; ++q) v[q] = warp_sum<R>(v[q]);
    }
    if (nw == 1) return;
    __syncthreads();
    if (warp < nw && (threadIdx.x & 31) == 0)
#pragma unroll
        for (int q = 0; q < NV; ++q) scr[q * ORTH_WARPS + warp] = v[q];
    __syncthreads();
    if (warp == 0) {
#pragma unroll
        for (int q = 0; q < NV; ++q) {
            R t = threadIdx.x < nw ? scr[q * ORTH_WARPS + threadIdx.x] : (R)0;
#pragma unroll
            for (int o = ORTH_WARPS / 2; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
            v[q] = t;
        }
    }
}

// p[i0] + p[i0 + stride] + ... (indices below end), added in that order;
// the loads go out eight at a time, so a sum over the partials of a grid
// costs one L2 round trip instead of one per term (an add waiting for its
// load stalls the warp's next load: the loop form issued them one by one)
template <class R>
__device__ __forceinline__ R strided_sum(const R *p, int i0, int end, int stride) {
    R t = (R)0;
    for (int b0 = i0; b0 < end; b0 += 8 * stride) {
        R v[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int b = b0 + q * stride;
            v[q] = b < end ? __ldcg(p + b) : (R)0;
        }
#pragma unroll
        for (int q = 0; q < 8; ++q)
            if (b0 + q * stride < end) t += v[q];
    }
    return t;
}

// sums of the G per-CTA partials of NV columns p[q*G + b], same order in
// every CTA; warp q reduces column q, results broadcast through bc[]
template <class R, int NV>
__device__ __forceinline__ void grid_totals(const R *p, int G, R *bc, R (&out)[NV]) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (warp < NV) {
        R t = strided_sum<R>(p + (int64_t)warp * G, lane, G, 32);
        t = warp_sum<R>(t);
        if (lane == 0) bc[warp] = t;
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < NV; ++q) out[q] = bc[q];
}

// hs[l] = sum_b p[l*G + b] for l < ncol (four columns per warp in flight;
// all their loads issued before the first add)
template <class R>
__device__ __forceinline__ void grid_columns(const R *p, int G, int ncol, R *hs) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int l0 = warp; l0 < ncol; l0 += 4 * ORTH_WARPS) {
        R t[4] = {(R)0, (R)0, (R)0, (R)0};
        for (int b0 = lane; b0 < G; b0 += 8 * 32) {
            R v[4][8];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int l = l0 + u * ORTH_WARPS;
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    const int b = b0 + 32 * q;
                    v[u][q] = (l < ncol && b < G) ? __ldcg(p + (int64_t)l * G + b) : (R)0;
                }
            }
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int q = 0; q < 8; ++q) t[u] += v[u][q];
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const R s = warp_sum<R>(t[u]);
            const int l = l0 + u * ORTH_WARPS;
            if (lane == 0 && l < ncol) hs[l] = s;
        }
    }
}

// Sums of d[0..N) over groups of P lanes (butterfly with exchange while a lane
// holds more than one value, N <= P): d[0] ends as the group's sum of value
// (lane % P) * N / P.  The order of the additions, lanes P/2 apart first, does
// not depend on N.
template <class R, int N, int P>
__device__ __forceinline__ R multi_reduce(R (&d)[N], int lane) {
    static_assert(N <= P, "every value needs a lane");
#pragma unroll
    for (int s = P / 2, cnt = N; s >= 1; s >>= 1) {
        if (cnt > 1) {
            const bool upper = (lane & s) != 0;
            cnt >>= 1;
#pragma unroll
            for (int c = 0; c < N / 2; ++c)
                if (c < cnt) {
                    const R send = upper ? d[c] : d[c + cnt];
                    const R keep = upper ? d[c + cnt] : d[c];
                    d[c] = keep + __shfl_xor_sync(0xffffffffu, send, s);
                }
        } else {
            d[0] += __shfl_xor_sync(0xffffffffu, d[0], s);
        }
    }
    return d[0];
}

// Tagged exchange between the CTAs of k_orth.  A grid barrier costs an atomic
// per CTA on one address and a poll (1.6 us over 152 CTAs), and the partials
// are read and summed by everybody only after it (0.6-1.2 us more).  In k_orth
// the values are all that travels (every CTA works on its own rows), so no
// fence is needed: every CTA stores its values as 64-bit words (32 bits of
// value, 32 of epoch); the last CTA polls them, sums and stores the totals as
// tagged words, which the others poll: barrier and sum in two hops.  A CTA
// stores epoch e+1 only after it has read the totals of e, and the last CTA its
// totals of e+1 only after every word of e+1, so one buffer of each is enough.
// Epochs grow from launch to launch (*xep); a run starts with words and epoch
// zeroed.  With the column sums shared out (xchg_columns): FP64 solves of 3 958
// states 3.28 -> 3.12 ms, of 66 600 10.07 -> 9.85 ms.  Where the exchange has
// to publish other writes too (k_chunk32), its fences make it slower than the
// barrier: 2.8 us against 2.6 us for barrier and sum, 7 us with seven values;
// and every CTA polling all words, 152 x 152 readers of the same lines, took
// 4 us.
constexpr int XMAX = 192;        // CTAs of a cooperative launch at most
constexpr int XCOLS = 9;         // words per epoch (double: two a value), the last for the flag

template <class R>
struct XW { static constexpr int words = sizeof(R) / 4; };

__device__ __forceinline__ void st_word(uint64_t *p, uint32_t v, unsigned ep) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"((uint64_t)v | ((uint64_t)ep << 32)) : "memory");
}
__device__ __forceinline__ uint64_t ld_word(const uint64_t *p) {
    uint64_t w;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(w) : "l"(p) : "memory");
    return w;
}
// value q of a set of `n` values, words `stride` apart: word k of the value at p + (q * words + k) * stride
__device__ __forceinline__ void st_value(uint64_t *p, int64_t, float v, unsigned ep) {
    st_word(p, __float_as_uint(v), ep);
}
__device__ __forceinline__ void st_value(uint64_t *p, int64_t stride, double v, unsigned ep) {
    st_word(p, (uint32_t)__double2loint(v), ep);
    st_word(p + stride, (uint32_t)__double2hiint(v), ep);
}
// polls until the value carries the epoch; false when the limit ran out
__device__ __forceinline__ bool ld_value(const uint64_t *p, int64_t, unsigned ep, float &v, const int *err, uint32_t spin) {
    uint32_t it = 0;
    for (;;) {
        const uint64_t w = ld_word(p);
        if ((unsigned)(w >> 32) == ep) {
            v = __uint_as_float((uint32_t)w);
            return true;
        }
        if (++it > spin || ((it & 255u) == 0 && *(volatile const int *)err)) return false;
    }
}
__device__ __forceinline__ bool ld_value(const uint64_t *p, int64_t stride, unsigned ep, double &v, const int *err,
                                         uint32_t spin) {
    uint32_t it = 0;
    for (;;) {
        const uint64_t w0 = ld_word(p), w1 = ld_word(p + stride);
        if ((unsigned)(w0 >> 32) == ep && (unsigned)(w1 >> 32) == ep) {
            v = __hiloint2double((int)(uint32_t)w1, (int)(uint32_t)w0);
            return true;
        }
        if (++it > spin || ((it & 255u) == 0 && *(volatile const int *)err)) return false;
    }
}

// x[q] = the value at p + lane + 32 q (for those below G): all words in flight
// at once, where one ld_value after the other takes an L2 round trip each
template <class R, int Q>
__device__ __forceinline__ bool ld_values(const uint64_t *p, int64_t stride, int lane, int G, unsigned ep, R (&x)[Q],
                                          const int *err, uint32_t spin) {
    constexpr int W = XW<R>::words;
    uint32_t it = 0;
    for (;;) {
        uint64_t w[Q][W];
        bool all = true;
#pragma unroll
        for (int q = 0; q < Q; ++q)
#pragma unroll
            for (int k = 0; k < W; ++k)
                w[q][k] = lane + 32 * q < G ? ld_word(p + k * stride + lane + 32 * q) : (uint64_t)ep << 32;
#pragma unroll
        for (int q = 0; q < Q; ++q) {
#pragma unroll
            for (int k = 0; k < W; ++k) all = all && (unsigned)(w[q][k] >> 32) == ep;
            if constexpr (W == 1) x[q] = __uint_as_float((uint32_t)w[q][0]);
            else x[q] = __hiloint2double((int)(uint32_t)w[q][1], (int)(uint32_t)w[q][0]);
        }
        if (all) return true;
        if (++it > spin || ((it & 255u) == 0 && *(volatile const int *)err)) return false;
    }
}

// out[q] = sum over the CTAs of v[q] (valid in thread 0), in the order of
// grid_totals; xs: [NV][G] in shared memory.  Only the values travel: no
// barrier, no fence.  flag (may be null): the last CTA's value (thread 0), on
// return everybody's.  False when a wait ran out (sets *err).
template <class R, int NV>
__device__ __forceinline__ bool xchg_totals(uint64_t *xtot, unsigned &ep, const R (&v)[NV], int G, R *xs, R *bc,
                                            R (&out)[NV], int *err, uint32_t spin, int *flag = nullptr) {
    constexpr int W = XW<R>::words;
    static_assert(NV * W < XCOLS, "words per CTA");
    __shared__ int xflag;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int last = G - 1;
    uint64_t *res = xtot + (size_t)XCOLS * XMAX;     // the totals
    ++ep;
    bool good = true;
    __syncthreads();                                 // xs, bc and xflag of the last exchange are read
    if ((int)blockIdx.x != last) {
        if (tid == 0) {
#pragma unroll
            for (int q = 0; q < NV; ++q) st_value(xtot + (size_t)(q * W) * XMAX + blockIdx.x, XMAX, v[q], ep);
        }
        if (tid < NV) {
            R x = (R)0;
            good = ld_value(res + tid * W, 1, ep, x, err, spin);
            bc[tid] = x;
        }
        if (flag && tid == NV) {
            float f = 0.f;
            good = ld_value(res + XCOLS - 1, 0, ep, f, err, spin);
            xflag = __float_as_int(f);
        }
        if (!good) atomicExch(err, 1);
    } else {
        if (tid == 0)
#pragma unroll
            for (int q = 0; q < NV; ++q) xs[q * G + last] = v[q];
        for (int k = tid; k < NV * last; k += ORTH_THREADS) {
            const int q = k / last, b = k - q * last;
            R x = (R)0;
            good = good && ld_value(xtot + (size_t)(q * W) * XMAX + b, XMAX, ep, x, err, spin);
            xs[q * G + b] = x;
        }
        if (!good) atomicExch(err, 1);
        if (!__syncthreads_and(good)) good = false;
        if (warp < NV && good) {
            R t = (R)0;
            for (int b = lane; b < G; b += 32) t += xs[warp * G + b];
            t = warp_sum<R>(t);
            if (lane == 0) {
                bc[warp] = t;
                st_value(res + warp * W, 1, t, ep);
                if (flag && warp == 0) {
                    st_word(res + XCOLS - 1, (uint32_t)*flag, ep);
                    xflag = *flag;
                }
            }
        }
    }
    if (!__syncthreads_and(good)) return false;
    if (flag) *flag = xflag;
#pragma unroll
    for (int q = 0; q < NV; ++q) out[q] = bc[q];
    return true;
}

// hs[l] = sum over the CTAs of column l's partial (l < ncol), which every CTA
// has stored at xpart (st_value, epoch ep + 1): CTA l mod G sums column l, in
// the order of grid_columns, and stores the total as tagged words at xcol,
// which all poll (summed by every CTA instead, 100 FP64 columns took each SM's
// FP64 pipe 10 us).  A CTA writes its partials and totals of a later epoch only
// after it has read all totals of this one, so one buffer of each is enough.
template <class R>
__device__ __forceinline__ bool xchg_columns(const uint64_t *xpart, uint64_t *xcol, unsigned &ep, int G, int ncol, R *hs,
                                             int *err, uint32_t spin) {
    constexpr int W = XW<R>::words;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    ++ep;
    bool good = true;
    for (int l = blockIdx.x + warp * G; l < ncol; l += ORTH_WARPS * G) {
        const uint64_t *p = xpart + (size_t)l * W * XMAX;
        R x[XMAX / 32];
        good = good && ld_values<R, XMAX / 32>(p, XMAX, lane, G, ep, x, err, spin);
        R t = (R)0;
#pragma unroll
        for (int q = 0; q < XMAX / 32; ++q)
            if (lane + 32 * q < G) t += x[q];
        good = __all_sync(0xffffffffu, good);
        t = warp_sum<R>(t);
        if (lane == 0 && good) st_value(xcol + (size_t)l * W, 1, t, ep);
    }
    for (int l = tid; l < ncol; l += ORTH_THREADS) {
        R x = (R)0;
        good = good && ld_value(xcol + (size_t)l * W, 1, ep, x, err, spin);
        hs[l] = x;
    }
    if (!good) atomicExch(err, 1);
    return __syncthreads_and(good);
}

// One item of cta_dots: CW columns from l0 over the rows [r0, r1).  P lanes go
// along the rows and 32 / P side by side along the columns, so a lane holds
// CW P / 32 sums; rows beyond a lane's would only add zeros, so the result is
// bit for bit that of P = 32.
template <class T, int CW, int P>
__device__ __forceinline__ void dots_item(const T *__restrict__ V, int m, const T *__restrict__ w, int64_t n, int l0,
                                          int64_t r0, int64_t r1, int ncol, T *red) {
    constexpr int N = CW * P / 32;
    const int lane = threadIdx.x & 31, rl = lane % P, lb = l0 + (lane / P) * N;
    T acc[N];
#pragma unroll
    for (int c = 0; c < N; ++c) acc[c] = (T)0;
    if (lb + N <= m) {
        for (int64_t r = r0 + rl; r < r1; r += P) {
            const T wv = w[r];
            const T *vr = V + (int64_t)lb * n + r;
#pragma unroll
            for (int c = 0; c < N; ++c) acc[c] += vr[(int64_t)c * n] * wv;
        }
    } else {
        for (int64_t r = r0 + rl; r < r1; r += P) {
            const T wv = w[r];
#pragma unroll
            for (int c = 0; c < N; ++c) {
                const int l = lb + c;
                if (l < m) acc[c] += V[(int64_t)l * n + r] * wv;
                else if (l < ncol) acc[c] += wv * wv;
            }
        }
    }
    const T s = multi_reduce<T, N, P>(acc, lane);
    const int l = lb + rl * N / P;
    if (rl % (P / N) == 0 && l < ncol) red[l] = s;
}

// CTA partials of h[l] = V[l] . w (l < m) over rows [i0, i1), plus w.w as
// column m when `ww`; handed to store(l, sum).  Work items are (CW-column
// group, row quarter), a warp each.  A DADD on the whole warp holds an SM
// quarter's FP64 pipe for 64 cycles whatever its lanes hold, so with a few
// rows per quarter (12 per CTA at 1 800 states) the lanes go along the columns
// instead, and the totals are exchanged in two hops (xchg_columns): a step that
// projects at every iteration, 1 500 states, 30 columns: 31 -> 16 us, a chain of
// 20 spins with 40 states kept 21.8 -> 17.6 ms.
template <class T, int CW, class Store>
__device__ __forceinline__ void cta_dots(const T *__restrict__ V, int m, const T *__restrict__ w, int64_t n,
                                         int64_t i0, int64_t i1, bool ww, T *red, Store store) {
    const int warp = threadIdx.x >> 5;
    const int ncol = m + (ww ? 1 : 0);
    const int ng = (ncol + CW - 1) / CW;
    const int nq = ng >= ORTH_WARPS ? 1 : ORTH_WARPS / ng;
    const int rs = ng * CW;
    const unsigned len = (unsigned)(i1 - i0), qlen = (len + nq - 1) / nq;   // a CTA's rows: 32-bit divisions
    const int nqe = qlen > 0 ? (int)((len + qlen - 1) / qlen) : 1;          // quarters with rows
    for (int item = warp; item < ng * nqe; item += ORTH_WARPS) {
        const int g = item % ng, q = item / ng;
        const int64_t r0 = i0 + (int64_t)q * qlen, r1 = min(i1, r0 + qlen);
        T *rq = red + q * rs;
        if (qlen > 16) dots_item<T, CW, 32>(V, m, w, n, g * CW, r0, r1, ncol, rq);
        else if (qlen > 4) dots_item<T, CW, 16>(V, m, w, n, g * CW, r0, r1, ncol, rq);
        else dots_item<T, CW, 4>(V, m, w, n, g * CW, r0, r1, ncol, rq);
    }
    __syncthreads();
    for (int l = threadIdx.x; l < ncol; l += ORTH_THREADS) {
        T s = (T)0;
        for (int q = 0; q < nqe; ++q) s += red[q * rs + l];
        store(l, s);
    }
}

// w -= V_m h over rows [i0, i1); returns this thread's share of w.w
template <class T>
__device__ __forceinline__ T cta_update(const T *__restrict__ V, int m, T *__restrict__ w, int64_t n, int64_t i0,
                                        int64_t i1, const T *hs) {
    T ss = (T)0;
    for (int64_t i = i0 + threadIdx.x; i < i1; i += ORTH_THREADS) {
        T x = w[i];
#pragma unroll 32
        for (int l = 0; l < m; ++l) x -= V[(int64_t)l * n + i] * hs[l];
        w[i] = x;
        ss += x * x;
    }
    return ss;
}

template <class T>
struct OrthCW { static constexpr int value = sizeof(T) == 4 ? 32 : 16; };

// also the exchanged values of a CTA (xchg_totals), up to PA_COLS + 1 of XMAX CTAs
__host__ __device__ inline int orth_redsz(int pstride, int cw) {
    const int dots = ORTH_WARPS * cw > pstride + cw ? ORTH_WARPS * cw : pstride + cw;
    return dots > (PA_COLS + 1) * XMAX ? dots : (PA_COLS + 1) * XMAX;
}

// A Krylov basis of more columns than this leaves no room for the recurrence:
// its solve projects at every step
constexpr int PRO_MAX_PS = 4096;

// floats of the omega recurrence in shared memory: estimates of v_j, v_{j-1},
// v_{j+1}, alpha, beta
__host__ __device__ inline size_t pro_floats(int pstride) {
    return pstride <= PRO_MAX_PS ? 5 * (size_t)((pstride + 3) & ~3) : 0;
}

// shared memory of the orthogonalisation in bytes: hs, red, scratch (T), the
// recurrence
__host__ __device__ inline size_t orth_smem(int pstride, int cw, size_t tsize) {
    const size_t t = (size_t)(pstride + orth_redsz(pstride, cw) + 8 * ORTH_WARPS + 16) * tsize;
    return ((t + 15) & ~(size_t)15) + pro_floats(pstride) * sizeof(float);
}

// The recurrence's shared arrays
struct ProSmem {
    float *so, *sp, *sn, *sa, *sb;
    const bool on;
    __device__ ProSmem(void *base, int ps) : on(ps <= PRO_MAX_PS) {
        const int st = (ps + 3) & ~3;
        so = (float *)base;
        sp = so + st;
        sn = sp + st;
        sa = sn + st;
        sb = sa + st;
    }
    // state of step j from global memory (estimates, alpha_k, beta_k, k < j)
    __device__ __forceinline__ void load(const float *pro, int ps, const double *alpha, const double *beta, int j) {
        for (int k = threadIdx.x; on && k < j; k += blockDim.x) {
            so[k] = __ldcg(pro + k);
            sp[k] = __ldcg(pro + ps + k);
            sa[k] = (float)__ldcg(alpha + k);
            sb[k] = (float)__ldcg(beta + k);
        }
    }
    // (one thread) alpha_j, beta_j
    __device__ __forceinline__ void set(int j, float alpha, float beta) {
        if (!on) return;
        sa[j] = alpha;
        sb[j] = beta;
    }
    // does v_{j+1} lose more than `limit`?
    template <class T>
    __device__ __forceinline__ bool over(int j, float limit = (float)Pro<T>::DELTA) {
        return on ? pro_step<T>(so, sp, sa, sb, sn, j, limit) : true;
    }
    // step j projects
    template <class T>
    __device__ __forceinline__ void projected(int j) {
        for (int k = threadIdx.x; on && k <= j; k += blockDim.x) sn[k] = (float)Pro<T>::EPS1;
    }
    // after step j: the new estimates become v_{j+1}'s
    __device__ __forceinline__ void advance() {
        float *t = sp;
        sp = so;
        so = sn;
        sn = t;
    }
    __device__ __forceinline__ void store(float *pro, int ps, int j, int force) const {
        for (int k = threadIdx.x; on && k <= j; k += blockDim.x) {
            pro[k] = so[k];
            pro[ps + k] = sp[k];
        }
        if (threadIdx.x == 0) *(int *)(pro + 2 * ps) = force;
    }
};

// FP64 superblocks of fewer states than this project at every step: the
// truncation errors of small chains (1 - sum lambda, 1e-12) follow the last
// bits of the ground state, so their arithmetic stays what it was.  An FP32
// basis projects at every step once it fills an eighth of its space: close to
// exhausting it the estimates' model no longer holds.
constexpr int64_t PRO_MIN_N = 3072;
template <class T>
__host__ __device__ __forceinline__ bool pro_always(int m, int64_t n, int ps) {
    return ps > PRO_MAX_PS || (sizeof(T) == 8 ? n < PRO_MIN_N : 8 * (int64_t)m > n);
}

// Rows of a thread whose loads go out together (a store to w would order the
// next row's loads behind it; a CTA has five rows a thread at 398 000 states)
constexpr int ROWS = 4;

template <class T, int CW>
__global__ void __launch_bounds__(ORTH_THREADS, 1) k_orth(OrthArgs a) {
    int *flags = a.flags;
    // the launch's state, loads issued together
    const int stop = *(volatile int *)&flags[F_STOP];
    const int j = a.jdev ? *(volatile const int *)a.jdev : a.j, m = j + 1;
    unsigned ep = *(volatile unsigned *)a.xep;       // advanced when the launch ends
    int force = __ldcg((const int *)(a.pro + 2 * a.pstride));
    if (stop) return;                                // set before this launch: uniform
    extern __shared__ __align__(16) unsigned char osm_raw[];
    T *osm = (T *)osm_raw;
    const int ps = a.pstride;
    T *hs = osm;
    T *red = hs + ps;
    T *scr = red + orth_redsz(ps, CW);               // [8 x 16] block sums, then [16] broadcasts
    T *bc = scr + 8 * ORTH_WARPS;
    T *xs = red;                                     // between two uses of red
    ProSmem pro(osm_raw + (orth_smem(ps, CW, sizeof(T)) - pro_floats(ps) * sizeof(float)), ps);
    const int G = gridDim.x, blk = blockIdx.x, tid = threadIdx.x;
    const int64_t n = a.n;
    const int64_t chunk = (n + G - 1) / G;
    const int64_t i0 = min(n, (int64_t)blk * chunk), i1 = min(n, i0 + chunk);
    const int nw = (int)min((int64_t)ORTH_WARPS, max((int64_t)1, (chunk + 31) / 32));   // warps with rows
    T *V = (T *)a.V, *w = (T *)a.w;
    const T *vj = V + (int64_t)j * n;
    const T *vjm = V + (int64_t)(j > 0 ? j - 1 : 0) * n;
    int *err = flags + F_ERR;
    constexpr int W = XW<T>::words;
    auto column = [&](int l, T t) { st_value(a.xpart + (size_t)l * W * XMAX + blk, XMAX, t, ep + 1); };
    // leaving: the next launch's epochs follow this one's.  A wait that ran out
    // is reported through the mapped flag mirror, which the host reads before
    // any result.
    auto leave = [&](bool failed) {
        if (tid != 0) return;
        if (failed) {
            a.h_flags[F_ERR] = 1;
            __threadfence_system();
        } else if (blk == 0) {
            *a.xep = ep;
        }
    };
    const T *au = (const T *)a.anc_u, *ar = (const T *)a.anc_r, *ay = (const T *)a.defl;
    const bool anc = sizeof(T) == 4 && au != nullptr;   // the refinement's bases are FP32
    const int nd = anc ? a.ndefl : 0;

    // the host's stop request (host memory: issued first, consumed just
    // before the first barrier so the read overlaps the first phase)
    int host_stop = 0;
    if (blk == G - 1 && tid == 0) host_stop = *(volatile const int *)(a.h_flags + F_NFLAGS);
    // alpha = v_j . w; anchored also u.w, r.v_j and y_k.w
    T av[PA_COLS];
#pragma unroll
    for (int q = 0; q < PA_COLS; ++q) av[q] = (T)0;
    for (int64_t b0 = i0 + tid; b0 < i1; b0 += ROWS * ORTH_THREADS) {
        T wv[ROWS], vv[ROWS], uv[ROWS], rv[ROWS];
#pragma unroll
        for (int u = 0; u < ROWS; ++u) {
            const int64_t i = b0 + u * ORTH_THREADS;
            const bool ok = i < i1;
            wv[u] = ok ? w[i] : (T)0;
            vv[u] = ok ? vj[i] : (T)0;
            uv[u] = anc && ok ? au[i] : (T)0;
            rv[u] = anc && ok ? ar[i] : (T)0;
        }
        if constexpr (sizeof(T) == 4) {
            if (a.tc) {                              // H v_j's tensor-core part, plane 0 first
                float d[ROWS];
#pragma unroll
                for (int u = 0; u < ROWS; ++u) d[u] = b0 + u * ORTH_THREADS < i1 ? a.tc[b0 + u * ORTH_THREADS] : 0.f;
                for (int p = 1; p < a.tcn; ++p)
#pragma unroll
                    for (int u = 0; u < ROWS; ++u)
                        if (b0 + u * ORTH_THREADS < i1) d[u] += a.tc[(int64_t)p * n + b0 + u * ORTH_THREADS];
#pragma unroll
                for (int u = 0; u < ROWS; ++u) {
                    wv[u] += d[u];
                    if (b0 + u * ORTH_THREADS < i1) w[b0 + u * ORTH_THREADS] = wv[u];
                }
            }
        }
#pragma unroll
        for (int u = 0; u < ROWS; ++u) {
            const int64_t i = b0 + u * ORTH_THREADS;
            if (i >= i1) break;
            av[0] += vv[u] * wv[u];
            if (anc) {
                av[1] += uv[u] * wv[u];
                av[2] += rv[u] * vv[u];
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (k < nd) av[3 + k] += ay[(int64_t)k * n + i] * wv[u];
            }
        }
    }
    const T beta_m = j > 0 ? (T)__ldcg(a.beta + j - 1) : (T)0;
    const bool always = a.every || pro_always<T>(m, n, ps);
    if (!always) pro.load(a.pro, ps, a.alpha, a.beta, j);
    // no exchange here needs a fence: every CTA works on its own rows, and only
    // the values and the last CTA's stop request travel
    T tot[PA_COLS];
    bool ok;
    if constexpr (sizeof(T) == 4) {
        if (anc) {
            block_sums<T, PA_COLS>(av, scr, nw);
            ok = xchg_totals<T, PA_COLS>(a.xtot, ep, av, G, xs, bc, tot, err, a.spin, &host_stop);
            if (blk == 0 && tid == 0) a.h_m[j] = (double)tot[2];
        }
    }
    if (!anc) {
        T a1[1] = {av[0]}, t1[1];
        block_sums<T, 1>(a1, scr, nw);
        ok = xchg_totals<T, 1>(a.xtot, ep, a1, G, xs, bc, t1, err, a.spin, &host_stop);
#pragma unroll
        for (int q = 0; q < PA_COLS; ++q) tot[q] = (T)0;
        tot[0] = t1[0];
    }
    if (!ok) { leave(true); return; }
    if (host_stop) {
        if (blk == 0 && tid == 0) flags[F_STOP] = 1;
        leave(false);
        return;
    }
    const T alpha0 = tot[0];
    // three-term step (and the anchor projections); ww = w.w, and what is left
    // of w along u and y_k, taken off when w is normalised: alpha v_j and
    // beta v_{j-1} bring back alpha and beta times the rounding-level products
    // u.v_j and u.v_{j-1}, which would grow from step to step
    T ew[1 + ANC_MAX];
#pragma unroll
    for (int q = 0; q < 1 + ANC_MAX; ++q) ew[q] = (T)0;
    for (int64_t b0 = i0 + tid; b0 < i1; b0 += ROWS * ORTH_THREADS) {
        T wv[ROWS], vv[ROWS], pv[ROWS], uv[ROWS];
#pragma unroll
        for (int u = 0; u < ROWS; ++u) {
            const int64_t i = b0 + u * ORTH_THREADS;
            const bool ok = i < i1;
            wv[u] = ok ? w[i] : (T)0;
            vv[u] = ok ? vj[i] : (T)0;
            pv[u] = ok && j > 0 ? vjm[i] : (T)0;
            uv[u] = anc && ok ? au[i] : (T)0;
        }
#pragma unroll
        for (int u = 0; u < ROWS; ++u) {
            const int64_t i = b0 + u * ORTH_THREADS;
            if (i >= i1) break;
            T x = wv[u] - alpha0 * vv[u];
            if (j > 0) x -= beta_m * pv[u];
            if (anc) {
                x -= tot[1] * uv[u];
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (k < nd) x -= tot[3 + k] * ay[(int64_t)k * n + i];
                ew[1] += uv[u] * x;
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (k < nd) ew[2 + k] += ay[(int64_t)k * n + i] * x;
            }
            w[i] = x;
            if (!always) ew[0] += x * x;
        }
    }
    T bb[1] = {(T)0};
    bool project = always;
    if (!always || anc) {
        if constexpr (sizeof(T) == 4) {
            if (anc) {
                block_sums<T, 1 + ANC_MAX>(ew, scr, nw);
                ok = xchg_totals<T, 1 + ANC_MAX>(a.xtot, ep, ew, G, xs, bc, ew, err, a.spin);
                bb[0] = ew[0];
            }
        }
        if (!anc) {
            T s1[1] = {ew[0]};
            block_sums<T, 1>(s1, scr, nw);
            ok = xchg_totals<T, 1>(a.xtot, ep, s1, G, xs, bc + 8, bb, err, a.spin);
        }
        if (!ok) { leave(true); return; }
    }
    if (!always) {
        // does this step project?  (same decision in every CTA; beta in FP32
        // is enough for the estimates)
        if (tid == 0) pro.set(j, (float)alpha0, sqrtf((float)bb[0]));
        __syncthreads();
        const bool over = pro.template over<T>(j, a.delta);
        project = over || force;
        if (project) {
            force = over && !force;
            pro.template projected<T>(j);
        }
    }
    T hj = (T)0;
    if (project) {
        __syncthreads();
        T ww = (T)0;
        for (int pass = 0; pass < 2; ++pass) {       // a second time when the first took more than half (same in every CTA)
            cta_dots<T, CW>(V, m, w, n, i0, i1, pass == 0, red, column);
            if (!xchg_columns<T>(a.xpart, a.xcol, ep, G, pass == 0 ? m + 1 : m, hs, err, a.spin)) {
                leave(true);
                return;
            }
            if (pass == 0) ww = hs[m];
            hj += hs[j];
            T s1[1] = {cta_update<T>(V, m, w, n, i0, i1, hs)};
            block_sums<T, 1>(s1, scr, nw);
            if (!xchg_totals<T, 1>(a.xtot, ep, s1, G, xs, bc + 9 + pass, bb, err, a.spin)) { leave(true); return; }
            if (!(bb[0] < (T)0.5 * ww)) break;
        }
    }
    const T alpha_j = alpha0 + hj;
    // one warp takes the root and the reciprocal: on all sixteen they would
    // hold the FP64 pipe for over a microsecond
    if (tid < 32) {
        const T bt = sqrt(bb[0]);
        const T iv = (T)1 / bt;
        if (tid == 0) {
            bc[11] = bt;
            bc[12] = iv;
        }
    }
    __syncthreads();
    const T beta_j = bc[11];
    bool brk = false;
    if (m < a.mmax) {
        const T scale = fmax(fabs(alpha_j), beta_m);
        brk = !(beta_j > (T)1e-13 * fmax(scale, (T)1e-30));
        if (!brk) {
            const T inv = bc[12];
            T *vn = V + (int64_t)m * n;
            T *vc = (T *)a.vcur;
            for (int64_t b0 = i0 + tid; b0 < i1; b0 += ROWS * ORTH_THREADS) {
                T wv[ROWS], uv[ROWS];
#pragma unroll
                for (int u = 0; u < ROWS; ++u) {
                    const int64_t i = b0 + u * ORTH_THREADS;
                    wv[u] = i < i1 ? w[i] : (T)0;
                    uv[u] = anc && i < i1 ? au[i] : (T)0;
                }
#pragma unroll
                for (int u = 0; u < ROWS; ++u) {
                    const int64_t i = b0 + u * ORTH_THREADS;
                    if (i >= i1) break;
                    T x = wv[u];
                    if (anc) {
                        x -= ew[1] * uv[u];
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            if (k < nd) x -= ew[2 + k] * ay[(int64_t)k * n + i];
                    }
                    x *= inv;
                    vn[i] = x;
                    if (vc) vc[i] = x;
                }
            }
        }
    }
    if (blk == 0) {
        if (!always) {
            pro.advance();
            pro.store(a.pro, ps, j, force);          // every CTA read its copy before the first barrier
        }
        if (tid == 0) {
            if (a.jdev) *a.jdev = j + 1;             // every CTA read j before the first barrier
            a.alpha[j] = (double)alpha_j;
            a.beta[j] = (double)beta_j;
            a.h_alpha[j] = (double)alpha_j;
            a.h_beta[j] = (double)beta_j;
            if (brk) {
                flags[F_BREAK] = m;
                flags[F_STOP] = 2;
                a.h_flags[F_BREAK] = m;
                a.h_flags[F_STOP] = 2;
                __threadfence_system();
            }
        }
    }
    leave(false);
}

// ---------------------------------------------------------------------------
// Persistent chunk kernel of the mixed method (FP32 basis, all sectors on
// FP32 CUDA-core tiles): one cooperative launch runs iterations
// [j0, jend), each as
//   H*psi          work items (32x32 tiles, the long ones split into an H_L
//                  and an H_R + A x B part written to two slot vectors)
//                  shared out over the CTAs, two items per CTA at a time (two
//                  256-thread groups, named barriers); the input is the
//                  previous w'' scaled by 1/beta, the alpha partials come out
//                  of the item epilogues
//   barrier
//   three-term step on the CTA's rows (w = slots - alpha v_j - beta v_{j-1},
//   less the anchored refinement's components along u and y_k), beta^2 = w.w
//   barrier; beta, the omega estimates; at a projecting step the CGS dots,
//   a barrier, column sums, w -= V h, beta^2 partials, a barrier (and again
//   when the projection removed more than half)
// so an iteration costs two grid barriers and no launch.  V rows are only
// touched by the CTA that owns them; the work vectors alternate between two
// buffers so that the items reading w''_{j-1} (all rows) never race with the
// writes of w''_j.  The normalisation v_j = w''_{j-1} / beta_{j-1} is written
// into V[j] by the owner CTA in iteration j.  alpha, beta, the anchor
// couplings and the flags reach the host-visible arrays when the launch ends.

struct ChunkArgs {
    OrthArgs o;                  // V, n, mmax, pstride, alpha/beta, part, bar, flags, mirrors, anchors
    float *buf[2];               // w buffers, iteration j reads buf[j & 1], writes buf[(j+1) & 1]
    float *slot[3];              // H v_j parts
    int j0, jend;
    int first_from_v;            // iteration j0 reads V[j0] itself (start or restart)
    const ItemRec *items;
    int nitems;
    Hv32Ops op;
    // shared-memory copy of the CTA's rows of the last two basis vectors and
    // of the work vector (vc = 2; 0: everything from global memory), `cs`
    // floats per vector
    int vc = 0, cs = 0;
};

constexpr int CHUNK_MAXIT = 16;  // iterations per launch (>= CHECK)

__host__ __device__ inline size_t chunk_smem(int pstride) {
    return 2 * sizeof(Item32Smem) + orth_smem(pstride, OrthCW<float>::value, sizeof(float));
}

// offset of the row cache in k_chunk32's dynamic shared memory
__host__ __device__ inline size_t chunk_cache_off(int pstride) { return (chunk_smem(pstride) + 15) & ~(size_t)15; }

// dynamic shared memory k_chunk32 may take: the 227 KB of one CTA less room
// for its static arrays
constexpr size_t CHUNK_SMEM_MAX = 232448 - 2048;

// NSS_CHUNK_CACHE=0 turns the row cache off (comparisons, experiments)
inline bool chunk_cache_enabled() {
    const char *e = std::getenv("NSS_CHUNK_CACHE");
    return !(e && std::atoi(e) == 0);
}

template <bool ANC>
__global__ void __launch_bounds__(ORTH_THREADS, 1) k_chunk32(ChunkArgs a) {
    constexpr int CW = OrthCW<float>::value;
    int *flags = a.o.flags;
    unsigned epoch = 0;
    if (*(volatile int *)&flags[F_STOP]) {           // set before this launch: uniform
        grid_exit(a.o.bar);
        return;
    }
    extern __shared__ __align__(16) unsigned char chunk_raw[];
    Item32Smem *ism = (Item32Smem *)chunk_raw;
    float *osm = (float *)(chunk_raw + 2 * sizeof(Item32Smem));
    __shared__ float rec_a[CHUNK_MAXIT], rec_b[CHUNK_MAXIT], rec_m[CHUNK_MAXIT];
    const int ps = a.o.pstride;
    float *hs = osm;
    float *red = hs + ps;
    float *scr = red + orth_redsz(ps, CW);
    float *bc = scr + 8 * ORTH_WARPS;
    ProSmem pro(chunk_raw + (chunk_smem(ps) - pro_floats(ps) * sizeof(float)), ps);
    const int G = gridDim.x, blk = blockIdx.x, tid = threadIdx.x, grp = tid >> 8, lt = tid & 255;
    const int64_t n = a.o.n;
    const int64_t chunk = (n + G - 1) / G;
    const int64_t i0 = min(n, (int64_t)blk * chunk), i1 = min(n, i0 + chunk);
    const int nw = (int)min((int64_t)ORTH_WARPS, max((int64_t)1, (chunk + 31) / 32));   // warps with rows
    float *V = (float *)a.o.V;
    float *pA = (float *)a.o.part, *pH = pA + PA_COLS * G, *pB = pH + (int64_t)ps * G, *pH2 = pB + G,
          *pB2 = pH2 + (int64_t)ps * G, *pW = pB2 + G;
    int *err = flags + F_ERR;
    const float *ar = (const float *)a.o.anc_r;
    const AncCols ac{(const float *)a.o.anc_u, (const float *)a.o.defl, a.o.ndefl, n};
    // row cache: the three-term step reads the CTA's rows of v_{j-1} and of
    // the previous w from shared memory instead of L2 (one round of loads
    // less per step); global V and w stay complete
    const bool yc = a.vc > 0;
    const int cs = a.cs;
    float *vcache = (float *)(chunk_raw + chunk_cache_off(ps));   // V[l] at slot l & 1
    float *ycache = vcache + 2 * (size_t)cs;
    float beta_prev = a.j0 > 0 ? (float)a.o.beta[a.j0 - 1] : 0.f;
    pro.load(a.o.pro, ps, a.o.alpha, a.o.beta, a.j0);
    // u.v_j, y_k.v_j and u.v_{j-1}, y_k.v_{j-1}: rounding level, but alpha v_j
    // and beta v_{j-1} in the three-term step would let them grow
    constexpr int NA = ANC ? ANC_MAX : 0;            // anchor columns
    __shared__ float dc[ANC_MAX], dm[ANC_MAX];
    if (tid < NA) {
        dc[tid] = __ldcg(a.o.pro + 2 * ps + 1 + tid);
        dm[tid] = __ldcg(a.o.pro + 2 * ps + 1 + ANC_MAX + tid);
    }
    // the group's first work item, as a rule its only one
    __shared__ ItemRec irec[2];
    const int ti0 = blk + grp * G;
    const bool one = ti0 + 2 * G >= a.nitems;
    if (ti0 < a.nitems && lt == 0) irec[grp] = a.items[ti0];
    __syncthreads();
    int force = __ldcg((const int *)(a.o.pro + 2 * ps));
    int done = 0, brk_m = 0;
    // CTA 0 publishes the completed iterations (device arrays, host mirrors)
    auto publish = [&]() {
        if (tid == 0 && *(volatile int *)err) {
            a.o.h_flags[F_ERR] = 1;
            __threadfence_system();
        }
        if (blk == 0 && done > 0) {
            pro.store(a.o.pro, ps, a.j0 + done - 1, force);
            if (tid < NA) {
                a.o.pro[2 * ps + 1 + tid] = dc[tid];
                a.o.pro[2 * ps + 1 + ANC_MAX + tid] = dm[tid];
            }
        }
        if (blk == 0 && tid == 0) {
            for (int q = 0; q < done; ++q) {
                const int j = a.j0 + q;
                a.o.alpha[j] = (double)rec_a[q];
                a.o.beta[j] = (double)rec_b[q];
                a.o.h_alpha[j] = (double)rec_a[q];
                a.o.h_beta[j] = (double)rec_b[q];
                if constexpr (ANC) a.o.h_m[j] = (double)rec_m[q];
            }
            if (brk_m) {
                flags[F_BREAK] = brk_m;
                flags[F_STOP] = 2;
                a.o.h_flags[F_BREAK] = brk_m;
                a.o.h_flags[F_STOP] = 2;
            }
            __threadfence_system();
        }
        grid_exit(a.o.bar);
    };
    for (int jj = a.j0; jj < a.jend; ++jj) {
        const int m = jj + 1;
        const bool first = jj == a.j0 && a.first_from_v;
        const float *x = first ? V + (int64_t)jj * n : a.buf[jj & 1];
        const float sc = first ? 1.f : 1.f / beta_prev;
        float *y = a.buf[(jj + 1) & 1];
        int host_stop = 0;
        if (blk == 0 && tid == 0) host_stop = *(volatile const int *)(a.o.h_flags + F_NFLAGS);
        // H v_j into the slots; alpha, u.w and y_k.w partials from the items
        float ap[1 + NA];
#pragma unroll
        for (int q = 0; q < 1 + NA; ++q) ap[q] = 0.f;
        // longest items first, one to every CTA before a second joins it (two
        // neighbours of the order per CTA: 1.90 against 1.67 ms at 15 200
        // states, 22 CTAs busy with 44 items)
        for (int ti = ti0; ti < a.nitems; ti += 2 * G) {
            const ItemRec it = ti == ti0 ? irec[grp] : a.items[ti];
            hv32_item<NA>(it, x, a.slot, a.op, ism[grp], lt, GroupSync{1 + grp}, sc, ac, ap, one && jj > a.j0);
        }
        block_sums<float, 1 + NA>(ap, scr);
        if (tid == 0)
#pragma unroll
            for (int q = 0; q < 1 + NA; ++q) pA[q * G + blk] = ap[q];
        if (blk == 0 && tid == 0) flags[F_HOST] = host_stop;
        if (!grid_sync(a.o.bar, epoch, err, a.o.spin)) { publish(); return; }
        const int stop = __ldcg(&flags[F_HOST]);     // looked at below, with the totals
        const float *s0 = a.slot[0], *s1 = a.slot[1], *s2 = a.slot[2];
        // the three-term step's H v_j of the thread's first row, loaded before
        // the alpha total so that the two L2 round trips overlap
        const int64_t if0 = i0 + tid;
        float hv0 = 0.f;
        if (if0 < i1) hv0 = s0[if0] + s1[if0] + s2[if0];
        float tot[1 + NA];
        grid_totals<float, 1 + NA>(pA, G, bc, tot);
        if (stop) {
            if (blk == 0 && tid == 0) flags[F_STOP] = 1;
            publish();
            return;
        }
#pragma unroll
        for (int q = 0; q < NA; ++q) tot[1 + q] -= tot[0] * dc[q] + beta_prev * dm[q];
        const float alpha0 = tot[0];
        // v_j into V (own rows), three-term step, anchor projections; w.w,
        // u.w, y_k.w and r.v_j
        float sv[2 + NA];
#pragma unroll
        for (int q = 0; q < 2 + NA; ++q) sv[q] = 0.f;
        {
            float *vj = V + (int64_t)jj * n;
            const float *vjm = V + (int64_t)(jj > 0 ? jj - 1 : 0) * n;
            // own rows of x: the cached w of the previous iteration of this launch
            const bool xc = yc && jj > a.j0;
            float *vcj = vcache + (jj & 1) * (size_t)cs;
            const float *vcm = vcache + ((jj + 1) & 1) * (size_t)cs;
            for (int64_t i = if0; i < i1; i += ORTH_THREADS) {
                const int r = (int)(i - i0);
                const float v = (xc ? ycache[r] : x[i]) * sc;
                if (!first) vj[i] = v;
                float w = (i == if0 ? hv0 : (s0[i] + s1[i] + s2[i])) - alpha0 * v;
                if (jj > 0) w -= beta_prev * (xc ? vcm[r] : vjm[i]);
                if constexpr (ANC) {
                    sv[1] += ar[i] * v;
                    w -= tot[1] * ac.u[i];
#pragma unroll
                    for (int k = 0; k < ANC_MAX - 1; ++k)
                        if (k < ac.nd) w -= tot[2 + k] * ac.y[(int64_t)k * n + i];
                    sv[2] += ac.u[i] * w;
#pragma unroll
                    for (int k = 0; k < ANC_MAX - 1; ++k)
                        if (k < ac.nd) sv[3 + k] += ac.y[(int64_t)k * n + i] * w;
                }
                y[i] = w;
                if (yc) {
                    vcj[r] = v;
                    ycache[r] = w;
                }
                sv[0] += w * w;
            }
        }
        if constexpr (ANC) {
            block_sums<float, 2 + NA>(sv, scr, nw);
            if (tid == 0)
#pragma unroll
                for (int q = 0; q < 2 + NA; ++q) pW[q * G + blk] = sv[q];
        } else {
            float s1[1] = {sv[0]};
            block_sums<float, 1>(s1, scr, nw);
            if (tid == 0) pW[blk] = s1[0];
        }
        if (!grid_sync(a.o.bar, epoch, err, a.o.spin)) { publish(); return; }
        if constexpr (ANC) {
            grid_totals<float, 2 + NA>(pW, G, bc + 8, sv);
        } else {
            float t1[1];
            grid_totals<float, 1>(pW, G, bc + 8, t1);
            sv[0] = t1[0];
        }
        float bb = sv[0];
        const float mj = sv[1];
        if (tid == 0) pro.set(jj, alpha0, sqrtf(bb));
        __syncthreads();
        // does this step project?  (same decision in every CTA)
        const bool over = pro.over<float>(jj);
        float hj = 0.f;
        if (over || force || pro_always<float>(m, n, ps)) {
            force = over && !force;
            pro.projected<float>(jj);
            // w -= V h
            auto update = [&]() -> float {
                float ss = 0.f;
                for (int64_t i = i0 + tid; i < i1; i += ORTH_THREADS) {
                    float w = y[i];
#pragma unroll 32
                    for (int l = 0; l < m; ++l) w -= V[(int64_t)l * n + i] * hs[l];
                    y[i] = w;
                    if (yc) ycache[i - i0] = w;
                    ss += w * w;
                }
                return ss;
            };
            cta_dots<float, CW>(V, m, y, n, i0, i1, false, red, [&](int l, float t) { pH[(int64_t)l * G + blk] = t; });
            if (!grid_sync(a.o.bar, epoch, err, a.o.spin)) { publish(); return; }
            grid_columns<float>(pH, G, m, hs);
            __syncthreads();
            hj = hs[jj];
            const float ww = bb;
            {
                float s1[1] = {update()};
                block_sums<float, 1>(s1, scr, nw);
                if (tid == 0) pB[blk] = s1[0];
            }
            if (!grid_sync(a.o.bar, epoch, err, a.o.spin)) { publish(); return; }
            float t1[1];
            grid_totals<float, 1>(pB, G, bc + 15, t1);
            bb = t1[0];
            if (bb < 0.5f * ww) {   // second projection (same decision in every CTA)
                cta_dots<float, CW>(V, m, y, n, i0, i1, false, red, [&](int l, float t) { pH2[(int64_t)l * G + blk] = t; });
                if (!grid_sync(a.o.bar, epoch, err, a.o.spin)) { publish(); return; }
                grid_columns<float>(pH2, G, m, hs);
                __syncthreads();
                hj += hs[jj];
                float s1[1] = {update()};
                block_sums<float, 1>(s1, scr, nw);
                if (tid == 0) pB2[blk] = s1[0];
                if (!grid_sync(a.o.bar, epoch, err, a.o.spin)) { publish(); return; }
                grid_totals<float, 1>(pB2, G, bc + 6, t1);
                bb = t1[0];
            }
        }
        const float alpha_j = alpha0 + hj;
        const float beta_j = sqrtf(bb);
        bool brk = false;
        if (m < a.o.mmax) {
            const float scale = fmaxf(fabsf(alpha_j), jj > 0 ? beta_prev : 0.f);
            brk = !(beta_j > 1e-13f * fmaxf(scale, 1e-30f));
        }
        if (blk == 0 && tid == 0) {
            rec_a[done] = alpha_j;
            rec_b[done] = beta_j;
            rec_m[done] = mj;
        }
        if (tid == 0) pro.set(jj, alpha_j, beta_j);
        pro.advance();
        if (tid < NA) {
            dm[tid] = dc[tid];
            dc[tid] = bc[8 + 2 + tid] / beta_j;      // the totals of sv
        }
        ++done;
        if (brk) {
            brk_m = m;
            __syncthreads();
            publish();
            return;
        }
        beta_prev = beta_j;
        __syncthreads();
    }
    publish();
}

// ---------------------------------------------------------------------------
// Batched persistent kernel: several independent mixed-precision solves (one
// context each) advance together, one launch per chunk of iterations.  The
// H*psi work items of all solves are shared out over all CTAs (longest
// first); each solve's rows belong to its own range of CTAs, which run its
// three-term step, projections and updates.  The grid barriers are global,
// so every CTA takes the same barrier sequence: the per-solve decisions that
// change it (second projection, breakdown, end of the chunk) are recomputed
// by every CTA from the solves' partial sums, in the same order, so all CTAs
// agree.  The omega estimates belong to a solve's own CTAs, so their verdict
// reaches the others one step later: v_{j+1} over the threshold makes the
// steps j+1 and j+2 project, with the threshold a quarter of the one of the
// single-solve kernels for that step of growth.  All solves project together:
// one solve's projection already costs everybody its two barriers, and solves
// that start over at the same time come due at about the same time.  Solves stop within a launch only at their chunk end or at a
// breakdown; the host checks convergence between launches.

struct BatchSolve {
    ChunkArgs c;                 // per-solve arguments (c.o.bar unused)
    float *pitem;                // [2 c.nitems] alpha and u.w partials of the solve's items
    int cta0, ncta;              // CTAs owning the solve's rows
    int active;                  // takes part in this launch
    int pad;
};

struct BatchArgs {
    const BatchSolve *s;
    int ns;
    int nitems;                  // items of all active solves
    const int2 *gitems;          // (solve, item) in processing order
    float *st;                   // [ST_WORDS ns] per-solve scalars published inside an iteration (batch_words.hpp)
    unsigned *bar;               // global barrier
    int *err;
    int steps;                   // iterations of this launch
    uint32_t spin;               // poll limit of the grid barriers (wait_limit)
    unsigned *qcnt;              // [CHUNK_MAXIT] item queue heads, zero at launch
};

constexpr int BATCH_MAX = 160;   // solves per launch (each needs a CTA)

__global__ void __launch_bounds__(ORTH_THREADS, 1) k_batch32(BatchArgs B) {
    constexpr int CW = OrthCW<float>::value;
    extern __shared__ __align__(16) unsigned char batch_raw[];
    Item32Smem *ism = (Item32Smem *)batch_raw;
    float *osm = (float *)(batch_raw + 2 * sizeof(Item32Smem));
    __shared__ float rec_a[CHUNK_MAXIT], rec_b[CHUNK_MAXIT], rec_m[CHUNK_MAXIT];
    __shared__ float bprev[BATCH_MAX], balpha[BATCH_MAX], bbb[BATCH_MAX];
    __shared__ int alive[BATCH_MAX], p2[BATCH_MAX], brkm[BATCH_MAX];
    __shared__ int my_s, any_p2;
    __shared__ int qn[2];
    const int blk = blockIdx.x, tid = threadIdx.x, grp = tid >> 8, lt = tid & 255;
    const int ns = B.ns;
    unsigned epoch = 0;
    if (tid == 0) {
        my_s = -1;
        for (int s = 0; s < ns; ++s)
            if (B.s[s].active && blk >= B.s[s].cta0 && blk < B.s[s].cta0 + B.s[s].ncta) my_s = s;
    }
    for (int s = tid; s < ns; s += ORTH_THREADS) {
        const BatchSolve &S = B.s[s];
        const int j0 = S.c.j0;
        alive[s] = S.active && !*(volatile int *)&S.c.o.flags[F_STOP] && S.c.jend > j0;
        bprev[s] = j0 > 0 ? (float)S.c.o.beta[j0 - 1] : 0.f;
        brkm[s] = 0;
    }
    __syncthreads();
    const int me = my_s;
    // this CTA's own solve (if any)
    const BatchSolve *Mp = me >= 0 ? &B.s[me] : nullptr;
    const int Gs = Mp ? Mp->ncta : 1, lb = Mp ? blk - Mp->cta0 : 0;
    const int ps = Mp ? Mp->c.o.pstride : 8;
    float *hs = osm;
    float *red = hs + ps;
    float *scr = red + orth_redsz(ps, CW);
    float *bc = scr + 8 * ORTH_WARPS;
    ProSmem pro(batch_raw + (chunk_smem(ps) - pro_floats(ps) * sizeof(float)), ps);
    const int64_t n = Mp ? Mp->c.o.n : 0;
    const int64_t chunk = (n + Gs - 1) / Gs;
    const int64_t i0 = min(n, (int64_t)lb * chunk), i1 = min(n, i0 + chunk);
    if (Mp) pro.load(Mp->c.o.pro, ps, Mp->c.o.alpha, Mp->c.o.beta, Mp->c.j0);
    float dc = Mp ? __ldcg(Mp->c.o.pro + 2 * ps + 1) : 0.f;            // u.v_j, u.v_{j-1} (see k_chunk32)
    float dm = Mp ? __ldcg(Mp->c.o.pro + 2 * ps + 1 + ANC_MAX) : 0.f;
    int owed = Mp ? __ldcg((const int *)(Mp->c.o.pro + 2 * ps)) : 0;   // projections its estimates still ask for
    float *V = Mp ? (float *)Mp->c.o.V : nullptr;
    float *pA = Mp ? (float *)Mp->c.o.part : nullptr;
    float *pH = pA + PA_COLS * Gs, *pB = pH + (int64_t)ps * Gs, *pH2 = pB + Gs, *pB2 = pH2 + (int64_t)ps * Gs,
          *pW = pB2 + Gs;
    const float *au = Mp ? (const float *)Mp->c.o.anc_u : nullptr;
    const float *ar = Mp ? (const float *)Mp->c.o.anc_r : nullptr;
    const bool anc = au != nullptr;          // no deflation vectors: one state a solve
    int done = 0;
    for (int step = 0; step < B.steps; ++step) {
        // ---- H*psi of every running solve, all items over all CTAs: each
        // thread group takes the next item off a global queue (longest
        // first), fetching the index after next while it works on one
        if (lt == 0) qn[grp] = (int)atomicAdd(B.qcnt + step, 1u);
        GroupSync{1 + grp}();
        for (int gi = qn[grp]; gi < B.nitems;) {
            int nxt = 0;
            if (lt == 0) nxt = (int)atomicAdd(B.qcnt + step, 1u);
            const int2 g = B.gitems[gi];
            const BatchSolve &S = B.s[g.x];
            const int tj = S.c.j0 + step;
            if (alive[g.x] && tj < S.c.jend) {
                const bool first = tj == S.c.j0 && S.c.first_from_v;
                const float *x = first ? (const float *)S.c.o.V + (int64_t)tj * S.c.o.n : S.c.buf[tj & 1];
                const float sc = first ? 1.f : 1.f / bprev[g.x];
                const AncCols ac{(const float *)S.c.o.anc_u, nullptr, 0, 0};
                float ap[2] = {0.f, 0.f};
                hv32_item<1>(S.c.items[g.y], x, S.c.slot, S.c.op, ism[grp], lt, GroupSync{1 + grp}, sc, ac, ap,
                             false);
                // group sums of the alpha and u.w partials (named barrier of the group)
                const float a0 = warp_sum<float>(ap[0]), a1 = warp_sum<float>(ap[1]);
                if ((lt & 31) == 0) {
                    scr[grp * 16 + (lt >> 5)] = a0;
                    scr[grp * 16 + 8 + (lt >> 5)] = a1;
                }
                GroupSync{1 + grp}();
                if (lt < 2) {
                    float t = 0.f;
                    for (int q = 0; q < 8; ++q) t += scr[grp * 16 + 8 * lt + q];
                    S.pitem[(int64_t)lt * S.c.nitems + g.y] = t;
                }
            }
            GroupSync{1 + grp}();
            if (lt == 0) qn[grp] = nxt;
            GroupSync{1 + grp}();
            gi = qn[grp];
        }
        if (!grid_sync(B.bar, epoch, B.err, B.spin)) break;
        const bool run = me >= 0 && alive[me] && Mp->c.j0 + step < Mp->c.jend;
        const int jj = Mp ? Mp->c.j0 + step : 0, m = jj + 1;
        const bool first = run && jj == Mp->c.j0 && Mp->c.first_from_v;
        const float *x = run ? (first ? V + (int64_t)jj * n : Mp->c.buf[jj & 1]) : nullptr;
        const float sc = first ? 1.f : (me >= 0 ? 1.f / bprev[me] : 1.f);
        float *y = run ? Mp->c.buf[(jj + 1) & 1] : nullptr;
        const int nw = (int)min((int64_t)ORTH_WARPS, max((int64_t)1, (chunk + 31) / 32));
        float alpha0 = 0.f, mj = 0.f, hj = 0.f, ud = 0.f;
        if (run) {
            float uw = 0.f;
            {   // alpha (and u.w) from the item partials, fixed order
                if (tid < 64) {
                    float t = strided_sum<float>(Mp->pitem + (int64_t)(tid >> 5) * Mp->c.nitems, tid & 31, Mp->c.nitems, 32);
                    t = warp_sum<float>(t);
                    if ((tid & 31) == 0) bc[tid >> 5] = t;
                }
                __syncthreads();
                alpha0 = bc[0];
                uw = bc[1] - alpha0 * dc - (jj > 0 ? bprev[me] * dm : 0.f);
            }
            float *vj = V + (int64_t)jj * n;
            const float *vjm = V + (int64_t)(jj > 0 ? jj - 1 : 0) * n;
            const float *s0 = Mp->c.slot[0], *s1 = Mp->c.slot[1], *s2 = Mp->c.slot[2];
            float sv[3] = {0.f, 0.f, 0.f};
            for (int64_t i = i0 + tid; i < i1; i += ORTH_THREADS) {
                const float v = x[i] * sc;
                if (!first) vj[i] = v;
                float w = (s0[i] + s1[i] + s2[i]) - alpha0 * v;
                if (jj > 0) w -= bprev[me] * vjm[i];
                if (anc) {
                    sv[1] += ar[i] * v;
                    w -= uw * au[i];
                    sv[2] += au[i] * w;
                }
                y[i] = w;
                sv[0] += w * w;
            }
            block_sums<float, 3>(sv, scr, nw);
            if (tid == 0) {
                pW[lb] = sv[0];
                pW[Gs + lb] = sv[1];
                pW[2 * Gs + lb] = sv[2];
                if (lb == 0) {
                    B.st[ST_WORDS * me + ST_ALPHA] = alpha0;
                    B.st[ST_WORDS * me + ST_HJ] = 0.f;          // h_j of a projection
                }
            }
        }
        if (!grid_sync(B.bar, epoch, B.err, B.spin)) break;
        // every CTA: w.w and whether the step projects, of every solve
        if (tid == 0) any_p2 = 0;
        __syncthreads();
        for (int s = tid; s < ns; s += ORTH_THREADS) {
            const BatchSolve &S = B.s[s];
            p2[s] = 0;
            if (!alive[s] || S.c.j0 + step >= S.c.jend) continue;
            const float *pWs = (const float *)S.c.o.part + (PA_COLS + 2 * (int64_t)S.c.o.pstride + 2) * S.ncta;
            bbb[s] = strided_sum<float>(pWs, 0, S.ncta, 1);
            balpha[s] = __ldcg(B.st + ST_WORDS * s + ST_ALPHA);
            const int ow = step == 0 ? __ldcg((const int *)(S.c.o.pro + 2 * S.c.o.pstride))
                                     : __float_as_int(__ldcg(B.st + ST_WORDS * s + owed_word(step - 1)));
            p2[s] = 1;
            if (ow > 0 || pro_always<float>(S.c.j0 + step + 1, S.c.o.n, S.c.o.pstride)) any_p2 = 1;
        }
        __syncthreads();
        auto update = [&]() -> float {
            float ss = 0.f;
            for (int64_t i = i0 + tid; i < i1; i += ORTH_THREADS) {
                float w = y[i];
#pragma unroll 32
                for (int l = 0; l < m; ++l) w -= V[(int64_t)l * n + i] * hs[l];
                y[i] = w;
                ss += w * w;
            }
            return ss;
        };
        if (run) {
            float t2[2];
            grid_totals<float, 2>(pW + Gs, Gs, bc + 2, t2);
            mj = t2[0];
            ud = t2[1];
            if (tid == 0) pro.set(jj, alpha0, sqrtf(bbb[me]));
            __syncthreads();
            const bool over = pro.over<float>(jj, 0.25f * Pro<float>::DELTA);
            if (any_p2) {
                pro.projected<float>(jj);
                if (owed > 0) --owed;
            } else if (over) {
                owed = 2;
            }
        }
        // the projections, up to two rounds (the second for the solves that
        // lost more than half); pH / pB, then pH2 / pB2
        for (int round = 0; round < 2 && any_p2; ++round) {
            const bool mine = run && p2[me];
            float *ph = round == 0 ? pH : pH2, *pb = round == 0 ? pB : pB2;
            if (mine)
                cta_dots<float, CW>(V, m, y, n, i0, i1, false, red,
                                    [&](int l, float t) { ph[(int64_t)l * Gs + lb] = t; });
            if (!grid_sync(B.bar, epoch, B.err, B.spin)) { done = -1; break; }
            if (mine) {
                grid_columns<float>(ph, Gs, m, hs);
                __syncthreads();
                hj += hs[jj];
                if (lb == 0 && tid == 0) B.st[ST_WORDS * me + ST_HJ] = hj;
                float s1[1] = {update()};
                block_sums<float, 1>(s1, scr, nw);
                if (tid == 0) pb[lb] = s1[0];
            }
            if (!grid_sync(B.bar, epoch, B.err, B.spin)) { done = -1; break; }
            if (tid == 0) any_p2 = 0;
            __syncthreads();
            for (int s = tid; s < ns; s += ORTH_THREADS) {
                if (!p2[s]) continue;
                const BatchSolve &S = B.s[s];
                const float *pBs = (const float *)S.c.o.part +
                                   (PA_COLS + (round + 1) * (int64_t)S.c.o.pstride + round) * S.ncta;
                const float t = strided_sum<float>(pBs, 0, S.ncta, 1);
                const bool again = round == 0 && t < 0.5f * bbb[s];
                bbb[s] = t;
                balpha[s] = __ldcg(B.st + ST_WORDS * s + ST_ALPHA) + __ldcg(B.st + ST_WORDS * s + ST_HJ);
                p2[s] = again;
                if (again) any_p2 = 1;
            }
            __syncthreads();
        }
        if (done < 0) {                              // a barrier ran out
            done = 0;
            break;
        }
        // every CTA: beta, breakdown, next scale of every solve that ran
        for (int s = tid; s < ns; s += ORTH_THREADS) {
            const BatchSolve &S = B.s[s];
            if (!alive[s] || S.c.j0 + step >= S.c.jend) continue;
            const float beta = sqrtf(bbb[s]);
            const int ms = S.c.j0 + step + 1;
            if (ms < S.c.o.mmax) {
                const float scale = fmaxf(fabsf(balpha[s]), S.c.j0 + step > 0 ? bprev[s] : 0.f);
                if (!(beta > 1e-13f * fmaxf(scale, 1e-30f))) {
                    brkm[s] = ms;
                    alive[s] = 0;
                }
            }
            bprev[s] = beta;
        }
        __syncthreads();
        if (run) {
            if (lb == 0 && tid == 0) {
                rec_a[done] = balpha[me];
                rec_b[done] = bprev[me];
                rec_m[done] = mj;
                B.st[ST_WORDS * me + owed_word(step)] = __int_as_float(owed);   // read by all in the next step
            }
            if (tid == 0) pro.set(jj, balpha[me], bprev[me]);
            dm = dc;
            dc = anc ? ud / bprev[me] : 0.f;
            pro.advance();
            ++done;
        }
    }
    // publish the completed iterations of the own solve
    __syncthreads();
    if (me >= 0 && lb == 0 && done > 0) {
        pro.store(Mp->c.o.pro, ps, Mp->c.j0 + done - 1, owed);
        if (tid == 0) {
            Mp->c.o.pro[2 * ps + 1] = dc;
            Mp->c.o.pro[2 * ps + 1 + ANC_MAX] = dm;
        }
    }
    if (me >= 0 && lb == 0 && tid == 0) {
        const ChunkArgs &a = Mp->c;
        for (int q = 0; q < done; ++q) {
            const int j = a.j0 + q;
            a.o.alpha[j] = (double)rec_a[q];
            a.o.beta[j] = (double)rec_b[q];
            a.o.h_alpha[j] = (double)rec_a[q];
            a.o.h_beta[j] = (double)rec_b[q];
            if (anc) a.o.h_m[j] = (double)rec_m[q];
        }
        if (brkm[me]) {
            a.o.flags[F_BREAK] = brkm[me];
            a.o.flags[F_STOP] = 2;
            a.o.h_flags[F_BREAK] = brkm[me];
            a.o.h_flags[F_STOP] = 2;
        }
        __threadfence_system();
    }
    grid_exit(B.bar);
}

// Ritz vectors: out[e] = sum_l V[l] s_e[l]   (FP64 accumulation, FP64 out)
template <class T>
__global__ void __launch_bounds__(256) k_ritz(const T *__restrict__ V, int m, int64_t n,
                                              const double *__restrict__ svec, int sstride, int ne,
                                              double *__restrict__ out) {
    extern __shared__ double ss[];   // [ne][m]
    for (int t = threadIdx.x; t < ne * m; t += blockDim.x) ss[t] = svec[(int64_t)(t / m) * sstride + (t % m)];
    __syncthreads();
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        double acc[4] = {0, 0, 0, 0};
        for (int l = 0; l < m; ++l) {
            const double v = (double)V[(int64_t)l * n + i];
            for (int e = 0; e < ne && e < 4; ++e) acc[e] = fma(v, ss[e * m + l], acc[e]);
        }
        for (int e = 0; e < ne && e < 4; ++e) out[(int64_t)e * n + i] = acc[e];
    }
}

// FP64 refinement: r[0] = psi.w, r[1] = w.w, r[2] = psi.psi (grid reduction)
__global__ void __launch_bounds__(256) k_rq(const double *__restrict__ psi, const double *__restrict__ w, int64_t n,
                                            double *__restrict__ part, double *__restrict__ r, unsigned *counter) {
    const int tid = threadIdx.x;
    double a = 0.0, b = 0.0, c = 0.0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + tid; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        a = fma(psi[i], w[i], a);
        b = fma(w[i], w[i], b);
        c = fma(psi[i], psi[i], c);
    }
    a = warp_sum<double>(a);
    b = warp_sum<double>(b);
    c = warp_sum<double>(c);
    __shared__ double red[3][8];
    if ((tid & 31) == 0) { red[0][tid >> 5] = a; red[1][tid >> 5] = b; red[2][tid >> 5] = c; }
    __syncthreads();
    if (tid < 3) {
        double t = 0.0;
        for (int q = 0; q < 8; ++q) t += red[tid][q];
        part[(int64_t)tid * gridDim.x + blockIdx.x] = t;
    }
    if (!last_block(counter)) return;
    for (int q = 0; q < 3; ++q) {
        const double t = lastblock_sum(part + (int64_t)q * gridDim.x, gridDim.x);
        if (tid == 0) r[q] = t;
    }
    if (tid == 0) *counter = 0u;
}

// ||w - theta psi||^2 (grid reduction); theta = r[0]/r[2]
__global__ void __launch_bounds__(256) k_resid(const double *__restrict__ psi, const double *__restrict__ w, int64_t n,
                                               double *__restrict__ part, double *__restrict__ r, unsigned *counter) {
    const int tid = threadIdx.x;
    const double th = r[0] / r[2];
    double a = 0.0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + tid; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const double d = w[i] - th * psi[i];
        a = fma(d, d, a);
    }
    a = warp_sum<double>(a);
    __shared__ double red[8];
    if ((tid & 31) == 0) red[tid >> 5] = a;
    __syncthreads();
    if (tid == 0) {
        double t = 0.0;
        for (int q = 0; q < 8; ++q) t += red[q];
        part[blockIdx.x] = t;
    }
    if (!last_block(counter)) return;
    const double t = lastblock_sum(part, gridDim.x);
    if (tid != 0) return;
    r[3] = t;
    *counter = 0u;
}

// Anchor residual: w <- w - theta0 psi with theta0 = r[0]/r[2] (from k_rq),
// and r[4] = ||w||^2 (grid reduction)
__global__ void __launch_bounds__(256) k_anchor_r(const double *__restrict__ psi, double *__restrict__ w, int64_t n,
                                                  double *__restrict__ part, double *__restrict__ r, unsigned *counter) {
    const int tid = threadIdx.x;
    const double th = r[0] / r[2];
    double a = 0.0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + tid; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const double d = w[i] - th * psi[i];
        w[i] = d;
        a = fma(d, d, a);
    }
    a = warp_sum<double>(a);
    __shared__ double red[8];
    if ((tid & 31) == 0) red[tid >> 5] = a;
    __syncthreads();
    if (tid == 0) {
        double t = 0.0;
        for (int q = 0; q < 8; ++q) t += red[q];
        part[blockIdx.x] = t;
    }
    if (!last_block(counter)) return;
    const double t = lastblock_sum(part, gridDim.x);
    if (tid != 0) return;
    r[4] = t;
    *counter = 0u;
}

// Gram matrix of k <= 4 FP64 vectors against k others: r[i*k+j] = U_i . W_j
// (grid reduction; part holds k*k columns of gridDim.x partials)
__global__ void __launch_bounds__(256) k_gram(const double *__restrict__ U, const double *__restrict__ W, int k,
                                              int64_t n, double *__restrict__ part, double *__restrict__ r,
                                              unsigned *counter) {
    const int tid = threadIdx.x;
    double acc[16];
#pragma unroll
    for (int q = 0; q < 16; ++q) acc[q] = 0.0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + tid; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        double u[4], w[4];
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            u[a] = a < k ? U[(int64_t)a * n + i] : 0.0;
            w[a] = a < k ? W[(int64_t)a * n + i] : 0.0;
        }
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
            for (int b = 0; b < 4; ++b) acc[a * 4 + b] = fma(u[a], w[b], acc[a * 4 + b]);
    }
    __shared__ double red[16][8];
#pragma unroll
    for (int q = 0; q < 16; ++q) {
        const double v = warp_sum<double>(acc[q]);
        if ((tid & 31) == 0) red[q][tid >> 5] = v;
    }
    __syncthreads();
    if (tid < k * k) {
        const int a = tid / k, b = tid % k;
        double t = 0.0;
        for (int q = 0; q < 8; ++q) t += red[a * 4 + b][q];
        part[(int64_t)tid * gridDim.x + blockIdx.x] = t;
    }
    if (!last_block(counter)) return;
    for (int q = 0; q < k * k; ++q) {
        const double t = lastblock_sum(part + (int64_t)q * gridDim.x, gridDim.x);
        if (tid == 0) r[q] = t;
    }
    if (tid == 0) *counter = 0u;
}

// X <- X Q for k <= 4 FP64 vectors (Q column-major k x k)
struct Rot4 {
    double q[16];
};
__global__ void __launch_bounds__(256) k_rot(double *__restrict__ X, int k, int64_t n, Rot4 Q) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        double x[4], y[4];
#pragma unroll
        for (int a = 0; a < 4; ++a) x[a] = a < k ? X[(int64_t)a * n + i] : 0.0;
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            double t = 0.0;
#pragma unroll
            for (int a = 0; a < 4; ++a) t = fma(x[a], Q.q[b * 4 + a], t);
            y[b] = t;
        }
#pragma unroll
        for (int b = 0; b < 4; ++b)
            if (b < k) X[(int64_t)b * n + i] = y[b];
    }
}

// Eigenvalues (ascending) and orthonormal eigenvectors (columns of q,
// column-major k x k) of a symmetric k x k matrix a (row-major, destroyed),
// k <= 4, by cyclic Jacobi rotations.
void sym_eig_small(int k, double *a, double *lam, double *q) {
    if (k < 1 || k > 4) return;   // callers pass 1..4
    for (int i = 0; i < k; ++i)
        for (int j = 0; j < k; ++j) q[j * k + i] = i == j ? 1.0 : 0.0;
    for (int sweep = 0; sweep < 50; ++sweep) {
        double off = 0.0, tot = 0.0;
        for (int i = 0; i < k; ++i)
            for (int j = 0; j < k; ++j) {
                tot += a[i * k + j] * a[i * k + j];
                if (i != j) off += a[i * k + j] * a[i * k + j];
            }
        if (off <= 1e-34 * tot) break;
        for (int p = 0; p < k; ++p)
            for (int r = p + 1; r < k; ++r) {
                const double apr = a[p * k + r];
                if (apr == 0.0) continue;
                const double tau = (a[r * k + r] - a[p * k + p]) / (2.0 * apr);
                const double t = (tau >= 0.0 ? 1.0 : -1.0) / (std::fabs(tau) + std::sqrt(1.0 + tau * tau));
                const double cs = 1.0 / std::sqrt(1.0 + t * t), sn = t * cs;
                for (int i = 0; i < k; ++i) {   // columns p, r
                    const double x = a[i * k + p], y = a[i * k + r];
                    a[i * k + p] = cs * x - sn * y;
                    a[i * k + r] = sn * x + cs * y;
                }
                for (int j = 0; j < k; ++j) {   // rows p, r
                    const double x = a[p * k + j], y = a[r * k + j];
                    a[p * k + j] = cs * x - sn * y;
                    a[r * k + j] = sn * x + cs * y;
                }
                for (int i = 0; i < k; ++i) {
                    const double x = q[p * k + i], y = q[r * k + i];
                    q[p * k + i] = cs * x - sn * y;
                    q[r * k + i] = sn * x + cs * y;
                }
            }
    }
    // ascending by the diagonal: insertion sort (equal values keep their order)
    int ord[4] = {0, 1, 2, 3};
    for (int j = 1; j < k; ++j) {
        const int x = ord[j];
        int i = j;
        for (; i > 0 && a[x * k + x] < a[ord[i - 1] * k + ord[i - 1]]; --i) ord[i] = ord[i - 1];
        ord[i] = x;
    }
    double qs[16];
    for (int j = 0; j < k; ++j) {
        lam[j] = a[ord[j] * k + ord[j]];
        for (int i = 0; i < k; ++i) qs[j * k + i] = q[ord[j] * k + i];
    }
    for (int t = 0; t < k * k; ++t) q[t] = qs[t];
}

// out = (float)(x * s)
__global__ void k_to32(float *__restrict__ out, const double *__restrict__ x, double s, int64_t n) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        out[i] = (float)(x[i] * s);
}

// The FP32 vectors of an anchored run: v = (float)(r s), the start vector,
// u32 = (float)u, r32 = (float)r
__global__ void k_anchor32(float *__restrict__ v, float *__restrict__ u32, float *__restrict__ r32,
                           const double *__restrict__ u, const double *__restrict__ r, double s, int64_t n) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        v[i] = (float)(r[i] * s);
        u32[i] = (float)u[i];
        r32[i] = (float)r[i];
    }
}

// The start of a batched solve's run: k_pro_reset, and zeros in the flags, beta
// and the product slots that no item may write (one launch instead of four
// calls a solve)
__global__ void k_run_reset(float *pro, int ps, float eps1, int *flags, double *beta, int nbeta, float *slots, int64_t nslots) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, nt = (int64_t)gridDim.x * blockDim.x;
    for (int64_t k = t; k < 2 * ps; k += nt) pro[k] = eps1;
    if (t < PRO_TAIL) pro[2 * ps + t] = 0.f;
    if (t < F_NFLAGS) flags[t] = 0;
    for (int64_t k = t; k < nbeta; k += nt) beta[k] = 0.0;
    for (int64_t k = t; k < nslots; k += nt) slots[k] = 0.f;
}

// Ritz vectors of ne states from the coefficients svec[e * m + l] in shared
// memory: all states in one pass over the basis, or one after the other where
// their coefficients do not fit together
template <class T>
int launch_ritz(Ctx &c, const T *V, int m, int64_t n, const double *svec, int ne, double *out, cudaStream_t st,
                int64_t &launches) {
    const int at_once = (size_t)ne * m * sizeof(double) <= CHUNK_SMEM_MAX ? ne : 1;
    const size_t smem = (size_t)at_once * m * sizeof(double);
    NSS_CUDA_TRY(c, allow_smem((const void *)k_ritz<T>, smem));
    for (int e = 0; e < ne; e += at_once) {
        ++launches;
        k_ritz<T><<<NBLK, 256, smem, st>>>(V, m, n, svec + (int64_t)e * m, m, at_once, out + (int64_t)e * n);
    }
    NSS_CUDA_TRY(c, cudaGetLastError());
    return NSS_OK;
}

// x <- x / ||x|| on stream st (two launches)
template <class T>
void normalize_dev(DevLanczos &z, T *x, int64_t n, cudaStream_t st, int64_t &launches) {
    k_sumsq<T><<<NBLK, 256, 0, st>>>(x, n, z.part, z.scal + S_NRM, z.counter);
    k_scale<T><<<NBLK, 256, 0, st>>>(x, n, z.scal + S_NRM);
    launches += 1;   // the caller counted one launch for the normalisation
}

// words of a workspace's exchange area (w: words per value)
inline size_t x_words(int pstride, int w) {
    return 1 + (size_t)XCOLS * (XMAX + 1) + (size_t)w * pstride * (1 + XMAX);
}

// per-eigenvector scratch row of svec
inline int svec_stride(int cap) { return 4 * (cap + 1); }

// Memory for a Lanczos workspace.  A DMRG run solves another size at every
// step; allocating and freeing two dozen arrays took 100 to 260 us a step
// (of 2 ms in a chain of 20 spins), so they are sections of one block that the
// context keeps while it fits: with a quarter to spare (64 MB at most), given
// back when less than a quarter of it would be used (above 64 MB) and with the
// context.  A context with a budget allocates each array for itself, so that
// what it holds is what the solve needs.
int workspace(Ctx &c, const std::vector<std::pair<void **, size_t>> &want) {
    if (c.budget) {
        for (auto &w : want) {
            char *p = nullptr;
            NSS_CUDA_TRY(c, ctx_alloc(c, &p, w.second));
            *w.first = p;
        }
        return NSS_OK;
    }
    auto up = [](size_t b) { return (b + 255) & ~(size_t)255; };
    size_t need = 0;
    for (auto &w : want) need += up(w.second);
    constexpr size_t SMALL = (size_t)64 << 20;
    if (need > c.lz_arena_bytes || (c.lz_arena_bytes > SMALL && need < c.lz_arena_bytes / 4)) {
        ctx_free(c, c.lz_arena);
        c.lz_arena = nullptr;
        c.lz_arena_bytes = 0;
        const size_t roomy = std::max(need + std::min(need / 4, SMALL), (size_t)8 << 20);
        if (ctx_alloc(c, &c.lz_arena, roomy) == cudaSuccess) {
            c.lz_arena_bytes = roomy;
        } else {
            cudaGetLastError();                      // no room for the spare part
            NSS_CUDA_TRY(c, ctx_alloc(c, &c.lz_arena, need));
            c.lz_arena_bytes = need;
        }
    }
    size_t at = 0;
    for (auto &w : want) {
        *w.first = c.lz_arena + at;
        at += up(w.second);
    }
    return NSS_OK;
}

int ensure_lanczos(Ctx &c, int64_t n, int cap, bool mixed) {
    DevLanczos &z = c.lz;
    // reuse only buffers shaped for this mode: the FP64 method needs a whole
    // FP64 basis in V, the mixed one an FP32 basis in V32
    if (z.V && z.n == n && z.cap >= cap && (mixed ? (z.V32 != nullptr) : z.full64)) return NSS_OK;
    lanczos_release(c, true);
    z.n = n;
    z.cap = cap;
    std::vector<std::pair<void **, size_t>> want;    // the workspace's arrays and their bytes
    auto add = [&](auto *p, size_t count) { want.push_back({(void **)p, std::max<size_t>(count * sizeof(**p), 16)}); };
    if (mixed) {
        add(&z.V32, (size_t)(cap + 1) * n);
        add(&z.w32, (size_t)n);
        add(&z.anc32, (size_t)6 * n);   // FP32 anchor, residual, deflation set
        add(&z.V, (size_t)n);   // FP64 refinement scratch
        z.full64 = false;
    } else {
        add(&z.V, (size_t)(cap + 1) * n);
        z.full64 = true;
    }
    int dev = 0, nsm = 0;
    NSS_CUDA_TRY(c, cudaGetDevice(&dev));
    NSS_CUDA_TRY(c, cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    const int pstride = cap + 8;   // m+1 columns plus the anchored refinement's extras
    const int cw = mixed ? OrthCW<float>::value : OrthCW<double>::value;
    const size_t smem = orth_smem(pstride, cw, mixed ? sizeof(float) : sizeof(double));
    const void *fn = mixed ? (const void *)k_orth<float, OrthCW<float>::value>
                           : (const void *)k_orth<double, OrthCW<double>::value>;
    NSS_CUDA_TRY(c, allow_smem(fn, smem));
    int occ = 0;
    NSS_CUDA_TRY(c, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fn, ORTH_THREADS, smem));
    if (occ < 1) {
        c.err = "nss_eigh: Krylov basis too large for the orthogonalisation kernel's shared memory";
        return NSS_ERR_INVALID;
    }
    z.orth_grid = std::min(nsm, XMAX);      // one CTA per SM, all resident (cooperative launch)
    z.orth_smem = smem;
    z.chunk_ok = false;
    if (mixed) {
        // the persistent chunk kernel of the mixed method
        const size_t csm = chunk_smem(pstride);
        // the row cache: the CTA's rows of the work vector and of the last two
        // basis vectors, where they fit beside the rest
        const int64_t rows = (n + nsm - 1) / nsm;
        const int cs = (int)((rows + 3) & ~(int64_t)3);
        const size_t coff = chunk_cache_off(pstride), vbytes = (size_t)cs * sizeof(float);
        int vc = 0;
        if (chunk_cache_enabled() && coff + 3 * vbytes <= CHUNK_SMEM_MAX) vc = 2;
        const size_t csm_vc = vc > 0 ? coff + (size_t)(vc + 1) * vbytes : csm;
        for (const void *fn : {(const void *)k_chunk32<false>, (const void *)k_chunk32<true>})
            NSS_CUDA_TRY(c, allow_smem(fn, std::max(csm, csm_vc)));
        int occ2 = 0;
        NSS_CUDA_TRY(c, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ2, (const void *)k_chunk32<true>, ORTH_THREADS,
                                                                      csm_vc));
        if (occ2 < 1 && vc > 0) {   // no room for the cache after all: run without it
            vc = 0;
            NSS_CUDA_TRY(c, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ2, (const void *)k_chunk32<true>, ORTH_THREADS,
                                                                          csm));
        }
        if (occ2 >= 1) {
            add(&z.wbuf32, (size_t)2 * n);
            add(&z.slot32, (size_t)3 * n);
            z.chunk_smem = csm;
            z.chunk_vc = vc;
            z.chunk_cs = vc > 0 ? cs : 0;
            z.chunk_smem_vc = vc > 0 ? csm_vc : csm;
            z.chunk_ok = true;
        }
    }
    add(&z.w, (size_t)n);
    double *vcur = nullptr;
    add(&vcur, (size_t)n);
    add(&z.jdev, 1);
    // exchange words: epoch (one word), totals, column partials, column totals
    z.xwords = x_words(pstride, mixed ? 1 : 2);
    add(&z.xch, z.xwords);
    add(&z.pro, (size_t)2 * pstride + PRO_TAIL);
    add(&z.evecs, (size_t)4 * n);
    // scalars, projection coefficients, restart scratch alpha/beta, refinement
    add(&z.scal, (size_t)S_NSCAL + 4 * (cap + 2) + 8);
    const size_t part = std::max((size_t)(cap + 2) * NBLK, (size_t)(2 * pstride + 2 * PA_COLS + 2) * (size_t)nsm);
    add(&z.part, part);
    add(&z.counter, 4);
    add(&z.alpha, (size_t)cap + 1);
    add(&z.beta, (size_t)cap + 1);
    add(&z.theta, 8);
    add(&z.resid, 8);
    add(&z.svec, (size_t)4 * svec_stride(cap));
    add(&z.flags, F_NFLAGS);
    // host-mapped mirrors: flags + the host's stop request; alpha, beta, anchor couplings m
    const size_t hflags = 256, hbytes = hflags + 3 * (size_t)(cap + 1) * sizeof(double);
    static_assert((F_NFLAGS + 8) * sizeof(int) <= 256, "flag mirror");
    if (hbytes > c.lz_host_bytes) {
        if (c.lz_host) cudaFreeHost(c.lz_host);
        c.lz_host = nullptr;
        c.lz_host_bytes = 0;
        NSS_CUDA_TRY(c, cudaHostAlloc((void **)&c.lz_host, hbytes, cudaHostAllocMapped));
        c.lz_host_bytes = hbytes;
    }
    char *dh = nullptr;
    NSS_CUDA_TRY(c, cudaHostGetDevicePointer((void **)&dh, c.lz_host, 0));
    if (int rc = workspace(c, want)) {
        z.vcur = vcur;
        lanczos_release(c, true);
        return rc;
    }
    z.vcur = vcur;
    z.h_flags = (int *)c.lz_host;
    z.h_ab = (double *)(c.lz_host + hflags);
    z.d_h_flags = (int *)dh;
    z.d_h_ab = (double *)(dh + hflags);
    NSS_CUDA_TRY(c, cudaMemsetAsync(z.counter, 0, 4 * sizeof(unsigned), c.stream));
    return NSS_OK;
}

// the FP64 scratch of the mixed refinement's Rayleigh-Ritz step (4 vectors)
int ensure_rrw(Ctx &c, int64_t n) {
    DevLanczos &z = c.lz;
    if (z.rrw) return NSS_OK;
    NSS_CUDA_TRY(c, ctx_alloc(c, &z.rrw, (size_t)4 * n));
    return NSS_OK;
}

template <class T>
int hv_t(Ctx &c, const T *v, T *hv, const int *stop);
template <>
int hv_t<double>(Ctx &c, const double *v, double *hv, const int *stop) { return hv_device(c, v, hv, stop); }
template <>
int hv_t<float>(Ctx &c, const float *v, float *hv, const int *stop) {
    return hv_device_fp32(c, v, hv, stop, false);    // k_orth adds the tensor-core planes
}

// Anchored refinement of one eigenvector (mixed precision, second phase):
// the FP64 anchor u with theta0 = u.H.u and r = H u - theta0 u; the caller
// has put r/|r| (FP32) into V[0].  The result c0 u + sum_l c_l V[l] goes to
// `out` (may alias u).
struct AnchorSpec {
    const double *u;             // FP64 anchor (the combination uses it)
    const float *u32, *r32, *defl32;   // FP32 copies for the projections in k_orth
    int ndefl;
    double theta0;
    double *out;
};

// out = c[0] u + sum_l c[l+1] V[l]   (FP64 accumulation)
template <class T>
__global__ void __launch_bounds__(256) k_ritz_anchor(const T *__restrict__ V, int m, int64_t n,
                                                     const double *__restrict__ cvec, const double *u, double *out) {
    extern __shared__ double cs[];   // [m+1]
    for (int t = threadIdx.x; t <= m; t += blockDim.x) cs[t] = cvec[t];
    __syncthreads();
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        double acc = cs[0] * u[i];
        for (int l = 0; l < m; ++l) acc = fma((double)V[(int64_t)l * n + i], cs[l + 1], acc);
        out[i] = acc;
    }
}

// The Lanczos iterations on a basis of type T; leaves theta (Ritz values),
// svec (their T_m eigenvectors, stride m) and the Ritz vectors (FP64) in c.lz.
// With `anc` it runs the anchored refinement instead (one eigenvector).
// cluster_max > neigen (mixed first phase): the Ritz pairs just above the
// wanted ones whose values lie within CLUSTER_GAP (relative) of their lower
// neighbour are returned as well, up to cluster_max in all; *ne_out gets the
// number of Ritz vectors left in evecs.
constexpr double CLUSTER_GAP = 1e-4;
template <class T>
int run_lanczos(Ctx &c, T *V, T *w, int neigen, int mmax, double tol, uint64_t seed, int *numop_out,
                int *m_out, const AnchorSpec *anc = nullptr, int cluster_max = 0, int *ne_out = nullptr,
                const double *start = nullptr) {
    DevLanczos &z = c.lz;
    const int64_t n = c.sb.n;
    const int cap = z.cap;
    double *h1 = z.scal + S_NSCAL;
    double *rs_alpha = h1 + 2 * (cap + 2), *rs_beta = rs_alpha + (cap + 2);
    cudaStream_t st = c.stream;
    volatile int *hf = z.h_flags;
    double *ha = z.h_ab, *hb = z.h_ab + (cap + 1);
    // no kernel of this context is running: the previous solve synchronised
    for (int i = 0; i < F_NFLAGS + 8; ++i) hf[i] = 0;
    for (int i = 0; i <= cap; ++i) ha[i] = hb[i] = 0.0;
    NSS_CUDA_TRY(c, cudaMemsetAsync(z.flags, 0, F_NFLAGS * sizeof(int), st));
    NSS_CUDA_TRY(c, cudaMemsetAsync(z.beta, 0, (cap + 1) * sizeof(double), st));
    NSS_CUDA_TRY(c, cudaMemsetAsync(z.counter, 0, 4 * sizeof(unsigned), st));
    // epochs start over: no word of an earlier run may carry one of this run's
    NSS_CUDA_TRY(c, cudaMemsetAsync(z.xch, 0, z.xwords * sizeof(uint64_t), st));
    const int vb = 608;   // 4 CTAs per SM for elementwise kernels
    uint64_t restarts = 0;
    if (anc) {
        neigen = 1;
    } else {
        ++c.launches;
        if (start && sizeof(T) == sizeof(float))   // a given FP64 start vector (mixed refinement)
            k_to32<<<vb, 256, 0, st>>>((float *)(void *)V, start, 1.0, n);
        else
            k_random<T><<<vb, 256, 0, st>>>(V, n, seed, restarts);
        ++c.launches;
        normalize_dev<T>(z, V, n, st, c.launches);
    }
    const size_t dots_smem = (size_t)(cap + 2) * sizeof(double) + SUB * sizeof(T);
    const size_t upd_smem = (size_t)(cap + 2) * sizeof(double);
    allow_smem((const void *)k_dots<T>, dots_smem);
    allow_smem((const void *)k_update<T>, upd_smem);
    constexpr int CW = OrthCW<T>::value;
    OrthArgs oa;
    oa.V = V;
    oa.w = w;
    oa.n = n;
    oa.j = 0;
    oa.mmax = mmax;
    oa.pstride = cap + 8;
    oa.alpha = z.alpha;
    oa.beta = z.beta;
    oa.part = z.part;
    oa.bar = z.counter + 2;
    oa.flags = z.flags;
    oa.h_alpha = z.d_h_ab;
    oa.h_beta = z.d_h_ab + (cap + 1);
    oa.h_flags = z.d_h_flags;
    oa.anc_u = anc ? (const void *)anc->u32 : nullptr;
    oa.anc_r = anc ? (const void *)anc->r32 : nullptr;
    oa.defl = anc ? (const void *)anc->defl32 : nullptr;
    oa.ndefl = anc ? anc->ndefl : 0;
    oa.h_m = z.d_h_ab + 2 * (cap + 1);
    oa.spin = wait_limit();
    oa.jdev = nullptr;
    oa.pro = z.pro;
    oa.delta = Pro<T>::DELTA;
    if (sizeof(T) == sizeof(double)) {
        oa.delta = std::min(oa.delta, 0.5f * (float)tol);
        oa.every = oa.delta < PRO_EVERY * Pro<T>::EPS1;
    }
    oa.xep = (unsigned *)z.xch;
    oa.xtot = z.xch + 1;
    oa.xcol = oa.xtot + (size_t)XCOLS * (XMAX + 1);
    oa.xpart = oa.xcol + (size_t)XW<T>::words * (cap + 8);
    if (sizeof(T) == sizeof(float) && c.sb.mma_nitems) {
        oa.tc = c.sb.d_mma_out;
        oa.tcn = c.sb.mma_nplanes;
    }
    // the launched chunks keep vcur current too, so that a replayed chunk
    // can follow one
    oa.vcur = c.use_graphs ? z.vcur : nullptr;
    const double *hm = z.h_ab + 2 * (cap + 1);
    std::vector<double> cvec;
    // Chunks of CHECK iterations, each ending with an event; the host checks
    // chunk k on T_m while the GPU runs chunk k+1.
    cudaEvent_t evs[2];
    cudaEventCreateWithFlags(&evs[0], cudaEventDisableTiming);
    cudaEventCreateWithFlags(&evs[1], cudaEventDisableTiming);
    // mixed method without tensor-core sectors: one persistent launch per chunk
    const bool use_chunk = sizeof(T) == sizeof(float) && z.chunk_ok && c.sb.mma_nitems == 0;
    struct ChunkTiming {
        cudaEvent_t a, b;
        int j0, jend;
    };
    std::vector<ChunkTiming> ctime;
    if (use_chunk)   // slot 1 and 2 regions that no item writes must read as zero
        NSS_CUDA_TRY(c, cudaMemsetAsync(z.slot32 + n, 0, (size_t)2 * n * sizeof(float), st));
    bool from_v = true;   // the next chunk starts from V[j0] (start, restart)
    int jdev_next = -1;   // the step that queued replays leave in *jdev (-1: not known)
    auto enqueue_chunk = [&](int j0, int slot) -> int {
        const int jend = std::min(mmax, j0 + CHECK);
        if (from_v) {
            ++c.launches;
            k_pro_reset<<<1, 512, 0, st>>>(z.pro, cap + 8, Pro<T>::EPS1);
        }
        if (use_chunk && jend > j0) {
            ChunkArgs ca;
            ca.o = oa;
            ca.buf[0] = z.wbuf32;
            ca.buf[1] = z.wbuf32 + n;
            ca.j0 = j0;
            ca.jend = jend;
            ca.first_from_v = from_v ? 1 : 0;
            ca.slot[0] = z.slot32;
            ca.slot[1] = z.slot32 + n;
            ca.slot[2] = z.slot32 + 2 * n;
            ca.items = c.sb.d_items32;
            ca.nitems = c.sb.nitems32;
            ca.op = hv32_ops(c.sb);
            ca.vc = z.chunk_vc;
            ca.cs = z.chunk_cs;
            from_v = false;
            void *args[] = {&ca};
            ChunkTiming ct{nullptr, nullptr, j0, jend};
            if (c.time_chunks) {
                cudaEventCreate(&ct.a);
                cudaEventCreate(&ct.b);
                cudaEventRecord(ct.a, st);
            }
            cudaError_t e = cudaLaunchCooperativeKernel(anc ? (const void *)k_chunk32<true> : (const void *)k_chunk32<false>, dim3(z.orth_grid),
                                                        dim3(ORTH_THREADS), args, z.chunk_smem_vc, st);
            if (c.time_chunks) {
                cudaEventRecord(ct.b, st);
                ctime.push_back(ct);
            }
            ++c.launches;
            if (e != cudaSuccess) {
                c.err = std::string("nss_eigh: cooperative launch failed: ") + cudaGetErrorString(e);
                return -1;
            }
            cudaEventRecord(evs[slot], st);
            return jend;
        }
        // a whole chunk of a plain (not anchored) Lanczos run replays the
        // CUDA graph of CHECK iterations captured for this superblock,
        // precision and iteration cap (the step and the input vector live on
        // the device); the first chunk of a key runs as launches and captures
        // the graph for the next ones
        const int prec = sizeof(T) == sizeof(float) ? 1 : 0;
        const bool key_ok = z.gx && z.gx_gen == c.sb.gen && z.gx_prec == prec && z.gx_mmax == mmax &&
                            z.gx_anc == oa.anc_u && z.gx_ndefl == oa.ndefl && z.gx_spin == oa.spin && z.gx_delta == oa.delta;
        const bool graphable = c.use_graphs && !z.gx_failed && jend - j0 == CHECK && oa.anc_u == nullptr;
        if (graphable && key_ok) {
            if (from_v)
                NSS_CUDA_TRY_R(c, cudaMemcpyAsync(z.vcur, V + (int64_t)j0 * n, (size_t)n * sizeof(T),
                                                  cudaMemcpyDeviceToDevice, st), -1);
            if (jdev_next != j0) {                   // else the replay before left it there
                k_seti<<<1, 1, 0, st>>>(z.jdev, j0);
                ++c.launches;
            }
            NSS_CUDA_TRY_R(c, cudaGraphLaunch(z.gx, st), -1);
            jdev_next = jend;
            c.launches += z.gx_launches;
            ++c.graph_replays;
            from_v = false;
            cudaEventRecord(evs[slot], st);
            return jend;
        }
        for (int jj = j0; jj < jend; ++jj) {
            if (hv_t<T>(c, V + (int64_t)jj * n, w, z.flags + F_STOP)) return -1;
            oa.j = jj;
            void *args[] = {&oa};
            cudaError_t e = cudaLaunchCooperativeKernel((const void *)k_orth<T, CW>, dim3(z.orth_grid),
                                                        dim3(ORTH_THREADS), args, z.orth_smem, st);
            ++c.launches;
            if (e != cudaSuccess) {
                c.err = std::string("nss_eigh: cooperative launch failed: ") + cudaGetErrorString(e);
                return -1;
            }
        }
        from_v = false;
        cudaEventRecord(evs[slot], st);
        if (graphable && !key_ok) {
            // record (not run) the iterations of a chunk: H*psi of vcur, then
            // k_orth stepping *jdev and writing the next vector to vcur
            if (z.gx) {
                cudaGraphExecDestroy(z.gx);
                z.gx = nullptr;
            }
            OrthArgs og = oa;
            og.jdev = z.jdev;
            og.vcur = z.vcur;
            const int64_t l0 = c.launches;
            cudaGraph_t g = nullptr;
            bool ok = cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal) == cudaSuccess;
            for (int it = 0; ok && it < CHECK; ++it) {
                if (hv_t<T>(c, (const T *)z.vcur, w, z.flags + F_STOP)) ok = false;
                void *args[] = {&og};
                if (ok && cudaLaunchCooperativeKernel((const void *)k_orth<T, CW>, dim3(z.orth_grid),
                                                      dim3(ORTH_THREADS), args, z.orth_smem, st) != cudaSuccess)
                    ok = false;
            }
            const cudaError_t ee = cudaStreamEndCapture(st, &g);
            ok = ok && ee == cudaSuccess && g && cudaGraphInstantiate(&z.gx, g, 0) == cudaSuccess;
            if (g) cudaGraphDestroy(g);
            cudaGetLastError();                      // a failed capture leaves nothing behind
            if (ok) {
                z.gx_gen = c.sb.gen;
                z.gx_prec = prec;
                z.gx_mmax = mmax;
                z.gx_anc = oa.anc_u;
                z.gx_ndefl = oa.ndefl;
                z.gx_spin = oa.spin;
                z.gx_delta = oa.delta;
                z.gx_launches = (int)(c.launches - l0);
                ++c.graph_captures;
            } else {
                if (z.gx) cudaGraphExecDestroy(z.gx);
                z.gx = nullptr;
                z.gx_failed = true;
                c.err.clear();
            }
            c.launches = l0;
        }
        return jend;
    };
    std::vector<double> theta(4, 0.0), resid(4, 0.0), upper(4, 0.0), svec, work;
    bool have_upper = false;
    int m_done = 1, rc = NSS_OK, ne_done = 1;
    bool converged = false;
    int slot = 0;
    int pend_end = enqueue_chunk(0, slot);
    if (pend_end < 0) rc = NSS_ERR_CUDA;
    while (pend_end >= 0) {
        const int next_end = (pend_end < mmax) ? enqueue_chunk(pend_end, slot ^ 1) : -2;
        if (next_end == -1) { rc = NSS_ERR_CUDA; break; }
        cudaError_t ce = cudaEventSynchronize(evs[slot]);
        if (ce != cudaSuccess) { c.err = cudaGetErrorString(ce); rc = NSS_ERR_CUDA; break; }
        if (hf[F_ERR]) {   // a bounded barrier wait ran out: nothing of this solve is trusted
            c.err = "nss_eigh: a grid barrier of the orthogonalisation kernel timed out (results discarded)";
            rc = NSS_ERR_CUDA;
            break;
        }
        // a breakdown inside this chunk ends it early; one flagged by the
        // chunk running ahead belongs to the next check
        int m = pend_end;
        const bool brk = hf[F_STOP] == 2 && hf[F_BREAK] <= pend_end;
        if (brk) m = hf[F_BREAK];
        const int ne = std::min(neigen, m);
        int conv = 0;
        if (anc) {
            // lowest eigenpair of [[theta0, m^T], [m, T_m]]
            cvec.resize((size_t)m + 1);
            double lam = 0.0, res = 0.0;
            if (arrow_lowest(anc->theta0, hm, ha, hb, m, hb[m - 1], &lam, cvec.data(), &res, work)) {
                theta[0] = lam;
                resid[0] = res;
                if (res <= tol * std::max(std::fabs(lam), 1e-300) || brk) conv = 1;
            }
        } else {
            svec.resize((size_t)ne * m);
            tridiag_lowest(ha, hb, m, ne, hb[m - 1], theta.data(), svec.data(), resid.data(),
                           (have_upper && ne == neigen) ? upper.data() : nullptr, work);
            for (int e = 0; e < ne; ++e) upper[e] = theta[e];
            have_upper = ne == neigen;
            for (int e = 0; e < ne; ++e)
                if (resid[e] <= tol * std::max(std::fabs(theta[e]), 1e-300)) ++conv;
        }
        m_done = m;
        ne_done = ne;
        if (conv >= ne || (int64_t)m >= n) {
            hf[F_NFLAGS] = 1;                        // stop request for the queued kernels
            std::atomic_thread_fence(std::memory_order_seq_cst);
            converged = true;
            break;
        }
        if (brk) {
            // invariant subspace without convergence: continue from a random
            // vector orthogonal to V (the chunk run ahead has already exited)
            NSS_CUDA_TRY(c, cudaStreamSynchronize(st));
            ++restarts;
            T *vn = V + (int64_t)m_done * n;
            ++c.launches;
            k_random<T><<<vb, 256, 0, st>>>(vn, n, seed, restarts);
            NSS_CUDA_TRY(c, cudaMemsetAsync(z.flags, 0, F_NFLAGS * sizeof(int), st));
            for (int pass = 0; pass < 2; ++pass) {
                NSS_CUDA_TRY(c, cudaMemsetAsync(z.scal + S_ALPHA, 0, sizeof(double), st));
                c.launches += 2;
                k_dots<T><<<NBLK, 256, dots_smem, st>>>(V, m_done, vn, n, z.part, h1, z.scal, z.counter, z.flags,
                                                        0, 0, z.beta);
                k_update<T><<<NBLK, 256, upd_smem, st>>>(V, m_done, vn, n, h1, z.part, z.scal, z.counter, z.flags,
                                                         rs_alpha, rs_beta, 0);
            }
            ++c.launches;
            normalize_dev<T>(z, vn, n, st, c.launches);
            NSS_CUDA_TRY(c, cudaMemsetAsync(z.beta + (m_done - 1), 0, sizeof(double), st));
            NSS_CUDA_TRY(c, cudaMemsetAsync(z.flags, 0, F_NFLAGS * sizeof(int), st));
            NSS_CUDA_TRY(c, cudaStreamSynchronize(st));
            hb[m_done - 1] = 0.0;
            hf[F_STOP] = 0;
            hf[F_BREAK] = 0;
            from_v = true;
            jdev_next = -1;       // the chunk ended early
            slot = 0;
            pend_end = enqueue_chunk(m_done, slot);
            if (pend_end < 0) { rc = NSS_ERR_CUDA; break; }
            continue;
        }
        if (next_end < 0) break;   // iteration cap reached without convergence
        slot ^= 1;
        pend_end = next_end;
    }
    cudaError_t ce = cudaStreamSynchronize(st);
    cudaEventDestroy(evs[0]);
    cudaEventDestroy(evs[1]);
    for (const ChunkTiming &ct : ctime) {
        // launches that completed iterations of the basis the solve kept
        if (ce == cudaSuccess && ct.j0 < m_done) {
            float ms = 0.f;
            cudaEventElapsedTime(&ms, ct.a, ct.b);
            const int je = std::min(ct.jend, m_done);
            c.chunk_ms += ms;
            ++c.chunk_launches;
            c.chunk_iters += je - ct.j0;
            for (int jj = ct.j0; jj < je; ++jj) c.chunk_cols += jj + 1;
        }
        cudaEventDestroy(ct.a);
        cudaEventDestroy(ct.b);
    }
    if ((rc || ce != cudaSuccess) && z.gx) {   // a failed run keeps no graph
        cudaGraphExecDestroy(z.gx);
        z.gx = nullptr;
    }
    if (rc) return rc;
    if (ce != cudaSuccess) { c.err = cudaGetErrorString(ce); return NSS_ERR_CUDA; }
    int dflags[F_NFLAGS];
    NSS_CUDA_TRY(c, cudaMemcpy(dflags, z.flags, sizeof(dflags), cudaMemcpyDeviceToHost));
    if (dflags[F_ERR]) {
        c.err = "nss_eigh: a grid barrier of the orthogonalisation kernel timed out (results discarded)";
        return NSS_ERR_CUDA;
    }
    *numop_out = m_done;
    *m_out = m_done;
    if (!converged) {
        c.err = "nss_eigh: no convergence within nitermax=" + std::to_string(mmax) + " iterations";
        return NSS_ERR_NOCONV;
    }
    if (anc) {
        if (cvec.size() != (size_t)m_done + 1) {
            c.err = "nss_eigh: the anchored refinement found no eigenpair";
            return NSS_ERR_NOCONV;
        }
        NSS_CUDA_TRY(c, cudaMemcpyAsync(z.svec, cvec.data(), cvec.size() * sizeof(double), cudaMemcpyHostToDevice, st));
        c.launches += 2;
        NSS_CUDA_TRY(c, allow_smem((const void *)k_ritz_anchor<T>, cvec.size() * sizeof(double)));
        k_ritz_anchor<T><<<NBLK, 256, cvec.size() * sizeof(double), st>>>(V, m_done, n, z.svec, anc->u, anc->out);
        normalize_dev<double>(z, anc->out, n, st, c.launches);
        NSS_CUDA_TRY(c, cudaGetLastError());
        NSS_CUDA_TRY(c, cudaStreamSynchronize(st));
        z.last_anchor_theta = theta[0];
        return NSS_OK;
    }
    if (cluster_max > ne_done && m_done > ne_done && (int64_t)cluster_max * cluster_max <= cap + 2) {
        // near-degenerate partners of the wanted pairs (see cluster_max)
        const int ntry = std::min(cluster_max, m_done);
        std::vector<double> th2(ntry), sv2((size_t)ntry * m_done), rs2(ntry);
        tridiag_lowest(ha, hb, m_done, ntry, hb[m_done - 1], th2.data(), sv2.data(), rs2.data(), nullptr, work);
        double scale = 0.0;
        for (int e = 0; e < ntry; ++e) scale = std::max(scale, std::fabs(th2[e]));
        int k = ne_done;
        while (k < ntry && th2[k] - th2[k - 1] <= CLUSTER_GAP * scale) ++k;
        if (k > ne_done) {
            for (int e = 0; e < k; ++e) {
                theta[e] = th2[e];
                resid[e] = rs2[e];
            }
            svec.assign(sv2.begin(), sv2.begin() + (size_t)k * m_done);
            ne_done = k;
        }
    }
    if (ne_out) *ne_out = ne_done;
    const int ne = ne_done;
    NSS_CUDA_TRY(c, cudaMemcpyAsync(z.theta, theta.data(), ne * sizeof(double), cudaMemcpyHostToDevice, st));
    NSS_CUDA_TRY(c, cudaMemcpyAsync(z.resid, resid.data(), ne * sizeof(double), cudaMemcpyHostToDevice, st));
    NSS_CUDA_TRY(c, cudaMemcpyAsync(z.svec, svec.data(), (size_t)ne * m_done * sizeof(double),
                                    cudaMemcpyHostToDevice, st));
    if (int rc2 = launch_ritz<T>(c, V, m_done, n, z.svec, ne, z.evecs, st, c.launches)) return rc2;
    // a basis kept orthogonal by estimates gives Ritz vectors that are orthogonal
    // to some m times their threshold (2.5e-13 between three states); projected,
    // to rounding
    const bool project = sizeof(T) == sizeof(double) && !oa.every && !pro_always<T>(m_done, n, oa.pstride);
    const size_t d64_smem = (size_t)(cap + 2) * sizeof(double) + SUB * sizeof(double);
    if (project && ne > 1) {
        NSS_CUDA_TRY(c, allow_smem((const void *)k_dots<double>, d64_smem));
        NSS_CUDA_TRY(c, allow_smem((const void *)k_update<double>, upd_smem));
        NSS_CUDA_TRY(c, cudaMemsetAsync(z.flags, 0, F_NFLAGS * sizeof(int), st));
    }
    for (int e = 0; e < ne; ++e) {
        double *u = z.evecs + (int64_t)e * n;
        if (project && e > 0) {
            NSS_CUDA_TRY(c, cudaMemsetAsync(z.scal + S_ALPHA, 0, sizeof(double), st));
            c.launches += 2;
            k_dots<double><<<NBLK, 256, d64_smem, st>>>(z.evecs, e, u, n, z.part, h1, z.scal, z.counter, z.flags, 0, 0, z.beta);
            k_update<double><<<NBLK, 256, upd_smem, st>>>(z.evecs, e, u, n, h1, z.part, z.scal, z.counter, z.flags, rs_alpha,
                                                          rs_beta, 0);
        }
        ++c.launches;
        normalize_dev<double>(z, u, n, st, c.launches);
    }
    NSS_CUDA_TRY(c, cudaGetLastError());
    // the pageable sources above are consumed before this returns
    NSS_CUDA_TRY(c, cudaStreamSynchronize(st));
    return NSS_OK;
}

}  // namespace

// keep: the block of the workspace's arrays and the host mirrors stay for the next
void lanczos_release(Ctx &c, bool keep) {
    DevLanczos &z = c.lz;
    if (z.gx) cudaGraphExecDestroy(z.gx);
    ctx_free(c, z.rrw);
    ctx_free(c, z.pitem);
    if (c.budget) {
        void *ptrs[] = {z.V, z.w, z.V32, z.w32, z.anc32, z.wbuf32, z.slot32, z.evecs, z.scal, z.part, z.counter,
                        z.alpha, z.beta, z.theta, z.resid, z.svec, z.flags, z.vcur, z.jdev, z.pro, z.xch};
        for (void *p : ptrs) ctx_free(c, p);
    }
    if (!keep) {
        ctx_free(c, c.lz_arena);
        c.lz_arena = nullptr;
        c.lz_arena_bytes = 0;
        if (c.lz_host) cudaFreeHost(c.lz_host);
        c.lz_host = nullptr;
        c.lz_host_bytes = 0;
    }
    z = DevLanczos{};
}

int lanczos_eigh(Ctx &c, int neigen, int nitermax, double tol, uint64_t seed, int precision,
                 double *evals_host, int *numop) {
    DevSb &s = c.sb;
    if (!s.valid) { c.err = "nss_eigh: no superblock uploaded"; return NSS_ERR_STATE; }
    const int64_t n = s.n;
    if (neigen < 1 || neigen > 4) { c.err = "nss_eigh: neigen must be in [1,4]"; return NSS_ERR_INVALID; }
    if (neigen > n) neigen = (int)n;
    if (nitermax <= 0) nitermax = 512;
    int mmax = (int)std::min<int64_t>(n, nitermax);
    if (mmax < neigen) mmax = neigen;
    if (tol <= 0.0) tol = 1e-15;
    const bool mixed = precision == NSS_PREC_MIXED;
    int rc = ensure_lanczos(c, n, mmax + 1, mixed);
    if (rc) return rc;
    DevLanczos &z = c.lz;
    c.chunk_ms = 0.0;
    c.graph_replays = 0;
    c.graph_captures = 0;
    c.chunk_launches = 0;
    c.chunk_iters = 0;
    c.chunk_cols = 0.0;
    cudaStream_t st = c.stream;
    // the tensor-core pipeline's error word belongs to this solve
    if (s.d_tc_err) NSS_CUDA_TRY(c, cudaMemsetAsync(s.d_tc_err, 0, sizeof(int), st));
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    cudaEventRecord(e0, st);
    int numop_ = 0, m_done = 0, kcl = 1;
    if (!mixed) {
        rc = run_lanczos<double>(c, z.V, z.w, neigen, mmax, tol, seed, &numop_, &m_done);
    } else {
        // after a solve that needed a near-degenerate partner (consecutive
        // DMRG steps have alike spectra) the FP32 phase also converges the
        // next Ritz pair, so that the pair is resolved when it stops
        const int want32 = std::min(4, neigen + (c.last_pair ? 1 : 0));
        rc = run_lanczos<float>(c, z.V32, z.w32, want32, mmax, std::max(tol, mixed_tol()), seed, &numop_, &m_done,
                                nullptr, std::min(4, want32 + 2), &kcl);
        if (rc == NSS_ERR_NOCONV && want32 > neigen) {
            // the extra pair did not converge within nitermax: the wanted ones alone
            int it0 = numop_;
            rc = run_lanczos<float>(c, z.V32, z.w32, neigen, mmax, std::max(tol, mixed_tol()), seed, &numop_, &m_done,
                                    nullptr, std::min(4, neigen + 2), &kcl);
            numop_ += it0;
        }
    }
    const int ne = (int)std::min<int64_t>(neigen, std::max(m_done, 1));
    if (!rc && mixed) {
        // Iterative refinement of the FP32 Ritz vectors to FP64 quality.  Each
        // pass takes every vector u (deflated against the ones before it) as
        // an FP64 anchor: theta0 = u.H.u and r = H u - theta0 u in FP64; a
        // vector with ||r|| <= tol |theta0| is final, any other gets an FP32
        // Lanczos run on the complement of u started from r/|r|, with the
        // couplings u.H.v = r.v in FP64, solved on the host.  The FP32 errors
        // then only touch the correction, which shrinks by about
        // eps32 ||H|| / gap per pass, gap the distance to the nearest other
        // eigenvalue.  Near-degenerate partners (within CLUSTER_GAP of the
        // wanted pairs, e.g. the singlet and Sz=0 triplet of a spin-1
        // chain's edge spins, split by ~1e-7 relative) would make that factor
        // ~1: they are refined along, and before every later pass an FP64
        // Rayleigh-Ritz step on the cluster resolves the mixing among them
        // exactly, so only the gap to the rest of the spectrum matters.  The
        // passes end when every wanted vector meets the FP64 residual test;
        // after MAX_PASSES without that the solve is redone in FP64.
        constexpr int MAX_PASSES = 8;
        double *r = z.scal + S_NSCAL + 4 * (z.cap + 2);   // 8 refinement slots
        double *h1 = z.scal + S_NSCAL;
        double *rs_alpha = h1 + 2 * (z.cap + 2), *rs_beta = rs_alpha + (z.cap + 2);
        const size_t dots_smem = (size_t)(z.cap + 2) * sizeof(double) + SUB * sizeof(double);
        const size_t upd_smem = (size_t)(z.cap + 2) * sizeof(double);
        allow_smem((const void *)k_dots<double>, dots_smem);
        allow_smem((const void *)k_update<double>, upd_smem);
        // w -= Y (Y^T w) against the e vectors before it; returns via scal[S_BB]
        auto deflate = [&](double *vec, int e) -> int {
            NSS_CUDA_TRY(c, cudaMemsetAsync(z.flags, 0, F_NFLAGS * sizeof(int), st));
            NSS_CUDA_TRY(c, cudaMemsetAsync(z.scal + S_ALPHA, 0, sizeof(double), st));
            c.launches += 2;
            k_dots<double><<<NBLK, 256, dots_smem, st>>>(z.evecs, e, vec, n, z.part, h1, z.scal, z.counter, z.flags,
                                                         0, 0, z.beta);
            k_update<double><<<NBLK, 256, upd_smem, st>>>(z.evecs, e, vec, n, h1, z.part, z.scal, z.counter, z.flags,
                                                          rs_alpha, rs_beta, 0);
            return NSS_OK;
        };
        double th[4] = {0, 0, 0, 0}, res[4] = {0, 0, 0, 0};
        // FP64 check of wanted vector e (deflated against the ones before it
        // and normalised): th[e] = u.H.u, res[e] = ||H u - th u||; leaves
        // r = H u - th u in z.w (deflated for e > 0) and its norm in *beta0
        double rr_lam[4] = {0, 0, 0, 0};
        int rr_k = 0;                                // cluster size of the last Rayleigh-Ritz step
        bool rr_fresh = false;                       // rrw holds H U of the current U
        auto check = [&](int e, double *beta0) -> int {
            double *u = z.evecs + (int64_t)e * n;
            if (e > 0) {
                if (int rc2 = deflate(u, e)) return rc2;
                ++c.launches;
                normalize_dev<double>(z, u, n, st, c.launches);
            }
            if (e == 0 && rr_fresh) {
                // right after a Rayleigh-Ritz step H u_0 is known
                NSS_CUDA_TRY(c, cudaMemcpyAsync(z.w, z.rrw, (size_t)n * sizeof(double), cudaMemcpyDeviceToDevice, st));
            } else {
                if (int rc2 = hv_device(c, u, z.w)) return rc2;
                ++numop_;
            }
            rr_fresh = false;
            c.launches += 2;
            k_rq<<<NBLK, 256, 0, st>>>(u, z.w, n, z.part, r, z.counter);
            k_anchor_r<<<NBLK, 256, 0, st>>>(u, z.w, n, z.part, r, z.counter);
            double hr[8];
            NSS_CUDA_TRY(c, cudaMemcpyAsync(hr, r, 8 * sizeof(double), cudaMemcpyDeviceToHost, st));
            NSS_CUDA_TRY(c, cudaStreamSynchronize(st));
            th[e] = hr[0] / hr[2];
            res[e] = std::sqrt(std::max(hr[4], 0.0));
            double rr = hr[4];
            if (e > 0) {
                if (int rc2 = deflate(z.w, e)) return rc2;
                NSS_CUDA_TRY(c, cudaMemcpyAsync(&rr, z.scal + S_BB, sizeof(double), cudaMemcpyDeviceToHost, st));
                NSS_CUDA_TRY(c, cudaStreamSynchronize(st));
            }
            *beta0 = std::sqrt(std::max(rr, 0.0));
            return NSS_OK;
        };
        // anchored FP32 correction of wanted vector e, right after check(e)
        auto refine = [&](int e, double beta0) -> int {
            double *u = z.evecs + (int64_t)e * n;
            float *u32 = z.anc32, *r32 = z.anc32 + n, *y32 = z.anc32 + 2 * n;
            c.launches += 1 + e;
            k_anchor32<<<608, 256, 0, st>>>(z.V32, u32, r32, u, z.w, 1.0 / beta0, n);
            for (int f = 0; f < e; ++f)
                k_to32<<<608, 256, 0, st>>>(y32 + (int64_t)f * n, z.evecs + (int64_t)f * n, 1.0, n);
            AnchorSpec as{u, u32, r32, y32, e, th[e], u};
            int it2 = 0, m2 = 0;
            // the anchored problem is solved to 1e-6 of the vector's residual
            // (from the FP32 phase's 1e-7 that is the final tolerance: one
            // pass; a stalled pass cannot gain more than its FP32 floor)
            const double tol_pass = std::max(tol, 1e-6 * beta0 / std::max(std::fabs(th[e]), 1e-300));
            if (int rc2 = run_lanczos<float>(c, z.V32, z.w32, 1, mmax, tol_pass, seed, &it2, &m2, &as)) return rc2;
            numop_ += it2;
            return NSS_OK;
        };
        // FP64 Rayleigh-Ritz on the k cluster vectors: orthonormalise them,
        // W = H U (into the FP64 scratch), G = U^T W, U <- U Q with G's
        // eigenvectors Q in ascending order
        auto rayleigh_ritz = [&](int k) -> int {
            if (k < 1 || k > 4) { c.err = "nss_eigh: Rayleigh-Ritz over 1 to 4 vectors"; return NSS_ERR_INVALID; }
            ++c.launches;
            normalize_dev<double>(z, z.evecs, n, st, c.launches);
            for (int e = 1; e < k; ++e) {
                double *u = z.evecs + (int64_t)e * n;
                if (int rc2 = deflate(u, e)) return rc2;
                ++c.launches;
                normalize_dev<double>(z, u, n, st, c.launches);
            }
            for (int e = 0; e < k; ++e) {
                if (int rc2 = hv_device(c, z.evecs + (int64_t)e * n, z.rrw + (int64_t)e * n)) return rc2;
                ++numop_;
            }
            ++c.launches;
            k_gram<<<NBLK, 256, 0, st>>>(z.evecs, z.rrw, k, n, z.part, h1, z.counter);
            double g[16];
            NSS_CUDA_TRY(c, cudaMemcpyAsync(g, h1, (size_t)k * k * sizeof(double), cudaMemcpyDeviceToHost, st));
            NSS_CUDA_TRY(c, cudaStreamSynchronize(st));
            double a[16], q[16], lam[4];
            for (int i = 0; i < k; ++i)
                for (int j = 0; j < k; ++j) a[i * k + j] = 0.5 * (g[i * k + j] + g[j * k + i]);
            sym_eig_small(k, a, lam, q);
            for (int e = 0; e < k; ++e) rr_lam[e] = lam[e];
            rr_k = k;
            Rot4 R{};
            for (int i = 0; i < k; ++i)
                for (int j = 0; j < k; ++j) R.q[j * 4 + i] = q[j * k + i];
            c.launches += 2;
            k_rot<<<608, 256, 0, st>>>(z.evecs, k, n, R);
            k_rot<<<608, 256, 0, st>>>(z.rrw, k, n, R);   // H U along, for the next check
            NSS_CUDA_TRY(c, cudaGetLastError());
            rr_fresh = true;
            return NSS_OK;
        };
        // k: the cluster (wanted vectors and partners); the passes
        int k = kcl;
        if (!rc) rc = ensure_rrw(c, n);
        bool done = false, rr_due = k > ne, rerun = false;
        double prev[4] = {0, 0, 0, 0};
        int passes = 0;
        for (; passes < MAX_PASSES && !rc && !done; ++passes) {
            if (rr_due && (rc = rayleigh_ritz(k))) break;
            const bool rr_now = rr_due;
            rr_due = false;
            bool all = true, redo = false;
            for (int e = 0; e < ne && !rc; ++e) {
                double beta0 = 0.0;
                if ((rc = check(e, &beta0))) break;
                if (res[e] <= tol * std::fabs(th[e])) continue;
                all = false;
                // a correction that gained less than 20x: the vector is mixed
                // with a near-degenerate state the cluster lacks or resolves
                // no longer
                const bool stalled = passes > 0 && !rr_now && res[e] > 0.05 * prev[e];
                if (stalled && k > ne) {
                    rr_due = redo = true;
                    break;
                }
                if (stalled && ne == 1 && !rerun) {
                    // the FP32 phase stopped before it resolved the pair: a
                    // short FP32 Lanczos run from the vector, which lies
                    // almost inside the pair's plane, finds both states
                    rerun = true;
                    int it3 = 0, m3 = 0, k3 = 2;
                    const int rc3 = run_lanczos<float>(c, z.V32, z.w32, 2, std::min(mmax, 160), std::max(tol, mixed_tol()),
                                                       seed, &it3, &m3, nullptr, 4, &k3, z.evecs);
                    numop_ += it3;
                    if (rc3 == NSS_ERR_NOCONV) break;   // left to the passes' limit
                    if ((rc = rc3)) break;
                    k = std::max(k3, 2);
                    rr_due = redo = true;
                    break;
                }
                if (!(beta0 > 0.0)) continue;
                if ((rc = refine(e, beta0))) break;
            }
            if (rc) break;
            if (all) done = true;
            else if (!redo)
                for (int e = 0; e < ne; ++e) prev[e] = res[e];
        }
        c.refine_passes = passes;
        c.refine_cluster = k;
        c.last_pair = rr_k > ne && rr_lam[ne] - rr_lam[ne - 1] <= CLUSTER_GAP * std::fabs(rr_lam[0]);
        if (!rc && done) {
            for (int e = 0; e < ne; ++e) z.last_resid[e] = res[e];
            NSS_CUDA_TRY(c, cudaMemcpyAsync(z.theta, th, ne * sizeof(double), cudaMemcpyHostToDevice, st));
            NSS_CUDA_TRY(c, cudaStreamSynchronize(st));
        } else if (!rc) {
            // the FP32 corrections did not reach tol: the plain FP64 method
            ++c.mixed_fallbacks;
            if ((rc = ensure_lanczos(c, n, mmax + 1, false)) == NSS_OK) {
                int it64 = 0;
                rc = run_lanczos<double>(c, c.lz.V, c.lz.w, neigen, mmax, tol, seed, &it64, &m_done);
                numop_ += it64;
            }
        }
    }
    cudaEventRecord(e1, st);
    cudaError_t ce = cudaStreamSynchronize(st);
    float ms = 0.f;
    cudaEventElapsedTime(&ms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (rc) return rc;
    if (ce != cudaSuccess) { c.err = cudaGetErrorString(ce); return NSS_ERR_CUDA; }
    if ((mixed || c.sb.sp_nitems) && c.sb.d_tc_err) {
        int tc_err = 0;
        NSS_CUDA_TRY(c, cudaMemcpy(&tc_err, c.sb.d_tc_err, sizeof(int), cudaMemcpyDeviceToHost));
        if (tc_err) {
            c.err = "nss_eigh: a tensor-core pipeline wait timed out (results discarded)";
            return NSS_ERR_CUDA;
        }
    }
    if (evals_host) NSS_CUDA_TRY(c, cudaMemcpy(evals_host, z.theta, ne * sizeof(double), cudaMemcpyDeviceToHost));
    c.last_ms_eigh = ms;
    c.last_numop = numop_;
    if (mixed) tune_record(c, ms, numop_);
    z.last_iters = m_done;
    z.neigen_done = ne;
    if (numop) *numop = numop_;
    return NSS_OK;
}


// ---------------------------------------------------------------------------
// Batch engine (mixed precision): every solve keeps its own context
// (superblock, Krylov basis, host mirrors); one cooperative launch of
// k_batch32 per round runs CHECK iterations of every solve in flight, then
// the host checks each solve (tridiagonal or anchored problem) and moves it
// through FP32 Lanczos -> anchored refinement -> FP64 energy, as
// lanczos_eigh does for one context.  Solves can join between rounds
// (continuous batching: nss_batch_add) and leave when done (nss_batch_step
// reports them).  The per-round follow-up work of all solves (Ritz vectors,
// FP64 products, restarts) is queued back to back with one synchronisation.

namespace {

struct BatchState {
    Ctx *c = nullptr;
    int id = 0;
    int64_t n = 0;
    int mmax = 0, phase = 1, j0 = 0, m_done = 0, numop = 0, rc = 0;
    bool from_v = true, have_upper = false;
    double tol = 0.0, tol_final = 0.0, theta0 = 0.0, result = 0.0;
    uint64_t seed = 0, restarts = 0;
    std::vector<double> theta, resid, upper, svec, work, cvec;
    AnchorSpec as{};
};

}  // namespace

struct BatchEngine {
    Ctx *c0 = nullptr;           // owns the stream, the barrier and the argument buffers
    std::vector<BatchState> solves;
    int next_id = 1;
    BatchSolve *d_solves = nullptr, *h_solves = nullptr;
    int2 *d_gitems = nullptr, *h_gitems = nullptr;
    int cap_items = 0;
    float *d_st = nullptr;
    unsigned *d_q = nullptr;     // item queue heads of a launch
    double *h_res = nullptr;     // [BATCH_MAX][8] pinned refinement results
    int *h_tc = nullptr;         // [BATCH_MAX] pinned: the FP64 product gave up a wait
    cudaEvent_t forked = nullptr, joined[BATCH_MAX] = {};   // the solves' own streams leave and rejoin c0's
    size_t smem_set = 0;         // dynamic shared memory of its launches (the most any round needed)
    ~BatchEngine() {
        if (!c0) return;
        cudaStreamSynchronize(c0->stream);
        if (forked) cudaEventDestroy(forked);
        for (cudaEvent_t e : joined)
            if (e) cudaEventDestroy(e);
        ctx_free(*c0, d_solves);
        ctx_free(*c0, d_gitems);
        ctx_free(*c0, d_st);
        ctx_free(*c0, d_q);
        if (h_solves) cudaFreeHost(h_solves);
        if (h_gitems) cudaFreeHost(h_gitems);
        if (h_res) cudaFreeHost(h_res);
        if (h_tc) cudaFreeHost(h_tc);
    }
};

namespace {

int engine_init(BatchEngine &E, Ctx &c0) {
    E.c0 = &c0;
    // the barrier, error word and refinement scratch live in c0's Lanczos state
    if (!c0.lz.flags) {
        int rc = ensure_lanczos(c0, std::max<int64_t>(c0.sb.valid ? c0.sb.n : 1, 1), 8, true);
        if (rc) return rc;
    }
    NSS_CUDA_TRY(c0, ctx_alloc(c0, &E.d_solves, (size_t)BATCH_MAX));
    NSS_CUDA_TRY(c0, ctx_alloc(c0, &E.d_st, (size_t)ST_WORDS * BATCH_MAX));
    NSS_CUDA_TRY(c0, ctx_alloc(c0, &E.d_q, (size_t)CHUNK_MAXIT));
    NSS_CUDA_TRY(c0, cudaMallocHost((void **)&E.h_solves, sizeof(BatchSolve) * BATCH_MAX));
    NSS_CUDA_TRY(c0, cudaMallocHost((void **)&E.h_res, sizeof(double) * 8 * BATCH_MAX));
    NSS_CUDA_TRY(c0, cudaMallocHost((void **)&E.h_tc, sizeof(int) * BATCH_MAX));
    NSS_CUDA_TRY(c0, cudaEventCreateWithFlags(&E.forked, cudaEventDisableTiming));
    NSS_CUDA_TRY(c0, cudaMemsetAsync(c0.lz.counter, 0, 4 * sizeof(unsigned), c0.stream));
    NSS_CUDA_TRY(c0, cudaMemsetAsync(c0.lz.flags, 0, F_NFLAGS * sizeof(int), c0.stream));
    return NSS_OK;
}

int engine_start_run(BatchEngine &E, BatchState &B) {
    Ctx &c0 = *E.c0;
    DevLanczos &z = B.c->lz;
    volatile int *hf = z.h_flags;
    for (int i = 0; i < F_NFLAGS + 8; ++i) hf[i] = 0;
    for (int i = 0; i < 3 * (z.cap + 1); ++i) z.h_ab[i] = 0.0;
    cudaStream_t st = c0.stream;
    ++c0.launches;
    k_run_reset<<<(unsigned)std::min<int64_t>(152, (2 * B.n + 255) / 256), 256, 0, st>>>(
        z.pro, z.cap + 8, Pro<float>::EPS1, z.flags, z.beta, z.cap + 1, z.slot32 + B.n, 2 * B.n);
    B.j0 = 0;
    B.from_v = true;
    B.have_upper = false;
    return NSS_OK;
}

int engine_add(BatchEngine &E, Ctx &c, uint64_t seed, int nitermax, double tol, int *id) {
    Ctx &c0 = *E.c0;
    if ((int)E.solves.size() >= std::min(BATCH_MAX, c0.lz.orth_grid)) {
        c0.err = "nss_batch_add: the batch is full";
        return NSS_ERR_INVALID;
    }
    if (c.device != c0.device) { c0.err = "nss_batch_add: the context is on another device"; return NSS_ERR_INVALID; }
    if (!c.sb.valid) { c0.err = "nss_batch_add: the context has no superblock"; return NSS_ERR_STATE; }
    for (auto &S : E.solves)
        if (S.c == &c) { c0.err = "nss_batch_add: the context is already in the batch"; return NSS_ERR_INVALID; }
    if (tol <= 0.0) tol = 1e-15;
    if (nitermax <= 0) nitermax = 512;
    BatchState B;
    B.c = &c;
    B.id = E.next_id++;
    B.n = c.sb.n;
    B.mmax = (int)std::min<int64_t>(B.n, nitermax);
    B.tol = std::max(tol, mixed_tol());
    B.tol_final = tol;
    B.seed = seed;
    B.theta.assign(4, 0.0);
    B.resid.assign(4, 0.0);
    B.upper.assign(4, 0.0);
    int rc = ensure_lanczos(c, B.n, B.mmax + 1, true);
    if (rc) { c0.err = c.err; return rc; }
    NSS_CUDA_TRY(c0, cudaStreamSynchronize(c.stream));   // the engine works on its own stream
    DevLanczos &z = c.lz;
    if (!z.chunk_ok) { c0.err = "nss_batch_add: the persistent kernel does not fit this Krylov basis"; return NSS_ERR_INVALID; }
    if (!z.pitem || z.cap_pitem < c.sb.nitems32) {
        ctx_free(c, z.pitem);
        z.pitem = nullptr;
        NSS_CUDA_TRY(c0, ctx_alloc(c, &z.pitem, (size_t)2 * std::max(c.sb.nitems32, 1)));
        z.cap_pitem = c.sb.nitems32;
    }
    if ((rc = engine_start_run(E, B))) return rc;
    cudaStream_t st = c0.stream;
    c0.launches += 2;
    k_random<float><<<608, 256, 0, st>>>(z.V32, B.n, B.seed, 0);
    normalize_dev<float>(z, z.V32, B.n, st, c0.launches);
    NSS_CUDA_TRY(c0, cudaGetLastError());
    if (id) *id = B.id;
    E.solves.push_back(std::move(B));
    return NSS_OK;
}

// One round: a launch over every solve in flight, the host checks, the
// follow-up work.  Finished solves are removed and reported.
int engine_step(BatchEngine &E, int max_done, int *ndone, int *ids, double *energies, int *numops) {
    Ctx &c0 = *E.c0;
    cudaStream_t st = c0.stream;
    if (ndone) *ndone = 0;
    const int G = c0.lz.orth_grid;
    std::vector<int> act;
    for (int b = 0; b < (int)E.solves.size(); ++b)
        if ((E.solves[b].phase == 1 || E.solves[b].phase == 2) && E.solves[b].rc == 0) act.push_back(b);
    const int na = (int)act.size();
    if (na > 0) {
        double ntot = 0.0;
        for (int b : act) ntot += (double)E.solves[b].n;
        // CTAs per solve for its rows: one each, the rest in proportion to
        // the orthogonalisation's work, rows x basis columns (largest
        // remainders take the leftovers)
        std::vector<int> ncta(na, 1);
        {
            std::vector<double> wgt(na);
            double wtot = 0.0;
            for (int q = 0; q < na; ++q) {
                const BatchState &B = E.solves[act[q]];
                wgt[q] = (double)B.n * (double)(B.j0 + CHECK + 16);
                wtot += wgt[q];
            }
            int left = G - na;
            std::vector<std::pair<double, int>> rem;
            const int pool = left;
            for (int q = 0; q < na && pool > 0; ++q) {
                const double share = pool * wgt[q] / wtot;
                const int whole = std::min(left, (int)share);
                ncta[q] += whole;
                left -= whole;
                rem.push_back({share - whole, q});
            }
            std::stable_sort(rem.begin(), rem.end(), [](const auto &x, const auto &y) { return x.first > y.first; });
            for (size_t r = 0; r < rem.size() && left > 0; ++r, --left) ++ncta[rem[r].second];
        }
        int tot_items = 0;
        for (int b : act) tot_items += E.solves[b].c->sb.nitems32;
        if (tot_items > E.cap_items) {
            ctx_free(c0, E.d_gitems);
            E.d_gitems = nullptr;
            if (E.h_gitems) cudaFreeHost(E.h_gitems);
            E.h_gitems = nullptr;
            NSS_CUDA_TRY(c0, ctx_alloc(c0, &E.d_gitems, (size_t)tot_items));
            NSS_CUDA_TRY(c0, cudaMallocHost((void **)&E.h_gitems, sizeof(int2) * tot_items));
            E.cap_items = tot_items;
        }
        int cta = 0, ng = 0;
        size_t smem_max = 0;
        std::vector<std::pair<int, int2>> order;
        order.reserve(tot_items);
        for (int q = 0; q < na; ++q) {
            BatchState &B = E.solves[act[q]];
            Ctx &c = *B.c;
            DevLanczos &z = c.lz;
            smem_max = std::max(smem_max, z.chunk_smem);
            BatchSolve bs{};
            ChunkArgs &ca = bs.c;
            OrthArgs &oa = ca.o;
            oa.V = z.V32;
            oa.w = z.w32;
            oa.n = B.n;
            oa.j = B.j0;
            oa.mmax = B.mmax;
            oa.pstride = z.cap + 8;
            oa.alpha = z.alpha;
            oa.beta = z.beta;
            oa.part = z.part;
            oa.bar = nullptr;
            oa.flags = z.flags;
            oa.h_alpha = z.d_h_ab;
            oa.h_beta = z.d_h_ab + (z.cap + 1);
            oa.h_flags = z.d_h_flags;
            oa.h_m = z.d_h_ab + 2 * (z.cap + 1);
            oa.spin = wait_limit();
            oa.pro = z.pro;
            const bool anc = B.phase == 2;
            oa.anc_u = anc ? (const void *)B.as.u32 : nullptr;
            oa.anc_r = anc ? (const void *)B.as.r32 : nullptr;
            oa.defl = anc ? (const void *)B.as.defl32 : nullptr;
            oa.ndefl = 0;
            ca.buf[0] = z.wbuf32;
            ca.buf[1] = z.wbuf32 + B.n;
            ca.slot[0] = z.slot32;
            ca.slot[1] = z.slot32 + B.n;
            ca.slot[2] = z.slot32 + 2 * B.n;
            ca.j0 = B.j0;
            ca.jend = std::min(B.mmax, B.j0 + CHECK);
            ca.first_from_v = B.from_v ? 1 : 0;
            ca.items = c.sb.d_items32;
            ca.nitems = c.sb.nitems32;
            ca.op = hv32_ops(c.sb);
            bs.pitem = z.pitem;
            bs.cta0 = cta;
            bs.ncta = ncta[q];
            bs.active = 1;
            cta += ncta[q];
            E.h_solves[q] = bs;
            for (int li = 0; li < c.sb.nitems32; ++li) order.push_back({c.sb.item_cost[li], make_int2(q, li)});
            B.from_v = false;
        }
        std::stable_sort(order.begin(), order.end(),
                         [](const std::pair<int, int2> &x, const std::pair<int, int2> &y) { return x.first > y.first; });
        for (auto &o : order) E.h_gitems[ng++] = o.second;
        NSS_CUDA_TRY(c0, cudaMemcpyAsync(E.d_solves, E.h_solves, sizeof(BatchSolve) * na, cudaMemcpyHostToDevice, st));
        NSS_CUDA_TRY(c0, cudaMemcpyAsync(E.d_gitems, E.h_gitems, sizeof(int2) * std::max(ng, 1), cudaMemcpyHostToDevice,
                                         st));
        NSS_CUDA_TRY(c0, allow_smem((const void *)k_batch32, smem_max));
        E.smem_set = std::max(E.smem_set, smem_max);
        NSS_CUDA_TRY(c0, cudaMemsetAsync(E.d_q, 0, CHUNK_MAXIT * sizeof(unsigned), st));
        BatchArgs ba;
        ba.qcnt = E.d_q;
        ba.s = E.d_solves;
        ba.ns = na;
        ba.nitems = ng;
        ba.gitems = E.d_gitems;
        ba.st = E.d_st;
        ba.bar = c0.lz.counter + 2;
        ba.err = c0.lz.flags + F_ERR;
        ba.steps = CHECK;
        ba.spin = wait_limit();
        void *args[] = {&ba};
        cudaError_t e = cudaLaunchCooperativeKernel((const void *)k_batch32, dim3(G), dim3(ORTH_THREADS), args,
                                                    E.smem_set, st);
        ++c0.launches;
        if (e != cudaSuccess) {
            c0.err = std::string("nss_batch: cooperative launch failed: ") + cudaGetErrorString(e);
            return NSS_ERR_CUDA;
        }
        cudaError_t ce = cudaStreamSynchronize(st);
        if (ce != cudaSuccess) { c0.err = cudaGetErrorString(ce); return NSS_ERR_CUDA; }
        int err_flag = 0;
        NSS_CUDA_TRY(c0, cudaMemcpy(&err_flag, c0.lz.flags + F_ERR, sizeof(int), cudaMemcpyDeviceToHost));
        if (err_flag) {
            c0.err = "nss_batch: a grid barrier timed out (results discarded)";
            return NSS_ERR_CUDA;
        }
    }
    // host checks
    std::vector<int> p1, p2, p3;
    for (int b : act) {
        BatchState &B = E.solves[b];
        Ctx &c = *B.c;
        DevLanczos &z = c.lz;
        volatile int *hf = z.h_flags;
        const double *ha = z.h_ab, *hb = z.h_ab + (z.cap + 1), *hm = z.h_ab + 2 * (z.cap + 1);
        const int jend = std::min(B.mmax, B.j0 + CHECK);
        int m = jend;
        const bool brk = hf[F_STOP] == 2 && hf[F_BREAK] <= jend;
        if (brk) m = hf[F_BREAK];
        bool conv = false;
        if (B.phase == 1) {
            B.svec.resize((size_t)m);
            tridiag_lowest(ha, hb, m, 1, hb[m - 1], B.theta.data(), B.svec.data(), B.resid.data(),
                           B.have_upper ? B.upper.data() : nullptr, B.work);
            B.upper[0] = B.theta[0];
            B.have_upper = true;
            conv = B.resid[0] <= B.tol * std::max(std::fabs(B.theta[0]), 1e-300) || (int64_t)m >= B.n;
        } else {
            B.cvec.resize((size_t)m + 1);
            double lam = 0.0, res = 0.0;
            if (arrow_lowest(B.theta0, hm, ha, hb, m, hb[m - 1], &lam, B.cvec.data(), &res, B.work))
                conv = res <= B.tol_final * std::max(std::fabs(lam), 1e-300) || brk;
            else
                B.cvec.clear();
        }
        B.m_done = m;
        if (!conv) {
            if (brk && B.phase == 1) {
                // invariant subspace without convergence: restart from a random
                // vector orthogonal to the basis
                ++B.restarts;
                float *vn = z.V32 + (int64_t)m * B.n;
                const size_t dots_smem = (size_t)(z.cap + 2) * sizeof(double) + SUB * sizeof(float);
                const size_t upd_smem = (size_t)(z.cap + 2) * sizeof(double);
                allow_smem((const void *)k_dots<float>, dots_smem);
                allow_smem((const void *)k_update<float>, upd_smem);
                double *h1 = z.scal + S_NSCAL;
                double *rs_alpha = h1 + 2 * (z.cap + 2), *rs_beta = rs_alpha + (z.cap + 2);
                c0.launches += 6;
                k_random<float><<<608, 256, 0, st>>>(vn, B.n, B.seed, B.restarts);
                NSS_CUDA_TRY(c0, cudaMemsetAsync(z.flags, 0, F_NFLAGS * sizeof(int), st));
                for (int pass = 0; pass < 2; ++pass) {
                    NSS_CUDA_TRY(c0, cudaMemsetAsync(z.scal + S_ALPHA, 0, sizeof(double), st));
                    k_dots<float><<<NBLK, 256, dots_smem, st>>>(z.V32, m, vn, B.n, z.part, h1, z.scal, z.counter,
                                                                z.flags, 0, 0, z.beta);
                    k_update<float><<<NBLK, 256, upd_smem, st>>>(z.V32, m, vn, B.n, h1, z.part, z.scal, z.counter,
                                                                 z.flags, rs_alpha, rs_beta, 0);
                }
                normalize_dev<float>(z, vn, B.n, st, c0.launches);
                NSS_CUDA_TRY(c0, cudaMemsetAsync(z.beta + (m - 1), 0, sizeof(double), st));
                NSS_CUDA_TRY(c0, cudaMemsetAsync(z.flags, 0, F_NFLAGS * sizeof(int), st));
                ++c0.launches;
                k_pro_reset<<<1, 512, 0, st>>>(z.pro, z.cap + 8, Pro<float>::EPS1);
                z.h_ab[(z.cap + 1) + m - 1] = 0.0;
                hf[F_STOP] = 0;
                hf[F_BREAK] = 0;
                B.j0 = m;
                B.from_v = true;
            } else if (m >= B.mmax) {
                c.err = "nss_eigh: no convergence within nitermax=" + std::to_string(B.mmax) + " iterations";
                B.rc = NSS_ERR_NOCONV;
            } else {
                B.j0 = jend;
            }
            continue;
        }
        B.numop += m;
        (B.phase == 1 ? p1 : p2).push_back(b);
    }
    for (int b = 0; b < (int)E.solves.size(); ++b)
        if (E.solves[b].phase == 3) p3.push_back(b);
    // follow-up work, every solve on its own context's stream and scratch:
    // refinement results land in h_res.  Its kernels are latency (60 us a solve
    // of a few thousand states); one after the other on the engine's stream
    // they took a third of a batch's device time
    auto fork = [&](BatchState &B) -> int {
        if (B.c->stream != st) NSS_CUDA_TRY(c0, cudaStreamWaitEvent(B.c->stream, E.forked, 0));
        return NSS_OK;
    };
    auto join = [&](BatchState &B, int slot) -> int {
        if (B.c->stream == st) return NSS_OK;
        if (!E.joined[slot]) NSS_CUDA_TRY(c0, cudaEventCreateWithFlags(&E.joined[slot], cudaEventDisableTiming));
        NSS_CUDA_TRY(c0, cudaEventRecord(E.joined[slot], B.c->stream));
        NSS_CUDA_TRY(c0, cudaStreamWaitEvent(st, E.joined[slot], 0));
        return NSS_OK;
    };
    auto fp64_energy = [&](BatchState &B, int slot, bool anchor) -> int {
        Ctx &c = *B.c;
        DevLanczos &z = c.lz;
        const cudaStream_t s = c.stream;
        double *r = z.scal + S_NSCAL + 4 * (z.cap + 2);
        // the error word of a product on the tensor cores travels with the results
        const bool tc = c.sb.sp_nitems > 0;
        E.h_tc[slot] = 0;
        if (tc) NSS_CUDA_TRY(c0, cudaMemsetAsync(c.sb.d_tc_err, 0, sizeof(int), s));
        if (int r2 = hv_device(c, z.evecs, z.w)) { c0.err = c.err; return r2; }
        if (tc) NSS_CUDA_TRY(c0, cudaMemcpyAsync(E.h_tc + slot, c.sb.d_tc_err, sizeof(int), cudaMemcpyDeviceToHost, s));
        ++B.numop;
        c0.launches += 2;
        k_rq<<<NBLK, 256, 0, s>>>(z.evecs, z.w, B.n, z.part, r, z.counter);
        if (anchor) k_anchor_r<<<NBLK, 256, 0, s>>>(z.evecs, z.w, B.n, z.part, r, z.counter);
        else k_resid<<<NBLK, 256, 0, s>>>(z.evecs, z.w, B.n, z.part, r, z.counter);
        NSS_CUDA_TRY(c0, cudaMemcpyAsync(E.h_res + 8 * slot, r, 8 * sizeof(double), cudaMemcpyDeviceToHost, s));
        return NSS_OK;
    };
    if (!p1.empty() || !p2.empty() || !p3.empty()) NSS_CUDA_TRY(c0, cudaEventRecord(E.forked, st));
    int rc = NSS_OK;
    for (int b : p1) {
        BatchState &B = E.solves[b];
        DevLanczos &z = B.c->lz;
        const int m = B.m_done;
        const cudaStream_t s = B.c->stream;
        if ((rc = fork(B))) return rc;
        NSS_CUDA_TRY(c0, cudaMemcpyAsync(z.svec, B.svec.data(), (size_t)m * sizeof(double), cudaMemcpyHostToDevice, s));
        ++c0.launches;
        if ((rc = launch_ritz<float>(c0, z.V32, m, B.n, z.svec, 1, z.evecs, s, c0.launches))) return rc;
        normalize_dev<double>(z, z.evecs, B.n, s, c0.launches);
        if ((rc = fp64_energy(B, b, true)) || (rc = join(B, b))) return rc;
    }
    for (int b : p2) {
        BatchState &B = E.solves[b];
        DevLanczos &z = B.c->lz;
        const cudaStream_t s = B.c->stream;
        if ((rc = fork(B))) return rc;
        NSS_CUDA_TRY(c0, cudaMemcpyAsync(z.svec, B.cvec.data(), B.cvec.size() * sizeof(double), cudaMemcpyHostToDevice,
                                         s));
        c0.launches += 2;
        NSS_CUDA_TRY(c0, allow_smem((const void *)k_ritz_anchor<float>, B.cvec.size() * sizeof(double)));
        k_ritz_anchor<float><<<NBLK, 256, B.cvec.size() * sizeof(double), s>>>(z.V32, B.m_done, B.n, z.svec, z.evecs,
                                                                               z.evecs);
        normalize_dev<double>(z, z.evecs, B.n, s, c0.launches);
        if ((rc = fp64_energy(B, b, false)) || (rc = join(B, b))) return rc;
    }
    for (int b : p3)
        if ((rc = fork(E.solves[b])) || (rc = fp64_energy(E.solves[b], b, false)) || (rc = join(E.solves[b], b))) return rc;
    NSS_CUDA_TRY(c0, cudaStreamSynchronize(st));
    for (const std::vector<int> *p : {&p1, &p2, &p3})
        for (int b : *p)
            if (E.h_tc[b]) {
                c0.err = "nss_batch: a tensor-core pipeline wait timed out (results discarded)";
                return NSS_ERR_CUDA;
            }
    auto finish = [&](BatchState &B, int slot) -> int {
        const double *hr = E.h_res + 8 * slot;
        B.result = hr[0] / hr[2];
        DevLanczos &z = B.c->lz;
        z.last_resid[0] = std::sqrt(std::max(hr[3], 0.0));
        NSS_CUDA_TRY(c0, cudaMemcpyAsync(z.theta, &B.result, sizeof(double), cudaMemcpyHostToDevice, st));
        z.last_iters = B.m_done;
        z.neigen_done = 1;
        B.c->last_numop = B.numop;
        B.phase = 4;
        return NSS_OK;
    };
    for (int b : p1) {
        BatchState &B = E.solves[b];
        DevLanczos &z = B.c->lz;
        const double *hr = E.h_res + 8 * b;
        B.theta0 = hr[0] / hr[2];
        const double beta0 = std::sqrt(std::max(hr[4], 0.0));
        if (!(beta0 > B.tol_final * std::fabs(B.theta0))) {
            B.phase = 3;   // the FP32 vector is converged already: its FP64 energy next round
            continue;
        }
        float *u32 = z.anc32, *r32 = z.anc32 + B.n;
        ++c0.launches;
        k_anchor32<<<608, 256, 0, st>>>(z.V32, u32, r32, z.evecs, z.w, 1.0 / beta0, B.n);
        B.as = AnchorSpec{z.evecs, u32, r32, z.anc32 + 2 * B.n, 0, B.theta0, z.evecs};
        if ((rc = engine_start_run(E, B))) return rc;
        B.phase = 2;
    }
    for (int b : p2)
        if ((rc = finish(E.solves[b], b))) return rc;
    for (int b : p3)
        if ((rc = finish(E.solves[b], b))) return rc;
    // report and remove the finished solves
    int nd = 0;
    std::vector<BatchState> keep;
    for (auto &B : E.solves) {
        if ((B.phase == 4 || B.rc) && nd < max_done) {
            if (ids) ids[nd] = B.rc ? -B.id : B.id;
            if (energies) energies[nd] = B.result;
            if (numops) numops[nd] = B.numop;
            ++nd;
        } else {
            keep.push_back(std::move(B));
        }
    }
    E.solves = std::move(keep);
    if (ndone) *ndone = nd;
    return NSS_OK;
}

// After a failed round: nothing of it still runs, and no solve is held
void engine_drop(BatchEngine &E) {
    cudaStreamSynchronize(E.c0->stream);
    for (BatchState &B : E.solves) cudaStreamSynchronize(B.c->stream);
    E.solves.clear();
}

}  // namespace

BatchEngine *batch_create(Ctx &c0) {
    BatchEngine *E = new BatchEngine();
    if (engine_init(*E, c0)) {
        delete E;
        return nullptr;
    }
    return E;
}

void batch_destroy(BatchEngine *E) { delete E; }

int batch_add(BatchEngine *E, Ctx &c, uint64_t seed, int nitermax, double tol, int *id) {
    return engine_add(*E, c, seed, nitermax, tol, id);
}

int batch_step(BatchEngine *E, int max_done, int *ndone, int *ids, double *energies, int *numops) {
    const int rc = engine_step(*E, max_done, ndone, ids, energies, numops);
    if (rc) {
        // a failed round drops every solve in flight, so that the engine
        // holds no context its caller may now solve alone or release; the
        // shared barrier and error word start the next round cleared
        engine_drop(*E);
        if (ndone) *ndone = 0;
        Ctx &c0 = *E->c0;
        cudaMemsetAsync(c0.lz.counter, 0, 4 * sizeof(unsigned), c0.stream);
        cudaMemsetAsync(c0.lz.flags, 0, F_NFLAGS * sizeof(int), c0.stream);
    }
    return rc;
}

int batch_inflight(const BatchEngine *E) { return (int)E->solves.size(); }

int lanczos_eigh_batch(Ctx *const *cs, int nb, int nitermax, double tol, const uint64_t *seeds,
                       double *evals_host, int *numops) {
    if (nb < 1 || nb > BATCH_MAX) {
        cs[0]->err = "nss_eigh_batch: between 1 and " + std::to_string(BATCH_MAX) + " solves per batch";
        return NSS_ERR_INVALID;
    }
    BatchEngine E;
    int rc = engine_init(E, *cs[0]);
    if (rc) return rc;
    std::vector<int> ids(nb);
    for (int b = 0; b < nb; ++b)
        if ((rc = engine_add(E, *cs[b], seeds ? seeds[b] : 1234, nitermax, tol, &ids[b]))) return rc;
    std::vector<int> did(nb), nop(nb);
    std::vector<double> en(nb);
    int first_rc = NSS_OK;
    for (int round = 0; round < 1000000 && !E.solves.empty(); ++round) {
        int nd = 0;
        if ((rc = engine_step(E, nb, &nd, did.data(), en.data(), nop.data()))) {
            engine_drop(E);
            return rc;
        }
        for (int q = 0; q < nd; ++q) {
            const int id = did[q] < 0 ? -did[q] : did[q];
            const int b = (int)(std::find(ids.begin(), ids.end(), id) - ids.begin());
            if (b >= nb) continue;
            if (evals_host) evals_host[b] = en[q];
            if (numops) numops[b] = nop[q];
            if (did[q] < 0 && !first_rc) {
                first_rc = NSS_ERR_NOCONV;
                cs[0]->err = cs[b]->err;
            }
        }
    }
    return first_rc;
}

}  // namespace nss

// Tile bodies of the sector product H_sb psi shared by the stand-alone
// kernels (k_matvec.cu) and the persistent Lanczos kernel (k_lanczos.cu).
//
// One output tile is rows [row0, row0+TR) x columns [col0, col0+TC) of
// sector k, W_k[il][ir] (ir fastest).  The dense part is
//     H_L(k) W_k + W_k H_R(k)^T           (src/DMRG_SUPERBLOCK_SETUP.f90:767-796)
// and the A x B terms of the sector add A W_q B^T (:808-857), regrouped by
// the sector they write.  A tile is computed by a group of 256 threads that
// synchronise through a `Sync` functor: the whole CTA (__syncthreads) in the
// stand-alone kernels, a named barrier of 256 threads when two tiles share a
// CTA of the persistent kernel.
#pragma once

#include "device.cuh"

namespace nss {

struct CtaSync {
    __device__ __forceinline__ void operator()() const { __syncthreads(); }
};

// bar.sync id, 256: one of the two 256-thread groups of a 512-thread CTA
struct GroupSync {
    int id;
    __device__ __forceinline__ void operator()() const {
        asm volatile("bar.sync %0, 256;" ::"r"(id) : "memory");
    }
};

// A x B terms of one output tile, staged.  The block operators of the two
// sites at the centre bond have at most one stored element per row (the
// enlarged blocks are block (x) site), so for each term of the output sector
// the tile's rows of A and columns of B are staged in shared memory as
// (column, value) pairs, and each output then needs only independent
// gathers W_q[aj][bj], in flight together.  A row with more than one element
// sends that batch of terms to the general CSR loop.
constexpr int AB_MAXT = 16;

template <class V, int TR, int TC>
struct AbStage {
    int ac[AB_MAXT][TR], bc[AB_MAXT][TC];
    V av[AB_MAXT][TR], bv[AB_MAXT][TC];
    const V *wq[AB_MAXT];
    int drq[AB_MAXT];
    int multi;
};

// stage terms [tb, tb+nt) for rows row0.. and columns col0..; `lt` is the
// thread's index in its group of `nthr`; ends with a group barrier
template <class V, int TR, int TC, class Sync>
__device__ __forceinline__ void ab_stage(AbStage<V, TR, TC> &S, const V *__restrict__ v, int tb, int nt, int row0,
                                         int col0, int dl, int dr, const int *__restrict__ drs,
                                         const int64_t *__restrict__ off, const DevTerm *__restrict__ terms,
                                         const int *__restrict__ ab_rp, const int *__restrict__ ab_col,
                                         const V *__restrict__ ab_val, int lt, int nthr, Sync sync) {
    if (lt == 0) S.multi = 0;
    sync();
    for (int e = lt; e < nt * (TR + TC); e += nthr) {
        const int tt = e / (TR + TC), r = e % (TR + TC);
        const DevTerm tm = terms[tb + tt];
        int c = -1;
        V x = (V)0;
        if (r < TR) {
            const int il = row0 + r;
            if (il < dl) {
                const int p0 = ab_rp[tm.a_rp + il], p1 = ab_rp[tm.a_rp + il + 1];
                if (p1 > p0) { c = ab_col[p0]; x = ab_val[p0]; }
                if (p1 - p0 > 1) S.multi = 1;
            }
            S.ac[tt][r] = c;
            S.av[tt][r] = x;
        } else {
            const int ir = col0 + (r - TR);
            if (ir < dr) {
                const int p0 = ab_rp[tm.b_rp + ir], p1 = ab_rp[tm.b_rp + ir + 1];
                if (p1 > p0) { c = ab_col[p0]; x = ab_val[p0]; }
                if (p1 - p0 > 1) S.multi = 1;
            }
            S.bc[tt][r - TR] = c;
            S.bv[tt][r - TR] = x;
            if (r == TR) {
                S.wq[tt] = v + off[tm.in_sec];
                S.drq[tt] = drs[tm.in_sec];
            }
        }
    }
    sync();
}

// general loop for output (il, ir) over terms [tb, tb+nt): the reference's
// sum over the stored elements of A and B
template <class V>
__device__ __forceinline__ V ab_csr(V acc, const V *__restrict__ v, int tb, int nt, int il, int ir,
                                    const int *__restrict__ drs, const int64_t *__restrict__ off,
                                    const DevTerm *__restrict__ terms, const int *__restrict__ ab_rp,
                                    const int *__restrict__ ab_col, const V *__restrict__ ab_val) {
    for (int ti = tb; ti < tb + nt; ++ti) {
        const DevTerm tm = terms[ti];
        const V *Wq = v + off[tm.in_sec];
        const int drq = drs[tm.in_sec];
        const int *arp = ab_rp + tm.a_rp, *brp = ab_rp + tm.b_rp;
        for (int ja = arp[il]; ja < arp[il + 1]; ++ja) {
            const int aj = ab_col[ja];
            V cb = (V)0;
            for (int jb = brp[ir]; jb < brp[ir + 1]; ++jb) cb = fma(ab_val[jb], Wq[(int64_t)aj * drq + ab_col[jb]], cb);
            acc = fma(ab_val[ja], cb, acc);
        }
    }
    return acc;
}

// Shared memory of one FP32 tile group.
struct Tile32Smem {
    float sa[32][33];
    float sb[32][33];
    AbStage<float, 32, 32> S;
};

// Operands of the FP32 sector product (device pointers of DevSb).
struct Hv32Ops {
    const int *dls, *drs;
    const int64_t *off;
    const float *hl;
    const int64_t *hl_off;
    const float *hr;
    const int64_t *hr_off;
    const int *term_ptr;
    const DevTerm *terms;
    const int *ab_rp, *ab_col;
    const float *ab_val;
    // per work item of the persistent kernel: offset of its A x B table in
    // `ell` (-1: a row with several elements, use the CSR loop)
    const int *item_ell;
    const int2 *ell;             // (column, value bits) of A rows / B columns
    const int4 *term_hdr;        // per term: offset of its input sector (lo, hi), its Dr
};

// One 32x32 FP32 output tile t = (sector, row0, col0, flags) by 256 threads
// (lt = thread index in the group), each owning rows {ty, ty+16} x columns
// {tx, tx+16}.  A "terms only" tile (t.w & 1) skips the two dense products:
// the tensor-core GEMM forms them beside it, and they are added afterwards
// (k_add_planes, k_orth).
template <class Sync>
__device__ __forceinline__ void hv32_tile(int4 t, const float *__restrict__ v, float *__restrict__ hv,
                                          const Hv32Ops &op, Tile32Smem &sm, int lt, Sync sync) {
    const int k = t.x, row0 = t.y, col0 = t.z;
    const int dl = op.dls[k], dr = op.drs[k];
    const int64_t o = op.off[k];
    const float *W = v + o;
    const float *HL = op.hl + op.hl_off[k];
    const float *HR = op.hr + op.hr_off[k];
    const int ty = lt / 16, tx = lt % 16;
    float acc[2][2] = {{0.f, 0.f}, {0.f, 0.f}};
    const int kdl = (t.w & 1) ? 0 : dl, kdr = (t.w & 1) ? 0 : dr;
    // H_L W
    for (int j0 = 0; j0 < kdl; j0 += 32) {
        for (int e = lt; e < 32 * 32; e += 256) {
            const int r = e / 32, cc = e % 32;
            const int gi = row0 + r, gj = j0 + cc;
            sm.sa[r][cc] = (gi < dl && gj < dl) ? HL[(int64_t)gi * dl + gj] : 0.f;
            const int gj2 = j0 + r, gc = col0 + cc;
            sm.sb[r][cc] = (gj2 < dl && gc < dr) ? W[(int64_t)gj2 * dr + gc] : 0.f;
        }
        sync();
#pragma unroll 8
        for (int j = 0; j < 32; ++j) {
            const float a0 = sm.sa[ty][j], a1 = sm.sa[ty + 16][j], b0 = sm.sb[j][tx], b1 = sm.sb[j][tx + 16];
            acc[0][0] = fmaf(a0, b0, acc[0][0]);
            acc[0][1] = fmaf(a0, b1, acc[0][1]);
            acc[1][0] = fmaf(a1, b0, acc[1][0]);
            acc[1][1] = fmaf(a1, b1, acc[1][1]);
        }
        sync();
    }
    // W H_R^T
    for (int j0 = 0; j0 < kdr; j0 += 32) {
        for (int e = lt; e < 32 * 32; e += 256) {
            const int r = e / 32, cc = e % 32;
            const int gi = row0 + r, gj = j0 + cc;
            sm.sa[r][cc] = (gi < dl && gj < dr) ? W[(int64_t)gi * dr + gj] : 0.f;
            const int gr = col0 + r;                 // sb[j][x] = HR[col0+x][j0+j]
            sm.sb[cc][r] = (gr < dr && gj < dr) ? HR[(int64_t)gr * dr + gj] : 0.f;
        }
        sync();
#pragma unroll 8
        for (int j = 0; j < 32; ++j) {
            const float a0 = sm.sa[ty][j], a1 = sm.sa[ty + 16][j], b0 = sm.sb[j][tx], b1 = sm.sb[j][tx + 16];
            acc[0][0] = fmaf(a0, b0, acc[0][0]);
            acc[0][1] = fmaf(a0, b1, acc[0][1]);
            acc[1][0] = fmaf(a1, b0, acc[1][0]);
            acc[1][1] = fmaf(a1, b1, acc[1][1]);
        }
        sync();
    }
    // A x B terms, staged per batch of terms (see ab_stage)
    AbStage<float, 32, 32> &S = sm.S;
    for (int tb = op.term_ptr[k]; tb < op.term_ptr[k + 1]; tb += AB_MAXT) {
        const int nt = min(AB_MAXT, op.term_ptr[k + 1] - tb);
        ab_stage<float, 32, 32>(S, v, tb, nt, row0, col0, dl, dr, op.drs, op.off, op.terms, op.ab_rp, op.ab_col,
                                op.ab_val, lt, 256, sync);
        if (!S.multi) {
            for (int tt = 0; tt < nt; ++tt) {
                const float *Wq = S.wq[tt];
                const int drq = S.drq[tt];
#pragma unroll
                for (int rr = 0; rr < 2; ++rr)
#pragma unroll
                    for (int cc = 0; cc < 2; ++cc) {
                        const int aj = S.ac[tt][ty + 16 * rr], bj = S.bc[tt][tx + 16 * cc];
                        if (aj >= 0 && bj >= 0)
                            acc[rr][cc] = fmaf(S.av[tt][ty + 16 * rr] * S.bv[tt][tx + 16 * cc],
                                               Wq[(int64_t)aj * drq + bj], acc[rr][cc]);
                    }
            }
        } else {
            for (int rr = 0; rr < 2; ++rr)
                for (int cc = 0; cc < 2; ++cc) {
                    const int il = row0 + ty + 16 * rr, ir = col0 + tx + 16 * cc;
                    if (il < dl && ir < dr)
                        acc[rr][cc] = ab_csr<float>(acc[rr][cc], v, tb, nt, il, ir, op.drs, op.off, op.terms,
                                                    op.ab_rp, op.ab_col, op.ab_val);
                }
        }
        sync();
    }
    for (int rr = 0; rr < 2; ++rr)
        for (int cc = 0; cc < 2; ++cc) {
            const int il = row0 + ty + 16 * rr, ir = col0 + tx + 16 * cc;
            if (il < dl && ir < dr) hv[o + (int64_t)il * dr + ir] = acc[rr][cc];
        }
}

}  // namespace nss

namespace nss {

// Work items of the persistent kernel's H*psi phase.  An item is a 32x32
// output tile (x = sector, y = row0, z = col0) and a part (w):
//   HV_FULL   H_L W + W H_R^T + A x B terms       -> slot 0
//   HV_LEFT   H_L W                               -> slot 1
//   HV_RIGHT  W H_R^T                             -> slot 2
//   HV_TERMS  A x B terms                         -> slot 0
// Sectors whose tiles have long K loops (Dl or Dr > HV_SPLIT) are split into the
// last three so the parts run on different SMs; the result is slot 0 +
// slot 1 + slot 2 (regions of slots 1 and 2 that no item writes stay zero).
// An iteration lasts as long as its longest item, and a superblock has fewer
// items than the 304 groups of the grid; but a part costs a load round of its
// own, which a batch of solves, with more items than groups, pays: solves of
// 16 900 states (54 x 54 sectors) 1.99 -> 1.92 ms and of 66 600 2.30 -> 2.28 ms
// from 64 to 48; 32 is no better there and costs a batch of 16 3 %, a solve of
// 66 600 20 % (more items than groups).
enum { HV_FULL = 0, HV_LEFT = 1, HV_RIGHT = 2, HV_TERMS = 3 };
constexpr int HV_SPLIT = 48;
constexpr int HV_KMAX = 128;            // K extent staged at once
constexpr int SA_LD = HV_KMAX + 4;      // rows along K: float4 reads, eight rows apart in different banks
constexpr int SB_FULL = 64 * 32;        // a FULL item's second B operand in sb, rows SB_LD apart
constexpr int SB_LD = 64 + 4;

// A work item with everything it needs to start its operand loads, so that
// these depend on one load only: (sector, row0, col0, part), (Dl, Dr, first
// term, end term), (sector offset lo/hi, A x B table offset, 0), (H_L and
// H_R offsets lo/hi).
struct ItemRec {
    int4 a, b, c, d;
};

__device__ __forceinline__ int64_t lohi(int lo, int hi) { return (int64_t)(unsigned)lo | ((int64_t)hi << 32); }

struct __align__(16) Item32Smem {
    float sa[32 * SA_LD];               // A: rows x K
    float sb[32 * SA_LD];               // B: K x columns (H_L W) or columns x K (W H_R^T)
                                        // (W's part of both: then the tile's four K shares)
    union {
        struct {
            int2 ta[AB_MAXT][32], tb[AB_MAXT][32];   // (column, value) of A's rows, B's columns (col_pos)
            int4 hd[AB_MAXT];
        };
        AbStage<float, 32, 32> S;       // rows of several elements
    };
};

// A thread's columns are eight apart; stored side by side it reads them as one vector
__device__ __forceinline__ int col_pos(int x) { return 4 * (x & 7) + (x >> 3); }

// Asynchronous copies into shared memory (zero when !in; the address is then not read)
template <int BYTES>
__device__ __forceinline__ void cp_async(void *dst, const void *src, bool in) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src),
                 "n"(BYTES), "r"(in ? BYTES : 0)
                 : "memory");
}
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// dst[r * LD + c] = src[r * ld + c], r < 32, c < kn4: zero from `rows` and `kn` on
__device__ __forceinline__ void stage_rows(float *dst, int LD, const float *src, int64_t ld, int rows, int kn, int kn4,
                                           int lt) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int r = (lt >> 5) + 8 * q;
        const float *p = r < rows ? src + r * ld : src;
        for (int c = lt & 31; c < kn4; c += 32) {
            const bool in = r < rows && c < kn;
            cp_async<4>(dst + r * LD + c, in ? p + c : src, in);
        }
    }
}
// dst[k * 32 + col_pos(x)] = src[k * ld + x], x < 32, k < kn4: zero from `cols` and `kn` on
__device__ __forceinline__ void stage_cols(float *dst, const float *src, int64_t ld, int cols, int kn, int kn4, int lt) {
    const int x = lt & 31;
    for (int k = lt >> 5; k < kn4; k += 8) {
        const bool in = k < kn && x < cols;
        cp_async<4>(dst + k * 32 + col_pos(x), in ? src + k * ld + x : src, in);
    }
}

// acc[i][j] += A[4 ty + i][k] B[k][tx + 8 j] over the K steps of four s, s + 4,
// ... < n4; ROWS: B is stored as columns x K
template <bool ROWS>
__device__ __forceinline__ void item_mma(const float *sa, const float *sb, int ldb, int s, int n4, int ty, int tx,
                                         float (&acc)[4][4]) {
    for (; s < n4; s += 4) {
        const int k = 4 * s;
        float a[4][4], b[4][4];                      // [row][k], [k][column]
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float4 t = *reinterpret_cast<const float4 *>(sa + (4 * ty + i) * SA_LD + k);
            a[i][0] = t.x; a[i][1] = t.y; a[i][2] = t.z; a[i][3] = t.w;
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float4 t = *reinterpret_cast<const float4 *>(ROWS ? sb + (tx + 8 * q) * ldb + k : sb + (k + q) * 32 + 4 * tx);
            const float u[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (ROWS) b[j][q] = u[j];
                else b[q][j] = u[j];
            }
        }
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i][q], b[q][j], acc[i][j]);
    }
}

// The anchored refinement's vectors whose products with H v are wanted: u
// and nd deflation vectors y[k*n..] (u null: none)
struct AncCols {
    const float *u, *y;
    int nd;
    int64_t n;
};
constexpr int ANC_MAX = 5;              // u and up to four y

// One item by 256 threads (lt = thread index in the group).  An iteration of
// the persistent kernel waits for its slowest item, and a group has one item
// as a rule, so what counts is an item's latency: operands, A x B tables and
// the outputs' own W go out in one round of asynchronous copies; the gathers
// of the first four terms are in flight during the products.  In the products
// a thread holds 4 x 4 outputs for every fourth K step of four (eight floats
// read from shared memory for sixteen FMAs; at 2 x 2 outputs shared memory's
// 128 B a clock took 130 clk a step); the four shares are added in shared
// memory, after which a thread owns row r, columns {cx, cx + 8, cx + 16,
// cx + 24}.  keep: this group's last item was the same one, so the tiles of
// H_L and H_R and the tables are still in shared memory.  An item of 39 x 40 states and
// three terms 9.7k -> 6.2k clk, a part of K = 106 13.4k -> 6.5k; an iteration of
// 66 600 states 14.2 -> 9.3 us, solves of it 2.36 -> 1.87 ms, of 16 900 states
// 1.92 -> 1.56 ms.  The staging (2.2k to 2.8k) is the L2's latency: plain loads
// through registers took as long.
// The outputs times `scale` go to the item's slot; this thread's share of
// sum_i (v[i] scale) (out[i] scale) over its outputs is added to p[0], those
// of u.out and y_k.out to p[1..NA].
template <int NA, class Sync>
__device__ __forceinline__ void hv32_item(const ItemRec &it, const float *__restrict__ v, float *const *slots,
                                          const Hv32Ops &op, Item32Smem &sm, int lt, Sync sync, float scale,
                                          const AncCols &ac, float (&p)[1 + NA], bool keep) {
    const int row0 = it.a.y, col0 = it.a.z, part = it.a.w;
    const int dl = it.b.x, dr = it.b.y, t0 = it.b.z, t1 = it.b.w;
    const int64_t o = lohi(it.c.x, it.c.y);
    const float *W = v + o;
    const float *HL = op.hl + lohi(it.d.x, it.d.y) + (int64_t)row0 * dl;
    const float *HR = op.hr + lohi(it.d.z, it.d.w) + (int64_t)col0 * dr;
    const float *Wr = W + (int64_t)row0 * dr;
    const int rows = dl - row0, cols = dr - col0;
    const int r = lt >> 3, cx = lt & 7;
    const bool terms = part == HV_FULL || part == HV_TERMS;
    const int eo = terms ? it.c.z : -1;
    const int nt0 = min(AB_MAXT, t1 - t0);
    auto stage_terms = [&](int tb, int nt) {
        const int2 *src = op.ell + eo + (int64_t)(tb - t0) * 64;
        for (int e = lt; e < nt * 64; e += 256) {
            const int tt = e >> 6, x = e & 63;
            cp_async<8>(x < 32 ? &sm.ta[tt][x] : &sm.tb[tt][col_pos(x - 32)], src + e, true);
        }
        if (lt < nt) cp_async<16>(&sm.hd[lt], op.term_hdr + tb + lt, true);
    };
    // K range [kb, kb + kn) of a LEFT or RIGHT item; kh: H is there already
    auto stage_part = [&](int kb, int kn, bool kh) {
        const int kn4 = (kn + 3) & ~3;
        if (part == HV_LEFT) {
            if (!kh) stage_rows(sm.sa, SA_LD, HL + kb, dl, rows, kn, kn4, lt);
            stage_cols(sm.sb, W + (int64_t)kb * dr + col0, dr, cols, kn, kn4, lt);
        } else {
            stage_rows(sm.sa, SA_LD, Wr + kb, dr, rows, kn, kn4, lt);
            if (!kh) stage_rows(sm.sb, SA_LD, HR + kb, dr, cols, kn, kn4, lt);
        }
    };
    const int K = part == HV_LEFT ? dl : dr;
    if (!keep) sync();                               // the last item's reads are done
    if (part == HV_FULL) {
        const int kl4 = (dl + 3) & ~3, kr4 = (dr + 3) & ~3;
        if (!keep) {
            stage_rows(sm.sa, SA_LD, HL, dl, rows, dl, kl4, lt);
            stage_rows(sm.sb + SB_FULL, SB_LD, HR, dr, cols, dr, kr4, lt);
        }
        stage_cols(sm.sb, W + col0, dr, cols, dl, kl4, lt);
        stage_rows(sm.sa + 64, SA_LD, Wr, dr, rows, dr, kr4, lt);
    } else if (part != HV_TERMS) {
        stage_part(0, min(HV_KMAX, K), keep && K <= HV_KMAX);
    }
    if (eo >= 0 && nt0 > 0 && !(keep && t1 - t0 <= AB_MAXT)) stage_terms(t0, nt0);
    float wv[4], uv[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const bool in = r < rows && cx + 8 * j < cols;
        const int64_t at = (int64_t)r * dr + col0 + cx + 8 * j;
        wv[j] = in ? Wr[at] : 0.f;
        uv[j] = NA > 0 && ac.u && in ? ac.u[o + (int64_t)row0 * dr + at] : 0.f;
    }
    cp_async_wait();
    sync();
    // W_q[aj][bj] of term tt of the staged batch for the thread's outputs
    auto gather = [&](int tt, float (&g)[4]) {
        const int aj = sm.ta[tt][r].x;
        const int4 b0 = *reinterpret_cast<const int4 *>(&sm.tb[tt][4 * cx]);
        const int4 b1 = *reinterpret_cast<const int4 *>(&sm.tb[tt][4 * cx + 2]);
        const int4 hd = sm.hd[tt];
        const float *q = v + lohi(hd.x, hd.y) + (int64_t)aj * hd.z;
        g[0] = (aj | b0.x) >= 0 ? q[b0.x] : 0.f;
        g[1] = (aj | b0.z) >= 0 ? q[b0.z] : 0.f;
        g[2] = (aj | b1.x) >= 0 ? q[b1.x] : 0.f;
        g[3] = (aj | b1.z) >= 0 ? q[b1.z] : 0.f;
    };
    float g[4][4];
#pragma unroll
    for (int u = 0; u < 4; ++u)
        if (eo >= 0 && u < nt0) gather(u, g[u]);
    float y[4] = {0.f, 0.f, 0.f, 0.f};
    if (part != HV_TERMS) {
        const int tx = lt & 7, ty = ((lt >> 3) & 3) + 4 * ((lt >> 5) & 1), kq = lt >> 6;
        float acc[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
        if (part == HV_FULL) {
            const int nl = (dl + 3) >> 2, nr = (dr + 3) >> 2;
            item_mma<false>(sm.sa, sm.sb, 0, kq, nl, ty, tx, acc);
            item_mma<true>(sm.sa + 64, sm.sb + SB_FULL, SB_LD, (kq - nl) & 3, nr, ty, tx, acc);
        } else {
            for (int kb = 0; kb < K; kb += HV_KMAX) {
                const int kn = min(HV_KMAX, K - kb);
                if (kb > 0) {
                    sync();
                    stage_part(kb, kn, false);
                    cp_async_wait();
                    sync();
                }
                if (part == HV_LEFT) item_mma<false>(sm.sa, sm.sb, 0, kq, (kn + 3) >> 2, ty, tx, acc);
                else item_mma<true>(sm.sa, sm.sb, SA_LD, kq, (kn + 3) >> 2, ty, tx, acc);
            }
        }
        // the shares go where W was: H stays for the next iteration
        auto share = [&](int q, int row) -> float4 * {
            float *d = part == HV_RIGHT ? sm.sa + (q * 32 + row) * 32
                       : part == HV_LEFT || q < 2 ? sm.sb + (q * 32 + row) * 32 : sm.sa + row * SA_LD + 64 + (q - 2) * 32;
            return reinterpret_cast<float4 *>(d);
        };
        sync();
#pragma unroll
        for (int i = 0; i < 4; ++i) share(kq, 4 * ty + i)[tx] = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
        sync();
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float4 t = share(q, r)[cx];
            y[0] += t.x;
            y[1] += t.y;
            y[2] += t.z;
            y[3] += t.w;
        }
    }
    for (int tb = t0; terms && tb < t1; tb += AB_MAXT) {
        const int nt = min(AB_MAXT, t1 - tb);
        if (eo >= 0) {
            if (tb != t0) {
                sync();
                stage_terms(tb, nt);
                cp_async_wait();
                sync();
            }
            for (int t4 = 0; t4 < nt; t4 += 4) {
                if (tb != t0 || t4 != 0)
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        if (t4 + u < nt) gather(t4 + u, g[u]);
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (t4 + u < nt) {
                        const float av = __int_as_float(sm.ta[t4 + u][r].y);
                        const int4 b0 = *reinterpret_cast<const int4 *>(&sm.tb[t4 + u][4 * cx]);
                        const int4 b1 = *reinterpret_cast<const int4 *>(&sm.tb[t4 + u][4 * cx + 2]);
                        y[0] = fmaf(av * __int_as_float(b0.y), g[u][0], y[0]);
                        y[1] = fmaf(av * __int_as_float(b0.w), g[u][1], y[1]);
                        y[2] = fmaf(av * __int_as_float(b1.y), g[u][2], y[2]);
                        y[3] = fmaf(av * __int_as_float(b1.w), g[u][3], y[3]);
                    }
            }
        } else {
            AbStage<float, 32, 32> &S = sm.S;
            ab_stage<float, 32, 32>(S, v, tb, nt, row0, col0, dl, dr, op.drs, op.off, op.terms, op.ab_rp, op.ab_col,
                                    op.ab_val, lt, 256, sync);
            if (!S.multi) {
                for (int tt = 0; tt < nt; ++tt) {
                    const int aj = S.ac[tt][r];
                    const float *q = S.wq[tt] + (int64_t)aj * S.drq[tt];
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const int bj = S.bc[tt][cx + 8 * j];
                        if ((aj | bj) >= 0) y[j] = fmaf(S.av[tt][r] * S.bv[tt][cx + 8 * j], q[bj], y[j]);
                    }
                }
            } else {
                for (int j = 0; j < 4; ++j)
                    if (r < rows && cx + 8 * j < cols)
                        y[j] = ab_csr<float>(y[j], v, tb, nt, row0 + r, col0 + cx + 8 * j, op.drs, op.off, op.terms,
                                             op.ab_rp, op.ab_col, op.ab_val);
            }
            sync();
        }
    }
    float *out = slots[part == HV_LEFT ? 1 : (part == HV_RIGHT ? 2 : 0)] + o + (int64_t)row0 * dr;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        y[j] *= scale;
        if (r < rows && cx + 8 * j < cols) out[(int64_t)r * dr + col0 + cx + 8 * j] = y[j];
        else y[j] = 0.f;
        p[0] = fmaf(wv[j] * scale, y[j], p[0]);
        if constexpr (NA > 0) p[1] = fmaf(uv[j], y[j], p[1]);
    }
    if constexpr (NA > 1) {
#pragma unroll
        for (int k = 0; k < NA - 1; ++k)
            if (k < ac.nd) {
                const float *yk = ac.y + (int64_t)k * ac.n + o + (int64_t)row0 * dr + (int64_t)r * dr + col0 + cx;
                float z[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) z[j] = r < rows && cx + 8 * j < cols ? yk[8 * j] : 0.f;
#pragma unroll
                for (int j = 0; j < 4; ++j) p[2 + k] = fmaf(z[j], y[j], p[2 + k]);
            }
    }
}

}  // namespace nss

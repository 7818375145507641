// Superblock upload and the direct H_sb * psi product (plain FP64 path).
//
// Restates spMatVec_direct_main (src/DMRG_SUPERBLOCK_SETUP.f90:740-865) as one
// kernel over output tiles.  For output sector k, with W_k the row-major
// [Dl x Dr] view of the sector (i = ir + il*Dr + Offset, :770),
//     Out_k = H_L(k) W_k + W_k H_R(k)^T + sum_t A_t W_q(t) B_t^T,
// where the last sum runs over the terms whose RowOffset is sector k
// (:808-857, regrouped by output sector so each tile has one writer).
#include "device.cuh"
#include "hv_tile.cuh"
#include "host_sparse.hpp"
#include "sector_mma.cuh"
#include "sector_split.cuh"

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <map>

namespace nss {

int tc_min_dl_default() {
    const char *e = std::getenv("NSS_TC_MIN_DL");
    if (!e) return 1024;
    const int x = std::atoi(e);
    return x < 0 ? 0 : x;
}

void mma_tile_default(int *bn, bool *split) {
    const char *b = std::getenv("NSS_TC_BN");
    *bn = (b && std::atoi(b) == 128) ? 128 : 64;
    const char *sp = std::getenv("NSS_TC_SPLIT");
    *split = !(sp && std::atoi(sp) == 0);
}

int mma_kps_default() {
    const char *e = std::getenv("NSS_TC_KPS");
    return (e && std::atoi(e) == 2) ? 2 : 1;
}

bool mma_lolo_default() {
    const char *e = std::getenv("NSS_TC_LOLO");
    return e && std::atoi(e) != 0;
}

uint32_t wait_limit() {
    const char *e = std::getenv("NSS_WAIT_LIMIT");
    if (!e) return 1u << 22;
    const long x = std::atol(e);
    return x < 0 ? 0u : (uint32_t)std::min<long>(x, 1l << 30);
}

void ctx_free(Ctx &c, void *p) {
    if (!p) return;
    auto it = c.sizes.find(p);
    if (it != c.sizes.end()) {
        c.used -= it->second;
        c.sizes.erase(it);
    }
    cudaFree(p);
}

// The pool's device arrays are sections of one device arena, filled from
// one pinned staging buffer by one copy; both grow only and are kept from
// one upload to the next (a DMRG run uploads a new pool every step).
void sb_release(Ctx &c, bool free_arena) {
    c.sb = DevSb{};
    if (free_arena) {
        ctx_free(c, c.sp_mem);
        c.sp_mem = nullptr;
        c.sp_cap = 0;
        ctx_free(c, c.sb_arena);
        if (c.sb_stage) cudaFreeHost(c.sb_stage);
        c.sb_arena = nullptr;
        c.sb_stage = nullptr;
        c.sb_arena_cap = c.sb_stage_cap = 0;
    }
}

namespace {

uint64_t next_gen() {
    static std::atomic<uint64_t> gen{0};
    return ++gen;
}

}  // namespace

bool split_drop(Ctx &c) {
    if (!c.sp_mem) return false;
    ctx_free(c, c.sp_mem);           // waits for the device
    c.sp_mem = nullptr;
    c.sp_cap = 0;
    if (c.sb.sp_nitems) {
        c.sb.sp_nitems = 0;
        c.sb.gen = next_gen();       // graphs captured with it are void
    }
    return true;
}

namespace {

constexpr int TILE = 16;
constexpr int TILE32 = 32;
constexpr int HV_TR = 4, HV_TC = 8;    // output tile of a warp of k_hv_fp64
constexpr int HV_WARPS = 4;            // warps of its CTAs, one per quarter of an SM
constexpr int HV_SUB = (8 / HV_TR) * (32 / HV_TC);   // its tiles in a SplitTile
constexpr int HV_CTAS = 5;             // CTAs per SM at most

// Sections of the pool's arena: each array at a 256-byte boundary (at least
// 16 bytes, so that every pointer is distinct and valid), those with a host
// source first, so that one copy of `host` bytes fills them; the sections that
// the device fills follow (they are many times larger and not copied).
struct Stager {
    struct Item {
        void **dst;
        const void *src;
        size_t bytes, off;
    };
    std::vector<Item> items, dev;
    size_t host = 0, device = 0;
    // a section gathered from several host arrays (straight from the caller's
    // matrices: collecting them in a vector first cost a second copy and the
    // page faults of fresh memory, most of an upload's host time)
    struct Part {
        const void *src;
        size_t bytes, off;      // offset in the arena
    };
    std::vector<Part> parts;
    template <class T>
    void add_gather(T **dst, size_t count) {
        items.push_back({(void **)dst, nullptr, count * sizeof(T), host});
        host += (std::max<size_t>(count * sizeof(T), 16) + 255) / 256 * 256;
    }
    // the next `count` elements of the section `dst` was added for, at element `at`
    template <class T>
    void part(size_t item, const T *src, size_t count, size_t at) {
        if (count) parts.push_back({(const void *)src, count * sizeof(T), items[item].off + at * sizeof(T)});
    }
    template <class T>
    void add(T **dst, const std::vector<T> &v) {
        const size_t bytes = v.size() * sizeof(T);
        items.push_back({(void **)dst, (const void *)v.data(), bytes, host});
        host += (std::max<size_t>(bytes, 16) + 255) / 256 * 256;
    }
    // a section the device fills (no host source, not copied)
    template <class T>
    void add_dev(T **dst, size_t count) {
        const size_t bytes = count * sizeof(T);
        dev.push_back({(void **)dst, nullptr, bytes, device});
        device += (std::max<size_t>(bytes, 16) + 255) / 256 * 256;
    }
};

// Dense sector operators from their CSR rows: one warp per row of one
// sector's H_L or H_R (rows of both sides in one launch), 32 entries at a time,
// duplicates summed in their order as the host build did (one lane takes a
// batch that holds a column twice); the blocks are zeroed beforehand.  FP32
// copies follow in k_dense32.  (A thread per row wrote 300 entries one after
// the other: 62 us at Hubbard m = 250, 187 us at spin-1 m = 400.)
struct DenseRows {
    const int *rowptr;      // per side: all sectors' rows, global entry offsets
    const int *col;
    const double *val;
    const int *row_sec;     // sector of each row (global row index)
    const int64_t *row_first;   // first global row of each sector
};
__global__ void __launch_bounds__(256) k_densify(DenseRows L, DenseRows R, int nrow_l, int nrow_r,
                                                  const int *__restrict__ dls, const int *__restrict__ drs,
                                                  const int64_t *__restrict__ hl_off, const int64_t *__restrict__ hr_off,
                                                  double *__restrict__ hl, double *__restrict__ hr) {
    const int64_t t = blockIdx.x * (int64_t)(blockDim.x / 32) + threadIdx.x / 32;
    if (t >= (int64_t)nrow_l + nrow_r) return;       // whole warps
    const int lane = threadIdx.x & 31;
    const bool right = t >= nrow_l;
    const DenseRows &D = right ? R : L;
    const int g = (int)(right ? t - nrow_l : t);
    const int k = D.row_sec[g];
    const int d = right ? drs[k] : dls[k];
    const int i = (int)(g - D.row_first[k]);
    double *row = (right ? hr + hr_off[k] : hl + hl_off[k]) + (int64_t)i * d;
    const int p1 = D.rowptr[g + 1];
    for (int p0 = D.rowptr[g]; p0 < p1; p0 += 32) {
        const int p = p0 + lane;
        const int c = p < p1 ? D.col[p] : -1 - lane;
        const double x = p < p1 ? D.val[p] : 0.0;
        const bool twice = __popc(__match_any_sync(0xffffffffu, c)) > 1;
        if (!__any_sync(0xffffffffu, twice)) {
            if (p < p1) row[c] += x;
        } else if (lane == 0) {
            for (int q = p0; q < min(p1, p0 + 32); ++q) row[D.col[q]] += D.val[q];
        }
        __syncwarp();
    }
}

__global__ void __launch_bounds__(256) k_dense32(const double *__restrict__ x, float *__restrict__ y, int64_t n) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        y[i] = (float)x[i];
}

int stage_commit(Ctx &c, Stager &sg) {
    // the previous upload's copy out of the staging buffer may still be in
    // flight on the stream (two uploads with no solve between them)
    NSS_CUDA_TRY(c, cudaStreamSynchronize(c.stream));
    const size_t total = sg.host + sg.device;
    if (c.sb_arena_cap < total) {
        ctx_free(c, c.sb_arena);
        c.sb_arena = nullptr;
        c.sb_arena_cap = 0;
        const size_t cap = total + total / 4;   // headroom: the pool size varies from step to step
        NSS_CUDA_TRY(c, ctx_alloc(c, &c.sb_arena, cap));
        c.sb_arena_cap = cap;
    }
    if (c.sb_stage_cap < sg.host) {
        if (c.sb_stage) cudaFreeHost(c.sb_stage);
        c.sb_stage = nullptr;
        c.sb_stage_cap = 0;
        const size_t cap = sg.host + sg.host / 4;
        NSS_CUDA_TRY(c, cudaHostAlloc((void **)&c.sb_stage, cap, cudaHostAllocDefault));
        c.sb_stage_cap = cap;
    }
    // the staging copy in pieces of at most 1 MiB, spread over host threads
    struct Piece {
        char *dst;
        const char *src;
        size_t bytes;
    };
    std::vector<Piece> pieces;
    constexpr size_t PIECE = (size_t)1 << 20;
    auto cut = [&](const void *src, size_t off, size_t bytes) {
        for (size_t o = 0; o < bytes; o += PIECE)
            pieces.push_back({c.sb_stage + off + o, (const char *)src + o, std::min(PIECE, bytes - o)});
    };
    for (const auto &it : sg.items)
        if (it.src) cut(it.src, it.off, it.bytes);
    for (const auto &p : sg.parts) cut(p.src, p.off, p.bytes);
    parallel_for((int)pieces.size(), [&](int i) { std::memcpy(pieces[i].dst, pieces[i].src, pieces[i].bytes); },
                 sg.host > ((size_t)4 << 20));
    NSS_CUDA_TRY(c, cudaMemcpyAsync(c.sb_arena, c.sb_stage, sg.host, cudaMemcpyHostToDevice, c.stream));
    for (const auto &it : sg.items) {
        *it.dst = (void *)(c.sb_arena + it.off);
        c.sb.h2d_bytes += (int64_t)it.bytes;
    }
    for (const auto &it : sg.dev) *it.dst = (void *)(c.sb_arena + sg.host + it.off);
    return NSS_OK;
}

// shape and row pointers always; the column of every entry unless the
// caller built the matrices itself (cols_known)
bool csr_ok(const nss_csr &m, int nrow, int ncol, bool cols_known = false) {
    if (m.nrow != nrow || m.ncol != ncol) return false;
    if (nrow == 0) return true;
    if (!m.rowptr || m.rowptr[0] != 0) return false;
    int nnz = m.rowptr[nrow];
    if (nnz < 0 || (nnz > 0 && (!m.colidx || !m.vals))) return false;
    for (int i = 0; i < nrow; ++i)
        if (m.rowptr[i + 1] < m.rowptr[i]) return false;
    if (cols_known) return true;
    for (int j = 0; j < nnz; ++j)
        if (m.colidx[j] < 0 || m.colidx[j] >= ncol) return false;
    return true;
}

// every stored value finite (a NaN or Inf operator entry would poison every
// H*psi and the Lanczos scalars without any other sign)
bool csr_finite(const nss_csr &m) {
    const int nnz = m.nrow > 0 ? m.rowptr[m.nrow] : 0;
    for (int j = 0; j < nnz; ++j)
        if (!std::isfinite(m.vals[j])) return false;
    return true;
}

}  // namespace

// Validate and copy the operator pool.  Errors mirror the reference's stop
// conditions (wrong sizes, vecDim != m_sb) as NSS_ERR_INVALID.
int sb_upload(Ctx &c, const nss_sb_desc *d, bool trusted, bool allow_split) {
    if (!d || d->nsb <= 0 || d->tnso < 0 || !d->dls || !d->drs || !d->offset || !d->hleft ||
        !d->hright) {
        c.err = "nss_sb_upload: incomplete descriptor";
        return NSS_ERR_INVALID;
    }
    // kernels of the previous pool may still be reading the arena (a
    // batch runs several contexts' solves on one stream)
    NSS_CUDA_TRY(c, cudaDeviceSynchronize());
    sb_release(c, false);
    DevSb &s = c.sb;
    s.nsb = d->nsb;
    s.tnso = d->tnso;
    s.m_left = d->m_left;
    s.m_right = d->m_right;
    s.dls.assign(d->dls, d->dls + s.nsb);
    s.drs.assign(d->drs, d->drs + s.nsb);
    s.off.assign(d->offset, d->offset + s.nsb);
    int64_t pos = 0;
    std::map<int64_t, int> sec_at;
    for (int k = 0; k < s.nsb; ++k) {
        if (s.dls[k] <= 0 || s.drs[k] <= 0 || s.off[k] != pos) {
            c.err = "nss_sb_upload: sector dims/offsets inconsistent at sector " + std::to_string(k);
            return NSS_ERR_INVALID;
        }
        sec_at[pos] = k;
        pos += (int64_t)s.dls[k] * s.drs[k];
    }
    s.n = pos;
    // sector block maps (for the RDM)
    if (d->ai && d->bi) {
        int la = 0, lb = 0;
        for (int k = 0; k < s.nsb; ++k) {
            s.ai_off.push_back(la);
            s.bi_off.push_back(lb);
            la += s.dls[k];
            lb += s.drs[k];
        }
        s.ai_off.push_back(la);
        s.bi_off.push_back(lb);
        s.ai.assign(d->ai, d->ai + la);
        s.bi.assign(d->bi, d->bi + lb);
        for (int x : s.ai)
            if (x < 0 || x >= d->m_left) { c.err = "nss_sb_upload: ai out of range"; return NSS_ERR_INVALID; }
        for (int x : s.bi)
            if (x < 0 || x >= d->m_right) { c.err = "nss_sb_upload: bi out of range"; return NSS_ERR_INVALID; }
    }

    // dense sector operators: their CSR rows travel and the device scatters
    // them into zeroed row-major blocks (k_densify), FP32 copies after
    int64_t hl_tot = 0, hr_tot = 0, nnz_l = 0, nnz_r = 0, nrow_l = 0, nrow_r = 0;
    for (int k = 0; k < s.nsb; ++k) {
        const int dl = s.dls[k], dr = s.drs[k];
        if (!csr_ok(d->hleft[k], dl, dl, trusted) || !csr_ok(d->hright[k], dr, dr, trusted)) {
            c.err = "nss_sb_upload: Hleft/Hright shape or index error at sector " + std::to_string(k);
            return NSS_ERR_INVALID;
        }
        if (!trusted && (!csr_finite(d->hleft[k]) || !csr_finite(d->hright[k]))) {
            c.err = "nss_sb_upload: non-finite value in Hleft/Hright at sector " + std::to_string(k);
            return NSS_ERR_INVALID;
        }
        s.hl_off.push_back(hl_tot);
        s.hr_off.push_back(hr_tot);
        hl_tot += (int64_t)dl * dl;
        hr_tot += (int64_t)dr * dr;
        nnz_l += d->hleft[k].rowptr[dl];
        nnz_r += d->hright[k].rowptr[dr];
        nrow_l += dl;
        nrow_r += dr;
        s.flops_dense += 2.0 * dl * dr * ((double)dl + dr);
    }
    s.hl_off.push_back(hl_tot);
    s.hr_off.push_back(hr_tot);
    if (nnz_l > INT32_MAX || nnz_r > INT32_MAX) {
        c.err = "nss_sb_upload: more than 2^31 entries in the sector operators";
        return NSS_ERR_INVALID;
    }
    struct PackedRows {
        std::vector<int> rowptr, row_sec;
        std::vector<int64_t> row_first;
    } pk[2];
    for (int side = 0; side < 2; ++side) {
        PackedRows &P = pk[side];
        P.rowptr.reserve((size_t)(side ? nrow_r : nrow_l) + 1);
        P.rowptr.push_back(0);
        P.row_first.reserve(s.nsb);
        P.row_sec.reserve((size_t)(side ? nrow_r : nrow_l));
        int64_t rows = 0;
        for (int k = 0; k < s.nsb; ++k) {
            const nss_csr &M = side ? d->hright[k] : d->hleft[k];
            const int base = P.rowptr.back();
            P.row_first.push_back(rows);
            for (int i = 0; i < M.nrow; ++i) {
                P.rowptr.push_back(base + M.rowptr[i + 1]);
                P.row_sec.push_back(k);
            }
            rows += M.nrow;
        }
    }

    // A x B terms, regrouped by output sector
    std::vector<std::vector<DevTerm>> by_out(s.nsb);
    std::vector<int> rowptr;
    std::vector<int> col;
    std::vector<double> val;
    auto push_csr = [&](const nss_csr &m) {
        int64_t at = (int64_t)rowptr.size();
        int base = (int)col.size();
        for (int i = 0; i <= m.nrow; ++i) rowptr.push_back(base + m.rowptr[i]);
        int nnz = m.rowptr[m.nrow];
        col.insert(col.end(), m.colidx, m.colidx + nnz);
        val.insert(val.end(), m.vals, m.vals + nnz);
        return at;
    };
    const int nt = s.tnso * s.nsb;
    for (int idx = 0; idx < nt; ++idx) {
        const nss_csr &A = d->a[idx], &B = d->b[idx];
        if (A.nrow == 0 || B.nrow == 0) continue;   // status=.false. -> skipped (:810)
        auto ro = sec_at.find(d->row_offset[idx]);
        auto co = sec_at.find(d->col_offset[idx]);
        if (ro == sec_at.end() || co == sec_at.end()) {
            c.err = "nss_sb_upload: Row/ColOffset not at a sector start (term " + std::to_string(idx) + ")";
            return NSS_ERR_INVALID;
        }
        int o = ro->second, q = co->second;
        if (!csr_ok(A, s.dls[o], s.dls[q], trusted) || !csr_ok(B, s.drs[o], s.drs[q], trusted)) {
            c.err = "nss_sb_upload: A/B shape or index error (term " + std::to_string(idx) + ")";
            return NSS_ERR_INVALID;
        }
        if (!trusted && (!csr_finite(A) || !csr_finite(B))) {
            c.err = "nss_sb_upload: non-finite value in A/B (term " + std::to_string(idx) + ")";
            return NSS_ERR_INVALID;
        }
        DevTerm t;
        t.out_sec = o;
        t.in_sec = q;
        t.a_nrow = A.nrow; t.a_ncol = A.ncol;
        t.b_nrow = B.nrow; t.b_ncol = B.ncol;
        t.a_rp = push_csr(A);
        t.b_rp = push_csr(B);
        by_out[o].push_back(t);
        // the reference's loop count, src/DMRG_SUPERBLOCK_SETUP.f90:819-853
        s.flops_ab += 2.0 * ((double)B.rowptr[B.nrow] * A.ncol + (double)A.rowptr[A.nrow] * B.nrow);
    }
    s.term_ptr.push_back(0);
    for (int k = 0; k < s.nsb; ++k) {
        for (auto &t : by_out[k]) s.terms.push_back(t);
        s.term_ptr.push_back((int)s.terms.size());
    }
    // tiles (k_noalloc.cu)
    std::vector<int4> tiles;
    for (int k = 0; k < s.nsb; ++k)
        for (int r = 0; r < s.dls[k]; r += TILE)
            for (int cc = 0; cc < s.drs[k]; cc += TILE) tiles.push_back(make_int4(k, r, cc, 0));
    s.ntiles = (int)tiles.size();
    // k_hv_fp64's terms, with the first entry of every row, and its tiles,
    // longest first
    const bool split = allow_split && split_wanted(s);
    std::vector<HvTerm> hv_terms;
    std::vector<HvRec> hv_recs;
    std::vector<int> ell_col;
    std::vector<double> ell_val;
    for (const DevTerm &t : s.terms) {
        HvTerm h{s.off[t.in_sec], s.drs[t.in_sec], 0, 0, t.a_rp, t.b_rp, 0, 1};
        for (int side = 0; side < 2; ++side) {
            const int64_t rp = side == 0 ? t.a_rp : t.b_rp;
            const int nrow = side == 0 ? t.a_nrow : t.b_nrow;
            (side == 0 ? h.a : h.b) = (int)ell_col.size();
            for (int i = 0; i < nrow; ++i) {
                const int p0 = rowptr[rp + i], p1 = rowptr[rp + i + 1];
                ell_col.push_back(p1 > p0 ? col[p0] : -1);
                ell_val.push_back(p1 > p0 ? val[p0] : 0.0);
                if (p1 - p0 > 1) h.kind = std::max(h.kind, side == 0 ? 1 : 2);
                if (side == 1 && p1 > p0 && std::fabs(val[p0]) != 1.0) h.unit_b = 0;
            }
        }
        hv_terms.push_back(h);
    }
    std::vector<int> hv_csr(s.nsb, 0);
    for (int k = 0; k < s.nsb; ++k)
        for (int t = s.term_ptr[k]; t < s.term_ptr[k + 1]; ++t) hv_csr[k] |= hv_terms[t].kind > 0;
    if (!split) {
        for (int k = 0; k < s.nsb; ++k) {
            // FMAs per output: the two K loops and, per term, a row of A
            int cost = s.dls[k] + s.drs[k];
            for (int t = s.term_ptr[k]; t < s.term_ptr[k + 1]; ++t) {
                const DevTerm &tm = s.terms[t];
                cost += (rowptr[tm.a_rp + tm.a_nrow] - rowptr[tm.a_rp]) / std::max(tm.a_nrow, 1);
            }
            for (int r = 0; r < s.dls[k]; r += HV_TR)
                for (int cc = 0; cc < s.drs[k]; cc += HV_TC)
                    hv_recs.push_back(HvRec{s.dls[k], s.drs[k], r, cc, s.term_ptr[k], s.term_ptr[k + 1], hv_csr[k], cost, s.off[k],
                                            s.hl_off[k], s.hr_off[k]});
        }
        std::stable_sort(hv_recs.begin(), hv_recs.end(),
                         [](const HvRec &x, const HvRec &y) { return x.cost > y.cost; });
    }
    s.nhv = (int)hv_recs.size();

    // FP32 copies for the mixed path, and its 32x32 tiles.  The FP32 A/B
    // pool drops entries below 1e-12 of the largest entry of their matrix:
    // the renormalised sign operator P carries rounding-level off-diagonal
    // entries (up to 33 per row at m=256) whose contribution (~1e-17 of the
    // result) is far below FP32 rounding, while each of them costs a gather.
    // The FP64 pool keeps every entry, as the reference does.
    std::vector<int> rowptr32, col32;
    std::vector<float> val32;
    std::vector<DevTerm> terms32 = s.terms;
    for (DevTerm &t : terms32) {
        for (int which = 0; which < 2; ++which) {
            const int64_t rp = which == 0 ? t.a_rp : t.b_rp;
            const int nrow = which == 0 ? t.a_nrow : t.b_nrow;
            double mx = 0.0;
            for (int jj = rowptr[rp]; jj < rowptr[rp + nrow]; ++jj) mx = std::max(mx, std::fabs(val[jj]));
            const int64_t at = (int64_t)rowptr32.size();
            rowptr32.push_back((int)col32.size());
            for (int i = 0; i < nrow; ++i) {
                for (int jj = rowptr[rp + i]; jj < rowptr[rp + i + 1]; ++jj)
                    if (std::fabs(val[jj]) > 1e-12 * mx) {
                        col32.push_back(col[jj]);
                        val32.push_back((float)val[jj]);
                    }
                rowptr32.push_back((int)col32.size());
            }
            if (which == 0) t.a_rp = at;
            else t.b_rp = at;
        }
    }
    // Sectors on the tensor-core GEMM (k_sector_mma.cu) get their A x B
    // terms from "terms only" CUDA-core tiles (w = 1), listed first, which
    // k_hv_fp32 runs beside the GEMM; its output planes are added afterwards.
    MmaPlan plan;
    int tc_thr = c.tc_min_dl, tc_bn = c.mma_bn;
    c.tune_cand = -1;
    if (c.tc_auto) tune_choose(c, s, &tc_thr, &tc_bn);
    int nsm = 0;
    NSS_CUDA_TRY(c, cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, c.device));
    mma_layout(s, tc_thr, tc_bn, c.mma_split, nsm, plan);
    s.hv_nsm = nsm;
    s.hv_grid = s.nhv <= 2 * HV_WARPS * nsm ? (s.nhv + HV_WARPS - 1) / HV_WARPS
                                            : nsm * std::min(HV_CTAS, (s.nhv + HV_WARPS * nsm - 1) / (HV_WARPS * nsm));
    if (split) s.hv_grid = nsm * HV_CTAS;
    std::vector<char> on_tc(s.nsb, 0);
    for (int k : plan.sectors) on_tc[k] = 1;
    std::vector<int4> tiles32;
    for (int k = 0; k < s.nsb; ++k)
        if (on_tc[k])
            for (int r = 0; r < s.dls[k]; r += TILE32)
                for (int cc = 0; cc < s.drs[k]; cc += TILE32) tiles32.push_back(make_int4(k, r, cc, 1));
    for (int k = 0; k < s.nsb; ++k)
        if (!on_tc[k])
            for (int r = 0; r < s.dls[k]; r += TILE32)
                for (int cc = 0; cc < s.drs[k]; cc += TILE32) tiles32.push_back(make_int4(k, r, cc, 0));
    // work items of the persistent kernel: 32x32 tiles of every sector,
    // split into H_L, H_R and A x B parts when a K loop is long
    std::vector<int4> items32;
    for (int k = 0; k < s.nsb; ++k) {
        const bool split = std::max(s.dls[k], s.drs[k]) > HV_SPLIT;
        for (int r = 0; r < s.dls[k]; r += TILE32)
            for (int cc = 0; cc < s.drs[k]; cc += TILE32) {
                if (split) {
                    items32.push_back(make_int4(k, r, cc, HV_LEFT));
                    items32.push_back(make_int4(k, r, cc, HV_RIGHT));
                    items32.push_back(make_int4(k, r, cc, HV_TERMS));   // without terms: zeros, the slot is read
                } else {
                    items32.push_back(make_int4(k, r, cc, HV_FULL));
                }
            }
    }
    // longest first, so the split halves start at once
    std::stable_sort(items32.begin(), items32.end(), [&](const int4 &x, const int4 &y) {
        auto cost = [&](const int4 &t) {
            const int dl = s.dls[t.x], dr = s.drs[t.x];
            return t.w == HV_LEFT ? dl : (t.w == HV_RIGHT ? dr : (t.w == HV_TERMS ? 48 : dl + dr + 48));
        };
        return cost(x) > cost(y);
    });
    // A x B tables of the items that carry terms: for each term of the
    // sector, the (column, value) of the tile's 32 rows of A and 32 columns
    // of B in the FP32 pool (-1: empty row); items with a row of several
    // elements keep -1 and use the CSR loop
    std::vector<int> item_ell(items32.size(), -1);
    std::vector<int2> ell;
    for (size_t ii = 0; ii < items32.size(); ++ii) {
        const int4 it = items32[ii];
        if (it.w != HV_FULL && it.w != HV_TERMS) continue;
        const int k = it.x, dl = s.dls[k], dr = s.drs[k];
        const size_t base = ell.size();
        bool ok = true;
        for (int ti = s.term_ptr[k]; ti < s.term_ptr[k + 1] && ok; ++ti) {
            const DevTerm &tm = terms32[ti];
            for (int side = 0; side < 2 && ok; ++side) {
                const int64_t rp = side == 0 ? tm.a_rp : tm.b_rp;
                const int lim = side == 0 ? dl : dr, first = side == 0 ? it.y : it.z;
                for (int r = 0; r < 32; ++r) {
                    const int g = first + r;
                    int2 e = make_int2(-1, 0);
                    if (g < lim) {
                        const int p0 = rowptr32[rp + g], p1 = rowptr32[rp + g + 1];
                        if (p1 - p0 > 1) { ok = false; break; }
                        if (p1 > p0) {
                            float fv = val32[p0];
                            int bits;
                            std::memcpy(&bits, &fv, sizeof(bits));
                            e = make_int2(col32[p0], bits);
                        }
                    }
                    ell.push_back(e);
                }
            }
        }
        if (ok) item_ell[ii] = (int)base;
        else ell.resize(base);
    }
    if (ell.empty()) ell.push_back(make_int2(-1, 0));
    std::vector<int4> term_hdr(std::max<size_t>(terms32.size(), 1), make_int4(0, 0, 0, 0));
    for (size_t ti = 0; ti < terms32.size(); ++ti) {
        const int64_t of = s.off[terms32[ti].in_sec];
        term_hdr[ti] = make_int4((int)(uint32_t)(of & 0xffffffff), (int)(of >> 32), s.drs[terms32[ti].in_sec], 0);
    }
    std::vector<ItemRec> recs(items32.size());
    for (size_t ii = 0; ii < items32.size(); ++ii) {
        const int4 it = items32[ii];
        const int k = it.x;
        const int64_t of = s.off[k], hlo = s.hl_off[k], hro = s.hr_off[k];
        auto lo = [](int64_t x) { return (int)(uint32_t)(x & 0xffffffff); };
        auto hi = [](int64_t x) { return (int)(x >> 32); };
        recs[ii].a = it;
        recs[ii].b = make_int4(s.dls[k], s.drs[k], s.term_ptr[k], s.term_ptr[k + 1]);
        recs[ii].c = make_int4(lo(of), hi(of), item_ell[ii], 0);
        recs[ii].d = make_int4(lo(hlo), hi(hlo), lo(hro), hi(hro));
    }
    s.nitems32 = (int)items32.size();
    s.item_cost.resize(items32.size());
    for (size_t ii = 0; ii < items32.size(); ++ii) {
        const int4 t = items32[ii];
        const int dl = s.dls[t.x], dr = s.drs[t.x];
        s.item_cost[ii] = t.w == HV_LEFT ? dl : (t.w == HV_RIGHT ? dr : (t.w == HV_TERMS ? 48 : dl + dr + 48));
    }
    s.ntiles32 = (int)tiles32.size();
    std::vector<int> tc_err(1, 0);
    SplitPlan sp;
    if (split) split_layout(s, rowptr, col, val, hv_csr, nsm, sp);

    Stager sg;
    sg.add_dev(&s.d_hl32, (size_t)hl_tot);
    sg.add_dev(&s.d_hr32, (size_t)hr_tot);
    sg.add(&s.d_ab_val32, val32);
    sg.add(&s.d_ab_rowptr32, rowptr32);
    sg.add(&s.d_ab_col32, col32);
    sg.add(&s.d_terms32, terms32);
    sg.add(&s.d_tiles32, tiles32);
    sg.add(&s.d_items32, recs);
    sg.add(&s.d_item_ell, item_ell);
    sg.add(&s.d_ell, ell);
    sg.add(&s.d_term_hdr, term_hdr);
    sg.add(&s.d_tc_err, tc_err);
    sg.add_dev(&s.d_mma_pool, (size_t)(plan.items.empty() ? 0 : plan.plane_rows * MM_KC));
    sg.add_dev(&s.d_mma_out, (size_t)(plan.items.empty() ? 0 : plan.nplanes * s.n));
    sg.add(&s.d_mma_items, plan.items);
    sg.add(&s.d_mma_rng, plan.rng);
    sg.add(&s.d_mma_wt, plan.wt);
    sg.add(&s.d_mma_sec, plan.ps);
    sg.add(&s.d_dls, s.dls);
    sg.add(&s.d_drs, s.drs);
    sg.add(&s.d_off, s.off);
    sg.add(&s.d_hl_off, s.hl_off);
    sg.add(&s.d_hr_off, s.hr_off);
    sg.add_dev(&s.d_hl, (size_t)hl_tot);
    sg.add_dev(&s.d_hr, (size_t)hr_tot);
    DenseRows dr_dev[2];
    for (int side = 0; side < 2; ++side) {
        sg.add((int **)&dr_dev[side].rowptr, pk[side].rowptr);
        const size_t it = sg.items.size();
        sg.add_gather((int **)&dr_dev[side].col, (size_t)(side ? nnz_r : nnz_l));
        sg.add_gather((double **)&dr_dev[side].val, (size_t)(side ? nnz_r : nnz_l));
        size_t at = 0;
        for (int k = 0; k < s.nsb; ++k) {
            const nss_csr &M = side ? d->hright[k] : d->hleft[k];
            const size_t nz = (size_t)M.rowptr[M.nrow];
            sg.part(it, M.colidx, nz, at);
            sg.part(it + 1, M.vals, nz, at);
            at += nz;
        }
        sg.add((int **)&dr_dev[side].row_sec, pk[side].row_sec);
        sg.add((int64_t **)&dr_dev[side].row_first, pk[side].row_first);
    }
    sg.add(&s.d_term_ptr, s.term_ptr);
    sg.add(&s.d_terms, s.terms);
    sg.add(&s.d_ab_rowptr, rowptr);
    sg.add(&s.d_ab_col, col);
    sg.add(&s.d_ab_val, val);
    sg.add(&s.d_tiles, tiles);
    sg.add(&s.d_sp_items, sp.items);
    sg.add(&s.d_sp_rng, sp.rng);
    sg.add(&s.d_sp_sitems, sp.sitems);
    sg.add(&s.d_sp_srng, sp.srng);
    sg.add(&s.d_sp_jobs_w, sp.jobs_w);
    sg.add(&s.d_sp_jobs_hl, sp.jobs_hl);
    sg.add(&s.d_sp_jobs_hr, sp.jobs_hr);
    sg.add(&s.d_sp_terms, sp.terms);
    sg.add(&s.d_sp_tcol, sp.tcol);
    sg.add(&s.d_sp_tval, sp.tval);
    sg.add(&s.d_sp_dptr, sp.dptr);
    sg.add(&s.d_sp_dcol, sp.dcol);
    sg.add(&s.d_sp_dval, sp.dval);
    sg.add(&s.d_sp_tiles, sp.tiles);
    sg.add(&s.d_hv_recs, hv_recs);
    sg.add(&s.d_hv_terms, hv_terms);
    sg.add(&s.d_ell_col, ell_col);
    sg.add(&s.d_ell_val, ell_val);
    int rc;
    // a superblock that fits without the tensor-core product's tables is taken without
    if ((rc = stage_commit(c, sg))) return split && rc == NSS_ERR_NOMEM ? sb_upload(c, d, trusted, false) : rc;
    NSS_CUDA_TRY(c, cudaMemsetAsync(s.d_hl, 0, (size_t)hl_tot * sizeof(double), c.stream));
    NSS_CUDA_TRY(c, cudaMemsetAsync(s.d_hr, 0, (size_t)hr_tot * sizeof(double), c.stream));
    {
        const int64_t nr = nrow_l + nrow_r;
        c.launches += 3;
        k_densify<<<(unsigned)((nr + 7) / 8), 256, 0, c.stream>>>(dr_dev[0], dr_dev[1], (int)nrow_l, (int)nrow_r,
                                                                      s.d_dls, s.d_drs, s.d_hl_off, s.d_hr_off,
                                                                      s.d_hl, s.d_hr);
        k_dense32<<<608, 256, 0, c.stream>>>(s.d_hl, s.d_hl32, hl_tot);
        k_dense32<<<608, 256, 0, c.stream>>>(s.d_hr, s.d_hr32, hr_tot);
        NSS_CUDA_TRY(c, cudaGetLastError());
    }
    if ((rc = mma_finish(c, plan))) return rc;
    if ((rc = split_finish(c, sp))) return rc;
    NSS_CUDA_TRY(c, cudaStreamSynchronize(c.stream));
    s.gen = next_gen();
    s.valid = true;
    return NSS_OK;
}

// A warp per 4 x 8 output tile, a thread an output.
// The FP64 pipe takes a warp's FMA every 64 cycles (1.0-1.2 TFLOP/s over the
// GPU) and bounds the kernel: the K loops stop at the sector's edge, and the
// next 32 columns of K are loaded into registers while the current ones are
// multiplied.  What is left is balance: every quarter of an SM has a pipe of its
// own.  Up to two tiles for each (2 * 4 * 152) the CTAs get four each; above,
// every SM the same number of CTAs (at most five), and what is above one tile a
// warp is dealt backwards through the order, longest first.  The launch leaves
// nothing behind, so products replayed from graphs do not meet; a queue of
// tiles in memory took as long (one launch after another on one stream: 73.6
// us against 72.5 dealt at 90 554 states, Hubbard m = 297; 80.1 against 78.3 at
// 99 902).  At most 3 / 4 / 5 / 6 CTAs an SM: 85.2 / 76.0 / 72.9 / 101.4 us at
// 90 554 states (the sixth is not resident), no difference at 57 902.
// Tiles of 8 x 16 on four warps, one CTA each, left SMs with five CTAs beside
// others with four, and waited for each other at barriers.
// A x B terms: Out[ai][bi] += A[ai][aj] B[bi][bj] W_q[aj][bj] (:808-857).  Where
// all rows hold one entry, four terms' loads are in flight; where rows of A hold
// more (the renormalised sign operator leaves rounding-level entries in its
// whole block, 40 a row), a row's eight lanes hold two entries each, eight
// gathers in flight, instead of every thread walking the row by itself; a
// factor of +-1 is a sign flip and no FP64 multiplication.  (Gathers a round
// ahead of the FMAs need 126 registers and were slower: 57.7 against 51.5 us.)
// Bit for bit the results of 16 x 16 tiles on eight warps, in us, one launch
// after another on one stream: Hubbard 66 600 states 88 -> 60 (8 x 16) -> 51.3,
// spin-1/2 39 200 states 28.0 (8 x 16) -> 22.6, spin-1 61 200 states 37.3 -> 34.6.
__device__ __forceinline__ double hv_times(double b, double x, bool unit) {
    if (!unit) return b * x;
    return __hiloint2double(__double2hiint(x) ^ (__double2hiint(b) & 0x80000000), __double2loint(x));
}

struct HvOps {
    const double *hl, *hr;
    const HvTerm *terms;
    const int *ell_col;
    const double *ell_val;
    const int *ab_rp, *ab_col;
    const double *ab_val;
};

// What k_hv_fp64 computes of a product on the tensor cores: every tile when
// that gave up or did not run (words null), else those on its list, of which the
// sides that are good come from the planes of digit sums.  A tile is an eighth
// of a SplitTile.  A listed tile's K loops and terms are shared out over the
// four warps of a CTA, one on each quarter of its SM: there are few of them as a
// rule, and a warp by itself takes 16 us for 500 products a side.
struct HvRedo {
    const SplitTile *tiles;
    const int *words;            // sb.d_sp_redo
    const int64_t *planes;
    const int *planes0, *exps;
    int64_t n;
};

template <bool REDO>
__global__ void __launch_bounds__(32 * HV_WARPS) k_hv_fp64(const double *__restrict__ v, double *__restrict__ hv,
                                                           const HvRec *__restrict__ recs, HvRedo redo, HvOps op,
                                                           int ntiles, int nsm, const int *stop) {
    if (stop && *stop) return;   // the Lanczos loop has already finished (the same for every CTA)
    bool listed = false;
    if constexpr (REDO) {
        listed = redo.words && !redo.words[SP_REDO_ERR];
        if (listed) ntiles = redo.words[SP_REDO_COUNT];
    }
    constexpr int KC = 32;
    __shared__ double sa_[HV_WARPS][HV_TR][KC + 1];
    __shared__ double sb_[HV_WARPS][KC][HV_TC + 1];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, grid = gridDim.x;
    double(*sa)[KC + 1] = sa_[warp];
    double(*sb)[HV_TC + 1] = sb_[warp];
    const int ty = lane / HV_TC, tx = lane % HV_TC;
    // longest tiles first, a CTA's four a grid apart in the order; the warp that
    // may be left without one is another in each CTA of an SM.  What is above
    // one tile a warp is dealt backwards, so that the warps with the longest
    // first tile get the shortest second one.
    const int all = REDO && listed ? grid : HV_WARPS * grid;
    const int mine = REDO && listed ? blockIdx.x : (int)((warp + blockIdx.x / nsm) % HV_WARPS) * grid + blockIdx.x;
    for (int r = 0; r * all < ntiles; ++r) {
        const int tile = r * all + (r & 1 ? all - 1 - mine : mine);
        if (tile >= ntiles) continue;
        HvRec t;
        SplitTile s;
        int sides = 3;
        if constexpr (REDO) {
            const int word = listed ? redo.words[SP_REDO_LIST + tile] : 4 * tile + 3, id = word >> 2, sub = id % HV_SUB;
            sides = word & 3;
            s = redo.tiles[id / HV_SUB];
            t = HvRec{s.dl, s.dr, s.row0 + HV_TR * (sub / (32 / HV_TC)), s.col0 + HV_TC * (sub % (32 / HV_TC)), s.t0, s.t1, s.csr,
                      0, s.off, s.hlo, s.hro};
            if (t.row0 >= t.dl || t.col0 >= t.dr) continue;   // (not of the list)
            if (listed) {
                const int t0 = t.t0, nt = t.t1 - t0;
                t.t0 = t0 + nt * warp / HV_WARPS;
                t.t1 = t0 + nt * (warp + 1) / HV_WARPS;
            }
        } else {
            t = recs[tile];
        }
        const int dl = t.dl, dr = t.dr;
        const double *W = v + t.off, *HL = op.hl + t.hlo, *HR = op.hr + t.hro;
        const int il = t.row0 + ty, ir = t.col0 + tx;
        const int c0 = (dl + KC - 1) / KC, c1 = (dr + KC - 1) / KC;
        double ra[HV_TR], rb[HV_TC];
        // chunk c of the K loops: H_L W (sum_j HL[il][j] W[j][ir], :784-796), then
        // W H_R^T (sum_j W[il][j] HR[ir][j], :767-779)
        auto load = [&](int c) {
            const bool left = c < c0;
            const int j0 = (left ? c : c - c0) * KC, K = left ? dl : dr, gk = j0 + lane;
            const double *A = (left ? HL : W) + (int64_t)t.row0 * K + gk;
#pragma unroll
            for (int q = 0; q < HV_TR; ++q) ra[q] = t.row0 + q < dl && gk < K ? A[(int64_t)q * K] : 0.0;
            if (left) {
                const int gj = j0 + ty;
                const double *B = W + (int64_t)gj * dr + ir;
#pragma unroll
                for (int q = 0; q < HV_TC; ++q)
                    rb[q] = gj + HV_TR * q < dl && ir < dr ? B[(int64_t)(HV_TR * q) * dr] : 0.0;
            } else {
                const double *B = HR + (int64_t)t.col0 * dr + gk;
#pragma unroll
                for (int q = 0; q < HV_TC; ++q) rb[q] = t.col0 + q < dr && gk < dr ? B[(int64_t)q * dr] : 0.0;
            }
        };
        double acc = 0.0, part = 0.0;                // part (redo): a side's sum, the sides are added
        int first = REDO && !(sides & 1) ? c0 : 0, last = REDO && !(sides & 2) ? c0 : c0 + c1;
        if (REDO && listed) {
            const int c = first, nc = last - first;
            first = c + nc * warp / HV_WARPS;
            last = c + nc * (warp + 1) / HV_WARPS;
        }
        if (!REDO || first < last) load(first);
        for (int c = first; c < last; ++c) {
            const bool left = c < c0;
            if constexpr (REDO)
                if (c == c0) {
                    part = acc;
                    acc = 0.0;
                }
            const int kn = min(KC, left ? dl - c * KC : dr - (c - c0) * KC);
#pragma unroll
            for (int q = 0; q < HV_TR; ++q) sa[q][lane] = ra[q];
#pragma unroll
            for (int q = 0; q < HV_TC; ++q) {
                if (left) sb[ty + HV_TR * q][tx] = rb[q];
                else sb[lane][q] = rb[q];
            }
            __syncwarp();
            if (c + 1 < last) load(c + 1);
#pragma unroll 8
            for (int j = 0; j < kn; ++j) acc = fma(sa[ty][j], sb[j][tx], acc);
            __syncwarp();
        }
        const bool in = il < dl && ir < dr;
        if constexpr (REDO) {
            part += acc;
            acc = 0.0;
            if (in && warp == 0)                     // (sides = 3 where every warp has a tile)
                for (int side = 0; side < 2; ++side)
                    if (!(sides >> side & 1)) {      // left: H_L row, W column; right: W row, H_R row
                        const int64_t e = t.off + (int64_t)ir * dl + il + side * redo.n;
                        const int x0 = s.exp + (side ? dl + dr + il : il), x1 = s.exp + (side ? dl + ir : 2 * dl + dr + ir);
                        part += fixed_to_double(redo.planes0[e], redo.planes[e], redo.exps[x0] + redo.exps[x1] - 56);
                    }
        }
        if (!t.csr) {
            for (int tb = t.t0; tb < t.t1; tb += 4) {
                int aj[4], bj[4];
                double f[4], w[4];
                HvTerm tm[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) tm[q] = op.terms[min(tb + q, t.t1 - 1)];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const bool on = in && tb + q < t.t1;
                    aj[q] = on ? op.ell_col[tm[q].a + il] : -1;
                    bj[q] = on ? op.ell_col[tm[q].b + ir] : -1;
                    f[q] = on ? hv_times(op.ell_val[tm[q].b + ir], op.ell_val[tm[q].a + il], tm[q].unit_b) : 0.0;
                }
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    w[q] = aj[q] >= 0 && bj[q] >= 0 ? v[tm[q].off + (int64_t)aj[q] * tm[q].drq + bj[q]] : 0.0;
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    if (aj[q] >= 0 && bj[q] >= 0) acc = fma(f[q], w[q], acc);
            }
        } else {
            for (int ti = t.t0; ti < t.t1; ++ti) {
                const HvTerm tm = op.terms[ti];
                const double *Wq = v + tm.off;
                if (tm.kind == 2) {                  // rows of B with several entries
                    if (in)
                        for (int ja = op.ab_rp[tm.a_rp + il]; ja < op.ab_rp[tm.a_rp + il + 1]; ++ja) {
                            const int64_t row = (int64_t)op.ab_col[ja] * tm.drq;
                            double cb = 0.0;
                            for (int jb = op.ab_rp[tm.b_rp + ir]; jb < op.ab_rp[tm.b_rp + ir + 1]; ++jb)
                                cb = fma(op.ab_val[jb], Wq[row + op.ab_col[jb]], cb);
                            acc = fma(op.ab_val[ja], cb, acc);
                        }
                    continue;
                }
                const int bj = in ? op.ell_col[tm.b + ir] : -1;
                const double bv = in ? op.ell_val[tm.b + ir] : 0.0;
                const int p0 = il < dl ? op.ab_rp[tm.a_rp + il] : 0;
                const int cnt = il < dl ? op.ab_rp[tm.a_rp + il + 1] - p0 : 0;
                int most = cnt;                      // of the tile's rows, HV_TC lanes each
#pragma unroll
                for (int o = HV_TC; o < 32; o <<= 1) most = max(most, __shfl_xor_sync(0xffffffffu, most, o));
                for (int base = 0; base < most; base += 2 * HV_TC) {
                    int ec[2];                       // entries base + tx, base + HV_TC + tx of the lane's row
                    double ev[2];
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const bool mine = base + h * HV_TC + tx < cnt;
                        ec[h] = mine ? op.ab_col[p0 + base + h * HV_TC + tx] : 0;
                        ev[h] = mine ? op.ab_val[p0 + base + h * HV_TC + tx] : 0.0;
                    }
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const int b0 = base + h * HV_TC;
                        if (b0 >= most) break;
                        double g[HV_TC];
#pragma unroll
                        for (int x = 0; x < HV_TC; ++x) {
                            const int c = __shfl_sync(0xffffffffu, ec[h], x, HV_TC);
                            g[x] = bj >= 0 && b0 + x < cnt ? Wq[(int64_t)c * tm.drq + bj] : 0.0;
                        }
#pragma unroll
                        for (int x = 0; x < HV_TC; ++x) {
                            const double a = __shfl_sync(0xffffffffu, ev[h], x, HV_TC);
                            if (bj >= 0 && b0 + x < cnt) acc = fma(a, hv_times(bv, g[x], tm.unit_b), acc);
                        }
                    }
                }
            }
        }
        if constexpr (REDO) {
            acc += part;
            if (listed) {
                __shared__ double shares[HV_WARPS][32];
                shares[warp][lane] = acc;
                __syncthreads();
                acc = (shares[0][lane] + shares[1][lane]) + (shares[2][lane] + shares[3][lane]);
                __syncthreads();
                if (warp) continue;
            }
        }
        if (in) hv[t.off + (int64_t)il * dr + ir] = acc;
    }
}

// FP32 variant for the mixed-precision Lanczos phase: 32x32 output tiles,
// each thread owns rows {ty, ty+16} x cols {tx, tx+16}; FP32 operands and
// accumulation (GB300 issues FP32 FMAs 64x faster than FP64 ones).
__global__ void __launch_bounds__(256) k_hv_fp32(const float *__restrict__ v, float *__restrict__ hv,
                                                 const int4 *__restrict__ tiles, Hv32Ops op, const int *stop) {
    if (stop && *stop) return;   // the Lanczos loop has already finished
    __shared__ Tile32Smem sm;
    hv32_tile(tiles[blockIdx.x], v, hv, op, sm, threadIdx.x, CtaSync{});
}

Hv32Ops hv32_ops(const DevSb &s) {
    Hv32Ops op;
    op.dls = s.d_dls;
    op.drs = s.d_drs;
    op.off = s.d_off;
    op.hl = s.d_hl32;
    op.hl_off = s.d_hl_off;
    op.hr = s.d_hr32;
    op.hr_off = s.d_hr_off;
    op.term_ptr = s.d_term_ptr;
    op.terms = s.d_terms32;
    op.ab_rp = s.d_ab_rowptr32;
    op.ab_col = s.d_ab_col32;
    op.ab_val = s.d_ab_val32;
    op.item_ell = s.d_item_ell;
    op.ell = s.d_ell;
    op.term_hdr = s.d_term_hdr;
    return op;
}

// hv[i] += the tensor-core planes' sum at i (plane 0 first; zero outside the
// tensor-core sectors)
__global__ void __launch_bounds__(256) k_add_planes(float *__restrict__ hv, const float *__restrict__ planes,
                                                    int64_t n, int np, const int *stop) {
    if (stop && *stop) return;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        float d = planes[i];
        for (int p = 1; p < np; ++p) d += planes[(int64_t)p * n + i];
        hv[i] += d;
    }
}

int hv_device_fp32(Ctx &c, const float *d_v, float *d_hv, const int *stop, bool add_planes) {
    DevSb &s = c.sb;
    if (!s.valid) {
        c.err = "nss_hv: no superblock uploaded";
        return NSS_ERR_STATE;
    }
    if (s.mma_nitems == 0) {
        if (s.ntiles32 > 0) {
            k_hv_fp32<<<s.ntiles32, 256, 0, c.stream>>>(d_v, d_hv, s.d_tiles32, hv32_ops(s), stop);
            c.launches += 1;
            NSS_CUDA_TRY(c, cudaGetLastError());
        }
        return NSS_OK;
    }
    // tensor-core sectors: the CUDA-core tiles (their A x B terms, and the
    // small sectors) run on a side stream beside the W packing and the GEMM;
    // the GEMM's planes are added when both are done
    if (!c.hv_side) {
        NSS_CUDA_TRY(c, cudaStreamCreateWithFlags(&c.hv_side, cudaStreamNonBlocking));
        NSS_CUDA_TRY(c, cudaEventCreateWithFlags(&c.hv_fork, cudaEventDisableTiming));
        NSS_CUDA_TRY(c, cudaEventCreateWithFlags(&c.hv_join, cudaEventDisableTiming));
    }
    NSS_CUDA_TRY(c, cudaEventRecord(c.hv_fork, c.stream));
    NSS_CUDA_TRY(c, cudaStreamWaitEvent(c.hv_side, c.hv_fork, 0));
    if (s.ntiles32 > 0) {
        k_hv_fp32<<<s.ntiles32, 256, 0, c.hv_side>>>(d_v, d_hv, s.d_tiles32, hv32_ops(s), stop);
        c.launches += 1;
    }
    NSS_CUDA_TRY(c, cudaEventRecord(c.hv_join, c.hv_side));
    if (int rc = hv_device_mma(c, d_v, stop)) return rc;
    NSS_CUDA_TRY(c, cudaStreamWaitEvent(c.stream, c.hv_join, 0));
    if (!add_planes) return NSS_OK;
    int nsm = 0;
    NSS_CUDA_TRY(c, cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, c.device));
    k_add_planes<<<(unsigned)std::min<int64_t>(4 * nsm, (s.n + 255) / 256), 256, 0, c.stream>>>(
        d_hv, s.d_mma_out, s.n, s.mma_nplanes, stop);
    c.launches += 1;
    NSS_CUDA_TRY(c, cudaGetLastError());
    return NSS_OK;
}

int hv_device(Ctx &c, const double *d_v, double *d_hv, const int *stop, bool standalone) {
    DevSb &s = c.sb;
    if (!s.valid) {
        c.err = "nss_hv: no superblock uploaded";
        return NSS_ERR_STATE;
    }
    const HvOps op{s.d_hl, s.d_hr, s.d_hv_terms, s.d_ell_col, s.d_ell_val, s.d_ab_rowptr, s.d_ab_col, s.d_ab_val};
    if (s.sp_ntiles) {
        bool tc = s.sp_nitems > 0;                   // else all of it here
        if (tc && standalone) {
            // a product that is being captured may be replayed beside others: it
            // keeps to its own vectors
            cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
            NSS_CUDA_TRY(c, cudaStreamIsCapturing(c.stream, &cap));
            tc = cap == cudaStreamCaptureStatusNone;
        }
        if (tc)
            if (int rc = hv_device_split(c, d_v, d_hv, stop, standalone)) return rc;
        if (tc && !standalone) return NSS_OK;
        k_hv_fp64<true><<<s.hv_grid, 32 * HV_WARPS, 0, c.stream>>>(
            d_v, d_hv, nullptr,
            HvRedo{s.d_sp_tiles, tc ? s.d_sp_redo : nullptr, s.d_sp_out, s.d_sp_out0, s.d_sp_exp, s.n}, op,
            s.sp_ntiles * HV_SUB, s.hv_nsm, stop);
    } else {
        k_hv_fp64<false><<<s.hv_grid, 32 * HV_WARPS, 0, c.stream>>>(d_v, d_hv, s.d_hv_recs, HvRedo{}, op, s.nhv, s.hv_nsm,
                                                                    stop);
    }
    c.launches += 1;
    NSS_CUDA_TRY(c, cudaGetLastError());
    return NSS_OK;
}

}  // namespace nss

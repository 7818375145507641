// FP64 sector product on the tensor cores (k_sector_split.cu): the records
// shared with the superblock upload (k_matvec.cu), and the host plan that sizes
// the upload arena's sections.
#pragma once

#include <cstdint>
#include <vector>

#include "device.cuh"

namespace nss {

constexpr int SP_M = 128;      // UMMA M: rows of il per work item
constexpr int SP_KC = 64;      // K columns per slab (128 bytes of bf16)
constexpr int SP_D = 7;        // digits of an operand element
constexpr int SP_KMAX = 4096;  // largest contracted dimension (the 64-bit sums)

// One work item: the product of one 128 x BN tile of one phase, H_L W (output
// plane 0) or W H_R^T (plane 1).  Row indices address the digit pool.
struct SplitItem {
    int a_row, b_row;            // slab 0, digit 0 of the A and B operands
    int a_rows, b_rows;          // their rows per digit slab (Dl, Dr)
    int k;                       // contracted dimension
    int dl, dr;                  // the sector
    int m0, n0;                  // output tile origin (il, ir)
    int plane;
    int64_t off;                 // sector offset in psi
};

// One packing job: SP_ROWS rows of an operand, from rows (kind 0) or columns
// (kind 1) of a row-major matrix.
constexpr int SP_ROWS = 16;
struct SplitJob {
    int64_t src;                 // first element of the matrix
    int ld, rows, k;             // row length; rows and contracted dimension of the operand
    int r0, kind;
    int row, exp;                // slab 0, digit 0 row in the pool; scale exponent of row 0
    int pad;
};

// One A x B term with its dominant entries and its rounding-level rest
struct SplitTerm {
    int general;                 // rows with several sizeable entries: CSR loop
    int a, b;                    // per row of A / of B: (column, value) at a + il, b + ir
    int dust;                    // dptr[dust + il] .. dptr[dust + il + 1]: small entries of A's row (-1: none)
    int term;                    // DevTerm of the CSR loop
    int drq, ew, pad;            // the input sector: Dr, scale exponents of its W rows,
    int64_t off;                 // offset in psi
};

// One 8 x 32 output tile of the last kernel, eight tiles of k_hv_fp64
struct SplitTile {
    int row0, col0, dl, dr, t0, t1;
    int exp;                     // the sector's scale exponents: H_L rows, H_R rows, W rows, W columns
    int csr;                     // HvRec::csr of the sector
    int64_t off, hlo, hro;
};

struct SplitPlan {
    std::vector<SplitItem> items;      // grouped by CTA
    std::vector<int2> rng;             // per CTA: its items [x, y)
    std::vector<SplitJob> jobs_w, jobs_hl, jobs_hr;
    int64_t pool_rows = 0;
    int nexp = 0, bn = 64, grid = 0, kmax = 0;
    // A x B terms
    std::vector<SplitTerm> terms;
    std::vector<int> tcol, dptr, dcol;
    std::vector<double> tval;
    std::vector<float> dval;
    std::vector<SplitTile> tiles;
};

// whether the superblock's FP64 products take this path: from 40 MFLOP of
// dense work.  Measured (us a product, CUDA cores against this): spin-1 N =
// 25 300 (9 MFLOP) 22.9 / 23.0, 100 200 (62) 74 / 29, 398 000 (480) 455 / 56,
// 1.18 million (2 430) 2 108 / 154.  Superblocks between 10 and 40 MFLOP would
// gain up to a factor of two; they stay on the CUDA cores, whose results whole
// runs at those sizes are pinned to in their last digits.  NSS_SPLIT64 = 0 / 1
// forces a path (comparisons, tests).
bool split_wanted(const DevSb &s);
// the plan from the superblock's tables and its CSR pool (rowptr, col, val)
// (csr: HvRec::csr per sector)
void split_layout(const DevSb &s, const std::vector<int> &rowptr, const std::vector<int> &col,
                  const std::vector<double> &val, const std::vector<int> &csr, int nsm, SplitPlan &p);
// digits of H_L and H_R and the tensor maps, after the dense blocks are built
int split_finish(Ctx &c, const SplitPlan &p);
// hv = H v on c.stream.  A wait that ran out is reported in *err; clear: the
// first kernel sets it to zero.
int hv_device_split(Ctx &c, const double *d_v, double *d_hv, const int *stop, int *err, bool clear);

}  // namespace nss

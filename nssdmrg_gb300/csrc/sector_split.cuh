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
constexpr int SP_SN = 256;     // largest tile width of the sums of |H||W|
constexpr int SP_KMAX = 4096;  // largest contracted dimension (the 64-bit sums)
constexpr int SP_BADEXP = 1 << 20;         // scale exponent of a row with an Inf or NaN
constexpr int SP_ZEROEXP = -(1 << 20);     // ... of a row of zeros

// (s0 2^42 + r) 2^e rounded to nearest even, in integer arithmetic; 0 below the normal range
__device__ __forceinline__ double fixed_to_double(int s0, int64_t r, int e) {
    uint64_t l = ((uint64_t)(int64_t)s0 << 42) + (uint64_t)r;
    int64_t h = (int64_t)(s0 >> 22) + (r >> 63) + (l < (uint64_t)r ? 1 : 0);
    const uint64_t sign = (uint64_t)h & 0x8000000000000000ull;
    if (sign) {
        l = 0 - l;
        h = ~h + (l == 0 ? 1 : 0);
    }
    if (((uint64_t)h | l) == 0) return 0.0;
    // normalised: the leading bit at bit 63 of u, the rest below it in l
    uint64_t u = (uint64_t)h;
    int lz;
    if (u) {
        lz = __clzll((long long)u);                  // at least 36: h has 28 bits
        u = (u << lz) | (l >> (64 - lz));
        l <<= lz;
    } else {
        const int z = __clzll((long long)l);
        u = l << z;
        l = 0;
        lz = 64 + z;
    }
    uint64_t m = u >> 11;
    const uint32_t low = (uint32_t)u & 0x7ffu;
    if (low > 0x400u || (low == 0x400u && (l || (m & 1)))) ++m;
    const int ex = 127 - lz + e + 1023;
    if (ex <= 0) return __longlong_as_double((long long)sign);          // below the normal range
    if (ex >= 2047) return __longlong_as_double((long long)(sign | 0x7ff0000000000000ull));
    return __longlong_as_double((long long)(sign | (((uint64_t)(ex - 1) << 52) + m)));
}

// One work item: the product of one 128 x BN tile of one phase, H_L W (output
// plane 0) or W H_R^T (plane 1), or of their absolute values (128 x sn).
// Row indices address the digit pool.
struct SplitItem {
    int a_row, b_row;            // slab 0 of the A and B operands (digit 0 or absolute values)
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
    int abs;                     // slab 0, row 0 of its absolute values in the pool
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
    std::vector<SplitItem> sitems;     // sums of |H||W|: 128 x sn tiles
    int sn = SP_SN;
    std::vector<int2> srng;
    int sgrid = 0;
    // A x B terms
    std::vector<SplitTerm> terms;
    std::vector<int> tcol, dptr, dcol;
    std::vector<double> tval;
    std::vector<float> dval;
    std::vector<SplitTile> tiles;
};

// whether the superblock's FP64 products take this path: from 40 MFLOP of
// dense work.  Measured, us a product, one after another on one stream, CUDA
// cores / this in a solve / this for a caller (every element checked):
//   spin-1    25 300 states     9 MFLOP    16.5 / 24 / 36
//            100 200           62          59.5 / 30 / 43
//            397 700          480         410   / 58 / 76
//          1 178 000        2 430       2 008   / 158 / 194
//   spin-1/2  88 500           70          59.5 / 30 / 44
//            615 700        1 150         910   / 74 / 111
//   Hubbard  106 700           48          87   / 40 / 57
// For a caller's vector graded over twelve decades 84, 322, 1 349 (spin-1 from
// 100 200 states), 85, 656 and 103.  Superblocks between 15 and 40 MFLOP would
// gain up to a factor of two in a solve; they stay on the CUDA cores, whose
// results whole runs at those sizes are pinned to in their last digits.
// NSS_SPLIT64 = 0 / 1 forces a path (comparisons, tests).
bool split_wanted(const DevSb &s);
// the plan from the superblock's tables, its CSR pool (rowptr, col, val) and
// HvRec::csr of the sectors
void split_layout(const DevSb &s, const std::vector<int> &rowptr, const std::vector<int> &col,
                  const std::vector<double> &val, const std::vector<int> &csr, int nsm, SplitPlan &p);
// memory, digits of H_L and H_R and the tensor maps, after the dense blocks are
// built; without room for them sb.sp_nitems stays 0
int split_finish(Ctx &c, const SplitPlan &p);
// hv = H v on c.stream.  standalone: a wait that ran out and the tiles that are
// left to k_hv_fp64 go to sb.d_sp_redo (cleared first); else the former to
// sb.d_tc_err and the product is accurate relative to the rows' largest elements.
int hv_device_split(Ctx &c, const double *d_v, double *d_hv, const int *stop, bool standalone);
// sb.d_sp_redo; the list holds 4 tile + sides to sum (1: H_L W, 2: W H_R^T)
constexpr int SP_REDO_ERR = 0, SP_REDO_COUNT = 1, SP_REDO_LIST = 2;

}  // namespace nss

// Smoothed-aggregation prolongator of one multigrid level and the Galerkin product
// A_c = P^T A P with it (Vanek, Mandel & Brezina 1996).
//
// P = (I - omega D^-1 A) Q: every fine row reaches the aggregates of its matrix
// neighbours. The sparse products W = A P and A_c = P^T W are formed row by row, their patterns once
// and their values again when only the matrix values change; rows of more columns than a warp's hash set holds
// take lists of operand pairs sorted by the (row, column) of the entry they contribute to
// (expand, sort, compress). Every sum has a fixed order (no atomics: results do not
// depend on timing).
#pragma once

#include <cstdint>

#include "kernels.hpp"

namespace fx {

// fine block (row i, col j) and its values: planar BSR3 (3x3 levels) or row-major 6x6
struct FineView {
    int bs = 3;
    int n = 0;
    int64_t nblocks = 0;
    const int32_t* blk_row = nullptr;  // per block
    const int32_t* blk_col = nullptr;  // per block (6x6 levels); planar levels use cols4
    const double* vals = nullptr;
    const int32_t* row_ptr = nullptr;
    // planar
    const int32_t* goff = nullptr;
    const int32_t* cols4 = nullptr;
    __device__ __forceinline__ int col(int64_t b, int i) const {
        if (bs == 6) return blk_col[b];
        return cols4[4 * (int64_t)goff[i] + (b - row_ptr[i])];
    }
    // row r of block b
    template <int BS>
    __device__ __forceinline__ void load_row(int64_t b, int i, int r, double* v) const {
        if (BS == 6) {
#pragma unroll
            for (int k = 0; k < 6; ++k) v[k] = __ldg(vals + b * 36 + r * 6 + k);
        } else {
            const int k = (int)(b - __ldg(row_ptr + i));
            const int64_t g0 = __ldg(goff + i);
            const int64_t ng = __ldg(goff + i + 1) - g0;
            const double* base = vals + (g0 * 9 + 3 * r * ng + k / 4) * 4 + (k & 3);
#pragma unroll
            for (int t = 0; t < 3; ++t) v[t] = __ldg(base + t * ng * 4);
        }
    }
};

// Entries of a sparse product, ascending (row, col), with the operand pairs that each sums:
// pairs[seg[e] .. seg[e+1]) = (first operand << 32) | second operand.
struct PairList {
    int64_t n = 0;
    DBuf<int32_t> row, col;
    DBuf<int64_t> seg;
    DBuf<uint64_t> pairs;
};

// Transfer of a level to the next: P's entries by fine row (ptr, col; val: row-major blocks, what
// the products read; val32: the cycle's interleaved copy) and by aggregate (t_ptr, t_row, t_val32),
// t_ent: the entry), see transfer.cuh, and W's pattern with the largest rows of W and A_c (by_rows), or
// the pair lists of W = A P and A_c = P^T W.
struct Transfer {
    int n = 0, na = 0, bs = 3;
    int64_t nnz = 0;
    DBuf<int32_t> ptr, col, t_ptr, t_row, t_ent;
    DBuf<double> val;
    DBuf<double2> val32, t_val32;
    bool by_rows = false;
    DBuf<int32_t> w_ptr, w_col;
    int most_w = 0, most_c = 0;
    PairList w, c;
};

// P of the level `F` with aggregates agg (per fine row) and tentative prolongator Q
// (BS x 6 per fine row): smoothed with omega and the block inverses dinv, or (not `smooth`, or where the
// smoothed product would not fit 32-bit item indices) Q itself. Fills t and c_ptr (na + 1), c_cols: the
// block pattern of A_c. Returns whether P is smoothed; *ncb = blocks of A_c.
bool build_transfer(const FineView& F, int na, const int32_t* agg, const double* Q, const double* dinv, double omega,
                    bool smooth, Transfer& t, DBuf<int32_t>& c_ptr, DBuf<int32_t>& c_cols, int64_t* ncb,
                    DBuf<uint8_t>& tmp, cudaStream_t s);
// c_vals (36 per block of the pattern c_ptr, c_cols) = P^T A P
void galerkin_product(const FineView& F, const Transfer& t, const int32_t* c_ptr, const int32_t* c_cols,
                      double* c_vals, cudaStream_t s);

}  // namespace fx

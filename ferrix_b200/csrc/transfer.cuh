// Grid transfer of one multigrid level, shared by the per-step kernels and the
// persistent / cooperative coarse kernels, which must produce the same sums.
//
// The prolongator P of a level (block rows of BS DOFs) has BS x 6 blocks as entries, by fine row
// (row i: entries p_ptr[i] .. p_ptr[i+1], ascending aggregate) and, for the restriction P^T, by
// aggregate (ascending fine row). The cycle reads each order from a copy of its own in which 32
// consecutive entries are interleaved by 16-byte pairs (P32): a warp with a lane per entry then
// reads whole consecutive lines. (Entry after entry, every lane's pairs were 144 or 288 bytes apart
// and each load touched 32 lines: 205k-DOF C3D4, 212k entries, 13-15 us a transfer, bound by
// L1 tag lookups.)
#pragma once

#include <cstdint>

#include "device.cuh"

namespace fx {

// pair q (of 3 BS: row q / 3, columns 2 (q % 3), + 1) of entry e in the interleaved layout
template <int BS>
__host__ __device__ __forceinline__ int64_t p32(int64_t e, int q) {
    return ((e >> 5) * (3 * BS) + q) * 32 + (e & 31);
}
template <int BS>
__host__ __device__ constexpr int64_t p32_size(int64_t n) {  // pairs
    return (n + 31) / 32 * 32 * (3 * BS);
}

// One virtual warp's share of an aggregate's P^T r: t[c] = sum over the entries p0 + 32 v + lane,
// p0 + 32 (v + kRestrictWarps) + lane, ... of (P block)^T r(row), each entry whole in one lane,
// the lanes' sums added by an xor tree (every lane ends with the six sums). An aggregate's
// sum is its kRestrictWarps virtual warps' in order: the per-step kernel gives each its own
// warp, one round of loads for the ~100 entries of an aggregate; the persistent and
// cooperative kernels run them one after another in one warp.
// CG: r is written by other CTAs of the same launch (read through L2).
constexpr int kRestrictWarps = 4;
// wait: called in every lane before r is read, with the first entry's loads in flight.
template <int BS, bool CG, typename Wait = NoWait>
__device__ __forceinline__ void restrict_agg(const int32_t* __restrict__ t_row, const double2* __restrict__ t_val,
                                             const double* r, int p0, int p1, int v, int lane, double (&t)[6],
                                             Wait wait = Wait()) {
    const int first = p0 + 32 * v + lane;
    if (first >= p1) wait();
#pragma unroll
    for (int c = 0; c < 6; ++c) t[c] = 0.0;
    for (int p = first; p < p1; p += 32 * kRestrictWarps) {
        const double* rr = r + (int64_t)BS * __ldg(t_row + p);
        double2 w[3 * BS];
#pragma unroll
        for (int q = 0; q < 3 * BS; ++q) w[q] = __ldg(t_val + p32<BS>(p, q));
        if (p == first) wait();
        double rv[BS];
#pragma unroll
        for (int k = 0; k < BS; ++k) rv[k] = CG ? __ldcg(rr + k) : rr[k];
#pragma unroll
        for (int k = 0; k < BS; ++k)
#pragma unroll
            for (int h = 0; h < 3; ++h) {
                t[2 * h] = __fma_rn(w[3 * k + h].x, rv[k], t[2 * h]);
                t[2 * h + 1] = __fma_rn(w[3 * k + h].y, rv[k], t[2 * h + 1]);
            }
    }
#pragma unroll
    for (int c = 0; c < 6; ++c) t[c] = warp_sum(t[c]);
}

// row k of entry e's block times x_c(col): what one entry adds to fine DOF k of its row
__device__ __forceinline__ double entry_dot(const double2 v[3], const double2 w[3]) {
    double d = __dmul_rn(v[0].x, w[0].x);
    d = __fma_rn(v[0].y, w[0].y, d);
    d = __fma_rn(v[1].x, w[1].x, d);
    d = __fma_rn(v[1].y, w[1].y, d);
    d = __fma_rn(v[2].x, w[2].x, d);
    return __fma_rn(v[2].y, w[2].y, d);
}

// (P x_c) of fine DOF (j, k): the row's entries in order (the persistent and cooperative
// kernels; the per-step kernel adds the same products in the same order from shared memory)
template <int BS>
__device__ __forceinline__ double prolong_dof(const int32_t* __restrict__ p_ptr, const int32_t* __restrict__ p_col,
                                              const double2* __restrict__ p_val, const double* xc, int j, int k) {
    double t = 0.0;
    const int e1 = __ldg(p_ptr + j + 1);
    for (int e = __ldg(p_ptr + j); e < e1; ++e) {
        const double2* x = reinterpret_cast<const double2*>(xc + (int64_t)__ldg(p_col + e) * 6);
        double2 v[3], w[3];
#pragma unroll
        for (int h = 0; h < 3; ++h) {
            v[h] = __ldg(p_val + p32<BS>(e, 3 * k + h));
            w[h] = __ldcg(x + h);
        }
        t = __dadd_rn(t, entry_dot(v, w));
    }
    return t;
}

}  // namespace fx

// Aggregation multigrid setup and V-cycle (see amg.hpp).
#include <cub/cub.cuh>

#include <algorithm>
#include <type_traits>
#include <cmath>
#include <cstring>

#include <cuda_fp16.h>

#include <vector>

#include "amg.hpp"
#include "coarse_row.cuh"
#include "corner.cuh"
#include "transfer.cuh"

namespace fx {

namespace {

constexpr int kCoarseMaxDof = 1200;  // dense inverse at or below this size
constexpr int kMaxLevels = 8;
// Prolongator smoothing weight omega = kSmoothOmega / lmax with lmax the level's estimate, which
// is 1.1 times the power iteration's value: 4/3 over the latter, the optimum of the analysis
constexpr double kLmaxMargin = 1.1;
constexpr double kSmoothOmega = 4.0 / 3.0 * kLmaxMargin;
// Transfers are smoothed but where the caller asks for aggregates of fewer than kSmoothMembers members on a level of
// more than kSmoothRows rows: smoothed ones reach so many small aggregates there that the Galerkin product costs
// more than it saves (205k-DOF C3D4 box with 4 / 8 / 16 nodes per aggregate 90 / 27 / 16.4 ms a solve, unsmoothed 17.8 /
// 12.5 / 11.0; with 24 11.6 and 11.7). The levels below follow the first, but below a corner level (96k-DOF
// C3D20 box, 8 nodes: 13.6 ms, 12.2 smoothed).
constexpr int64_t kSmoothMembers = 20, kSmoothRows = 5000;

// Whether FP16's rounding spoils the cycle, as it does on slender and stretched meshes and across stiffness contrasts
// (smoother_precision), shows in a V-cycle of the same residual with FP32 values: the energy of the difference of the two
// is 0.6 to 1,000 times r.z then, else 1e-5 to 3e-2. It is looked at, with smoothing that the caller left open, where from kTry16
// iterations on (then after twice as many each) the residual's fall so far lets expect more than 4 kTry16 in
// all, or twice those done; above kSpoilt16 the solve goes on with FP32 values from the residual at hand. A cantilever of 4 x 4 x 160
// regular C3D20 elements (43k DOF) did not converge in 3,000 iterations, 24 in FP64 (4.4 ms);
// 44 and 5.7 ms this way.
constexpr long long kTry16 = 16;
constexpr double kSpoilt16 = 0.1;

template <typename Op>
void cub_call(Op op, DBuf<uint8_t>& tmp, cudaStream_t s) {
    size_t bytes = 0;
    FX_CUDA_CHECK(op(nullptr, bytes));
    if (tmp.n < bytes) tmp.alloc(bytes, s);
    FX_CUDA_CHECK(op(tmp.ptr, bytes));
}

// ------------------------------------------------------------------ aggregation

// order-preserving integer image of a double, and back
__device__ __forceinline__ unsigned long long ordered(double v) {
    const unsigned long long u = (unsigned long long)__double_as_longlong(v);
    return (u >> 63) ? ~u : u | 0x8000000000000000ull;
}
__host__ __device__ __forceinline__ unsigned long long unordered_bits(unsigned long long u) {
    return (u >> 63) ? u & 0x7fffffffffffffffull : ~u;
}

// box[0..2] = componentwise minimum of the n points c, box[3..5] = maximum, as ordered integers (set to
// all ones / zero before). One pass over all SMs (one CTA took 79 us for 139k nodes).
__global__ void __launch_bounds__(256) k_box(int n, const double* __restrict__ c, unsigned long long* __restrict__ box) {
    unsigned long long lo[3] = {~0ull, ~0ull, ~0ull}, hi[3] = {0, 0, 0};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const unsigned long long v = ordered(c[3 * (int64_t)i + d]);
            lo[d] = min(lo[d], v);
            hi[d] = max(hi[d], v);
        }
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        for (int o = 16; o > 0; o >>= 1) {
            lo[d] = min(lo[d], __shfl_xor_sync(0xffffffffu, lo[d], o));
            hi[d] = max(hi[d], __shfl_xor_sync(0xffffffffu, hi[d], o));
        }
        if ((threadIdx.x & 31) == 0) {
            atomicMin(box + d, lo[d]);
            atomicMax(box + 3 + d, hi[d]);
        }
    }
}

// Cells of a level: the bounding box cut into k[d] equal parts per direction (none is a sliver at
// the box's far side; with cells of one edge the 205k-DOF C3D4 box had 3,060 instead of 2,464)
struct CellGrid {
    int k[3];
    double inv[3];  // parts per length
};

__global__ void k_cell_keys(int n, const double* __restrict__ c, const unsigned long long* __restrict__ box,
                            CellGrid g, uint64_t* __restrict__ keys, int32_t* __restrict__ ids) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint64_t key = 0;
#pragma unroll
    for (int d = 2; d >= 0; --d) {
        const double o = __longlong_as_double((long long)unordered_bits(box[d]));
        const double f = floor((c[3 * (int64_t)i + d] - o) * g.inv[d]);
        const int q = f > 0.0 ? (f < (double)g.k[d] ? (int)f : g.k[d] - 1) : 0;
        key = key * (uint64_t)g.k[d] + (uint64_t)q;
    }
    keys[i] = key;
    ids[i] = i;
}

__global__ void k_heads64(int n, const uint64_t* __restrict__ keys, int32_t* __restrict__ head) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) head[i] = (i == 0 || keys[i] != keys[i - 1]) ? 1 : 0;
}

// agg[node] = rank of its cell; agg_ptr[a] = first sorted position of aggregate a
__global__ void k_agg_assign(int n, const int32_t* __restrict__ rank1, const int32_t* __restrict__ head,
                             const int32_t* __restrict__ sorted_ids, int32_t* __restrict__ agg,
                             int32_t* __restrict__ agg_ptr) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int a = rank1[i] - 1;
    agg[sorted_ids[i]] = a;
    if (head[i]) agg_ptr[a] = i;
}

__global__ void k_agg_centroid(int na, const int32_t* __restrict__ ptr, const int32_t* __restrict__ nodes,
                               const double* __restrict__ c, double* __restrict__ cent) {
    int a = blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= na) return;
    double s0 = 0, s1 = 0, s2 = 0;
    int m = ptr[a + 1] - ptr[a];
    for (int k = ptr[a]; k < ptr[a + 1]; ++k) {
        int j = nodes[k];
        s0 += c[3 * j];
        s1 += c[3 * j + 1];
        s2 += c[3 * j + 2];
    }
    cent[3 * a] = s0 / m;
    cent[3 * a + 1] = s1 / m;
    cent[3 * a + 2] = s2 / m;
}

// Near-null-space row (d, col) of a member: level 0 rigid-body modes about the
// centroid; above, the member's R block from the previous QR.
__device__ __forceinline__ double nullspace_row(int bs, int j, int d, int col, const double* c, const double* cent,
                                                int a, const double* Rprev) {
    if (bs == 6) return Rprev[(size_t)j * 36 + d * 6 + col];
    double x = c[3 * j] - cent[3 * a], y = c[3 * j + 1] - cent[3 * a + 1], z = c[3 * j + 2] - cent[3 * a + 2];
    if (col < 3) return d == col ? 1.0 : 0.0;
    if (col == 3) return d == 0 ? -y : (d == 1 ? x : 0.0);   // rotation about z
    if (col == 4) return d == 1 ? -z : (d == 2 ? y : 0.0);   // rotation about x
    return d == 0 ? z : (d == 2 ? -x : 0.0);                  // rotation about y
}

// One warp per aggregate: Q (rows of the members) and R (6x6) by modified Gram-Schmidt, twice. The
// rows (at most kQrRows) are orthogonalised in shared memory, each lane its own rows, and written
// once; larger aggregates in place in Q (SH false). In global memory throughout, the passes' round
// trips took 95-108 us per level.
constexpr int kQrRows = 256, kQrWarps = 2;
template <bool SH>
__device__ __forceinline__ void agg_qr(int a, int lane, const int32_t* __restrict__ ptr,
                                       const int32_t* __restrict__ nodes, int bs, const double* __restrict__ c,
                                       const double* __restrict__ cent, const double* __restrict__ Rprev,
                                       double* __restrict__ Q, double* __restrict__ Rnext, double* sh) {
    const int p0 = ptr[a], m = ptr[a + 1] - ptr[a];
    const int rows = m * bs;
    auto qidx = [&](int r, int col) -> int64_t {
        if (SH) return (int64_t)col * kQrRows + r;
        return ((int64_t)nodes[p0 + r / bs] * bs + (r % bs)) * 6 + col;
    };
    double* W = SH ? sh : Q;
    for (int r = lane; r < rows; r += 32) {
        int j = nodes[p0 + r / bs];
        for (int col = 0; col < 6; ++col) W[qidx(r, col)] = nullspace_row(bs, j, r % bs, col, c, cent, a, Rprev);
    }
    __syncwarp();
    double R[36];
#pragma unroll
    for (int k = 0; k < 36; ++k) R[k] = 0.0;
#pragma unroll
    for (int col = 0; col < 6; ++col) {
        double n0 = 0.0;
        for (int r = lane; r < rows; r += 32) {
            double v = W[qidx(r, col)];
            n0 += v * v;
        }
        n0 = sqrt(warp_sum(n0));
        for (int pass = 0; pass < 2; ++pass)
#pragma unroll
            for (int k = 0; k < col; ++k) {
                double dot = 0.0;
                for (int r = lane; r < rows; r += 32) dot += W[qidx(r, k)] * W[qidx(r, col)];
                dot = warp_sum(dot);
                R[k * 6 + col] += dot;
                for (int r = lane; r < rows; r += 32) W[qidx(r, col)] -= dot * W[qidx(r, k)];
            }
        double nr = 0.0;
        for (int r = lane; r < rows; r += 32) {
            double v = W[qidx(r, col)];
            nr += v * v;
        }
        nr = sqrt(warp_sum(nr));
        const bool keep = n0 > 0.0 && nr > 1e-10 * n0;
        R[col * 6 + col] = keep ? nr : 0.0;
        for (int r = lane; r < rows; r += 32) W[qidx(r, col)] = keep ? W[qidx(r, col)] / nr : 0.0;
    }
    if (SH)
        for (int r = lane; r < rows; r += 32) {
            const int64_t o = ((int64_t)nodes[p0 + r / bs] * bs + (r % bs)) * 6;
#pragma unroll
            for (int col = 0; col < 6; ++col) Q[o + col] = W[qidx(r, col)];
        }
    if (lane == 0)
#pragma unroll
        for (int k = 0; k < 36; ++k) Rnext[(size_t)a * 36 + k] = R[k];
}

__global__ void __launch_bounds__(32 * kQrWarps) k_agg_qr(int na, const int32_t* __restrict__ ptr,
                                                          const int32_t* __restrict__ nodes, int bs,
                                                          const double* __restrict__ c,
                                                          const double* __restrict__ cent,
                                                          const double* __restrict__ Rprev, double* __restrict__ Q,
                                                          double* __restrict__ Rnext) {
    __shared__ double sh[kQrWarps][6 * kQrRows];
    const int w = threadIdx.x >> 5, a = blockIdx.x * kQrWarps + w, lane = threadIdx.x & 31;
    if (a >= na) return;  // warp-uniform
    if ((ptr[a + 1] - ptr[a]) * bs <= kQrRows)
        agg_qr<true>(a, lane, ptr, nodes, bs, c, cent, Rprev, Q, Rnext, sh[w]);
    else
        agg_qr<false>(a, lane, ptr, nodes, bs, c, cent, Rprev, Q, Rnext, nullptr);
}

__global__ void k_expand_rows(int n, const int32_t* __restrict__ row_ptr, int32_t* __restrict__ blk_row) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    for (int b = row_ptr[i]; b < row_ptr[i + 1]; ++b) blk_row[b] = i;
}

// block inverse of the 6x6 diagonal blocks; DOFs with a vanishing pivot (rank-
// deficient aggregates) get zero rows/columns in the inverse
__global__ void k_block_inv6(int n, const int32_t* __restrict__ row_ptr, const int32_t* __restrict__ cols,
                             const double* __restrict__ vals, double* __restrict__ dinv) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double A[36], X[36];
    for (int k = 0; k < 36; ++k) {
        A[k] = 0.0;
        X[k] = 0.0;
    }
    for (int b = row_ptr[i]; b < row_ptr[i + 1]; ++b)
        if (cols[b] == i)
            for (int k = 0; k < 36; ++k) A[k] = vals[(int64_t)b * 36 + k];
    double dmax = 0.0;
    for (int k = 0; k < 6; ++k) dmax = fmax(dmax, fabs(A[k * 7]));
    bool dead[6];
    for (int k = 0; k < 6; ++k) {
        dead[k] = !(fabs(A[k * 7]) > 1e-12 * dmax);
        if (dead[k]) {
            for (int t = 0; t < 6; ++t) A[k * 6 + t] = A[t * 6 + k] = 0.0;
            A[k * 7] = 1.0;
        }
        X[k * 7] = 1.0;
    }
    // Gauss-Jordan (SPD block, no pivoting)
    for (int k = 0; k < 6; ++k) {
        double p = A[k * 7];
        if (p == 0.0) p = 1.0;
        double ip = 1.0 / p;
        for (int t = 0; t < 6; ++t) {
            A[k * 6 + t] *= ip;
            X[k * 6 + t] *= ip;
        }
        for (int r = 0; r < 6; ++r)
            if (r != k) {
                double f = A[r * 6 + k];
                for (int t = 0; t < 6; ++t) {
                    A[r * 6 + t] -= f * A[k * 6 + t];
                    X[r * 6 + t] -= f * X[k * 6 + t];
                }
            }
    }
    for (int k = 0; k < 6; ++k)
        if (dead[k])
            for (int t = 0; t < 6; ++t) X[k * 6 + t] = X[t * 6 + k] = 0.0;
    for (int k = 0; k < 36; ++k) dinv[(int64_t)i * 36 + k] = X[k];
}

// ------------------------------------------------------------------ level operators

// The cycle's copy of a 6x6 level's values (coarse_row6): per block row 18 planes of 16-byte pairs
__global__ void __launch_bounds__(128) k_planar6(int n, const int32_t* __restrict__ row_ptr,
                                                 const double* __restrict__ vals, double2* __restrict__ out) {
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (i >= n) return;
    const int64_t b0 = row_ptr[i];
    const int nb = row_ptr[i + 1] - (int)b0;
    for (int it = lane; it < 18 * nb; it += 32) {
        const int q = it / nb, k = it - q * nb;
        out[b0 * 18 + it] = __ldg(reinterpret_cast<const double2*>(vals) + (b0 + k) * 18 + q);
    }
}

// b_c = P^T r_f: a CTA of kRestrictWarps warps per aggregate (restrict_agg).
// Coarse Chebyshev start fused into the restriction (cs.dinv != null): with
// b = P^T r the first pre-smoothing step of the coarse level from x = 0 is
// d = c2 D^-1 b, xs = d, r = b (what k_cheb_start does there).
template <int BS>
__global__ void __launch_bounds__(32 * kRestrictWarps)
    k_restrict(const int32_t* __restrict__ t_ptr, const int32_t* __restrict__ t_row, const double2* __restrict__ t_val,
               const double* rf, double* __restrict__ bc, CoarseStart cs) {
    __shared__ double sh[kRestrictWarps][6];
    const int a = blockIdx.x, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    double t[6];
    restrict_agg<BS, false>(t_row, t_val, rf, t_ptr[a], t_ptr[a + 1], w, lane, t, ChainWait());
    if (lane == 0)
#pragma unroll
        for (int c = 0; c < 6; ++c) sh[w][c] = t[c];
    __syncthreads();
    if (threadIdx.x >= 6) return;
#pragma unroll
    for (int c = 0; c < 6; ++c) {
        t[c] = sh[0][c];
#pragma unroll
        for (int k = 1; k < kRestrictWarps; ++k) t[c] += sh[k][c];
    }
    const int64_t o = (int64_t)a * 6 + lane;
    double tk = t[0];
#pragma unroll
    for (int c = 1; c < 6; ++c)
        if (lane == c) tk = t[c];
    bc[o] = tk;
    if (cs.dinv) {
        const double* Di = cs.dinv + (int64_t)a * 36 + lane * 6;
        double v = 0.0;
#pragma unroll
        for (int j = 0; j < 6; ++j) v += Di[j] * t[j];
        v *= cs.c2;
        cs.d[o] = v;
        cs.xs[o] = v;
        cs.r[o] = tk;
    }
}

// x_f += alpha P x_c; x4 != null (3x3 levels): the FP32 copy of the new x_f for the smoother's
// gathers, scaled by sqrt(a_ii) where sq4 is given. A CTA takes kProlongRows<BS> rows: a thread per
// entry (2-8 entries a row at the 3x3 levels, up to ~27 above) forms the entry's BS products into
// shared memory, then a thread per DOF adds its row's in order.
template <int BS>
constexpr int kProlongRows = BS == 3 ? 64 : 16;
template <int BS>
__global__ void __launch_bounds__(256) k_prolong(int n, const int32_t* __restrict__ p_ptr,
                                                 const int32_t* __restrict__ p_col, const double2* __restrict__ p_val,
                                                 const double* xc, double* xf, double alpha,
                                                 float* __restrict__ x4, const float4* __restrict__ sq4) {
    constexpr int ST = BS | 1;  // odd stride: no bank conflicts
    __shared__ double sh[256 * ST];
    const int r0 = blockIdx.x * kProlongRows<BS>, r1 = min(r0 + kProlongRows<BS>, n);
    const int e0 = p_ptr[r0], e1 = p_ptr[r1];
    const int j = r0 + (int)threadIdx.x / BS, c = (int)threadIdx.x % BS;
    const bool own = (int)threadIdx.x < kProlongRows<BS> * BS && j < r1;
    const int64_t k = (int64_t)j * BS + c;
    int p0 = 0, p1 = 0;
    double x0 = 0.0, q = 1.0, t = 0.0;
    if (own) {
        p0 = p_ptr[j];
        p1 = p_ptr[j + 1];
        if (BS == 3 && x4 && sq4) q = (double)reinterpret_cast<const float*>(sq4)[4 * (int64_t)j + c];
    }
    double2 v[3 * BS];
    int col = 0;
    auto load = [&](int e) {
        if (e >= e1) return;
        col = __ldg(p_col + e);
#pragma unroll
        for (int u = 0; u < 3 * BS; ++u) v[u] = __ldg(p_val + p32<BS>(e, u));
    };
    load(e0 + (int)threadIdx.x);
    chain_wait();
    if (own) x0 = xf[k];
    for (int tile = e0; tile < e1; tile += 256) {  // CTA-uniform
        const int e = tile + (int)threadIdx.x;
        if (tile > e0) load(e);
        if (e < e1) {
            double2 w[3];
            const double2* x = reinterpret_cast<const double2*>(xc + (int64_t)col * 6);
#pragma unroll
            for (int h = 0; h < 3; ++h) w[h] = x[h];
#pragma unroll
            for (int u = 0; u < BS; ++u) sh[threadIdx.x * ST + u] = entry_dot(v + 3 * u, w);
        }
        __syncthreads();
        for (int p = max(p0, tile); p < min(p1, tile + 256); ++p) t = __dadd_rn(t, sh[(p - tile) * ST + c]);
        __syncthreads();
    }
    if (!own) return;
    const double xn = x0 + alpha * t;
    xf[k] = xn;
    if (BS == 3 && x4) x4[4 * (int64_t)j + c] = (float)(xn * q);
}

// ------------------------------------------------------------------ coarsest level

// A (zeroed) = the dense matrix of a block CSR; a warp per block row, lanes over its values (a thread
// per row took 39-187 us on the rows of up to a hundred blocks that a smoothed transfer gives)
template <int BS>
__global__ void __launch_bounds__(128) k_dense_from_bsr(int n, const int32_t* __restrict__ row_ptr,
                                                        const int32_t* __restrict__ cols,
                                                        const double* __restrict__ vals, double* __restrict__ A) {
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (i >= n) return;
    const int64_t nd = (int64_t)BS * n;
    const int64_t v0 = (int64_t)row_ptr[i] * (BS * BS), v1 = (int64_t)row_ptr[i + 1] * (BS * BS);
    for (int64_t v = v0 + lane; v < v1; v += 32) {
        const int64_t b = v / (BS * BS);
        const int e = (int)(v - b * (BS * BS)), r = e / BS, c = e - r * BS;
        A[(BS * (int64_t)i + r) * nd + (int64_t)BS * cols[b] + c] = vals[v];
    }
}

// the same from a planar level's BSR3
__global__ void __launch_bounds__(128) k_dense_from_planar(int n, const int32_t* __restrict__ row_ptr,
                                                           const int32_t* __restrict__ goff,
                                                           const int32_t* __restrict__ cols,
                                                           const double* __restrict__ vals, double* __restrict__ A) {
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (i >= n) return;
    const int64_t nd = 3 * (int64_t)n, g0 = goff[i], ng = goff[i + 1] - g0;
    const int nb = row_ptr[i + 1] - row_ptr[i];
    for (int it = lane; it < 9 * nb; it += 32) {
        const int e = it / nb, k = it - e * nb;
        A[(3 * (int64_t)i + e / 3) * nd + 3 * (int64_t)cols[4 * g0 + k] + e % 3] =
            vals[(g0 * 9 + e * ng + k / 4) * 4 + (k & 3)];
    }
}

// Coarsest level: blocked Gauss-Jordan inverse of the dense SPD matrix (no pivoting), kPanel
// pivots per launch. With P the inverse of the pivot block A[K, K], panel K maps A to
//   B[K, K] = P, B[K, j] = P A[K, j], B[i, K] = -A[i, K] P, B[i, j] = A[i, j] - A[i, K] P A[K, j].
// A and B alternate between two buffers, so that every tile is computed from A alone by its own
// CTA and a panel is one launch; the CTA that holds the next pivot block inverts it as
// soon as it is updated. DOFs without stiffness (k_dense_decouple) are decoupled first and get
// zero rows/columns in the inverse.
constexpr int kPanel = 32;
constexpr int kTileRows = 64;  // rows of a tile (kPanel columns): P A[K, j] is formed once per tile

// dead[k] = 1 for the DOFs to decouple. 6x6 levels: a diagonal below 1e-12 of the largest, the columns that
// a rank-deficient aggregate's factorisation left empty. Planar levels: none but a zero diagonal (a
// node of no element). There the largest is the constraints' penalty, 1e6 times the stiffest
// material's, and the inverse is the only thing that acts on a soft material's nodes: with the 6x6 levels'
// rule, steel beside a material 4e6 times softer did not converge.
__global__ void __launch_bounds__(1024) k_dense_decouple(int nd, double rel, double* __restrict__ A,
                                                         uint8_t* __restrict__ dead, double* __restrict__ diag) {
    __shared__ double s_red[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    double m = 0.0;
    for (int k = threadIdx.x; k < nd; k += blockDim.x) m = fmax(m, fabs(A[(int64_t)k * nd + k]));
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (lane == 0) s_red[warp] = m;
    __syncthreads();
    double dmax = 0.0;
    for (int w = 0; w < nw; ++w) dmax = fmax(dmax, s_red[w]);
    int any = 0;
    for (int k = threadIdx.x; k < nd; k += blockDim.x) {
        dead[k] = !(fabs(A[(int64_t)k * nd + k]) > rel * dmax);
        any |= dead[k];
    }
    if (__syncthreads_or(any)) {  // (rank-deficient aggregates only: the pass over A takes ~50 us at 700 DOF)
        for (int r = warp; r < nd; r += nw)
            for (int c = lane; c < nd; c += 32)
                if (dead[r] || dead[c]) A[(int64_t)r * nd + c] = (r == c) ? 1.0 : 0.0;
    }
    __syncthreads();
    for (int k = threadIdx.x; k < nd; k += blockDim.x) diag[k] = A[(int64_t)k * nd + k];  // before elimination
}

// A pivot of the elimination below kSingularPivot of its row's original
// diagonal means the coarse operator is singular: the rigid-body modes of an
// insufficiently constrained model lie in the coarse space (an SPD coarse
// matrix keeps each pivot at or above 1 / cond of the original diagonal).
constexpr double kSingularPivot = 1e-12;

// P = inverse of the pivot block that the 256 threads hold (thread (ty, tx): entries (ty + 8 u, tx)),
// b pivots from k0, the rest the identity; *singular |= 1 when a pivot is not above
// kSingularPivot times its original diagonal. Two pivots per step: their rows and columns go
// through alternating shared buffers (one barrier a step), everything else stays in registers,
// and the chain of a step (exchange, reciprocal, update) is paid 16 times instead of 32.
__device__ __forceinline__ void invert_pivot(double (&a)[4], int k0, int b, const double* __restrict__ diag,
                                             int* __restrict__ singular, double* __restrict__ P) {
    __shared__ double s_row[2][2][kPanel], s_col[2][2][kPanel];
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    for (int t = 0; t < b; t += 2) {  // (b odd: the last step's second pivot is an identity row)
        const int q = (t >> 1) & 1;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int r = ty + 8 * u;
            if ((tx & ~1) == t) s_col[q][tx & 1][r] = a[u];
            if ((r & ~1) == t) s_row[q][r & 1][tx] = a[u];
        }
        __syncthreads();
        const double p00 = s_row[q][0][t], p01 = s_row[q][0][t + 1], p10 = s_row[q][1][t], p11 = s_row[q][1][t + 1];
        const double det = p00 * p11 - p01 * p10, id = 1.0 / det;
        const double i00 = p11 * id, i01 = -p01 * id, i10 = -p10 * id, i11 = p00 * id;
        if (threadIdx.x == 0 &&
            (!(p00 > kSingularPivot * diag[k0 + t]) ||
             (t + 1 < b && !(det > kSingularPivot * diag[k0 + t + 1] * p00))))
            *singular = 1;
        const double r0 = s_row[q][0][tx], r1 = s_row[q][1][tx];
        const bool pc = (tx & ~1) == t;  // a pivot column: the inverse's own entries
        const double m0 = pc ? ((tx & 1) ? i01 : i00) : i00 * r0 + i01 * r1;
        const double m1 = pc ? ((tx & 1) ? i11 : i10) : i10 * r0 + i11 * r1;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int r = ty + 8 * u;
            const double f0 = s_col[q][0][r], f1 = s_col[q][1][r];
            if ((r & ~1) == t) a[u] = (r & 1) ? m1 : m0;
            else a[u] = (pc ? 0.0 : a[u]) - f0 * m0 - f1 * m1;
        }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) P[(ty + 8 * u) * kPanel + tx] = a[u];
}

// the first pivot block's inverse
__global__ void __launch_bounds__(256) k_gj_first(int nd, const double* __restrict__ A, const double* __restrict__ diag,
                                                  int* __restrict__ singular, double* __restrict__ P) {
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int b = min(kPanel, nd);
    double a[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const int r = ty + 8 * u;
        a[u] = r < b && tx < b ? A[(int64_t)r * nd + tx] : (r == tx ? 1.0 : 0.0);
    }
    invert_pivot(a, 0, b, diag, singular, P);
}

// One panel: B from A and P (see above). Bound by the launch and, above ~1,000 DOF, by
// shared-memory loads of the two 32-deep products (pairs of the left factor per load). With
// separate launches for the pivot inverse (16-18 us), panel rows (9), update (8) and panel
// columns (4) instead: the NLGEOM beam of 16k DOF, with 85 inverses of 168 DOF, took 370 ms
// against 355, the 14,883-DOF cantilever 9.44 against 9.15 ms from deck text.
__global__ void __launch_bounds__(256) k_gj_panel(int nd, int k0, const double* A, double* __restrict__ B,
                                                  const double* P, double* __restrict__ P_next,
                                                  const double* __restrict__ diag, int* __restrict__ singular) {
    __shared__ __align__(16) double Ps[kPanel][kPanel + 2];     // P, zero outside the panel
    __shared__ double Rs[kPanel][kPanel];                       // A[K, j0 + c], then P A[K, j0 + c]
    __shared__ __align__(16) double Ls[kTileRows][kPanel + 2];  // A[i0 + r, K]
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int i0 = blockIdx.y * kTileRows, j0 = blockIdx.x * kPanel;
    const int b = min(kPanel, nd - k0);
    const bool panel_col = j0 == k0;
    const int j = j0 + tx;
    chain_wait();
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const int r = ty + 8 * u;
        Ps[r][tx] = r < b && tx < b ? P[r * kPanel + tx] : 0.0;
        if (!panel_col) Rs[r][tx] = r < b && j < nd ? A[(int64_t)(k0 + r) * nd + j] : 0.0;
    }
    double a[kTileRows / 8];
#pragma unroll
    for (int u = 0; u < kTileRows / 8; ++u) {
        const int r = ty + 8 * u, i = i0 + r;
        Ls[r][tx] = i < nd && tx < b ? A[(int64_t)i * nd + k0 + tx] : 0.0;
        a[u] = i < nd && j < nd ? A[(int64_t)i * nd + j] : 0.0;
    }
    __syncthreads();
    double m[4] = {0.0, 0.0, 0.0, 0.0};  // R = P A[K, j], or P itself in the panel's own columns
    if (panel_col) {
#pragma unroll
        for (int u = 0; u < 4; ++u) m[u] = Ps[ty + 8 * u][tx];
    } else {
#pragma unroll
        for (int t = 0; t < kPanel; t += 2) {
            const double r0 = Rs[t][tx], r1 = Rs[t + 1][tx];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const double2 p = *reinterpret_cast<const double2*>(&Ps[ty + 8 * u][t]);
                m[u] += p.x * r0 + p.y * r1;
            }
        }
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < 4; ++u) Rs[ty + 8 * u][tx] = m[u];
    __syncthreads();
    double acc[kTileRows / 8];
#pragma unroll
    for (int u = 0; u < kTileRows / 8; ++u) acc[u] = 0.0;
#pragma unroll 4
    for (int t = 0; t < kPanel; t += 2) {
        const double r0 = Rs[t][tx], r1 = Rs[t + 1][tx];
#pragma unroll
        for (int u = 0; u < kTileRows / 8; ++u) {
            const double2 l = *reinterpret_cast<const double2*>(&Ls[ty + 8 * u][t]);
            acc[u] += l.x * r0 + l.y * r1;
        }
    }
#pragma unroll
    for (int u = 0; u < kTileRows / 8; ++u) {
        const int i = i0 + ty + 8 * u;
        if (i >= k0 && i < k0 + b) a[u] = Rs[i - k0][tx];
        else a[u] = (panel_col ? 0.0 : a[u]) - acc[u];
        if (i < nd && j < nd) B[(int64_t)i * nd + j] = a[u];
    }
    const int kn = k0 + kPanel;
    if (kn >= nd || j0 != kn || kn < i0 || kn >= i0 + kTileRows) return;  // CTA-uniform
    const int bn = min(kPanel, nd - kn);
    double pv[4];  // the next pivot block: rows kn - i0 .. of this tile (i0 and kn are multiples of 32)
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const double v = kn == i0 ? a[u] : a[4 + u];
        const int r = ty + 8 * u;
        pv[u] = r < bn && tx < bn ? v : (r == tx ? 1.0 : 0.0);
    }
    invert_pivot(pv, kn, bn, diag, singular, P_next);
}

__global__ void __launch_bounds__(256) k_dense_zero_dead(int nd, double* __restrict__ A,
                                                         const uint8_t* __restrict__ dead) {
    const int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (r >= nd) return;
    for (int c = lane; c < nd; c += 32)
        if (dead[r] || dead[c]) A[(int64_t)r * nd + c] = 0.0;
}

__global__ void k_dense_matvec(int nd, const double* __restrict__ A, const double* x, double* __restrict__ y) {
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (warp >= nd) return;
    const double t = dense_row_dot<false>(A + (int64_t)warp * nd, x, nd, lane, ChainWait());
    if (lane == 0) y[warp] = t;
}

// deterministic dot product of two vectors into out[0] (two launches)
__global__ void k_dot_part(int64_t n, const double* __restrict__ a, const double* __restrict__ b,
                           double* __restrict__ part) {
    __shared__ double sh[8];
    double t = 0.0;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        t += a[i] * b[i];
    t = warp_sum(t);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = t;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += sh[w];
        part[blockIdx.x] = s;
    }
}

// partial sums of (b.z, b.zold) as a V-cycle's last smoothing step leaves them (zold null: 0)
__global__ void __launch_bounds__(256) k_pair_part(int64_t n, const double* b, const double* z,
                                                   const double* zold, double* __restrict__ part);

// |a|^2 and |b|^2 in two launches (fixed order): partials of a in part[0 .. nb), of b in part[nb .. 2 nb)
__global__ void __launch_bounds__(256) k_norm2_part(int64_t n, const double* __restrict__ a,
                                                    const double* __restrict__ b, double* __restrict__ part, int nb) {
    __shared__ double sh[2][8];
    double t = 0.0, u = 0.0;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        t += a[i] * a[i];
        u += b[i] * b[i];
    }
    t = warp_sum(t);
    u = warp_sum(u);
    if ((threadIdx.x & 31) == 0) {
        sh[0][threadIdx.x >> 5] = t;
        sh[1][threadIdx.x >> 5] = u;
    }
    __syncthreads();
    if (threadIdx.x < 2) {
        double v = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) v += sh[threadIdx.x][w];
        part[threadIdx.x * nb + blockIdx.x] = v;
    }
}

__global__ void k_norm2_sum(int nb, const double* __restrict__ part, double* __restrict__ out) {
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;  // a warp per norm
    double t = 0.0;
    for (int k = lane; k < nb; k += 32) t += part[w * nb + k];
    t = warp_sum(t);
    if (lane == 0) out[w] = t;
}

// x = d / sqrt(*nrm2), the norm read on the device
__global__ void k_normalize(int64_t n, const double* __restrict__ nrm2, const double* d, double* x) {
    const double v = *nrm2;
    const double inv = v > 0.0 ? 1.0 / sqrt(v) : 1.0;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        x[i] = d[i] * inv;
}

__global__ void k_fill_hash(int64_t n, double* __restrict__ v) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint64_t h = (uint64_t)i * 0x9E3779B97F4A7C15ull;
    h ^= h >> 29;
    v[i] = (double)(h & 0xFFFFF) / 1048576.0 + 0.5;
}


unsigned grid_for(int64_t n, int t = 256) { return (unsigned)((n + t - 1) / t); }

// ---- outer PCG scalars: S[0] r.z of the last beta, S[2] r.D^-1 r, S[3] b.D^-1 b, S[6] breakdown, S[7] barrier
// timeout, S[8] r.z. The sums p.q, r.z and r.D^-1 r are left as partial sums by the launch that forms
// their terms and added by every CTA of the launch that needs them, in the same fixed order
// (cta_total): reducing them in the producing launch's last CTA (fence, counter, second read of
// the partials) ended three launches of every iteration with ~3 us of one CTA's latency.
__global__ void k_fin(int nb, const double* __restrict__ part, double* __restrict__ S, int what) {
    double t = 0.0;  // fixed lane assignment and tree: deterministic
    for (int k = threadIdx.x; k < nb; k += 32) t += part[k];
    t = warp_sum(t);
    if (threadIdx.x != 0) return;
    if (what == 1) {  // r.D^-1 r
        S[2] = t;
    } else if (what == 3) {  // initial r.z
        S[0] = t;
        S[8] = t;
    }
}

// Sum of n partial sums (entries of `stride` doubles; minus the second double of each with diff), in
// every thread of a CTA of 256.
__device__ __forceinline__ double cta_total(const double* part, int n, int stride, bool diff) {
    __shared__ double s_tot[8];
    double t = 0.0;
    for (int k = threadIdx.x; k < n; k += 256)
        t += diff ? part[(int64_t)k * stride] - part[(int64_t)k * stride + 1] : part[(int64_t)k * stride];
    t = warp_sum(t);
    if ((threadIdx.x & 31) == 0) s_tot[threadIdx.x >> 5] = t;
    __syncthreads();
    t = 0.0;
#pragma unroll
    for (int w = 0; w < 8; ++w) t += s_tot[w];
    __syncthreads();  // s_tot may be written again
    return t;
}

// partial r . D^-1 r without the update (start of the solve)
__global__ void k_rdr_part(int n, const double* __restrict__ r, const double* __restrict__ dinv,
                           double* __restrict__ part) {
    __shared__ double sh[8];
    double acc = 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const double* D = dinv + 9 * (int64_t)i;
        const double* rv = r + 3 * (int64_t)i;
        for (int c = 0; c < 3; ++c) acc += rv[c] * (D[3 * c] * rv[0] + D[3 * c + 1] * rv[1] + D[3 * c + 2] * rv[2]);
    }
    acc = warp_sum(acc);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += sh[w];
        part[blockIdx.x] = s;
    }
}

// p = z + beta p with beta = (r.z - r.z_old) / r.z_prev from the V-cycle's partial sums (pairs; z_old only
// in the flexible CG), r.z into S[8] and r.D^-1 r from the update's partial sums into S[2]
__global__ void __launch_bounds__(256) k_xpby(int64_t n, const double* z, double* S, const double* rz_part, int n_rz,
                                              bool flexible, const double* rd_part, int n_rd, double* p) {
    chain_wait();
    const double prev = S[0];  // (S[0] is moved on by the next update only)
    const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
    const double zv = i < n ? z[i] : 0.0, pv = i < n ? p[i] : 0.0;
    const double rz = cta_total(rz_part, n_rz, 2, false);
    const double num = flexible ? cta_total(rz_part, n_rz, 2, true) : rz;
    const double beta = prev > 0.0 ? num / prev : 0.0;
    if (i < n) p[i] = zv + beta * pv;
    if (blockIdx.x == 0) {
        const double rd = cta_total(rd_part, n_rd, 1, false);
        if (threadIdx.x == 0) {
            S[8] = rz;
            S[2] = rd;
        }
    }
}

// ------------------------------------------------------------------ level 0: fused operators
// One pass over the planar BSR3 matrix (8 lanes per block row, FP64 accumulation,
// values in VT = double or float) followed by a row-local epilogue:
//   kL0Resid  y = b - A v (y = A v without b)
//   kL0RUpd   r -= A v
//   kL0Cheb0  r = b - A v; d = c2 D^-1 r; xo = v + d             (first Chebyshev step from v = x)
//   kL0ChebK  r -= A v; d = c1 v + c2 D^-1 r; xo += d            (later steps, v = previous direction)
//   kL0Apply  y = A v
//   kL0Power  d = c2 D^-1 A v                                    (a step of the power iteration)
// With dot = 1 the CTAs leave partial sums of v.y (p.q), with dot = 2 of (b.xo, b.zold) (r.z and, in the
// flexible CG, r.z_old; the last V-cycle step of the outer CG).
enum : int { kL0Resid = 0, kL0RUpd = 1, kL0Cheb0 = 2, kL0ChebK = 3, kL0Apply = 4, kL0Power = 5 };

template <typename VT>
struct L0Op {
    int n;
    const int32_t* goff;
    const int32_t* cols;
    const VT* vals;
    const double* v;
    const double* b;
    double* y;
    double* r;
    double* d_out;
    double* xo;
    const double* dinv;
    double c1, c2;
    int dot;
    const double* zold;  // dot = 2 with a flexible outer CG: the previous preconditioned residual
    double* part;        // partial sums per CTA: one (dot = 1) or two doubles
    // FP32 smoother vectors (mixed precision): the gathered vector as float4 per
    // node (x, y, z, 0) and the new direction written into the same layout; with FP16
    // values and kL0H16Vec the directions are four halves per node (8 bytes) instead
    const float4* v4;
    float* d4_out;
    // FP16 values of the diagonally scaled matrix S A S (S = diag(a_ii)^-1/2): sqrt(a_ii)
    // per node; the gathered float4 vectors then hold sqrt(a_jj) v_j
    const float4* sq4;
    // FP16 smoother directions (kL0H16Vec): {2^k, 2^-k}, the V-cycle's scale of the
    // stored directions (null: 1)
    const float* hs;
};

__device__ __forceinline__ void ld4v(const float* p, float o[4]) {
    const float4 v = __ldcs(reinterpret_cast<const float4*>(p));
    o[0] = v.x;
    o[1] = v.y;
    o[2] = v.z;
    o[3] = v.w;
}
__device__ __forceinline__ void ld4v(const __half* p, float o[4]) {
    const uint2 v = __ldcs(reinterpret_cast<const uint2*>(p));
    const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&v.x));
    const float2 b = __half22float2(*reinterpret_cast<const __half2*>(&v.y));
    o[0] = a.x;
    o[1] = a.y;
    o[2] = b.x;
    o[3] = b.y;
}
__device__ __forceinline__ void unpack_h4(uint2 v, float o[4]) {
    const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&v.x));
    const float2 b = __half22float2(*reinterpret_cast<const __half2*>(&v.y));
    o[0] = a.x;
    o[1] = a.y;
    o[2] = b.x;
    o[3] = b.y;
}
template <typename T>
__device__ __forceinline__ void unpack_h4(uint2, T*) {}
__device__ __forceinline__ void ld4v(const double* p, double o[4]) {
    const double2 a = __ldcs(reinterpret_cast<const double2*>(p));
    const double2 b = __ldcs(reinterpret_cast<const double2*>(p) + 1);
    o[0] = a.x;
    o[1] = a.y;
    o[2] = b.x;
    o[3] = b.y;
}

// Fixed-order sums of (v, v2) over the CTA, left in part (two = false: v alone)
__device__ __forceinline__ void cta_partials(double v, double v2, bool two, double* part) {
    __shared__ double sh[2][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    v = warp_sum(v);
    v2 = warp_sum(v2);
    if (lane == 0) {
        sh[0][w] = v;
        sh[1][w] = v2;
    }
    __syncthreads();
    if (threadIdx.x < (two ? 2u : 1u)) {
        double t = 0.0;
        for (int k = 0; k < nw; ++k) t += sh[threadIdx.x][k];
        part[(two ? 2 : 1) * blockIdx.x + threadIdx.x] = t;
    }
}

__global__ void __launch_bounds__(256) k_pair_part(int64_t n, const double* b, const double* z,
                                                   const double* zold, double* __restrict__ part) {
    chain_wait();
    double t = 0.0, u = 0.0;
    for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < n; i += (int64_t)gridDim.x * 256) {
        t += b[i] * z[i];
        if (zold) u += b[i] * zold[i];
    }
    cta_partials(t, u, true, part);
}

#ifndef FX_L0_MIN_BLOCKS
#define FX_L0_MIN_BLOCKS 2
#endif
constexpr int kL0MinBlocks = FX_L0_MIN_BLOCKS;  // 256-thread CTAs resident per SM (2: at most 128 registers)
// The outer CG's q = K p (FP64 values, mode kL0Apply) compiled for its own CTAs per SM (2: on
// the 417k-DOF box a default solve took 51.5-51.7 ms, against 53.4 with 3 (80 registers)
// and 55.0 with 4 (64 registers, spilling))
#ifndef FX_L0_MIN_BLOCKS_APPLY
#define FX_L0_MIN_BLOCKS_APPLY 2
#endif
constexpr int kL0MinBlocksApply = FX_L0_MIN_BLOCKS_APPLY;
// FP16 values: its loads are half as wide as the FP32 form's, so it is latency-bound and
// needs more warps and more loads in flight. Measured per Chebyshev step on the 417k-DOF
// C3D20 box (B200): 57.7 us at 2 CTAs per SM; 54.8 at 3 (85 registers); 61.5 at 4 with
// spills; 50.5 at 4 with the row's epilogue operands loaded after the gathers (no spills
// at 64 registers); 48.1 with, in addition, each group's nine plane loads issued before
// its column ids (FX_L0_VFIRST_H). The FP32 / FP64 forms spill and slow down at those
// budgets, so they keep 2 CTAs per SM.
#ifndef FX_L0_VFIRST_H
#define FX_L0_VFIRST_H 1
#endif
#ifndef FX_L0_LATE_EPI_H
#define FX_L0_LATE_EPI_H 1
#endif
#ifndef FX_L0_MIN_BLOCKS_H
#define FX_L0_MIN_BLOCKS_H 4
#endif
constexpr int kL0MinBlocksH = FX_L0_MIN_BLOCKS_H;
// FP16 smoother: the Chebyshev directions as four halves per node (8 bytes) instead of
// a float4 (the prolongated iterate stays FP32). The directions shrink with the outer
// CG's residual, by 1e8 and more over a solve, so unscaled they fall below FP16's
// subnormal range and the smoothing stops; they are stored times a power of two taken
// from the residual the V-cycle smooths.
#ifndef FX_L0_H16VEC
#define FX_L0_H16VEC 1
#endif
constexpr bool kL0H16Vec = FX_L0_H16VEC != 0;
// With the FP16 smoother, the level-0 eigenvalue estimate's products also come from the FP16
// scaled matrix (1); else from an FP32 copy of the FP64 values made for it (0). On the
// 417k-DOF box: multigrid setup 5.17 -> 4.92 ms, the same 100 CG iterations.
#ifndef FX_AMG_EST_F16
#define FX_AMG_EST_F16 1
#endif
constexpr bool kAmgEstF16 = FX_AMG_EST_F16 != 0;
// the stored directions' 2-norm is about 2^kH16Exp: a direction entry overflows only if the
// residual grows by about 2^(15 - kH16Exp) from one outer iteration to the next, and the
// entries of a vector of 1e7 nodes still sit ~10 binades above the smallest normal FP16
constexpr int kH16Exp = 8;

// {2^k, 2^-k} with 2^k sqrt(rdr) in [2^(kH16Exp-1), 2^kH16Exp), rdr = r.D^-1 r of the
// residual the V-cycle smooths: the smoother's directions c D^-1 r scaled by sqrt(a_ii)
// have a 2-norm of about sqrt(rdr). A power of two scales exactly, so the FP16 roundings
// are those of an FP16 whose range is centred on the vector.
__device__ __forceinline__ float2 h16_scale(double rdr) {
    if (!(rdr > 0.0) || !isfinite(rdr)) return make_float2(1.0f, 1.0f);
    int e;
    frexp(sqrt(rdr), &e);
    const int k = max(-100, min(100, kH16Exp - e));
    return make_float2(ldexpf(1.0f, k), ldexpf(1.0f, -k));
}

// FP16 bits of x rounded to nearest, clamped to the finite range (a direction that
// outgrows the lagged scale saturates instead of turning the smoother's sums into inf)
__device__ __forceinline__ uint32_t h16_bits(float x) {
    return __half_as_ushort(__float2half_rn(fminf(fmaxf(x, -65504.0f), 65504.0f)));
}

#ifndef FX_L0_LANES
#define FX_L0_LANES 8
#endif
constexpr int kL0Lanes = FX_L0_LANES;          // lanes per block row (8 or 4)
constexpr int kL0RowsPerWarp = 32 / kL0Lanes;
constexpr int kL0LaneShift = kL0Lanes == 8 ? 3 : 2;
#ifndef FX_L0_UNROLL
#define FX_L0_UNROLL 2
#endif
constexpr int kL0Unroll = FX_L0_UNROLL;  // groups of a row in flight per lane

// G32: gathers from o.v4 (FP32, 16 B per node) and writes the direction into
// o.d4_out; the row's own FP64 values still come from o.v where the mode needs
// them (Cheb0: the iterate), else from o.v4.
template <typename VT, int MODE, bool G32 = false>
__global__ void __launch_bounds__(256, std::is_same<VT, __half>::value ? kL0MinBlocksH
                                      : (MODE == kL0Apply ? kL0MinBlocksApply : kL0MinBlocks))
    k_l0_op(L0Op<VT> o) {
    // FP16 values (of the scaled matrix): FP32 gathers of the scaled vectors, row sums
    // scaled back by sqrt(a_ii), directions written scaled
    constexpr bool H = std::is_same<VT, __half>::value;
    // FP16 values: the row-local epilogue operands are loaded after the gathers
    // (FX_L0_LATE_EPI_H), which frees their registers during the gather loop
    constexpr bool kL0LateEpi = H && FX_L0_LATE_EPI_H;
    constexpr bool kL0VFirst = H && FX_L0_VFIRST_H;
    // FP16 directions: written by the Chebyshev steps, gathered by all but the step from
    // the (FP32) iterate; 2^-k is applied to the row sums, after the gathers
    constexpr bool kH16 = H && G32 && kL0H16Vec;
    constexpr bool kH16g = kH16 && (MODE == kL0ChebK || MODE == kL0RUpd);
    const int sub = threadIdx.x & (kL0Lanes - 1);
    const int row0 = (blockIdx.x * blockDim.x + threadIdx.x) >> kL0LaneShift;
    const int rows_per_grid = (gridDim.x * blockDim.x) >> kL0LaneShift;
    // uniform trip count per warp: the warp's rows share one base
    const int nb = ((o.n + kL0RowsPerWarp - 1) / kL0RowsPerWarp) * kL0RowsPerWarp;
    const double* v = o.v;
    double dsum = 0.0, dsum2 = 0.0;
    chain_wait();
    for (int base = row0 - (row0 & (kL0RowsPerWarp - 1)); base < nb; base += rows_per_grid) {
        const int row = base + (row0 & (kL0RowsPerWarp - 1));
        const bool valid = row < o.n;
        const int g0 = valid ? o.goff[row] : 0;
        const int ng = valid ? o.goff[row + 1] - g0 : 0;
        // row-local operands of the epilogue, loaded before the gathers so that their latency overlaps
        const int64_t o3 = 3 * (int64_t)row;
        const int c = sub < 3 ? sub : 0;
        const bool epi = valid && sub < 3;
        double src3[3] = {0.0, 0.0, 0.0}, Dr[3] = {0.0, 0.0, 0.0}, vc = 0.0, xoc = 0.0, bc = 0.0, zoc = 0.0;
        float4 sqi = make_float4(1.f, 1.f, 1.f, 0.f);
        float2 hsc = make_float2(1.f, 1.f);  // {2^k, 2^-k}: .x is read where the direction is stored
        auto load_epi = [&]() {
        if (H && epi) sqi = __ldg(o.sq4 + row);
        if (kH16g && epi && o.hs) hsc.y = o.hs[1];
        if (epi) {
            if (MODE == kL0Cheb0 || MODE == kL0ChebK) {
                const double* src = MODE == kL0Cheb0 ? o.b : o.r;
#pragma unroll
                for (int kk = 0; kk < 3; ++kk) {
                    src3[kk] = src[o3 + kk];
                    Dr[kk] = o.dinv[9 * (int64_t)row + 3 * c + kk];
                }
                if (G32 && MODE == kL0ChebK) {
                    const float* own = reinterpret_cast<const float*>(o.v4 + row);
                    if constexpr (kH16)
                        vc = (double)(__half2float(reinterpret_cast<const __half*>(o.v4)[4 * (int64_t)row + c]) *
                                      hsc.y);
                    else vc = (double)own[c];
                    if (H) vc /= (double)(c == 0 ? sqi.x : (c == 1 ? sqi.y : sqi.z));
                } else {
                    vc = v[o3 + c];
                }
                if (MODE == kL0ChebK) xoc = o.xo[o3 + c];
                if (o.dot) bc = o.b[o3 + c];
                if (o.dot && o.zold) zoc = o.zold[o3 + c];
            } else if (MODE == kL0Apply) {
                vc = v[o3 + c];
            } else if (MODE == kL0Power) {
#pragma unroll
                for (int kk = 0; kk < 3; ++kk) Dr[kk] = o.dinv[9 * (int64_t)row + 3 * c + kk];
            } else if (MODE == kL0Resid) {
                bc = o.b ? o.b[o3 + c] : 0.0;
            } else {
                src3[0] = o.r[o3 + c];
            }
        }
        };
        if (!kL0LateEpi) load_epi();
        double acc[3] = {0.0, 0.0, 0.0};
#pragma unroll kL0Unroll
        for (int g = sub; g < ng; g += kL0Lanes) {
            // FP16 values (kL0VFirst): the group's nine 8-byte plane loads are issued before
            // the column ids and the gathers that depend on them
            uint2 raw[kL0VFirst ? 9 : 1];
            if constexpr (kL0VFirst) {
                const __half* vh = reinterpret_cast<const __half*>(o.vals) + ((int64_t)g0 * 9 + g) * 4;
#pragma unroll
                for (int k = 0; k < 9; ++k)
                    raw[k] = __ldcs(reinterpret_cast<const uint2*>(vh + (int64_t)k * ng * 4));
            }
            const int4 cc = __ldg(reinterpret_cast<const int4*>(o.cols) + g0 + g);
            const int cj[4] = {cc.x, cc.y, cc.z, cc.w};
            // FP32 values with FP32 gathered vectors: the group's 4 blocks are summed in
            // FP32 (no FP64 conversions of the 36 values) and added to the FP64 row sums
            using GT = typename std::conditional<G32, float, double>::type;
            GT xv[4][3];
            if (G32) {
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    if constexpr (kH16g) {
                        const uint2 u = reinterpret_cast<const uint2*>(o.v4)[cj[q]];
                        const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&u.x));
                        xv[q][0] = a.x;
                        xv[q][1] = a.y;
                        xv[q][2] = __half2float(__ushort_as_half((unsigned short)(u.y & 0xffffu)));
                    } else {
                        const float4 t = o.v4[cj[q]];
                        xv[q][0] = t.x;
                        xv[q][1] = t.y;
                        xv[q][2] = t.z;
                    }
                }
            } else {
#pragma unroll
                for (int q = 0; q < 4; ++q)
#pragma unroll
                    for (int k = 0; k < 3; ++k) xv[q][k] = (GT)v[3 * (int64_t)cj[q] + k];
            }
            const VT* vb = o.vals + ((int64_t)g0 * 9 + g) * 4;
            const int64_t pl = (int64_t)ng * 4;
#pragma unroll
            for (int r = 0; r < 3; ++r) {
                using MT = typename std::conditional<H, float, VT>::type;
                MT m0[4], m1[4], m2[4];
                if constexpr (kL0VFirst) {
                    unpack_h4(raw[3 * r], m0);
                    unpack_h4(raw[3 * r + 1], m1);
                    unpack_h4(raw[3 * r + 2], m2);
                } else {
                    ld4v(vb + (3 * r) * pl, m0);
                    ld4v(vb + (3 * r + 1) * pl, m1);
                    ld4v(vb + (3 * r + 2) * pl, m2);
                }
                GT t = 0;
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    t += (GT)m0[q] * xv[q][0] + (GT)m1[q] * xv[q][1] + (GT)m2[q] * xv[q][2];
                acc[r] += (double)t;
            }
        }
#pragma unroll
        for (int s = kL0Lanes / 2; s > 0; s >>= 1)
#pragma unroll
            for (int r = 0; r < 3; ++r) acc[r] += __shfl_xor_sync(0xffffffffu, acc[r], s);
        if (kL0LateEpi) load_epi();
        // epilogue: lane c of the row's 8 handles component c
        if (H) {  // (A v)_i = sqrt(a_ii) (S A S (sqrt(a_jj) v_j))_i; FP16 directions: times 2^-k
            const double u = kH16g ? (double)hsc.y : 1.0;
            acc[0] *= (double)sqi.x * u;
            acc[1] *= (double)sqi.y * u;
            acc[2] *= (double)sqi.z * u;
        }
        const double axc = c == 0 ? acc[0] : (c == 1 ? acc[1] : acc[2]);
        __syncwarp();  // every lane's reads of r (above) are ordered before any lane writes r[c]
        if (!epi) continue;
        if (MODE == kL0Resid) {
            o.y[o3 + c] = o.b ? bc - axc : axc;
        } else if (MODE == kL0RUpd) {
            o.r[o3 + c] = src3[0] - axc;
        } else if (MODE == kL0Apply) {
            o.y[o3 + c] = axc;
            dsum += vc * axc;
        } else if (MODE == kL0Power) {
            const double z = o.c2 * (Dr[0] * acc[0] + Dr[1] * acc[1] + Dr[2] * acc[2]);
            if (G32) o.d4_out[4 * (int64_t)row + c] =
                (float)(H ? z * (double)(c == 0 ? sqi.x : (c == 1 ? sqi.y : sqi.z)) : z);
            if (!G32 || o.d_out) o.d_out[o3 + c] = z;
        } else {  // Chebyshev steps
            const double rr[3] = {src3[0] - acc[0], src3[1] - acc[1], src3[2] - acc[2]};
            const double z = Dr[0] * rr[0] + Dr[1] * rr[1] + Dr[2] * rr[2];
            o.r[o3 + c] = c == 0 ? rr[0] : (c == 1 ? rr[1] : rr[2]);
            const double dn = (MODE == kL0Cheb0 ? 0.0 : o.c1 * vc) + o.c2 * z;
            if (kH16) {
                if (o.hs) hsc.x = o.hs[0];
                reinterpret_cast<unsigned short*>(o.d4_out)[4 * (int64_t)row + c] = (unsigned short)h16_bits(
                    (float)(dn * (double)(c == 0 ? sqi.x : (c == 1 ? sqi.y : sqi.z))) * hsc.x);
            } else if (G32) o.d4_out[4 * (int64_t)row + c] = (float)(H ? dn * (double)(c == 0 ? sqi.x : (c == 1 ? sqi.y : sqi.z)) : dn);
            else o.d_out[o3 + c] = dn;
            const double xn = (MODE == kL0Cheb0 ? vc : xoc) + dn;
            o.xo[o3 + c] = xn;
            if (o.dot) {
                dsum += bc * xn;
                dsum2 += bc * zoc;
            }
        }
    }
    if (o.dot) cta_partials(dsum, dsum2, o.dot == 2, o.part);
}

// ---- K-cycle on a coarse level (one CTA; the level has at most a few 10k DOF)
// Two steps of a flexible CG for A x = b preconditioned by the next cycle:
//   z1 = B(b), v1 = A z1, alpha1 = z1.b / z1.v1, x = alpha1 z1, r = b - alpha1 v1;
//   z2 = B(r), v2 = A z2, w = z2 - (z2.v1 / z1.v1) z1, x += (w.r / w.Aw) w.
template <int NV>
__device__ __forceinline__ void block_sums(double (&v)[NV], double* sh /* [NV][32] */) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int k = 0; k < NV; ++k) v[k] = warp_sum(v[k]);
    if (lane == 0)
#pragma unroll
        for (int k = 0; k < NV; ++k) sh[k * 32 + w] = v[k];
    __syncthreads();
#pragma unroll
    for (int k = 0; k < NV; ++k) {  // every thread sums in the same fixed order
        double t = 0.0;
        for (int j = 0; j < nw; ++j) t += sh[k * 32 + j];
        v[k] = t;
    }
    __syncthreads();
}

__global__ void __launch_bounds__(1024) k_kcycle1(int64_t n, const double* __restrict__ b,
                                                  const double* __restrict__ z1, const double* __restrict__ v1,
                                                  double* __restrict__ x, double* __restrict__ r,
                                                  double* __restrict__ kc) {
    __shared__ double sh[2 * 32];
    double s[2] = {0.0, 0.0};
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) {
        s[0] += z1[i] * b[i];
        s[1] += z1[i] * v1[i];
    }
    block_sums<2>(s, sh);
    const double sigma = s[1];
    const double alpha = sigma > 0.0 && isfinite(sigma) ? s[0] / sigma : 0.0;
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) {
        x[i] = alpha * z1[i];
        r[i] = b[i] - alpha * v1[i];
    }
    if (threadIdx.x == 0) kc[0] = sigma;
}

__global__ void __launch_bounds__(1024) k_kcycle2(int64_t n, const double* __restrict__ z1,
                                                  const double* __restrict__ v1, const double* __restrict__ z2,
                                                  const double* __restrict__ v2, const double* __restrict__ r,
                                                  double* __restrict__ x, const double* __restrict__ kc) {
    __shared__ double sh[2 * 32];
    const double sigma = kc[0];
    double g[1] = {0.0};
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) g[0] += z2[i] * v1[i];
    block_sums<1>(g, sh);
    const double beta = sigma > 0.0 && isfinite(sigma) ? g[0] / sigma : 0.0;
    double s[2] = {0.0, 0.0};
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) {
        const double w = z2[i] - beta * z1[i];
        const double aw = v2[i] - beta * v1[i];
        s[0] += w * r[i];
        s[1] += w * aw;
    }
    block_sums<2>(s, sh);
    const double alpha = s[1] > 0.0 && isfinite(s[1]) ? s[0] / s[1] : 0.0;
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) x[i] += alpha * (z2[i] - beta * z1[i]);
}

// ---- coarse levels (row-major 6x6 block CSR): SpMV fused with the smoother
// update, one warp per block row, a lane per block of the row (coarse_row6); the
// same modes as the fine-level operator (kL0Resid, kL0RUpd, kL0Cheb0, kL0ChebK).
// Threads per CTA of the coarse-level kernels (warp per block row / aggregate).
#ifndef FX_LN_THREADS
#define FX_LN_THREADS 128
#endif
constexpr int kLnThreads = FX_LN_THREADS;
// CTAs per SM the coarse-level operators are compiled for: 4 x 128 threads leaves 128
// registers, enough for a lane's whole 6x6 block and its gathered 6-vector in flight
// without spills. On the 417k-DOF box a default solve took 51.9-52.4 ms with 4, against
// 52.9-53.2 with 6 (80 registers), 52.5-53.2 with 7 (72, spilling) and 52.3-52.5 with 8
// (64). The epilogue's operands are loaded after the row sums: before them, behind the wait for
// the kernel ahead, two of the modes spilled, at the same time per solve.
#ifndef FX_LN_MIN_BLOCKS
#define FX_LN_MIN_BLOCKS 4
#endif
constexpr int kLnMinBlocks = FX_LN_MIN_BLOCKS;
struct LnOp {
    int n;
    const int32_t* row_ptr;
    const int32_t* cols;
    const double2* vals;
    const double* v;
    const double* b;
    double* y;
    double* r;
    double* d_out;
    double* xo;
    const double* dinv;  // 6x6 block inverses
    double c1, c2;
};

template <int MODE>
__global__ void __launch_bounds__(kLnThreads, kLnMinBlocks) k_ln_op(LnOp o) {
    const int row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (row >= o.n) return;  // warp-uniform
    const int64_t o6 = 6 * (int64_t)row;
    const int c = lane < 6 ? lane : 0;
    const bool epi = lane < 6;
    double src6[6] = {0, 0, 0, 0, 0, 0}, Dr[6] = {0, 0, 0, 0, 0, 0}, vc = 0.0, xoc = 0.0, bc = 0.0;
    // lanes over the row's blocks; every lane ends with the six row sums
    const int b0 = o.row_ptr[row];
    double acc[6];
    coarse_row6<false>(o.cols, o.vals, o.v, b0, o.row_ptr[row + 1] - b0, lane, acc, ChainWait());
    // row-local operands of the epilogue
    if (epi) {
        if (MODE == kL0Cheb0 || MODE == kL0ChebK) {
            const double* src = MODE == kL0Cheb0 ? o.b : o.r;
#pragma unroll
            for (int k = 0; k < 6; ++k) {
                src6[k] = src[o6 + k];
                Dr[k] = o.dinv[36 * (int64_t)row + 6 * c + k];
            }
            vc = o.v[o6 + c];
            if (MODE == kL0ChebK) xoc = o.xo[o6 + c];
        } else if (MODE == kL0Power) {
#pragma unroll
            for (int k = 0; k < 6; ++k) Dr[k] = o.dinv[36 * (int64_t)row + 6 * c + k];
        } else if (MODE == kL0Resid) {
            bc = o.b ? o.b[o6 + c] : 0.0;
        } else {
            src6[0] = o.r[o6 + c];
        }
    }
    double axc = acc[0];
#pragma unroll
    for (int r = 1; r < 6; ++r)
        if (c == r) axc = acc[r];
    __syncwarp();  // every lane's reads of r are ordered before any lane writes r[c]
    if (!epi) return;
    if (MODE == kL0Resid) {
        o.y[o6 + c] = o.b ? bc - axc : axc;
    } else if (MODE == kL0RUpd) {
        o.r[o6 + c] = src6[0] - axc;
    } else if (MODE == kL0Power) {
        double z = 0.0;
#pragma unroll
        for (int k = 0; k < 6; ++k) z += Dr[k] * acc[k];
        o.d_out[o6 + c] = o.c2 * z;
    } else {
        double z = 0.0, rc = 0.0;
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            const double rk = src6[k] - acc[k];
            z += Dr[k] * rk;
            if (k == c) rc = rk;
        }
        o.r[o6 + c] = rc;
        const double dn = (MODE == kL0Cheb0 ? 0.0 : o.c1 * vc) + o.c2 * z;
        o.d_out[o6 + c] = dn;
        o.xo[o6 + c] = (MODE == kL0Cheb0 ? vc : xoc) + dn;
    }
}

// FP32 copy of a node's three components for the smoother's gathers; with the FP16
// scaled matrix (sq4 != null) multiplied by sqrt(a_ii) per component.
__device__ __forceinline__ float4 scaled4(const double t[3], const float4* __restrict__ sq4, int i) {
    if (!sq4) return make_float4((float)t[0], (float)t[1], (float)t[2], 0.0f);
    const float4 q = sq4[i];
    return make_float4((float)(t[0] * (double)q.x), (float)(t[1] * (double)q.y), (float)(t[2] * (double)q.z), 0.0f);
}

// Stores node i of a smoother direction: float4 per node, or with the FP16 scaled matrix
// (sq4 != null) and kL0H16Vec four halves per node (8 bytes), times hs = 2^k, in the same buffer.
__device__ __forceinline__ void store_dir4(float4* __restrict__ base, int i, const double t[3],
                                           const float4* __restrict__ sq4, float hs) {
    const float4 f = scaled4(t, sq4, i);
    if (kL0H16Vec && sq4) {
        uint2 u;
        u.x = h16_bits(f.x * hs) | (h16_bits(f.y * hs) << 16);
        u.y = h16_bits(f.z * hs);
        reinterpret_cast<uint2*>(base)[i] = u;
    } else {
        base[i] = f;
    }
}

// x4[i] = the float4 of node i's three components scaled by sqrt(a_ii) (the FP16
// operator's gathered vector), from an FP64 vector
__global__ void k_scaled4(int n, const double* __restrict__ x, const float4* __restrict__ sq4, float4* __restrict__ x4) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double t[3] = {x[3 * (int64_t)i], x[3 * (int64_t)i + 1], x[3 * (int64_t)i + 2]};
    x4[i] = scaled4(t, sq4, i);
}

// first smoothing step from x = 0 at any level: d = c2 D^-1 b; x = d; r = b
__global__ void k_cheb_start(int n, int bs, const double* __restrict__ dinv, const double* __restrict__ b,
                             double* __restrict__ r, double* __restrict__ d, double* __restrict__ x, double c2) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int64_t o = (int64_t)i * bs;
    const double* Di = dinv + (int64_t)i * bs * bs;
    for (int k = 0; k < bs; ++k) {
        double t = 0.0;
        for (int j = 0; j < bs; ++j) t += Di[k * bs + j] * b[o + j];
        t *= c2;
        d[o + k] = t;
        x[o + k] = t;
    }
    for (int k = 0; k < bs; ++k) r[o + k] = b[o + k];
}

// first pre-smoothing step from x = 0: d = c2 D^-1 b; x = d; r = b
// (d4 != null: the direction as float4 per node instead of d; hs != null: FP16 directions,
// whose scale for this V-cycle is taken from *rdr = b.D^-1 b and published in hs)
__global__ void k_l0_cheb_start(int n, const double* __restrict__ dinv, const double* __restrict__ b,
                                double* __restrict__ r, double* __restrict__ d, float4* __restrict__ d4,
                                double* __restrict__ x, double c2, const float4* __restrict__ sq4,
                                const double* __restrict__ rdr, float* __restrict__ hs) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float2 hsc = hs ? h16_scale(*rdr) : make_float2(1.0f, 1.0f);
    if (hs && i == 0) {  // read by the V-cycle's later launches only
        hs[0] = hsc.x;
        hs[1] = hsc.y;
    }
    const int64_t o3 = 3 * (int64_t)i;
    const double bb[3] = {b[o3], b[o3 + 1], b[o3 + 2]};
    const double* D = dinv + 9 * (int64_t)i;
    double t[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        t[c] = c2 * (D[3 * c] * bb[0] + D[3 * c + 1] * bb[1] + D[3 * c + 2] * bb[2]);
        r[o3 + c] = bb[c];
        x[o3 + c] = t[c];
    }
    if (d4) store_dir4(d4, i, t, sq4, hsc.x);
    else
        for (int c = 0; c < 3; ++c) d[o3 + c] = t[c];
}

// b = P^T r of the corner level (a group of lanes per corner) fused with the level's first
// pre-smoothing step from x = 0, as k_l0_cheb_start
__global__ void __launch_bounds__(256) k_corner_restrict(CornerView V, const double* rf,
                                                         double* __restrict__ b, const double* __restrict__ dinv,
                                                         double* __restrict__ r, double* __restrict__ x,
                                                         double* __restrict__ d, double c2) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x, i = t / kCornerLanes, sub = t % kCornerLanes;
    double v[3];
    corner_restrict_row<false>(V, rf, i < V.n ? i : -1, sub, v, ChainWait());
    if (i >= V.n || sub != 0) return;
    const int64_t o3 = 3 * (int64_t)i;
    const double* D = dinv + 9 * (int64_t)i;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const double u = c2 * (D[3 * c] * v[0] + D[3 * c + 1] * v[1] + D[3 * c + 2] * v[2]);
        b[o3 + c] = v[c];
        r[o3 + c] = v[c];
        x[o3 + c] = u;
        d[o3 + c] = u;
    }
}

// x += alpha P x_c from the corner level, and the FP32 copy of x for the smoother's gathers
__global__ void __launch_bounds__(256) k_corner_prolong(CornerView V, const double* xc,
                                                        double* xf, double alpha,
                                                        float4* __restrict__ x4, const float4* __restrict__ sq4) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= V.n_fine) return;
    double u[3];
    corner_prolong_node<false>(V, xc, j, u, ChainWait());
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        u[k] = xf[3 * (int64_t)j + k] + alpha * u[k];
        xf[3 * (int64_t)j + k] = u[k];
    }
    if (x4) x4[j] = scaled4(u, sq4, j);
}

// The CG update fused with the first step of the V-cycle that follows it:
// alpha = r.z / p.q from the operator's partial sums, x += alpha p, r -= alpha q, partial sums of
// r.D^-1 r, and with b = the new r: r0 = b, x0 = d = c2 D^-1 b (what k_l0_cheb_start does).
// hs != null (FP16 directions): the V-cycle's scale comes from S[2], the previous residual's
// r.D^-1 r (the new one is summed later), and is published in hs for the V-cycle's later launches.
// A thread per node, the node's operands loaded before the sum of the partials.
__global__ void __launch_bounds__(256) k_amg_update_start(int n, double* S,
                                                          const double* pq_part, int n_pq,
                                                          const double* p, const double* q,
                                                          double* x, double* r,
                                                          const double* __restrict__ dinv, double* __restrict__ part,
                                                          double* __restrict__ r0, double* __restrict__ x0,
                                                          double* __restrict__ d0, float4* __restrict__ d4,
                                                          double c2, const float4* __restrict__ sq4,
                                                          float* __restrict__ hs) {
    const int i = blockIdx.x * 256 + threadIdx.x;
    const bool own = i < n;
    const int64_t o3 = 3 * (int64_t)i;
    double pv[3], qv[3], xv[3], rv[3], D[9];
    if (own)
#pragma unroll
        for (int c = 0; c < 9; ++c) D[c] = dinv[9 * (int64_t)i + c];
    chain_wait();
    if (own) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            pv[c] = p[o3 + c];
            qv[c] = q[o3 + c];
            xv[c] = x[o3 + c];
            rv[c] = r[o3 + c];
        }
    }
    const double rz = S[8];
    const float2 hsc = hs ? h16_scale(S[2]) : make_float2(1.0f, 1.0f);
    const double pq = cta_total(pq_part, n_pq, 1, false);
    const bool ok = (pq > 0.0 && isfinite(pq)) || rz == 0.0;  // (rz = 0: the residual is zero, queued iterations idle)
    const double alpha = ok && rz != 0.0 ? rz / pq : 0.0;
    if (i == 0) {
        S[0] = rz;
        if (!ok) S[6] = 1.0;
        if (hs) {
            hs[0] = hsc.x;
            hs[1] = hsc.y;
        }
    }
    double acc = 0.0;
    if (own) {
        double t[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            x[o3 + c] = xv[c] + alpha * pv[c];
            rv[c] -= alpha * qv[c];
            r[o3 + c] = rv[c];
            r0[o3 + c] = rv[c];
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const double dr = D[3 * c] * rv[0] + D[3 * c + 1] * rv[1] + D[3 * c + 2] * rv[2];
            acc += rv[c] * dr;
            t[c] = c2 * dr;
            x0[o3 + c] = t[c];
        }
        if (d4) store_dir4(d4, i, t, sq4, hsc.x);
        else
            for (int c = 0; c < 3; ++c) d0[o3 + c] = t[c];
    }
    cta_partials(acc, 0.0, false, part);
}

// sqrt of the fine matrix's diagonal per DOF (float4 per node; 1 where a node has no
// diagonal block or a non-positive diagonal)
__global__ void k_diag_sqrt(int n, const int32_t* __restrict__ goff, const int32_t* __restrict__ diag_k,
                            const double* __restrict__ vals, float4* __restrict__ sq4) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int kk = diag_k[i];
    float o[3] = {1.f, 1.f, 1.f};
    if (kk >= 0) {
        const int64_t g0 = goff[i], ng = goff[i + 1] - g0;
        for (int c = 0; c < 3; ++c) {
            const double a = vals[(g0 * 9 + (int64_t)(4 * c) * ng + kk / 4) * 4 + (kk & 3)];
            if (a > 0.0) o[c] = (float)sqrt(a);
        }
    }
    sq4[i] = make_float4(o[0], o[1], o[2], 0.f);
}

// FP16 copy of the scaled matrix S A S, S = diag(sqrt(a_ii))^-1 with the float square
// roots of k_diag_sqrt (the smoother scales its vectors by the same values): |entries| <= 1
// for a symmetric positive definite matrix. Warp per block row; lane `it` takes plane
// e = it / ng of group g = it % ng, whose 4 values are the row's vec4 number it (planar
// layout), so a warp reads consecutive 32-byte vectors; the scale is an FP32 reciprocal
// of sqrt(a_ii) sqrt(a_jj) (its rounding, ~6e-8, is far below FP16's).
__global__ void k_vals_to_f16(int n, const int32_t* __restrict__ goff, const int32_t* __restrict__ cols,
                              const double* __restrict__ vals, const float4* __restrict__ sq4, __half* __restrict__ out) {
    const int row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (row >= n) return;
    const int64_t g0 = goff[row];
    const int ng = goff[row + 1] - (int)g0;
    const float4 sr = sq4[row];
    for (int it = lane; it < 9 * ng; it += 32) {
        const int e = it / ng, g = it - e * ng;
        const int4 cc = __ldg(reinterpret_cast<const int4*>(cols) + g0 + g);
        const int cj[4] = {cc.x, cc.y, cc.z, cc.w};
        const int cr = e / 3, ccomp = e - 3 * cr;
        const float si = cr == 0 ? sr.x : (cr == 1 ? sr.y : sr.z);
        const double2* src = reinterpret_cast<const double2*>(vals + (g0 * 9 + it) * 4);
        const double2 v01 = __ldcs(src), v23 = __ldcs(src + 1);
        const double v[4] = {v01.x, v01.y, v23.x, v23.y};
        __half h[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float4 t = __ldg(sq4 + cj[q]);
            const float sj = ccomp == 0 ? t.x : (ccomp == 1 ? t.y : t.z);
            h[q] = __double2half(v[q] * (double)(1.0f / (si * sj)));
        }
        uint2 packed;
        packed.x = (uint32_t)__half_as_ushort(h[0]) | ((uint32_t)__half_as_ushort(h[1]) << 16);
        packed.y = (uint32_t)__half_as_ushort(h[2]) | ((uint32_t)__half_as_ushort(h[3]) << 16);
        reinterpret_cast<uint2*>(out)[g0 * 9 + it] = packed;
    }
}

__global__ void k_f64_to_f32(int64_t n, const double* __restrict__ a, float* __restrict__ b) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        b[i] = (float)a[i];
}

}  // namespace

// ------------------------------------------------------------------ host side

// Grid of the level-0 operators: at most one wave of resident CTAs (grid-stride rows);
// h: the FP16-value kernels, which have their own register budget; apply: the outer CG's
// FP64 q = K p (kL0MinBlocksApply).
static unsigned l0_grid(int n, bool h = false, bool apply = false) {
    thread_local int cached_dev = -1, cached_cap[3] = {0, 0, 0};  // per host thread: contexts live on one thread each
    int dev = 0;
    FX_CUDA_CHECK(cudaGetDevice(&dev));
    if (dev != cached_dev) {
        int sms = 0, per_sm = 0, per_sm_h = 0, per_sm_a = 0;
        FX_CUDA_CHECK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        FX_CUDA_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_l0_op<double, kL0ChebK>, 256, 0));
        FX_CUDA_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm_h, k_l0_op<__half, kL0ChebK, true>, 256,
                                                                    0));
        FX_CUDA_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm_a, k_l0_op<double, kL0Apply>, 256, 0));
        cached_cap[0] = std::max(1, sms * std::max(1, per_sm));
        cached_cap[1] = std::max(1, sms * std::max(1, per_sm_h));
        cached_cap[2] = std::max(1, sms * std::max(1, per_sm_a));
        cached_dev = dev;
    }
    return (unsigned)std::min<int64_t>(grid_for((int64_t)n * kL0Lanes), cached_cap[apply ? 2 : (h ? 1 : 0)]);
}

// Slots of the partial-sum buffer a level-0 operator with a dot product needs: two per CTA
// of the largest level-0 grid (the FP16 kernels run more CTAs per SM than the others).
static int64_t l0_part_slots(int n) {
    return 2 * (int64_t)std::max({l0_grid(n, false), l0_grid(n, true), l0_grid(n, false, true)});
}

template <typename VT>
static L0Op<VT> l0_op(const AmgLevel& l, const VT* vals) {
    L0Op<VT> o{};
    o.n = l.n;
    o.goff = l.S0->goff.ptr;
    o.cols = l.S0->cols.ptr;
    o.vals = vals;
    o.dinv = l.dinv0;
    return o;
}

static LnOp ln_op(const AmgLevel& l) {
    LnOp o{};
    o.n = l.n;
    o.row_ptr = l.row_ptr.ptr;
    o.cols = l.cols.ptr;
    o.vals = l.pvals.ptr;
    o.dinv = l.dinv.ptr;
    return o;
}

static void level_spmv(const AmgLevel& l, const double* x, const double* b, double* y, cudaStream_t s) {
    if (l.S0) {
        L0Op<double> o = l0_op<double>(l, l.vals0);
        o.v = x;
        o.b = b;
        o.y = y;
        FX_LAUNCH((k_l0_op<double, kL0Resid>), l0_grid(l.n), 256, 0, s, o);
    } else {
        LnOp o = ln_op(l);
        o.v = x;
        o.b = b;
        o.y = y;
        FX_LAUNCH(k_ln_op<kL0Resid>, grid_for((int64_t)l.n * 32, kLnThreads), kLnThreads, 0, s, o);
    }
}

// Largest eigenvalue of D^-1 A by 12 power iterations from a fixed hashed start vector, one launch
// each: a step is x <- c2 D^-1 A x without a normalisation, and the eigenvalue is the ratio of the last two vectors' norms.
// (Normalised after every step, an iteration was six launches, ~18 us on a small level.) Planar levels have
// eigenvalues of at most the nodes of an element, 20, so that with c2 = 1/4 twelve steps grow a vector by at most 2.4e8;
// in FP32 it also holds the factors sqrt(a_ii) of the scaled matrix, up to 1e11 with the constraints' penalty on a
// stiffness of 1e16. The 6x6 levels, whose bound is the blocks of a row, are in FP64.
// Planar levels: the products come from the FP16 scaled matrix that the smoother reads, through
// float4 vectors, or from the FP32 copy or the FP64 values with FP64 vectors.
// warm: start from the vector the previous estimate on this level ended with (a
// refresh after a small change of the matrix) and iterate 4 times instead of 12.
static void estimate_lmax(AmgLevel& l, DBuf<double>& red, cudaStream_t s, bool warm) {
    constexpr double kStep = 0.25;
    const bool h16 = l.S0 && kAmgEstF16 && l.vals16 && l.sq4;
    const int64_t nd = (int64_t)l.n * l.bs;
    const int nb = 296;
    const bool from_ev = warm && l.ev.n == (size_t)nd;
    const int iters = from_ev ? 4 : 12;
    const double* x = from_ev ? l.ev.ptr : l.x.ptr;
    if (!from_ev) FX_LAUNCH(k_fill_hash, grid_for(nd), 256, 0, s, nd, l.x.ptr);
    float4* xa = reinterpret_cast<float4*>(l.x4.ptr);
    float4* xb = reinterpret_cast<float4*>(l.d4a.ptr);
    if (h16) FX_LAUNCH(k_scaled4, grid_for(l.n), 256, 0, s, l.n, x, l.sq4, xa);
    double* out[2] = {l.d.ptr, l.t.ptr};
    for (int it = 0; it < iters; ++it) {
        double* y = out[it & 1];
        // chained but for the first, which follows kernels that write what a chain may read early (set-up
        // of a 417k-DOF C3D20 box 2.98 and 2.86 ms, of a 45k-DOF FP64 solve 1.56 and 1.52)
        auto step = [&](auto k_power_step, unsigned grid, unsigned block, const auto& o) {
            if (it) FX_LAUNCH_CHAIN(k_power_step, grid, block, 0, s, o);
            else FX_LAUNCH(k_power_step, grid, block, 0, s, o);
        };
        if (h16) {
            L0Op<__half> o = l0_op<__half>(l, l.vals16);
            o.v4 = xa;
            o.d4_out = reinterpret_cast<float*>(xb);
            o.d_out = it >= iters - 2 ? y : nullptr;
            o.sq4 = l.sq4;
            o.c2 = kStep;
            step(k_l0_op<__half, kL0Power, true>, l0_grid(l.n, true), 256, o);
            std::swap(xa, xb);
        } else if (l.S0 && l.vals32) {
            L0Op<float> o = l0_op<float>(l, l.vals32);
            o.v = x;
            o.d_out = y;
            o.c2 = kStep;
            step(k_l0_op<float, kL0Power>, l0_grid(l.n), 256, o);
        } else if (l.S0) {
            L0Op<double> o = l0_op<double>(l, l.vals0);
            o.v = x;
            o.d_out = y;
            o.c2 = kStep;
            step(k_l0_op<double, kL0Power>, l0_grid(l.n), 256, o);
        } else {
            LnOp o = ln_op(l);
            o.v = x;
            o.d_out = y;
            o.c2 = kStep;
            step(k_ln_op<kL0Power>, grid_for((int64_t)l.n * 32, kLnThreads), kLnThreads, o);
        }
        x = y;
    }
    // |last|^2 and |last but one|^2
    if (red.n < 2 * (size_t)(nb + 1)) red.alloc(2 * (nb + 1), s);
    double* last = out[(iters - 1) & 1];
    FX_LAUNCH(k_norm2_part, nb, 256, 0, s, nd, last, out[iters & 1], red.ptr, nb);
    FX_LAUNCH(k_norm2_sum, 1, 64, 0, s, nb, red.ptr, red.ptr + 2 * nb);
    l.ev.alloc(nd, s);
    FX_LAUNCH(k_normalize, grid_for(nd), 256, 0, s, nd, red.ptr + 2 * nb, last, l.ev.ptr);
    double h[2] = {0.0, 0.0};
    FX_CUDA_CHECK(cudaMemcpyAsync(h, red.ptr + 2 * nb, sizeof(h), cudaMemcpyDeviceToHost, s));
    stream_wait(s, "amg eigenvalue estimate");
    const double q = h[0] / h[1] / (kStep * kStep);
    l.lmax = kLmaxMargin * (q > 0.0 && std::isfinite(q) ? std::sqrt(q) : 1.0);
}

// A level's matrix as the transfer kernels read it: the planar BSR3 at level 0,
// row-major 6x6 block CSR (with each block's row) above.
static FineView fine_view(const AmgLevel& l) {
    FineView F{};
    F.bs = l.bs;
    F.n = l.n;
    F.nblocks = l.nblocks;
    if (l.S0) {
        F.blk_row = l.S0->blk_row.ptr;
        F.vals = l.vals0;
        F.row_ptr = l.S0->row_ptr.ptr;
        F.goff = l.S0->goff.ptr;
        F.cols4 = l.S0->cols.ptr;
    } else {
        F.blk_row = l.blk_row.ptr;
        F.blk_col = l.cols.ptr;
        F.vals = l.vals.ptr;
        F.row_ptr = l.row_ptr.ptr;
    }
    return F;
}

// Dense inverse of the coarsest level's matrix (blocked Gauss-Jordan); fails
// with FX_NUMERICAL when the matrix is singular (rigid-body modes).
void Amg::coarsest_inverse(AmgLevel& l, cudaStream_t s) {
    const int64_t nd = (int64_t)l.n * l.bs;
    l.dense_inv.alloc((size_t)nd * nd, s);
    l.dense_inv.zero(s);
    if (l.S0)
        FX_LAUNCH(k_dense_from_planar, grid_for((int64_t)l.n * 32, 128), 128, 0, s, l.n, l.S0->row_ptr.ptr,
                  l.S0->goff.ptr, l.S0->cols.ptr, l.vals0, l.dense_inv.ptr);
    else
        FX_LAUNCH(k_dense_from_bsr<6>, grid_for((int64_t)l.n * 32, 128), 128, 0, s, l.n, l.row_ptr.ptr, l.cols.ptr,
                  l.vals.ptr, l.dense_inv.ptr);
    DBuf<uint8_t> dead;
    dead.alloc(nd, s);
    DBuf<double> diag0, other, pivot;
    DBuf<int> singular;
    diag0.alloc(nd, s);
    singular.alloc(1, s);
    singular.zero(s);
    other.alloc((size_t)nd * nd, s);
    pivot.alloc(2 * kPanel * kPanel, s);
    FX_LAUNCH(k_dense_decouple, 1, 1024, 0, s, (int)nd, l.S0 ? 0.0 : 1e-12, l.dense_inv.ptr, dead.ptr, diag0.ptr);
    double* P[2] = {pivot.ptr, pivot.ptr + kPanel * kPanel};
    FX_LAUNCH(k_gj_first, 1, 256, 0, s, (int)nd, l.dense_inv.ptr, diag0.ptr, singular.ptr, P[0]);
    const dim3 tiles(grid_for(nd, kPanel), grid_for(nd, kTileRows));
    for (int k0 = 0; k0 < (int)nd; k0 += kPanel) {
        FX_LAUNCH_CHAIN(k_gj_panel, tiles, 256, 0, s, (int)nd, k0, l.dense_inv.ptr, other.ptr, P[0], P[1], diag0.ptr,
                  singular.ptr);
        l.dense_inv.swap(other);
        std::swap(P[0], P[1]);
    }
    FX_LAUNCH(k_dense_zero_dead, grid_for(nd * 32), 256, 0, s, (int)nd, l.dense_inv.ptr, dead.ptr);
    int sing = 0;
    FX_CUDA_CHECK(cudaMemcpyAsync(&sing, singular.ptr, sizeof(int), cudaMemcpyDeviceToHost, s));
    stream_wait(s, "amg coarse inverse");
    if (sing)
        fail(FX_NUMERICAL, "Mathematical error: the multigrid coarse operator is singular (system not "
                           "positive definite). Check for rigid body modes!");
}

// The grid of cells with edges near `cell` over a box of these extents.
static CellGrid cell_grid(const double extent[3], double cell) {
    CellGrid g{};
    for (int d = 0; d < 3; ++d) {
        const double parts = extent[d] > 0.0 && cell > 0.0 ? extent[d] / cell : 1.0;
        g.k[d] = (int)std::min(1048576.0, std::max(1.0, std::floor(parts + 0.5)));
        g.inv[d] = extent[d] > 0.0 ? g.k[d] / extent[d] : 0.0;
    }
    return g;
}

// Edge of the aggregation cells of a level when the caller leaves it open: `extent` of the level's
// points, lo .. hi the edges that pay and mid the usual one. A level whose cells fit the dense
// coarsest solve ends the hierarchy, which saves the six launches per V-cycle of a level between
// (~2.5 us each on a small system), so the smallest such edge is taken while it is at most hi
// (with larger cells the CG needs more iterations than the launches are worth); otherwise mid.
// The cell count is that of a box of these extents, an upper bound for other shapes.
static double pick_cell(const double extent[3], double lo, double mid, double hi) {
    auto fits = [&](double c) {
        const CellGrid g = cell_grid(extent, c);
        return (double)g.k[0] * g.k[1] * g.k[2] * 6.0 <= kCoarseMaxDof;
    };
    if (!fits(hi)) return mid;
    if (fits(lo)) return lo;
    double a = lo, b = hi;
    for (int k = 0; k < 30; ++k) {
        const double m = 0.5 * (a + b);
        (fits(m) ? b : a) = m;
    }
    return b;
}

static void planar_values(AmgLevel& l, cudaStream_t s) {
    l.pvals.alloc((size_t)l.nblocks * 18, s);
    FX_LAUNCH(k_planar6, grid_for((int64_t)l.n * 32, 128), 128, 0, s, l.n, l.row_ptr.ptr, l.vals.ptr, l.pvals.ptr);
}

static void set_planar(AmgLevel& l, const PlanarIn& in) {
    l.n = in.S->n_rows;
    l.bs = 3;
    l.S0 = in.S;
    l.nblocks = in.S->n_blocks;
    l.vals0 = in.vals;
    l.dinv0 = in.dinv;
    l.vals32 = in.vals32;
    l.vals16 = in.vals16;
    l.sq4 = in.sq4;
}

static void planar_work(AmgLevel& l, bool result, cudaStream_t s) {
    const int64_t nd = 3 * (int64_t)l.n;
    for (DBuf<double>* v : {&l.x, &l.b, &l.r, &l.d, &l.t}) v->alloc(nd, s);
    if (result) l.xs.alloc(nd, s);
    if (!l.vals32 && !l.vals16) return;
    for (DBuf<float>* v : {&l.d4a, &l.d4b, &l.x4}) {
        v->alloc(4 * (size_t)l.n, s);
        v->zero(s);  // the fourth component stays 0
    }
}

void Amg::setup(const PlanarIn* in, const CornerLevel* corner, const double* xyz, double cell0, double node_volume,
                bool dense, cudaStream_t s, AmgStats* st) {
    EventTimer timer;
    timer.start(s);
    auto done = [&] {
        if (st) {
            st->levels = (int)L.size();
            st->sizes.clear();
            for (auto& l : L) st->sizes.push_back(l.n * l.bs);
            st->setup_ms = timer.stop_ms(s);
        }
    };
    L.clear();
    L.reserve(kMaxLevels + 1);
    planar_ = corner ? 2 : 1;
    corner_ = corner ? corner_view(*corner) : CornerView{};
    for (int m = 0; m < planar_; ++m) {
        L.emplace_back();
        set_planar(L[m], in[m]);
        planar_work(L[m], m > 0, s);
        if (m + 1 < planar_) {
            L[m].corner_next = true;
            L[m].pscale = 1.0 / kAmgOvercorrect;
            estimate_lmax(L[m], red_, s, false);
        }
    }
    if (dense && cell0 <= 0.0 && !tentative_ && dense_planar(L.back().n)) {
        AmgLevel& l = L.back();
        l.lmax = 1.0;  // (no smoothing here)
        l.coarsest = true;
        coarsest_inverse(l, s);
        done();
        return;
    }
    // the points of the last planar level and their bounding box (cell keys of every level are
    // taken from its lower corner)
    DBuf<double> coords, cent, Rprev, Rnext;
    DBuf<unsigned long long> box;
    const int n_points = L.back().n;
    coords.alloc(3 * (size_t)n_points, s);
    FX_CUDA_CHECK(cudaMemcpyAsync(coords.ptr, xyz, 3 * (size_t)n_points * sizeof(double), cudaMemcpyDeviceToDevice, s));
    box.alloc(6, s);
    FX_CUDA_CHECK(cudaMemsetAsync(box.ptr, 0xff, 3 * sizeof(unsigned long long), s));
    FX_CUDA_CHECK(cudaMemsetAsync(box.ptr + 3, 0, 3 * sizeof(unsigned long long), s));
    FX_LAUNCH(k_box, std::min(148u, grid_for(n_points)), 256, 0, s, n_points, coords.ptr, box.ptr);
    unsigned long long hbox[6];
    FX_CUDA_CHECK(cudaMemcpyAsync(hbox, box.ptr, sizeof(hbox), cudaMemcpyDeviceToHost, s));
    double cell = cell0, extent[3] = {0.0, 0.0, 0.0};
    bool smooth = true;
    for (int lev = planar_ - 1;; ++lev) {
        AmgLevel& l = L[lev];
        const int64_t nd = (int64_t)l.n * l.bs;
        if (!l.S0) {
            for (DBuf<double>* v : {&l.x, &l.b, &l.r, &l.d, &l.t, &l.xs}) v->alloc(nd, s);
            l.dinv.alloc((size_t)l.n * 36, s);
            FX_LAUNCH(k_block_inv6, grid_for(l.n, 128), 128, 0, s, l.n, l.row_ptr.ptr, l.cols.ptr, l.vals.ptr,
                      l.dinv.ptr);
        }
        if (!l.S0 && (nd <= kCoarseMaxDof || lev + 1 >= kMaxLevels)) {
            l.coarsest = true;
            coarsest_inverse(l, s);
            break;
        }
        if (!l.S0) planar_values(l, s);
        estimate_lmax(l, red_, s, false);  // (its host wait also covers the bounding box)
        if (lev == planar_ - 1)
            for (int d = 0; d < 3; ++d) {
                double lohi[2];
                for (int k = 0; k < 2; ++k) {
                    const unsigned long long u = unordered_bits(hbox[3 * k + d]);
                    std::memcpy(&lohi[k], &u, sizeof(double));
                }
                extent[d] = std::isfinite(lohi[1] - lohi[0]) ? std::max(0.0, lohi[1] - lohi[0]) : 0.0;
            }
        if (cell0 <= 0.0) {
            // 20 to 80 nodes per cell, else 27 (three per direction on a regular mesh); above, cells of
            // twice to 3.5 times the edge of the level before, else three times
            const double h = std::cbrt(node_volume);
            cell = lev == planar_ - 1 ? pick_cell(extent, std::cbrt(20.0) * h, 3.0 * h, std::cbrt(80.0) * h)
                                      : pick_cell(extent, 2.0 * cell, 3.0 * cell, 3.5 * cell);
        }
        // ---- aggregation by cells
        DBuf<uint64_t> keys, keys_s;
        DBuf<int32_t> ids, ids_s, head, rank1;
        int na = 0;
        while (true) {
            keys.alloc(l.n, s);
            keys_s.alloc(l.n, s);
            ids.alloc(l.n, s);
            ids_s.alloc(l.n, s);
            const CellGrid grid = cell_grid(extent, cell);
            int bits = 1;
            while (bits < 63 && std::ldexp(1.0, bits) < (double)grid.k[0] * grid.k[1] * grid.k[2]) ++bits;
            FX_LAUNCH(k_cell_keys, grid_for(l.n), 256, 0, s, l.n, coords.ptr, box.ptr, grid, keys.ptr, ids.ptr);
            cub_call([&](void* t, size_t& b) {
                return cub::DeviceRadixSort::SortPairs(t, b, keys.ptr, keys_s.ptr, ids.ptr, ids_s.ptr, l.n, 0, bits, s);
            }, tmp_, s);
            head.alloc(l.n, s);
            rank1.alloc(l.n, s);
            FX_LAUNCH(k_heads64, grid_for(l.n), 256, 0, s, l.n, keys_s.ptr, head.ptr);
            cub_call([&](void* t, size_t& b) { return cub::DeviceScan::InclusiveSum(t, b, head.ptr, rank1.ptr, l.n, s); },
                     tmp_, s);
            FX_CUDA_CHECK(cudaMemcpyAsync(&na, rank1.ptr + l.n - 1, sizeof(int), cudaMemcpyDeviceToHost, s));
            stream_wait(s, "amg aggregates");
            if (na < l.n) break;
            // cells too small to aggregate: grow and retry (a single cell in the end)
            if (l.n <= 1) fail(FX_GENERIC, "multigrid: a single block row cannot be coarsened");
            cell *= 1.5;
        }
        DBuf<int32_t> agg, agg_ptr;
        agg.alloc(l.n, s);
        agg_ptr.alloc(na + 1, s);
        FX_LAUNCH(k_agg_assign, grid_for(l.n), 256, 0, s, l.n, rank1.ptr, head.ptr, ids_s.ptr, agg.ptr, agg_ptr.ptr);
        FX_CUDA_CHECK(cudaMemcpyAsync(agg_ptr.ptr + na, &l.n, sizeof(int), cudaMemcpyHostToDevice, s));
        cent.alloc((size_t)na * 3, s);
        FX_LAUNCH(k_agg_centroid, grid_for(na), 256, 0, s, na, agg_ptr.ptr, ids_s.ptr, coords.ptr, cent.ptr);
        // ---- tentative prolongator
        DBuf<double> Q;
        Q.alloc((size_t)nd * 6, s);
        Rnext.alloc((size_t)na * 36, s);
        FX_LAUNCH(k_agg_qr, grid_for(na, kQrWarps), 32 * kQrWarps, 0, s, na, agg_ptr.ptr, ids_s.ptr, l.bs, coords.ptr,
                  cent.ptr, Rprev.ptr, Q.ptr, Rnext.ptr);
        // ---- smoothed prolongator, coarse pattern and Galerkin coarse matrix
        if (!l.S0) {
            l.blk_row.alloc(l.nblocks, s);
            FX_LAUNCH(k_expand_rows, grid_for(l.n), 256, 0, s, l.n, l.row_ptr.ptr, l.blk_row.ptr);
        }
        if (l.S0) smooth = cell0 <= 0.0 || l.n <= kSmoothRows || l.n >= kSmoothMembers * na;
        else if (planar_ == 2) smooth = true;
        smooth &= !tentative_;
        L.emplace_back();
        AmgLevel& c = L.back();
        AmgLevel& lf = L[L.size() - 2];
        const bool smoothed = build_transfer(fine_view(lf), na, agg.ptr, Q.ptr, lf.dinv_ptr(), kSmoothOmega / lf.lmax,
                                             smooth, lf.tr, c.row_ptr, c.cols, &c.nblocks, tmp_, s);
        lf.pscale = smoothed ? 1.0 / kAmgOvercorrect : 1.0;
        c.n = na;
        c.bs = 6;
        c.vals.alloc((size_t)c.nblocks * 36, s);
        galerkin_product(fine_view(lf), lf.tr, c.row_ptr.ptr, c.cols.ptr, c.vals.ptr, s);
        // next level points and near-null-space
        coords = std::move(cent);
        Rprev = std::move(Rnext);
        if (cell0 > 0.0) cell *= 2.0;
    }
    if ((int)L.size() > planar_ + 1) {  // K-cycle work vectors on the first 6x6 level
        AmgLevel& l1 = L[planar_];
        const int64_t nd1 = (int64_t)l1.n * l1.bs;
        for (auto& v : l1.kc) v.alloc(nd1, s);
        l1.kcs.alloc(8, s);
        l1.kcs.zero(s);
    }
    done();
}

void Amg::refresh(const PlanarIn* in, cudaStream_t s, AmgStats* st) {
    EventTimer timer;
    timer.start(s);
    for (int m = 0; m < planar_; ++m) set_planar(L[m], in[m]);
    for (size_t lev = 0; lev < L.size(); ++lev) {  // the numeric steps of setup(), in its order
        AmgLevel& l = L[lev];
        if (!l.S0)
            FX_LAUNCH(k_block_inv6, grid_for(l.n, 128), 128, 0, s, l.n, l.row_ptr.ptr, l.cols.ptr, l.vals.ptr,
                      l.dinv.ptr);
        if (l.coarsest) {
            coarsest_inverse(l, s);
            break;
        }
        if (!l.S0) planar_values(l, s);
        estimate_lmax(l, red_, s, true);
        if (!l.corner_next)
            galerkin_product(fine_view(l), l.tr, L[lev + 1].row_ptr.ptr, L[lev + 1].cols.ptr, L[lev + 1].vals.ptr, s);
    }
    if (st) {
        st->levels = (int)L.size();
        st->sizes.clear();
        for (auto& l : L) st->sizes.push_back(l.n * l.bs);
        st->setup_ms = timer.stop_ms(s);
    }
}

void Amg::keep(const PlanarIn& fine, AmgStats* st) {
    set_planar(L[0], fine);
    if (st) {
        st->levels = (int)L.size();
        st->sizes.clear();
        for (auto& l : L) st->sizes.push_back(l.n * l.bs);
        st->setup_ms = 0.0;
    }
}

// Chebyshev polynomial smoother on D^-1 A over [lmax/30, lmax] (degree = steps):
// d_1 = D^-1 r_0 / theta, then r_k = r_{k-1} - A d_k,
// d_{k+1} = rho_k rho_{k-1} d_k + (2 rho_k / delta) D^-1 r_k with
// rho_0 = delta / theta, rho_k = 1 / (2 theta / delta - rho_{k-1}); x += every d.
struct ChebCoef {
    double c2_start;
    double c1[8], c2[8];
};
// kind 1: fourth-kind Chebyshev smoother (Lottes, "Optimal polynomial smoothers
// for multigrid V-cycles", Numer. Linear Algebra Appl. 2023): d_1 = 4/(3 rho)
// D^-1 r_0, d_k = (2k-3)/(2k+1) d_{k-1} + (8k-4)/((2k+1) rho) D^-1 r_{k-1}, rho =
// the lambda_max estimate; no lower eigenvalue bound needed.
static ChebCoef cheb_coef(double lmax, int degree, int kind, double ratio) {
    if (kind == 1) {
        ChebCoef k{};
        k.c2_start = 4.0 / (3.0 * lmax);
        for (int s = 1; s < degree; ++s) {
            const int i = s + 1;  // step index of the recurrence (the start is step 1)
            k.c1[s] = (2.0 * i - 3.0) / (2.0 * i + 1.0);
            k.c2[s] = (8.0 * i - 4.0) / ((2.0 * i + 1.0) * lmax);
        }
        return k;
    }
    const double lmin = lmax / ratio;
    const double theta = 0.5 * (lmax + lmin), delta = 0.5 * (lmax - lmin);
    const double sigma = theta / delta;
    ChebCoef k{};
    k.c2_start = 1.0 / theta;
    double rho = 1.0 / sigma;
    for (int s = 1; s < degree; ++s) {
        const double rho1 = 1.0 / (2.0 * sigma - rho);
        k.c1[s] = rho1 * rho;
        k.c2[s] = 2.0 * rho1 / delta;
        rho = rho1;
    }
    return k;
}

// Cycle at a coarse level (6x6 blocks) for A x = b (b and x of that level's size):
// Chebyshev pre-smoothing from x = 0 into the scratch iterate xs (start kernel,
// then SpMVs fused with the updates), the residual, the coarse correction added
// to xs, and post-smoothing that reads xs and writes the result into x.
CoarseStart Amg::coarse_start(int m) const {
    CoarseStart cs{};
    const AmgLevel& c = L[m];
    if (c.coarsest || (kcycle_ && m == planar_)) return cs;  // dense solve; K-cycle calls the cycle on other vectors
    cs.dinv = c.dinv.ptr;
    cs.r = c.r.ptr;
    cs.d = c.d.ptr;
    cs.xs = c.xs.ptr;
    cs.c2 = cheb_coef(c.lmax, degree_, cheb_kind_, cheb_ratio_).c2_start;
    return cs;
}

void Amg::cycle(int lev, const double* b, double* x, cudaStream_t s, bool started) {
    AmgLevel& l = L[lev];
    const int64_t nd = (int64_t)l.n * l.bs;
    if (l.coarsest) {
        FX_LAUNCH_CHAIN(k_dense_matvec, grid_for(nd * 32, kLnThreads), kLnThreads, 0, s, (int)nd, l.dense_inv.ptr, b, x);
        return;
    }
    AmgLevel& c = L[lev + 1];
    // coarse_row6 reads the gathered 6-vectors as 16-byte pairs
    if ((reinterpret_cast<uintptr_t>(l.d.ptr) |
         reinterpret_cast<uintptr_t>(l.t.ptr) | reinterpret_cast<uintptr_t>(l.xs.ptr)) & 15)
        fail(FX_GENERIC, "multigrid: coarse-level buffers not 16-byte aligned");
    const ChebCoef k = cheb_coef(l.lmax, degree_, cheb_kind_, cheb_ratio_);
    const unsigned grid = grid_for((int64_t)l.n * 32, kLnThreads);
    double* dA = l.d.ptr;
    double* dB = l.t.ptr;
    double* xs = l.xs.ptr;
    if (!started)
        FX_LAUNCH(k_cheb_start, grid_for(l.n), 256, 0, s, l.n, l.bs, l.dinv.ptr, b, l.r.ptr, dA, xs, k.c2_start);
    for (int st = 1; st < degree_; ++st) {
        LnOp o = ln_op(l);
        o.v = dA;
        o.r = l.r.ptr;
        o.d_out = dB;
        o.xo = xs;
        o.c1 = k.c1[st];
        o.c2 = k.c2[st];
        FX_LAUNCH_CHAIN(k_ln_op<kL0ChebK>, grid, kLnThreads, 0, s, o);
        std::swap(dA, dB);
    }
    {
        LnOp o = ln_op(l);
        o.v = dA;
        o.r = l.r.ptr;
        FX_LAUNCH_CHAIN(k_ln_op<kL0RUpd>, grid, kLnThreads, 0, s, o);  // r = b - A xs
    }
    FX_LAUNCH_CHAIN(k_restrict<6>, (unsigned)l.tr.na, 32 * kRestrictWarps, 0, s, l.tr.t_ptr.ptr, l.tr.t_row.ptr,
              l.tr.t_val32.ptr, l.r.ptr, c.b.ptr, coarse_start(lev + 1));
    coarse(lev + 1, s);
    FX_LAUNCH_CHAIN(k_prolong<6>, grid_for(l.n, kProlongRows<6>), 256, 0, s, l.n, l.tr.ptr.ptr, l.tr.col.ptr,
              l.tr.val32.ptr, c.x.ptr, xs,
              alpha_ * pscale(l), nullptr, nullptr);
    {
        LnOp o = ln_op(l);
        o.v = xs;
        o.b = b;
        o.r = l.r.ptr;
        o.d_out = dA;
        o.xo = x;
        o.c2 = k.c2_start;
        FX_LAUNCH_CHAIN(k_ln_op<kL0Cheb0>, grid, kLnThreads, 0, s, o);
    }
    for (int st = 1; st < degree_; ++st) {
        LnOp o = ln_op(l);
        o.v = dA;
        o.r = l.r.ptr;
        o.d_out = dB;
        o.xo = x;
        o.c1 = k.c1[st];
        o.c2 = k.c2[st];
        FX_LAUNCH_CHAIN(k_ln_op<kL0ChebK>, grid, kLnThreads, 0, s, o);
        std::swap(dA, dB);
    }
}

// Coarse correction at 6x6 level m: L[m].x ~ A_m^-1 L[m].b, by a K-cycle at the first
// such level (when it is not the coarsest) and V-cycles below.
void Amg::coarse(int m, cudaStream_t s) {
    AmgLevel& l = L[m];
    if (!(kcycle_ && m == planar_ && !l.coarsest)) {
        cycle(m, l.b.ptr, l.x.ptr, s, coarse_start(m).dinv != nullptr);
        return;
    }
    const int64_t nd = (int64_t)l.n * l.bs;
    double *z1 = l.kc[0].ptr, *v1 = l.kc[1].ptr, *r = l.kc[2].ptr, *z2 = l.kc[3].ptr, *v2 = l.kc[4].ptr;
    cycle(m, l.b.ptr, z1, s);
    level_spmv(l, z1, nullptr, v1, s);
    FX_LAUNCH(k_kcycle1, 1, 1024, 0, s, nd, l.b.ptr, z1, v1, l.x.ptr, r, l.kcs.ptr);
    cycle(m, r, z2, s);
    level_spmv(l, z2, nullptr, v2, s);
    FX_LAUNCH(k_kcycle2, 1, 1024, 0, s, nd, z1, v1, z2, v2, r, l.x.ptr, l.kcs.ptr);
}

// The first 6x6 level's correction of the last planar level: restriction of its residual, the
// coarse cycle, prolongation into its iterate (and the FP32 copy for the smoother's gathers).
void Amg::first_coarse(cudaStream_t s) {
    AmgLevel& l = L[planar_ - 1];
    AmgLevel& c = L[planar_];
    const bool g32 = l.vals32 || l.vals16;
    if (fused_coarse_ && !kcycle_ && desc_.ptr) {  // one launch
        launch_coarse_grid(desc_.ptr, gbar_.ptr, gflag_, g32, degree_, alpha_, s);
        return;
    }
    FX_LAUNCH_CHAIN(k_restrict<3>, (unsigned)l.tr.na, 32 * kRestrictWarps, 0, s, l.tr.t_ptr.ptr, l.tr.t_row.ptr,
              l.tr.t_val32.ptr, l.r.ptr, c.b.ptr, coarse_start(planar_));
    coarse(planar_, s);
    FX_LAUNCH_CHAIN(k_prolong<3>, grid_for(l.n, kProlongRows<3>), 256, 0, s, l.n, l.tr.ptr.ptr, l.tr.col.ptr,
              l.tr.val32.ptr, c.x.ptr, l.x.ptr, alpha_ * pscale(l), g32 ? l.x4.ptr : nullptr, l.sq4);
}

// A planar level with the fused operators: pre-smoothing from x = 0 (one elementwise
// start, degree-1 fused steps, one fused residual update), coarse correction,
// post-smoothing written straight into z. With part != null (level 0) the last step also
// leaves the partial sums of r.z for the outer CG.
template <typename VT>
void Amg::vcycle_of(int m, const double* b, double* z, double* part, const double* zold, cudaStream_t s,
                    bool started) {
    AmgLevel& l = L[m];
    if (l.coarsest) {  // z = A^-1 b
        const int64_t nd = 3 * (int64_t)l.n;
        FX_LAUNCH_CHAIN(k_dense_matvec, grid_for(nd * 32, kLnThreads), kLnThreads, 0, s, (int)nd, l.dense_inv.ptr, b, z);
        if (part) FX_LAUNCH_CHAIN(k_pair_part, apply_grid(), 256, 0, s, nd, b, z, zold, part);
        return;
    }
    const VT* vals;
    if constexpr (std::is_same<VT, __half>::value) vals = l.vals16;
    else if constexpr (std::is_same<VT, float>::value) vals = l.vals32;
    else vals = l.vals0;
    const ChebCoef k = cheb_coef(l.lmax, degree_, cheb_kind_, cheb_ratio_);
    const unsigned grid = l0_grid(l.n, std::is_same<VT, __half>::value);
    // FP32 or FP16 values: the smoother's gathered vectors are FP32 (float4 per node),
    // with FP16 values FP16 directions (kL0H16Vec) scaled by the V-cycle's power of two
    constexpr bool g32 = !std::is_same<VT, double>::value;
    float* hs = std::is_same<VT, __half>::value ? h16_scale_slot() : nullptr;
    double* dA = l.d.ptr;
    double* dB = l.t.ptr;
    float4* dA4 = reinterpret_cast<float4*>(l.d4a.ptr);
    float4* dB4 = reinterpret_cast<float4*>(l.d4b.ptr);
    float4* x4 = reinterpret_cast<float4*>(l.x4.ptr);
    if (!started)
        FX_LAUNCH(k_l0_cheb_start, grid_for(l.n), 256, 0, s, l.n, l.dinv0, b, l.r.ptr, dA, g32 ? dA4 : nullptr,
                  l.x.ptr, k.c2_start, l.sq4, rdr_, hs);
    auto op = [&]() {
        L0Op<VT> o = l0_op<VT>(l, vals);
        o.sq4 = l.sq4;
        o.hs = hs;
        return o;
    };
    for (int st = 1; st < degree_; ++st) {
        L0Op<VT> o = op();
        o.v = dA;
        o.v4 = dA4;
        o.r = l.r.ptr;
        o.d_out = dB;
        o.d4_out = reinterpret_cast<float*>(dB4);
        o.xo = l.x.ptr;
        o.c1 = k.c1[st];
        o.c2 = k.c2[st];
        FX_LAUNCH_CHAIN((k_l0_op<VT, kL0ChebK, g32>), grid, 256, 0, s, o);
        std::swap(dA, dB);
        std::swap(dA4, dB4);
    }
    {
        L0Op<VT> o = op();
        o.v = dA;
        o.v4 = dA4;
        o.r = l.r.ptr;
        FX_LAUNCH_CHAIN((k_l0_op<VT, kL0RUpd, g32>), grid, 256, 0, s, o);  // r = b - A x
    }
    if (l.corner_next) {
        AmgLevel& c = L[m + 1];
        FX_LAUNCH_CHAIN(k_corner_restrict, grid_for((int64_t)c.n * kCornerLanes), 256, 0, s, corner_, l.r.ptr, c.b.ptr,
                        c.dinv0, c.r.ptr, c.x.ptr, c.d.ptr, cheb_coef(c.lmax, degree_, cheb_kind_, cheb_ratio_).c2_start);
        vcycle(m + 1, c.b.ptr, c.xs.ptr, nullptr, nullptr, s, true);
        FX_LAUNCH_CHAIN(k_corner_prolong, grid_for(l.n), 256, 0, s, corner_, c.result(), l.x.ptr, alpha_ * pscale(l),
                  g32 ? x4 : nullptr, l.sq4);
    } else {
        first_coarse(s);
    }
    for (int st = 0; st < degree_; ++st) {
        L0Op<VT> o = op();
        o.b = b;
        o.r = l.r.ptr;
        o.xo = z;
        if (st == 0) {  // from the iterate: r = b - A x, d = D^-1 r / theta, z = x + d
            o.v = l.x.ptr;
            o.v4 = x4;
            o.d_out = dA;
            o.d4_out = reinterpret_cast<float*>(dA4);
            o.c2 = k.c2_start;
        } else {
            o.v = dA;
            o.v4 = dA4;
            o.d_out = dB;
            o.d4_out = reinterpret_cast<float*>(dB4);
            o.c1 = k.c1[st];
            o.c2 = k.c2[st];
        }
        if (st == degree_ - 1 && part) {
            if (2 * (int64_t)grid > part_slots_)
                fail(FX_GENERIC, "multigrid: partial-sum buffer smaller than the smoother grid");
            o.dot = 2;
            o.zold = zold;
            o.part = part;
        }
        if (st == 0) FX_LAUNCH_CHAIN((k_l0_op<VT, kL0Cheb0, g32>), grid, 256, 0, s, o);
        else {
            FX_LAUNCH_CHAIN((k_l0_op<VT, kL0ChebK, g32>), grid, 256, 0, s, o);
            std::swap(dA, dB);
            std::swap(dA4, dB4);
        }
    }
}

void Amg::vcycle(int m, const double* b, double* z, double* part, const double* zold, cudaStream_t s, bool started) {
    if (L[m].vals16) vcycle_of<__half>(m, b, z, part, zold, s, started);
    else if (L[m].vals32) vcycle_of<float>(m, b, z, part, zold, s, started);
    else vcycle_of<double>(m, b, z, part, zold, s, started);
}

void Amg::apply(const double* r, double* z, double* part, const double* zold, cudaStream_t s, bool started) {
    vcycle(0, r, z, part, zold, s, started);
}

unsigned Amg::apply_grid() const { return l0_grid(L[0].n, L[0].vals16 != nullptr); }

Amg::Start0 Amg::start0() const {
    const AmgLevel& l = L[0];
    Start0 o{};
    o.r = l.r.ptr;
    o.x = l.x.ptr;
    o.d = l.d.ptr;
    o.d4 = l.vals32 || l.vals16 ? reinterpret_cast<float4*>(l.d4a.ptr) : nullptr;
    o.c2 = cheb_coef(l.lmax, degree_, cheb_kind_, cheb_ratio_).c2_start;
    o.sq4 = l.sq4;
    o.hs = l.vals16 ? h16_scale_slot() : nullptr;
    return o;
}

// the scale slot of FP16 smoother directions (null: the directions are FP32, or unscaled)
float* Amg::h16_scale_slot() const { return kL0H16Vec && rdr_ ? hs_ : nullptr; }

// ------------------------------------------------------------------ AMG-preconditioned CG (FP64)

double profile_smoother_op(const BsrStructure& S, const double* vals64, const double* dinv64, bool fp32, bool fp16,
                           int reps, cudaStream_t s, double* bytes) {
    fp32 = fp32 || fp16;
    const int n = S.n_rows;
    const int64_t nd = 3 * (int64_t)n;
    DBuf<float> v32;
    DBuf<__half> v16;
    DBuf<float4> sq4;
    if (fp16) {
        sq4.alloc((size_t)n, s);
        FX_LAUNCH(k_diag_sqrt, grid_for(n), 256, 0, s, n, S.goff.ptr, S.diag_k.ptr, vals64, sq4.ptr);
        v16.alloc((size_t)S.n_groups * 36, s);
        FX_LAUNCH(k_vals_to_f16, grid_for((int64_t)n * 32), 256, 0, s, n, S.goff.ptr, S.cols.ptr, vals64, sq4.ptr,
                  v16.ptr);
    } else if (fp32) {
        const int64_t nv = (int64_t)S.n_groups * 36;
        v32.alloc(nv, s);
        FX_LAUNCH(k_f64_to_f32, 148 * 8, 256, 0, s, nv, vals64, v32.ptr);
    }
    DBuf<double> v, r, d, xo;
    for (DBuf<double>* b : {&v, &r, &d, &xo}) {
        b->alloc(nd, s);
        FX_LAUNCH(k_fill_hash, grid_for(nd), 256, 0, s, nd, b->ptr);
    }
    DBuf<float> v4, d4;  // FP32 smoother vectors (float4 per node), as in the V-cycle
    if (fp32) {
        v4.alloc(4 * (size_t)n, s);
        d4.alloc(4 * (size_t)n, s);
        v4.zero(s);
        d4.zero(s);
    }
    AmgLevel l;
    l.n = n;
    l.S0 = &S;
    l.vals0 = vals64;
    l.dinv0 = dinv64;
    const unsigned grid = l0_grid(n, fp16);
    auto launch = [&]() {
        if (fp16) {
            L0Op<__half> o = l0_op<__half>(l, v16.ptr);
            o.v = v.ptr;
            o.v4 = reinterpret_cast<const float4*>(v4.ptr);
            o.r = r.ptr;
            o.d_out = d.ptr;
            o.d4_out = d4.ptr;
            o.xo = xo.ptr;
            o.c1 = 0.5;
            o.c2 = 1e-9;
            o.sq4 = sq4.ptr;
            FX_LAUNCH((k_l0_op<__half, kL0ChebK, true>), grid, 256, 0, s, o);
        } else if (fp32) {
            L0Op<float> o = l0_op<float>(l, v32.ptr);
            o.v = v.ptr;
            o.v4 = reinterpret_cast<const float4*>(v4.ptr);
            o.r = r.ptr;
            o.d_out = d.ptr;
            o.d4_out = d4.ptr;
            o.xo = xo.ptr;
            o.c1 = 0.5;
            o.c2 = 1e-9;
            FX_LAUNCH((k_l0_op<float, kL0ChebK, true>), grid, 256, 0, s, o);
        } else {
            L0Op<double> o = l0_op<double>(l, vals64);
            o.v = v.ptr;
            o.r = r.ptr;
            o.d_out = d.ptr;
            o.xo = xo.ptr;
            o.c1 = 0.5;
            o.c2 = 1e-9;
            FX_LAUNCH((k_l0_op<double, kL0ChebK>), grid, 256, 0, s, o);
        }
    };
    for (int k = 0; k < 3; ++k) launch();
    EventTimer t;
    t.start(s);
    for (int k = 0; k < reps; ++k) launch();
    const double ms = t.stop_ms(s) / reps;
    // compulsory bytes: matrix values + column indices once, row offsets, and per
    // node the gathered direction (24 B FP64 / 16 B float4), r read+write (48), the
    // new direction (24 / 16), iterate read+write (48) and the 3x3 block inverse (72)
    // (FP16: 2-byte values, the 16-byte scales of each row, and with kL0H16Vec 8-byte
    // directions gathered and written)
    const double vb = fp16 ? 2.0 : (fp32 ? 4.0 : 8.0);
    const double per_node = fp16 && kL0H16Vec ? 184.0 : (fp32 ? 200.0 : 216.0);
    *bytes = (double)S.n_blocks * (9.0 * vb + 4.0) + 4.0 * (n + 1) + per_node * n + (fp16 ? 16.0 * n : 0.0);
    return ms;
}

static ClTransfer cl_transfer(const AmgLevel& l, double pscale) {
    const Transfer& t = l.tr;
    return ClTransfer{t.na, t.ptr.ptr, t.col.ptr, t.t_ptr.ptr, t.t_row.ptr, t.val32.ptr, t.t_val32.ptr, pscale};
}

void Amg::describe(ClInst& o) const {
    o.n = L[0].n;
    o.levels = (int)L.size();
    o.planar = planar_;
    for (int m = 0; m < planar_; ++m) {
        const AmgLevel& l = L[m];
        ClPlanar& p = o.pl[m];
        p.n = l.n;
        p.goff = l.S0->goff.ptr;
        p.cols = l.S0->cols.ptr;
        p.vals64 = l.vals0;
        p.vals32 = l.vals32;
        p.dinv0 = l.dinv0;
        p.sq4 = l.sq4;
        p.lr = l.r.ptr;
        p.lx = l.x.ptr;
        p.ld = l.d.ptr;
        p.lt = l.t.ptr;
        p.b = l.b.ptr;
        p.z = l.xs.ptr;
        p.dense_inv = l.coarsest ? l.dense_inv.ptr : nullptr;
        p.d4a = l.d4a.ptr;
        p.d4b = l.d4b.ptr;
        p.x4 = l.x4.ptr;
        const ChebCoef k = cheb_coef(l.lmax, degree_, cheb_kind_, cheb_ratio_);
        p.c2_start = k.c2_start;
        for (int i = 0; i < 8; ++i) {
            p.c1[i] = k.c1[i];
            p.c2[i] = k.c2[i];
        }
    }
    o.corner = corner_;
    o.corner_scale = pscale(L[0]);
    o.tr = cl_transfer(L[planar_ - 1], pscale(L[planar_ - 1]));
    for (size_t m = planar_; m < L.size() && m < (size_t)kClMaxLevels; ++m) {
        const AmgLevel& l = L[m];
        ClLevel& c = o.lev[m];
        c.n = l.n;
        c.coarsest = l.coarsest ? 1 : 0;
        c.row_ptr = l.row_ptr.ptr;
        c.cols = l.cols.ptr;
        c.vals = l.pvals.ptr;
        c.dinv = l.dinv.ptr;
        c.dense_inv = l.dense_inv.ptr;
        c.tr = cl_transfer(l, pscale(l));
        c.x = l.x.ptr;
        c.b = l.b.ptr;
        c.r = l.r.ptr;
        c.d = l.d.ptr;
        c.t = l.t.ptr;
        c.xs = l.xs.ptr;
        for (const void* q : {(const void*)c.vals, (const void*)c.x, (const void*)c.b, (const void*)c.d,
                              (const void*)c.t, (const void*)c.xs})
            if (reinterpret_cast<uintptr_t>(q) & 15)  // coarse_row6's 16-byte loads
                fail(FX_GENERIC, "multigrid: coarse-level buffers not 16-byte aligned");
        if (!l.coarsest) {
            const ChebCoef k = cheb_coef(l.lmax, degree_, cheb_kind_, cheb_ratio_);
            c.c2_start = k.c2_start;
            for (int i = 0; i < 8; ++i) {
                c.c1[i] = k.c1[i];
                c.c2[i] = k.c2[i];
            }
        }
    }
}

const float* AmgPcg::fine_fp32(const BsrStructure& S, const double* vals64, cudaStream_t s) {
    const int64_t nv = (int64_t)S.n_groups * 36;
    vals32_.alloc(nv, s);
    FX_LAUNCH(k_f64_to_f32, 148 * 8, 256, 0, s, nv, vals64, vals32_.ptr);
    return vals32_.ptr;
}

void AmgPcg::prepare(const BsrStructure& S, const double* vals64, const double* dinv64, const double* xyz,
                     const CornerLevel* corner, double cell0, double node_volume, const PcgOptions& opt,
                     cudaStream_t s, AmgStats* st, bool reuse, bool persistent) {
    const int n = S.n_rows;
    const int64_t nd = 3 * (int64_t)n;
    if (opt.amg_degree < 1 || opt.amg_degree > 8) fail(FX_INVALID_ARGUMENT, "multigrid smoother degree must be 1..8");
    PlanarIn in[2];
    in[0].S = &S;
    in[0].vals = vals64;
    in[0].dinv = dinv64;
    if (corner) {
        in[1].S = &corner->S;
        in[1].vals = corner->vals.ptr;
        in[1].dinv = corner->minv.ptr;
    }
    if (!reuse) no16_ = false;
    const bool f16 = opt.amg_fp32 && opt.amg_fp16 > 0 && !persistent && !no16_;
    const bool keep = keeps(S, reuse) && amg.planar() == (corner ? 2 : 1);
    // the fine level's copies for the smoother; the corner level, as the 6x6 levels, stays FP64 (with FP16 there
    // a 417k-DOF C3D20 solve takes 20.4 instead of 21.5 ms to 1e-8)
    if (f16) {  // FP16 values of S A S and the scales
        sq4_.alloc((size_t)n, s);
        FX_LAUNCH(k_diag_sqrt, grid_for(n), 256, 0, s, n, S.goff.ptr, S.diag_k.ptr, vals64, sq4_.ptr);
        vals16_.alloc((size_t)S.n_groups * 36, s);
        FX_LAUNCH(k_vals_to_f16, grid_for((int64_t)n * 32), 256, 0, s, n, S.goff.ptr, S.cols.ptr, vals64, sq4_.ptr,
                  vals16_.ptr);
        in[0].vals16 = vals16_.ptr;
        in[0].sq4 = sq4_.ptr;
    }
    // FP32 values: the FP32 smoother's; with the FP16 smoother only when the eigenvalue
    // estimate reads them (kAmgEstF16 off) instead of the FP16 values
    if (opt.amg_fp32 && (!f16 || !kAmgEstF16)) in[0].vals32 = fine_fp32(S, vals64, s);
    amg.set_degree(opt.amg_degree);
    amg.set_tentative(opt.amg_tentative);
    kept_ = keep;
    if (keep) {
        amg.keep(in[0], st);
    } else if (reuse && amg.built_for == S.id && !amg.L.empty() && amg.L[0].n == n && amg.planar() == (corner ? 2 : 1)) {
        drop_graph();
        amg.refresh(in, s, st);
        fresh_ = true;
        stale_ = false;
    } else {
        drop_graph();
        amg.built_for = 0;  // (a failed setup leaves nothing to reuse)
        amg.setup(in, corner, corner ? corner->xyz.ptr : xyz, cell0, node_volume, corner || !persistent, s, st);
        amg.built_for = S.id;
        fresh_ = true;
        stale_ = false;
    }
    amg.set_cycle(opt.amg_kcycle);
    amg.set_smoother_kind(opt.amg_cheb_kind);
    amg.set_overcorrect(opt.amg_overcorrect, opt.amg_overcorrect_all);
    amg.set_cheb_ratio(opt.amg_cheb_ratio);
    S_ = &S;
    vals64_ = vals64;
    dinv64_ = dinv64;
    r_.alloc(nd, s);
    z_.alloc(nd, s);
    p_.alloc(nd, s);
    q_.alloc(nd, s);
    const int nb = 296;
    part_.alloc(std::max<int64_t>(nb, l0_part_slots(n)), s);
    amg.set_part_slots((int64_t)part_.n);
    rd_part_.alloc(grid_for(n), s);
    sc_.alloc(16, s);
    sc_.zero(s);
    hs_.alloc(2, s);
    amg.set_smoother_scale(f16 ? sc_.ptr + 2 : nullptr, f16 ? hs_.ptr : nullptr);  // S[2] = r.D^-1 r
    // the fused coarse cycle reads the hierarchy from a device descriptor, re-uploaded
    // after every setup / refresh (new eigenvalue estimates, new Chebyshev coefficients);
    // a barrier timeout sets S[7]
    amg.set_fused_coarse(opt.amg_fused_coarse && !opt.amg_kcycle, sc_.ptr + 7);
    if (opt.amg_fused_coarse && !opt.amg_kcycle) amg.upload_descriptor(s);
}

void AmgPcg::drop_graph() {
    if (gexec_) cudaGraphExecDestroy(gexec_);
    gexec_ = nullptr;
}

void Amg::upload_descriptor(cudaStream_t s) {
    ClInst h{};
    describe(h);
    desc_.upload(&h, 1, s);
    gbar_.alloc(1, s);
    gbar_.zero(s);
}

ClInst AmgPcg::describe(const double* b, double* x) const {
    ClInst o{};
    amg.describe(o);
    o.b = b;
    o.x = x;
    o.r = r_.ptr;
    o.z = z_.ptr;
    o.p = p_.ptr;
    o.q = q_.ptr;
    return o;
}

double AmgPcg::true_relres(const double* b, const double* x, cudaStream_t s) {
    const int n = S_->n_rows;
    const int nb = 296;
    level_spmv(amg.L[0], x, b, q_.ptr, s);
    FX_LAUNCH(k_rdr_part, nb, 256, 0, s, n, q_.ptr, dinv64_, part_.ptr);
    FX_LAUNCH(k_fin, 1, 32, 0, s, nb, part_.ptr, sc_.ptr, 1);
    FX_LAUNCH(k_rdr_part, nb, 256, 0, s, n, b, dinv64_, part_.ptr);
    FX_LAUNCH(k_fin, 1, 32, 0, s, nb, part_.ptr, sc_.ptr + 4, 1);
    double h[8];
    FX_CUDA_CHECK(cudaMemcpyAsync(h, sc_.ptr, sizeof(h), cudaMemcpyDeviceToHost, s));
    stream_wait(s, "amg true residual");
    return h[6] > 0.0 ? std::sqrt(std::max(0.0, h[2]) / h[6]) : 0.0;
}

int AmgPcg::solve(const BsrStructure& S, const double* vals64, const double* dinv64, const double* xyz,
                  const CornerLevel* corner, double cell0, double node_volume, const double* b, double* x, const PcgOptions& opt, cudaStream_t s,
                  int64_t* launches, long long* iters, double* relres, AmgStats* st, bool reuse) {
    const int n = S.n_rows;
    const int64_t nd = 3 * (int64_t)n;
    prepare(S, vals64, dinv64, xyz, corner, cell0, node_volume, opt, s, st, reuse);
    const int nb = 296;
    const unsigned g0 = l0_grid(n, false, true);  // q = K p
    if (2 * (int64_t)g0 > (int64_t)part_.n) fail(FX_GENERIC, "multigrid: partial-sum buffer smaller than the CG grid");
    FX_CUDA_CHECK(cudaMemsetAsync(x, 0, nd * sizeof(double), s));
    FX_CUDA_CHECK(cudaMemcpyAsync(r_.ptr, b, nd * sizeof(double), cudaMemcpyDeviceToDevice, s));
    // ||b||_D, z = V(b) with r.z, p = z
    FX_LAUNCH(k_rdr_part, nb, 256, 0, s, n, r_.ptr, dinv64, part_.ptr);
    FX_LAUNCH(k_fin, 1, 32, 0, s, nb, part_.ptr, sc_.ptr, 1);
    FX_CUDA_CHECK(cudaMemcpyAsync(sc_.ptr + 3, sc_.ptr + 2, sizeof(double), cudaMemcpyDeviceToDevice, s));
    z2_.alloc(nd, s);
    auto first_direction = [&] {
        amg.apply(r_.ptr, z_.ptr, nullptr, nullptr, s);
        FX_LAUNCH(k_dot_part, nb, 256, 0, s, nd, r_.ptr, z_.ptr, part_.ptr);
        FX_LAUNCH(k_fin, 1, 32, 0, s, nb, part_.ptr, sc_.ptr, 3);
        FX_CUDA_CHECK(cudaMemcpyAsync(p_.ptr, z_.ptr, nd * sizeof(double), cudaMemcpyDeviceToDevice, s));
    };
    first_direction();
    AmgLevel& l0 = amg.L[0];
    // flexible CG (the K-cycle makes the preconditioner vary slightly between
    // iterations): z alternates between two buffers so that r.z_old is at hand
    const unsigned gu = grid_for(n), gx = grid_for(nd);
    unsigned gz = amg.apply_grid();
    int parity = 0;
    auto iteration = [&]() {
        double* zn = parity ? z_.ptr : z2_.ptr;
        const double* zo = parity ? z2_.ptr : z_.ptr;
        if (amg.kcycle()) parity ^= 1;
        L0Op<double> o = l0_op<double>(l0, vals64);
        o.v = p_.ptr;
        o.y = q_.ptr;
        o.dot = 1;
        o.part = part_.ptr;
        FX_LAUNCH_CHAIN((k_l0_op<double, kL0Apply>), g0, 256, 0, s, o);  // q = A p, p.q
        const Amg::Start0 s0 = amg.start0();
        FX_LAUNCH_CHAIN(k_amg_update_start, gu, 256, 0, s, n, sc_.ptr, part_.ptr, (int)g0, p_.ptr, q_.ptr, x, r_.ptr, dinv64,
                  rd_part_.ptr, s0.r, s0.x, s0.d, s0.d4, s0.c2, s0.sq4, s0.hs);  // x, r; the V-cycle's first step
        amg.apply(r_.ptr, zn, part_.ptr, amg.kcycle() ? zo : nullptr, s, true);  // z, r.z
        FX_LAUNCH_CHAIN(k_xpby, gx, 256, 0, s, nd, zn, sc_.ptr, part_.ptr, (int)gz, amg.kcycle(), rd_part_.ptr, (int)gu,
                  p_.ptr);
    };
    // Two iterations per graph (z alternates in the flexible CG), one for large systems, where half an
    // iteration too many on average costs more than the gap between two graphs (2-3 us; 93k DOF: 29
    // iterations instead of 30, 7.55 and 7.38 ms a solve). Between host checks as many replays are queued as the
    // residual's fall so far says are surely needed (60 % of the estimate, at most 12 iterations, 4 where
    // an iteration takes several times the ~14 us that a check idles the GPU for): iterations queued
    // past the end cost more than checks.
    // (A device-side loop as a WHILE graph node, one or four iterations per body, measured 1-7 %
    // slower per iteration on B200 than host-polled replays.)
    const int per_graph = n > 30000 && !amg.kcycle() ? 1 : 2;
    // A hierarchy that ends with a planar level's dense inverse converges in 4 to 20 iterations of short
    // kernels: capturing and instantiating them costs more than it saves, and most beside other
    // threads that do the same (64 decks of 132 / 1,194 DOF as a batch 50 / 63 ms with graphs, 32 / 38 without;
    // alone 1.28 / 1.69 and 1.09 / 1.53; without the dense level, 64 x 1,512 DOF, 33 and 34).
    const bool graphs = opt.graphs && !debug_sync() && !amg.L[amg.planar() - 1].coarsest;
    const void* key[4] = {x, vals64, dinv64, r_.ptr};
    if (gexec_ && (!graphs || !std::equal(key, key + 4, graph_key_))) drop_graph();
    auto capture = [&] {
        if (!graphs || gexec_) return;
        cudaGraph_t g = nullptr;
        int64_t count = 0;
        int64_t* saved = g_launch_counter;
        FX_CUDA_CHECK(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
        g_launch_counter = &count;
        try {
            for (int k = 0; k < per_graph; ++k) iteration();
        } catch (...) {  // (a batch goes on with its other systems on this stream)
            g_launch_counter = saved;
            if (cudaStreamEndCapture(s, &g) == cudaSuccess && g) cudaGraphDestroy(g);
            cudaGetLastError();
            throw;
        }
        const cudaError_t ce = cudaStreamEndCapture(s, &g);
        g_launch_counter = saved;
        FX_CUDA_CHECK(ce);
        graph_launches_ = count;
        const cudaError_t ci = cudaGraphInstantiate(&gexec_, g, 0);
        cudaGraphDestroy(g);
        if (ci != cudaSuccess) gexec_ = nullptr;
        FX_CUDA_CHECK(ci);
        std::copy(key, key + 4, graph_key_);
    };
    capture();
    double h[9];
    long long it = 0;
    int rc = FX_OK;
    const double rtol2 = opt.rtol * opt.rtol;
    const long long max_iter = kept_ ? std::min<long long>(opt.max_iter, 2 * first_iters_ + 50) : opt.max_iter;
    long long try16 = kTry16;
    auto smooth_fp32 = [&](bool on) {
        l0.vals32 = on ? fine_fp32(S, vals64, s) : nullptr;
        l0.vals16 = on ? nullptr : vals16_.ptr;
        l0.sq4 = on ? nullptr : sq4_.ptr;
        amg.set_smoother_scale(on ? nullptr : sc_.ptr + 2, on ? nullptr : hs_.ptr);
        if (opt.amg_fused_coarse && !opt.amg_kcycle) amg.upload_descriptor(s);
    };
    auto host_dot = [&](const double* a, const double* c) {
        std::vector<double> parts(nb);
        FX_LAUNCH(k_dot_part, nb, 256, 0, s, nd, a, c, part_.ptr);
        part_.download(parts.data(), parts.size(), s);
        stream_wait(s, "amg pcg precision check");
        double t = 0.0;
        for (double v : parts) t += v;
        return t;
    };
    double seen = -1.0;  // r.D^-1 r at the check before, and the iterations queued since
    int queued = 0;
    while (true) {
        FX_CUDA_CHECK(cudaMemcpyAsync(h, sc_.ptr, sizeof(h), cudaMemcpyDeviceToHost, s));
        stream_wait(s, "amg pcg poll");
        if (h[7] != 0.0) fail(FX_TIMEOUT, "multigrid: a grid barrier of the coarse cycle timed out");
        if (h[6] != 0.0) {
            rc = FX_NUMERICAL;
            break;
        }
        if (h[3] <= 0.0 || h[2] <= rtol2 * h[3]) break;
        if (kept_ && h[8] < 0.0) {  // (AmgPcg::keeps)
            rc = FX_NUMERICAL;
            break;
        }
        if (it >= max_iter) {
            rc = FX_CONVERGENCE;
            break;
        }
        if (opt.amg_fp16 == 2 && l0.vals16 && it >= try16 &&
            std::log(h[2] / h[3]) > std::log(rtol2) * std::min(0.5, it / (4.0 * kTry16))) {
            try16 = 2 * it;
            smooth_fp32(true);
            double* last = amg.kcycle() ? z_.ptr : z2_.ptr;  // V(r) with FP16
            double* z32 = amg.kcycle() ? z2_.ptr : z_.ptr;   // (either holds nothing that is needed any more)
            amg.apply(r_.ptr, z32, nullptr, nullptr, s);
            const double rz = host_dot(r_.ptr, z32);
            launch_axpby(nd, 1.0, z32, -1.0, last, z32, s);
            level_spmv(l0, z32, nullptr, q_.ptr, s);
            if (host_dot(z32, q_.ptr) <= kSpoilt16 * rz) {
                smooth_fp32(false);
            } else {
                no16_ = true;
                drop_graph();
                gz = amg.apply_grid();
                first_direction();
                capture();
                seen = -1.0;
            }
        }
        int next = 4;
        if (seen > 0.0) {
            const double fall = std::log(h[2] / seen) / queued;  // per iteration
            const double left = fall < 0.0 ? std::log(rtol2 * h[3] / h[2]) / fall : 4.0;
            next = (int)(left < 20.0 ? 0.6 * left : 12.0);
            if (n > 30000) next = std::min(next, 4);
        }
        next = (int)std::min<long long>(std::max(next, 1), std::max<long long>(1, max_iter - it));
        const int replays = (next + per_graph - 1) / per_graph;
        for (int k = 0; k < replays; ++k) {
            if (gexec_) {
                FX_CUDA_CHECK(cudaGraphLaunch(gexec_, s));
                if (launches) *launches += graph_launches_;
            } else {
                for (int j = 0; j < per_graph; ++j) iteration();
            }
        }
        seen = h[2];
        queued = replays * per_graph;
        it += queued;
    }
    solved(it);
    // true residual of the assembled FP64 system in the block-Jacobi norm
    level_spmv(l0, x, b, q_.ptr, s);
    FX_LAUNCH(k_rdr_part, nb, 256, 0, s, n, q_.ptr, dinv64, part_.ptr);
    FX_LAUNCH(k_fin, 1, 32, 0, s, nb, part_.ptr, sc_.ptr, 1);
    FX_CUDA_CHECK(cudaMemcpyAsync(h, sc_.ptr, sizeof(h), cudaMemcpyDeviceToHost, s));
    stream_wait(s, "amg pcg final");
    if (iters) *iters = it;
    if (relres) *relres = h[3] > 0.0 ? std::sqrt(std::max(0.0, h[2]) / h[3]) : 0.0;
    return rc;
}

// A kernel of this file's module (preload_kernels() loads all of the module's kernels).
const void* kernels_anchor_amg() { return reinterpret_cast<const void*>(&k_xpby); }

}  // namespace fx

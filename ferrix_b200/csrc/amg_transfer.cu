// Smoothed prolongator and Galerkin product (see amg_transfer.hpp).
#include <cub/cub.cuh>

#include <type_traits>

#include "amg_transfer.hpp"
#include "common.hpp"
#include "transfer.cuh"

namespace fx {

namespace {

unsigned grid_for(int64_t n, int t = 256) { return (unsigned)((n + t - 1) / t); }

int bits_for(int64_t n) {
    int b = 1;
    while ((int64_t(1) << b) < n) ++b;
    return b;
}

template <typename Op>
void cub_call(Op op, DBuf<uint8_t>& tmp, cudaStream_t s) {
    size_t bytes = 0;
    FX_CUDA_CHECK(op(nullptr, bytes));
    if (tmp.n < bytes) tmp.alloc(bytes, s);
    FX_CUDA_CHECK(op(tmp.ptr, bytes));
}

// ------------------------------------------------------------------ row-wise products
// The usual path. A warp (or CTA) owns a row of the product: its distinct columns are collected in a
// hash set in shared memory, counted, and in a second pass written in ascending order; its values are
// accumulated in shared memory over the row's operands one after another (each operand's columns are
// distinct), so the sums' order is fixed. Nothing of the size of the products is sorted or stored. On a
// 205k-DOF C3D4 box the setup took 3.5 ms with the pair lists below (0.9 ms of it sorts, 0.8 ms sums that
// gather both operands of every pair) and 3.25 ms this way. Rows with more than kSetMax columns take the
// pair lists.

constexpr int kSet = 512, kSetMax = 384;  // slots of a warp's hash set, distinct columns it may hold
constexpr int kRowWarps = 8;
// A row of a planar level whose neighbours lie in more aggregates than this (a node that many elements meet; three cells
// in each direction are 27) keeps its tentative row. Smoothed, it joins every two of those aggregates, and the
// Galerkin product fills all their blocks: a 205k-DOF C3D4 box beside a ball about one node, whose row reaches 75 / 130 /
// 240 / 350 / 480 aggregates, took 20 / 31 / 64 / 110 / 177 ms a solve, and takes 17 / 23 / 29 / 37 / 45. (The whole
// level tentative: 20 / 25 / 31 / 38 / 45.)
constexpr int kLongRow = 64;

__device__ __forceinline__ void set_clear(int* set, int lane) {
    for (int k = lane; k < kSet; k += 32) set[k] = -1;
    __syncwarp();
}
// inserts key; false when the set is full
__device__ __forceinline__ bool set_insert(int* set, int key) {
    unsigned s = ((unsigned)key * 2654435761u) >> 23;  // 9 bits
    for (int probe = 0; probe < kSet; ++probe, s = (s + 1) & (kSet - 1)) {
        const int old = atomicCAS(set + s, -1, key);
        if (old == -1 || old == key) return true;
    }
    return false;
}
// number of keys in the set, in every lane
__device__ __forceinline__ int set_count(const int* set, int lane) {
    __syncwarp();
    int c = 0;
    for (int k = lane; k < kSet; k += 32) c += set[k] >= 0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    return c;
}
// the set's keys ascending to out (through list, kSetMax ints of shared memory)
__device__ __forceinline__ void set_write(const int* set, int* list, int lane, int32_t* __restrict__ out) {
    __syncwarp();
    int n = 0;
    for (int k = lane; k < kSet; k += 32) {
        const int key = set[k];
        const unsigned m = __ballot_sync(0xffffffffu, key >= 0);
        const int at = n + __popc(m & ((1u << lane) - 1));
        if (key >= 0 && at < kSetMax) list[at] = key;
        n += __popc(m);
    }
    n = min(n, kSetMax);
    __syncwarp();
    for (int a = lane; a < n; a += 32) {
        const int key = list[a];
        int rank = 0;
        for (int b = 0; b < n; ++b) rank += list[b] < key;
        out[rank] = key;
    }
    __syncwarp();
}

// column sources of a row
struct SrcP {  // P: aggregates of the row's neighbours, or its own alone (kLongRow; *long_rows = 1)
    FineView F;
    const int32_t* agg;
    int* long_rows;
    __device__ __forceinline__ bool fill(int i, int lane, int* set) const {
        bool ok = true;
        for (int b = F.row_ptr[i] + lane; b < F.row_ptr[i + 1]; b += 32) ok &= set_insert(set, agg[F.col(b, i)]);
        if (F.bs != 3) return ok;
        ok = __all_sync(0xffffffffu, ok);
        if (ok && set_count(set, lane) <= kLongRow) return true;
        __syncwarp();
        set_clear(set, lane);
        if (lane == 0) {
            set_insert(set, agg[i]);
            *long_rows = 1;
        }
        return true;
    }
};
struct SrcW {  // W = A P: the P rows of the row's neighbours
    FineView F;
    const int32_t *p_ptr, *p_col;
    __device__ __forceinline__ bool fill(int i, int lane, int* set) const {
        bool ok = true;
        for (int b = F.row_ptr[i] + lane; b < F.row_ptr[i + 1]; b += 32) {
            const int j = F.col(b, i);
            for (int e = p_ptr[j]; e < p_ptr[j + 1]; ++e) ok &= set_insert(set, p_col[e]);
        }
        return ok;
    }
};
struct SrcC {  // A_c = P^T W: the W rows of the aggregate's fine rows
    const int32_t *t_ptr, *t_row, *w_ptr, *w_col;
    __device__ __forceinline__ bool fill(int a, int lane, int* set) const {
        bool ok = true;
        for (int t = t_ptr[a] + lane; t < t_ptr[a + 1]; t += 32) {
            const int r = t_row[t];
            for (int w = w_ptr[r]; w < w_ptr[r + 1]; ++w) ok &= set_insert(set, w_col[w]);
        }
        return ok;
    }
};

// cnt[row] = distinct columns; most[0] = the largest, most[1] = 1 when a row has more than kSetMax
template <typename Src>
__global__ void __launch_bounds__(32 * kRowWarps) k_row_count(int n, Src src, int32_t* __restrict__ cnt,
                                                              int* __restrict__ most) {
    __shared__ int s_set[kRowWarps][kSet];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, row = blockIdx.x * kRowWarps + w;
    if (row >= n) return;  // warp-uniform
    set_clear(s_set[w], lane);
    const bool ok = src.fill(row, lane, s_set[w]);
    const int c = set_count(s_set[w], lane);
    const bool full = !__all_sync(0xffffffffu, ok) || c > kSetMax;
    if (lane == 0) {
        cnt[row] = c;
        atomicMax(most, c);
        if (full) most[1] = 1;
    }
}

template <typename Src>
__global__ void __launch_bounds__(32 * kRowWarps) k_row_write(int n, Src src, const int32_t* __restrict__ ptr,
                                                              int32_t* __restrict__ col) {
    __shared__ int s_set[kRowWarps][kSet], s_list[kRowWarps][kSetMax];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, row = blockIdx.x * kRowWarps + w;
    if (row >= n) return;  // warp-uniform
    set_clear(s_set[w], lane);
    src.fill(row, lane, s_set[w]);
    set_write(s_set[w], s_list[w], lane, col + ptr[row]);
}

// row[e] = r for the entries of row r
__global__ void k_entry_rows(int n, const int32_t* __restrict__ ptr, int32_t* __restrict__ row) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    for (int e = ptr[i]; e < ptr[i + 1]; ++e) row[e] = i;
}

// place of key in the ascending list (it is there)
__device__ __forceinline__ int place(const int32_t* list, int n, int key) {
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int m = (lo + hi) >> 1;
        if (list[m] < key) lo = m + 1;
        else hi = m;
    }
    return lo;
}

// P of row i (warp per row): A Q summed per aggregate over the row's blocks in order, four blocks' loads in
// flight, then P = (own aggregate: Q) - omega D^-1 (A Q). Lanes 0-17 hold output (r, c), and for 6x6
// blocks (r + 3, c) too.
template <int BS>
__global__ void __launch_bounds__(32 * kRowWarps) k_p_values(int n, int warps, int most, FineView F,
                                                             const int32_t* __restrict__ agg,
                                                             const double* __restrict__ Q,
                                                             const int32_t* __restrict__ p_ptr,
                                                             const int32_t* __restrict__ p_col,
                                                             const double* __restrict__ dinv, double omega,
                                                             double* __restrict__ out) {
    constexpr int V = BS * 6, H = BS / 3, FL = 4;
    extern __shared__ __align__(16) double sh[];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, i = blockIdx.x * warps + w;
    if (i >= n) return;  // warp-uniform
    double* acc = sh + (size_t)w * most * V;
    int* cols = reinterpret_cast<int*>(sh + (size_t)warps * most * V) + w * most;
    const int o0 = p_ptr[i], u = p_ptr[i + 1] - o0;
    for (int k = lane; k < u; k += 32) cols[k] = p_col[o0 + k];
    for (int k = lane; k < u * V; k += 32) acc[k] = 0.0;
    __syncwarp();
    const int b1 = F.row_ptr[i + 1];
    const int r = lane < 18 ? lane / 6 : 0, c = lane % 6;
    const bool act = lane < 18;
    bool tentative = false;  // kLongRow
    for (int b0 = F.row_ptr[i]; b0 < b1; b0 += 32) {
        int j = 0, at = 0;  // the next 32 blocks' columns and places
        bool other = false;
        if (b0 + lane < b1) {
            j = F.col(b0 + lane, i);
            at = place(cols, u, agg[j]);
            other = cols[at] != agg[j];
        }
        tentative = __any_sync(0xffffffffu, other);
        if (tentative) break;
        const int nb = min(32, b1 - b0);
        for (int q0 = 0; q0 < nb; q0 += FL) {  // warp-uniform
            double v[FL][H];
            int p[FL];
#pragma unroll
            for (int f = 0; f < FL; ++f) {
                const int q = min(q0 + f, nb - 1);
                const double* y = Q + (int64_t)__shfl_sync(0xffffffffu, j, q) * V + c;
                p[f] = __shfl_sync(0xffffffffu, at, q);
#pragma unroll
                for (int h = 0; h < H; ++h) {
                    double a[BS];
                    F.load_row<BS>(b0 + q, i, r + 3 * h, a);
                    v[f][h] = 0.0;
#pragma unroll
                    for (int k = 0; k < BS; ++k) v[f][h] += a[k] * __ldg(y + 6 * k);
                }
            }
            if (act)
#pragma unroll
                for (int f = 0; f < FL; ++f)
                    if (q0 + f < nb)
#pragma unroll
                        for (int h = 0; h < H; ++h) acc[p[f] * V + lane + 18 * h] += v[f][h];
        }
    }
    __syncwarp();
    const int mya = agg[i];
    const double* D = dinv + (int64_t)i * BS * BS;
    for (int k = lane; k < u * V; k += 32) {
        const int p = k / V, o = k - p * V, rr = o / 6, cc = o - 6 * rr;
        double z = 0.0;
#pragma unroll
        for (int m = 0; m < BS; ++m) z += D[rr * BS + m] * acc[p * V + 6 * m + cc];
        if (tentative) z = 0.0;
        out[(int64_t)o0 * V + k] = (cols[p] == mya ? Q[(int64_t)i * V + o] : 0.0) - omega * z;
    }
}

// W = A P of row i (warp per row): for each block b in order, a lane per column (y, c) of the P row of b's
// column: its BS values of the column (consecutive over the lanes) times the block (the same for
// all lanes) into BS sums. A lane per output element instead read both operands for every single
// product and was bound by the L1 cache (205k-DOF C3D4 box: 407 us).
template <int BS>
__global__ void __launch_bounds__(32 * kRowWarps) k_w_values(int n, int warps, int most, FineView F,
                                                             const int32_t* __restrict__ p_ptr,
                                                             const int32_t* __restrict__ p_col,
                                                             const double* __restrict__ P,
                                                             const int32_t* __restrict__ w_ptr,
                                                             const int32_t* __restrict__ w_col,
                                                             double* __restrict__ out) {
    constexpr int V = BS * 6;
    extern __shared__ __align__(16) double sh[];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, i = blockIdx.x * warps + w;
    if (i >= n) return;  // warp-uniform
    double* acc = sh + (size_t)w * most * V;
    int* cols = reinterpret_cast<int*>(sh + (size_t)warps * most * V) + w * most;
    const int o0 = w_ptr[i], u = w_ptr[i + 1] - o0;
    for (int k = lane; k < u; k += 32) cols[k] = w_col[o0 + k];
    for (int k = lane; k < u * V; k += 32) acc[k] = 0.0;
    __syncwarp();
    const int b1 = F.row_ptr[i + 1];
    for (int b0 = F.row_ptr[i]; b0 < b1; b0 += 32) {
        int y0 = 0, ny = 0;  // the next 32 blocks' P rows
        if (b0 + lane < b1) {
            const int j = F.col(b0 + lane, i);
            y0 = p_ptr[j];
            ny = p_ptr[j + 1] - y0;
        }
        const int nb = min(32, b1 - b0);
#pragma unroll 2
        for (int q = 0; q < nb; ++q) {  // warp-uniform
            const int yb = __shfl_sync(0xffffffffu, y0, q), yn = __shfl_sync(0xffffffffu, ny, q);
            double a[BS][BS];
#pragma unroll
            for (int r = 0; r < BS; ++r) F.load_row<BS>(b0 + q, i, r, a[r]);
            for (int t = lane; t < 6 * yn; t += 32) {
                const int y = yb + t / 6, c = t % 6;
                const int at = place(cols, u, __ldg(p_col + y));
                double x[BS];
#pragma unroll
                for (int k = 0; k < BS; ++k) x[k] = __ldg(P + (int64_t)y * V + 6 * k + c);
#pragma unroll
                for (int r = 0; r < BS; ++r) {
                    double v = 0.0;
#pragma unroll
                    for (int k = 0; k < BS; ++k) v += a[r][k] * x[k];
                    acc[at * V + 6 * r + c] += v;
                }
            }
            __syncwarp();
        }
    }
    for (int k = lane; k < u * V; k += 32) out[(int64_t)o0 * V + k] = acc[k];
}

// Values of coarse row a: acc[J] += P_p^T W_w over the aggregate's entries p, a contiguous share of them
// per warp of the CTA (the shares are added in order at the end). For each entry a lane per column
// (w, c) of its fine row's W row: BS values (consecutive over the lanes) times the transposed P block
// (the same for all lanes) into six sums.
constexpr int kCoarseWarps = 8;
template <int BS>
__global__ void __launch_bounds__(32 * kCoarseWarps)
    k_coarse_values(int most, const int32_t* __restrict__ t_ptr, const int32_t* __restrict__ t_ent,
                    const int32_t* __restrict__ t_row, const double* __restrict__ P,
                    const int32_t* __restrict__ w_ptr, const int32_t* __restrict__ w_col,
                    const double* __restrict__ W, const int32_t* __restrict__ c_ptr,
                    const int32_t* __restrict__ c_col, double* __restrict__ out) {
    constexpr int V = BS * 6;
    extern __shared__ __align__(16) double sh[];
    const int warps = blockDim.x >> 5, w = threadIdx.x >> 5, lane = threadIdx.x & 31, a = blockIdx.x;
    double* acc = sh + (size_t)w * most * 36;
    int* cols = reinterpret_cast<int*>(sh + (size_t)warps * most * 36);
    const int c0 = c_ptr[a], u = c_ptr[a + 1] - c0;
    for (int k = threadIdx.x; k < u; k += blockDim.x) cols[k] = c_col[c0 + k];
    for (int k = lane; k < u * 36; k += 32) acc[k] = 0.0;
    __syncthreads();
    const int t0 = t_ptr[a], nt = t_ptr[a + 1] - t0;
    const int s0 = t0 + (int)((int64_t)nt * w / warps), s1 = t0 + (int)((int64_t)nt * (w + 1) / warps);
    for (int sb = s0; sb < s1; sb += 32) {
        int pe = 0, w0 = 0, nw = 0;  // the next 32 entries and their W rows
        if (sb + lane < s1) {
            pe = t_ent[sb + lane];
            const int row = t_row[sb + lane];
            w0 = w_ptr[row];
            nw = w_ptr[row + 1] - w0;
        }
        const int ns = min(32, s1 - sb);
#pragma unroll 2
        for (int q = 0; q < ns; ++q) {  // warp-uniform
            const double* p = P + (int64_t)__shfl_sync(0xffffffffu, pe, q) * V;
            const int wb = __shfl_sync(0xffffffffu, w0, q), wn = __shfl_sync(0xffffffffu, nw, q);
            for (int t = lane; t < 6 * wn; t += 32) {
                const int y = wb + t / 6, c = t % 6;
                const int at = place(cols, u, __ldg(w_col + y));
                double v[6] = {0, 0, 0, 0, 0, 0};
#pragma unroll
                for (int k = 0; k < BS; ++k) {
                    const double x = __ldg(W + (int64_t)y * V + 6 * k + c);
#pragma unroll
                    for (int r = 0; r < 6; ++r) v[r] += __ldg(p + 6 * k + r) * x;
                }
#pragma unroll
                for (int r = 0; r < 6; ++r) acc[at * 36 + 6 * r + c] += v[r];
            }
            __syncwarp();
        }
    }
    __syncthreads();
    for (int k = threadIdx.x; k < u * 36; k += blockDim.x) {
        double t = sh[k];
        for (int q = 1; q < warps; ++q) t += sh[(size_t)q * most * 36 + k];
        out[(int64_t)c0 * 36 + k] = t;
    }
}

constexpr size_t kRowShared = 200 << 10;

// warps (1, 2, 4, 8) whose `per_warp` bytes fit the shared memory, at most `want`
int warps_that_fit(size_t per_warp, int want) {
    int w = want;
    while (w > 1 && per_warp * w > kRowShared) w >>= 1;
    return w;
}

// Row pattern of a product: ptr, col and the largest row; false when a row is too long.
template <typename Src>
bool row_pattern(int n, const Src& src, DBuf<int32_t>& ptr, DBuf<int32_t>& col, int64_t* nnz, int* most,
                 DBuf<uint8_t>& tmp, cudaStream_t s) {
    DBuf<int32_t> cnt;
    DBuf<int> d_most;
    cnt.alloc(n, s);
    d_most.alloc(2, s);
    d_most.zero(s);
    ptr.alloc(n + 1, s);
    FX_CUDA_CHECK(cudaMemsetAsync(ptr.ptr, 0, sizeof(int32_t), s));
    FX_LAUNCH(k_row_count<Src>, grid_for(n, kRowWarps), 32 * kRowWarps, 0, s, n, src, cnt.ptr, d_most.ptr);
    cub_call([&](void* t, size_t& b) { return cub::DeviceScan::InclusiveSum(t, b, cnt.ptr, ptr.ptr + 1, n, s); }, tmp,
             s);
    int32_t total = 0;
    int h[2];
    FX_CUDA_CHECK(cudaMemcpyAsync(&total, ptr.ptr + n, sizeof(int32_t), cudaMemcpyDeviceToHost, s));
    FX_CUDA_CHECK(cudaMemcpyAsync(h, d_most.ptr, sizeof(h), cudaMemcpyDeviceToHost, s));
    stream_wait(s, "amg transfer rows");
    if (h[1] || total < 0) return false;  // (negative: more than 2^31 entries)
    *nnz = total;
    *most = h[0];
    col.alloc(total, s);
    FX_LAUNCH(k_row_write<Src>, grid_for(n, kRowWarps), 32 * kRowWarps, 0, s, n, src, ptr.ptr, col.ptr);
    return true;
}

template <typename K, typename... A>
void launch_rows(K kernel, int bs, const FineView& F, int most, cudaStream_t s, A... args) {
    const size_t row = (size_t)most * (bs * 6 * sizeof(double) + sizeof(int));
    const int warps = warps_that_fit(row, kRowWarps);
    FX_LAUNCH(kernel, grid_for(F.n, warps), 32 * warps, warps * row, s, F.n, warps, most, F, args...);
}

static_assert(kSetMax * (36 * sizeof(double) + sizeof(int)) <= kRowShared, "a warp's longest row fits the shared memory");

// ------------------------------------------------------------------ products by pair lists

__device__ __forceinline__ uint64_t pack(int64_t x, int64_t y) { return ((uint64_t)x << 32) | (uint64_t)(uint32_t)y; }

// items of P: block (i, j) contributes A_ij Q_j to entry (i, agg j); unsmoothed: one item per row
template <typename KT>
__global__ void k_items_p(FineView F, const int32_t* __restrict__ agg, int cbits, KT* __restrict__ keys,
                          uint64_t* __restrict__ vals) {
    const int64_t b = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= F.nblocks) return;
    const int i = F.blk_row[b], j = F.col(b, i);
    keys[b] = (KT)(((uint64_t)i << cbits) | (uint64_t)agg[j]);
    vals[b] = pack(b, j);
}

template <typename KT>
__global__ void k_items_q(int n, const int32_t* __restrict__ agg, int cbits, KT* __restrict__ keys,
                          uint64_t* __restrict__ vals) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    keys[i] = (KT)(((uint64_t)i << cbits) | (uint64_t)agg[i]);
    vals[i] = pack(i, i);
}

// items of W = A P: block (i, j) meets every entry (j, J) of P: A_ij P_jJ into (i, J)
__global__ void k_count_w(FineView F, const int32_t* __restrict__ p_ptr, int64_t* __restrict__ cnt) {
    const int64_t b = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= F.nblocks) return;
    const int j = F.col(b, F.blk_row[b]);
    cnt[b] = p_ptr[j + 1] - p_ptr[j];
}

template <typename KT>
__global__ void k_items_w(FineView F, const int32_t* __restrict__ p_ptr, const int32_t* __restrict__ p_col,
                          const int64_t* __restrict__ end, int cbits, KT* __restrict__ keys,
                          uint64_t* __restrict__ vals) {
    const int64_t b = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= F.nblocks) return;
    const int i = F.blk_row[b], j = F.col(b, i);
    int64_t o = b ? end[b - 1] : 0;
    for (int e = p_ptr[j]; e < p_ptr[j + 1]; ++e, ++o) {
        keys[o] = (KT)(((uint64_t)i << cbits) | (uint64_t)p_col[e]);
        vals[o] = pack(b, e);
    }
}

// items of A_c = P^T W: entry (i, I) of P meets every entry (i, J) of W: P_iI^T W_iJ into (I, J)
__global__ void k_count_c(int64_t nnz, const int32_t* __restrict__ p_row, const int32_t* __restrict__ w_ptr,
                          int64_t* __restrict__ cnt) {
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= nnz) return;
    cnt[e] = w_ptr[p_row[e] + 1] - w_ptr[p_row[e]];
}

template <typename KT>
__global__ void k_items_c(int64_t nnz, const int32_t* __restrict__ p_row, const int32_t* __restrict__ p_col,
                          const int32_t* __restrict__ w_ptr, const int32_t* __restrict__ w_col,
                          const int64_t* __restrict__ end, int cbits, KT* __restrict__ keys,
                          uint64_t* __restrict__ vals) {
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= nnz) return;
    const int i = p_row[e];
    const uint64_t I = (uint64_t)p_col[e];
    int64_t o = e ? end[e - 1] : 0;
    for (int w = w_ptr[i]; w < w_ptr[i + 1]; ++w, ++o) {
        keys[o] = (KT)((I << cbits) | (uint64_t)w_col[w]);
        vals[o] = pack(e, w);
    }
}

template <typename KT>
__global__ void k_heads_items(int64_t n, const KT* __restrict__ keys, int32_t* __restrict__ head) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) head[i] = (i == 0 || keys[i] != keys[i - 1]) ? 1 : 0;
}

template <typename KT>
__global__ void k_entries(int64_t n, int64_t n_ent, const KT* __restrict__ keys, const int32_t* __restrict__ rank,
                          int cbits, int32_t* __restrict__ row, int32_t* __restrict__ col, int64_t* __restrict__ seg) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (i == 0) seg[n_ent] = n;
    if (i == 0 || keys[i] != keys[i - 1]) {
        const int e = rank[i] - 1;
        seg[e] = i;
        row[e] = (int32_t)(keys[i] >> cbits);
        col[e] = (int32_t)((uint64_t)keys[i] & ((uint64_t(1) << cbits) - 1));
    }
}

// ptr[r] = first of the n ascending keys that is >= r, r = 0 .. rows
__global__ void k_row_bounds(int64_t n, int rows, const int32_t* __restrict__ key, int32_t* __restrict__ ptr) {
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e > n) return;
    const int lo = e == 0 ? 0 : key[e - 1] + 1, hi = e == n ? rows : key[e];
    for (int r = lo; r <= hi; ++r) ptr[r] = (int32_t)e;
}

__global__ void k_iota(int64_t n, int32_t* __restrict__ v) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) v[i] = (int32_t)i;
}

__global__ void k_pick(int64_t n, const int32_t* __restrict__ idx, const int32_t* __restrict__ src,
                       int32_t* __restrict__ dst) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) dst[i] = src[idx[i]];
}

// out entry e (row i, BS x 6) = sum over its pairs (block b of row i, y) of A_b Y_y. A thread per
// (entry, block row): 6 sums and the 3 or 6 values of one block row in registers, so that
// enough threads are resident to cover the gathers (a thread per entry would hold 18 or 36 sums
// and leave a third of the threads).
template <int BS>
__global__ void __launch_bounds__(256) k_spmm_rows(int64_t n_ent, const int32_t* __restrict__ row,
                                                   const int64_t* __restrict__ seg,
                                                   const uint64_t* __restrict__ pairs, FineView F,
                                                   const double* __restrict__ Y, double* __restrict__ out) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t e = t / BS;
    const int r = (int)(t - e * BS);
    if (e >= n_ent) return;
    const int i = row[e];
    double acc[6] = {0, 0, 0, 0, 0, 0};
    for (int64_t s = seg[e]; s < seg[e + 1]; ++s) {
        const uint64_t p = __ldg(pairs + s);
        double a[BS];
        F.load_row<BS>((int64_t)(p >> 32), i, r, a);
        const double2* y = reinterpret_cast<const double2*>(Y + (int64_t)(p & 0xffffffffu) * (BS * 6));
#pragma unroll
        for (int k = 0; k < BS; ++k)
#pragma unroll
            for (int h = 0; h < 3; ++h) {
                const double2 v = __ldg(y + 3 * k + h);
                acc[2 * h] += a[k] * v.x;
                acc[2 * h + 1] += a[k] * v.y;
            }
    }
    double* o = out + (e * BS + r) * 6;
#pragma unroll
    for (int c = 0; c < 6; ++c) o[c] = acc[c];
}

// P = (own aggregate: Q) - omega D^-1 (A Q), in place over the A Q blocks; a thread per (entry, column)
template <int BS>
__global__ void k_smooth_p(int64_t nnz, const int32_t* __restrict__ row, const int32_t* __restrict__ col,
                           const int32_t* __restrict__ agg, const double* __restrict__ Q,
                           const double* __restrict__ dinv, double omega, double* __restrict__ val) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t e = t / 6;
    const int c = (int)(t - e * 6);
    if (e >= nnz) return;
    const int i = row[e];
    const bool own = col[e] == agg[i];
    double* v = val + e * (BS * 6);
    double a[BS];
#pragma unroll
    for (int k = 0; k < BS; ++k) a[k] = v[k * 6 + c];
    const double* D = dinv + (int64_t)i * BS * BS;
#pragma unroll
    for (int r = 0; r < BS; ++r) {
        double z = 0.0;
#pragma unroll
        for (int k = 0; k < BS; ++k) z += D[r * BS + k] * a[k];
        v[r * 6 + c] = (own ? Q[((int64_t)i * BS + r) * 6 + c] : 0.0) - omega * z;
    }
}

// c_vals block = sum over its pairs (entry p of P, entry w of W, same fine row) of P_p^T W_w.
// Warp per coarse block (tens to hundreds of pairs), lane k takes the k-th contiguous slice; the
// 36 sums are combined by a fixed butterfly.
template <int BS>
__global__ void __launch_bounds__(128) k_ptw(int64_t ncb, const int64_t* __restrict__ seg,
                                             const uint64_t* __restrict__ pairs, const double* __restrict__ P,
                                             const double* __restrict__ W, double* __restrict__ c_vals) {
    const int64_t cb = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (cb >= ncb) return;  // warp-uniform
    const int64_t s0 = seg[cb], s1 = seg[cb + 1];
    double acc[36];
#pragma unroll
    for (int k = 0; k < 36; ++k) acc[k] = 0.0;
    for (int64_t s = s0 + lane; s < s1; s += 32) {
        const uint64_t pr = __ldg(pairs + s);
        const double2* p = reinterpret_cast<const double2*>(P + (int64_t)(pr >> 32) * (BS * 6));
        const double2* w = reinterpret_cast<const double2*>(W + (int64_t)(pr & 0xffffffffu) * (BS * 6));
#pragma unroll
        for (int k = 0; k < BS; ++k) {
            double pv[6], wv[6];
#pragma unroll
            for (int h = 0; h < 3; ++h) {
                const double2 a = __ldg(p + 3 * k + h), b = __ldg(w + 3 * k + h);
                pv[2 * h] = a.x;
                pv[2 * h + 1] = a.y;
                wv[2 * h] = b.x;
                wv[2 * h + 1] = b.y;
            }
#pragma unroll
            for (int r = 0; r < 6; ++r)
#pragma unroll
                for (int c = 0; c < 6; ++c) acc[r * 6 + c] += pv[r] * wv[c];
        }
    }
#pragma unroll
    for (int k = 0; k < 36; ++k) {
        const double t = warp_sum(acc[k]);
        if (lane == 0) c_vals[cb * 36 + k] = t;
    }
}

// Sorts n items by key (kbits significant) and compresses them into entries. fill(keys, vals) writes
// the items, with 32-bit keys where kbits allows (a quarter of the sort's traffic).
template <typename KT, typename Fill>
void compress_t(int64_t n, int kbits, int cbits, PairList& out, DBuf<uint8_t>& tmp, cudaStream_t s, Fill&& fill) {
    DBuf<KT> keys, keys_s;
    DBuf<uint64_t> vals;
    keys.alloc(n, s);
    vals.alloc(n, s);
    fill(keys.ptr, vals.ptr);
    keys_s.alloc(n, s);
    out.pairs.alloc(n, s);
    cub_call([&](void* t, size_t& b) {
        return cub::DeviceRadixSort::SortPairs(t, b, keys.ptr, keys_s.ptr, vals.ptr, out.pairs.ptr, n, 0, kbits, s);
    }, tmp, s);
    keys.release();
    vals.release();
    DBuf<int32_t> head, rank;
    head.alloc(n, s);
    rank.alloc(n, s);
    FX_LAUNCH(k_heads_items<KT>, grid_for(n), 256, 0, s, n, keys_s.ptr, head.ptr);
    cub_call([&](void* t, size_t& b) { return cub::DeviceScan::InclusiveSum(t, b, head.ptr, rank.ptr, n, s); }, tmp,
             s);
    int32_t ne = 0;
    FX_CUDA_CHECK(cudaMemcpyAsync(&ne, rank.ptr + n - 1, sizeof(int32_t), cudaMemcpyDeviceToHost, s));
    stream_wait(s, "amg transfer entries");
    out.n = ne;
    out.row.alloc(ne, s);
    out.col.alloc(ne, s);
    out.seg.alloc(ne + 1, s);
    FX_LAUNCH(k_entries<KT>, grid_for(n), 256, 0, s, n, out.n, keys_s.ptr, rank.ptr, cbits, out.row.ptr, out.col.ptr,
              out.seg.ptr);
}

template <typename Fill>
void compress(int64_t n, int kbits, int cbits, PairList& out, DBuf<uint8_t>& tmp, cudaStream_t s, Fill&& fill) {
    if (kbits <= 32) compress_t<uint32_t>(n, kbits, cbits, out, tmp, s, fill);
    else compress_t<uint64_t>(n, kbits, cbits, out, tmp, s, fill);
}

// The cycle's interleaved copy of P: out entry e = block `order[e]` (order null: e). A thread per
// (entry, pair), entries fastest, so that the writes are consecutive.
template <int BS>
__global__ void k_interleave(int64_t nnz, const int32_t* __restrict__ order, const double* __restrict__ val,
                             double2* __restrict__ out) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t chunk = t / (96 * BS), e = chunk * 32 + (t & 31);
    const int q = (int)(t - chunk * (96 * BS)) >> 5;
    if (chunk * 32 >= nnz) return;
    double2 v = make_double2(0.0, 0.0);
    if (e < nnz) v = __ldg(reinterpret_cast<const double2*>(val) + (order ? (int64_t)order[e] : e) * (3 * BS) + q);
    out[t] = v;
}

// *total = sum of cnt, end = its inclusive prefix sums
int64_t scan_counts(const DBuf<int64_t>& cnt, DBuf<int64_t>& end, int64_t n, DBuf<uint8_t>& tmp, cudaStream_t s) {
    end.alloc(n, s);
    cub_call([&](void* t, size_t& b) { return cub::DeviceScan::InclusiveSum(t, b, cnt.ptr, end.ptr, n, s); }, tmp, s);
    int64_t total = 0;
    FX_CUDA_CHECK(cudaMemcpyAsync(&total, end.ptr + n - 1, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
    stream_wait(s, "amg transfer counts");
    return total;
}

constexpr int64_t kMaxItems = (int64_t(1) << 31) - 1;

}  // namespace

namespace {

// P's entries by aggregate (a stable sort: ascending fine row within one) and the cycle's copies
void transpose_and_interleave(Transfer& t, const int32_t* p_row, DBuf<uint8_t>& tmp, cudaStream_t s) {
    const int abits = bits_for(t.na > 1 ? t.na : 2);
    DBuf<int32_t> ids, col_s;
    ids.alloc(t.nnz, s);
    col_s.alloc(t.nnz, s);
    t.t_ent.alloc(t.nnz, s);
    t.t_row.alloc(t.nnz, s);
    t.t_ptr.alloc(t.na + 1, s);
    FX_LAUNCH(k_iota, grid_for(t.nnz), 256, 0, s, t.nnz, ids.ptr);
    cub_call([&](void* q, size_t& b) {
        return cub::DeviceRadixSort::SortPairs(q, b, t.col.ptr, col_s.ptr, ids.ptr, t.t_ent.ptr, (int)t.nnz, 0, abits,
                                               s);
    }, tmp, s);
    FX_LAUNCH(k_row_bounds, grid_for(t.nnz + 1), 256, 0, s, t.nnz, t.na, col_s.ptr, t.t_ptr.ptr);
    FX_LAUNCH(k_pick, grid_for(t.nnz), 256, 0, s, t.nnz, t.t_ent.ptr, p_row, t.t_row.ptr);
    const int64_t n32 = t.bs == 3 ? p32_size<3>(t.nnz) : p32_size<6>(t.nnz);
    t.val32.alloc(n32, s);
    t.t_val32.alloc(n32, s);
    if (t.bs == 3) {
        FX_LAUNCH(k_interleave<3>, grid_for(n32), 256, 0, s, t.nnz, nullptr, t.val.ptr, t.val32.ptr);
        FX_LAUNCH(k_interleave<3>, grid_for(n32), 256, 0, s, t.nnz, t.t_ent.ptr, t.val.ptr, t.t_val32.ptr);
    } else {
        FX_LAUNCH(k_interleave<6>, grid_for(n32), 256, 0, s, t.nnz, nullptr, t.val.ptr, t.val32.ptr);
        FX_LAUNCH(k_interleave<6>, grid_for(n32), 256, 0, s, t.nnz, t.t_ent.ptr, t.val.ptr, t.t_val32.ptr);
    }
}

// The smoothed transfer by rows; false (with t to be rebuilt) where a row is too long for it. *long_rows = 1
// where a row of P is (kLongRow).
bool build_by_rows(const FineView& F, int na, const int32_t* agg, const double* Q, const double* dinv, double omega,
                   Transfer& t, DBuf<int32_t>& c_ptr, DBuf<int32_t>& c_cols, int64_t* ncb, int* long_rows,
                   DBuf<uint8_t>& tmp, cudaStream_t s) {
    if (F.nblocks <= 0 || F.nblocks > kMaxItems / 2) return false;  // (32-bit row pointers below)
    const int bs = F.bs;
    int most_p = 0;
    t.most_w = t.most_c = 0;
    if (!row_pattern(F.n, SrcP{F, agg, long_rows}, t.ptr, t.col, &t.nnz, &most_p, tmp, s)) return false;
    t.val.alloc((size_t)t.nnz * bs * 6, s);
    if (bs == 3)
        launch_rows(k_p_values<3>, 3, F, most_p, s, agg, Q, (const int32_t*)t.ptr.ptr, (const int32_t*)t.col.ptr, dinv,
                    omega, t.val.ptr);
    else
        launch_rows(k_p_values<6>, 6, F, most_p, s, agg, Q, (const int32_t*)t.ptr.ptr, (const int32_t*)t.col.ptr, dinv,
                    omega, t.val.ptr);
    {
        DBuf<int32_t> p_row;
        p_row.alloc(t.nnz, s);
        FX_LAUNCH(k_entry_rows, grid_for(F.n), 256, 0, s, F.n, t.ptr.ptr, p_row.ptr);
        transpose_and_interleave(t, p_row.ptr, tmp, s);
    }
    if (!row_pattern(F.n, SrcW{F, t.ptr.ptr, t.col.ptr}, t.w_ptr, t.w_col, &t.w.n, &t.most_w, tmp, s)) return false;
    if (!row_pattern(na, SrcC{t.t_ptr.ptr, t.t_row.ptr, t.w_ptr.ptr, t.w_col.ptr}, c_ptr, c_cols, ncb, &t.most_c, tmp, s))
        return false;
    t.c.n = *ncb;
    return true;
}

}  // namespace

bool build_transfer(const FineView& F, int na, const int32_t* agg, const double* Q, const double* dinv, double omega,
                    bool smooth, Transfer& t, DBuf<int32_t>& c_ptr, DBuf<int32_t>& c_cols, int64_t* ncb,
                    DBuf<uint8_t>& tmp, cudaStream_t s) {
    const int n = F.n, bs = F.bs;
    const int abits = bits_for(na > 1 ? na : 2), nbits = bits_for(n > 1 ? n : 2);
    t.n = n;
    t.na = na;
    t.bs = bs;
    DBuf<int> long_rows;
    long_rows.alloc(1, s);
    long_rows.zero(s);
    t.by_rows = smooth && build_by_rows(F, na, agg, Q, dinv, omega, t, c_ptr, c_cols, ncb, long_rows.ptr, tmp, s);
    if (t.by_rows) return true;
    if (smooth) {  // (the pair lists would smooth the long rows too)
        int h = 0;
        FX_CUDA_CHECK(cudaMemcpyAsync(&h, long_rows.ptr, sizeof(int), cudaMemcpyDeviceToHost, s));
        stream_wait(s, "amg transfer rows");
        smooth = !h;
    }
    t.w_ptr.release();
    t.w_col.release();
    DBuf<int64_t> cnt, end;
    DBuf<int32_t> w_ptr;
    smooth = smooth && F.nblocks > 0;
    int64_t total = 0;
    PairList p;
    while (true) {
        const int64_t items = smooth ? F.nblocks : n;
        compress(items, nbits + abits, abits, p, tmp, s, [&](auto* keys, uint64_t* vals) {
            using KT = std::remove_pointer_t<decltype(keys)>;
            if (smooth) FX_LAUNCH(k_items_p<KT>, grid_for(items), 256, 0, s, F, agg, abits, keys, vals);
            else FX_LAUNCH(k_items_q<KT>, grid_for(items), 256, 0, s, n, agg, abits, keys, vals);
        });
        t.nnz = p.n;
        t.ptr.alloc(n + 1, s);
        FX_LAUNCH(k_row_bounds, grid_for(p.n + 1), 256, 0, s, p.n, n, p.row.ptr, t.ptr.ptr);
        if (F.nblocks == 0) break;
        cnt.alloc(F.nblocks, s);
        FX_LAUNCH(k_count_w, grid_for(F.nblocks), 256, 0, s, F, t.ptr.ptr, cnt.ptr);
        total = scan_counts(cnt, end, F.nblocks, tmp, s);
        if (total <= kMaxItems) break;
        if (!smooth) fail(FX_INVALID_ARGUMENT, "mesh too large for the multigrid's 32-bit item indices");
        smooth = false;  // too many products for 32-bit item indices: the tentative prolongator itself
    }
    // ---- values of P
    t.val.alloc((size_t)p.n * bs * 6, s);
    if (smooth) {
        if (bs == 3) {
            FX_LAUNCH(k_spmm_rows<3>, grid_for(p.n * 3), 256, 0, s, p.n, p.row.ptr, p.seg.ptr, p.pairs.ptr, F, Q,
                      t.val.ptr);
            FX_LAUNCH(k_smooth_p<3>, grid_for(p.n * 6), 256, 0, s, p.n, p.row.ptr, p.col.ptr, agg, Q, dinv, omega,
                      t.val.ptr);
        } else {
            FX_LAUNCH(k_spmm_rows<6>, grid_for(p.n * 6), 256, 0, s, p.n, p.row.ptr, p.seg.ptr, p.pairs.ptr, F, Q,
                      t.val.ptr);
            FX_LAUNCH(k_smooth_p<6>, grid_for(p.n * 6), 256, 0, s, p.n, p.row.ptr, p.col.ptr, agg, Q, dinv, omega,
                      t.val.ptr);
        }
    } else {
        FX_CUDA_CHECK(cudaMemcpyAsync(t.val.ptr, Q, (size_t)n * bs * 6 * sizeof(double), cudaMemcpyDeviceToDevice, s));
    }
    t.col = std::move(p.col);
    transpose_and_interleave(t, p.row.ptr, tmp, s);
    // ---- W = A P
    if (F.nblocks > 0) {
        compress(total, nbits + abits, abits, t.w, tmp, s, [&](auto* keys, uint64_t* vals) {
            using KT = std::remove_pointer_t<decltype(keys)>;
            FX_LAUNCH(k_items_w<KT>, grid_for(F.nblocks), 256, 0, s, F, t.ptr.ptr, t.col.ptr, end.ptr, abits, keys, vals);
        });
        w_ptr.alloc(n + 1, s);
        FX_LAUNCH(k_row_bounds, grid_for(t.w.n + 1), 256, 0, s, t.w.n, n, t.w.row.ptr, w_ptr.ptr);
        // ---- A_c = P^T W
        cnt.alloc(p.n, s);
        FX_LAUNCH(k_count_c, grid_for(p.n), 256, 0, s, p.n, p.row.ptr, w_ptr.ptr, cnt.ptr);
        total = scan_counts(cnt, end, p.n, tmp, s);
        if (total > kMaxItems) fail(FX_INVALID_ARGUMENT, "mesh too large for the multigrid's 32-bit item indices");
        compress(total, 2 * abits, abits, t.c, tmp, s, [&](auto* keys, uint64_t* vals) {
            using KT = std::remove_pointer_t<decltype(keys)>;
            FX_LAUNCH(k_items_c<KT>, grid_for(p.n), 256, 0, s, p.n, p.row.ptr, t.col.ptr, w_ptr.ptr, t.w.col.ptr,
                      end.ptr, abits, keys, vals);
        });
    }
    *ncb = t.c.n;
    c_ptr.alloc(na + 1, s);
    c_cols = std::move(t.c.col);
    if (t.c.n) FX_LAUNCH(k_row_bounds, grid_for(t.c.n + 1), 256, 0, s, t.c.n, na, t.c.row.ptr, c_ptr.ptr);
    else c_ptr.zero(s);
    t.w.col.release();
    return smooth;
}

void galerkin_product(const FineView& F, const Transfer& t, const int32_t* c_ptr, const int32_t* c_cols,
                      double* c_vals, cudaStream_t s) {
    if (!t.c.n) return;
    DBuf<double> W;
    W.alloc((size_t)t.w.n * t.bs * 6, s);
    if (t.by_rows) {
        // more warps per row where there are few rows (180 rows of 60 columns: 201 us with 8, 282 with 4)
        const int wc = warps_that_fit((size_t)t.most_c * (36 * sizeof(double) + sizeof(int)),
                                      t.na < 4 * 148 ? kCoarseWarps : kCoarseWarps / 2);
        const size_t bytes = (size_t)t.most_c * (wc * 36 * sizeof(double) + sizeof(int));
        if (t.bs == 3) {
            launch_rows(k_w_values<3>, 3, F, t.most_w, s, (const int32_t*)t.ptr.ptr, (const int32_t*)t.col.ptr,
                        (const double*)t.val.ptr, (const int32_t*)t.w_ptr.ptr, (const int32_t*)t.w_col.ptr, W.ptr);
            FX_LAUNCH(k_coarse_values<3>, (unsigned)t.na, 32 * wc, bytes, s, t.most_c, t.t_ptr.ptr, t.t_ent.ptr,
                      t.t_row.ptr, t.val.ptr, t.w_ptr.ptr, t.w_col.ptr, W.ptr, c_ptr, c_cols, c_vals);
        } else {
            launch_rows(k_w_values<6>, 6, F, t.most_w, s, (const int32_t*)t.ptr.ptr, (const int32_t*)t.col.ptr,
                        (const double*)t.val.ptr, (const int32_t*)t.w_ptr.ptr, (const int32_t*)t.w_col.ptr, W.ptr);
            FX_LAUNCH(k_coarse_values<6>, (unsigned)t.na, 32 * wc, bytes, s, t.most_c, t.t_ptr.ptr, t.t_ent.ptr,
                      t.t_row.ptr, t.val.ptr, t.w_ptr.ptr, t.w_col.ptr, W.ptr, c_ptr, c_cols, c_vals);
        }
        return;
    }
    if (t.bs == 3) {
        FX_LAUNCH(k_spmm_rows<3>, grid_for(t.w.n * 3), 256, 0, s, t.w.n, t.w.row.ptr, t.w.seg.ptr, t.w.pairs.ptr, F,
                  t.val.ptr, W.ptr);
        FX_LAUNCH(k_ptw<3>, grid_for(t.c.n * 32, 128), 128, 0, s, t.c.n, t.c.seg.ptr, t.c.pairs.ptr, t.val.ptr, W.ptr,
                  c_vals);
    } else {
        FX_LAUNCH(k_spmm_rows<6>, grid_for(t.w.n * 6), 256, 0, s, t.w.n, t.w.row.ptr, t.w.seg.ptr, t.w.pairs.ptr, F,
                  t.val.ptr, W.ptr);
        FX_LAUNCH(k_ptw<6>, grid_for(t.c.n * 32, 128), 128, 0, s, t.c.n, t.c.seg.ptr, t.c.pairs.ptr, t.val.ptr, W.ptr,
                  c_vals);
    }
}

void allow_shared_transfer() {
    for (const void* k : {reinterpret_cast<const void*>(&k_p_values<3>), reinterpret_cast<const void*>(&k_p_values<6>),
                          reinterpret_cast<const void*>(&k_w_values<3>), reinterpret_cast<const void*>(&k_w_values<6>),
                          reinterpret_cast<const void*>(&k_coarse_values<3>),
                          reinterpret_cast<const void*>(&k_coarse_values<6>)})
        FX_CUDA_CHECK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRowShared));
}

// A kernel of this file's module (preload_kernels() loads all of the module's kernels).
const void* kernels_anchor_amg_transfer() { return reinterpret_cast<const void*>(&k_iota); }

}  // namespace fx

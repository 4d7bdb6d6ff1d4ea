// Corner level of C3D20 meshes (see corner.hpp): structure, weights and Galerkin matrix.
#include <cuda_pipeline_primitives.h>

#include <cub/cub.cuh>

#include "common.hpp"
#include "corner.cuh"
#include "corner.hpp"

namespace fx {

namespace {

constexpr int kPairs8 = 36;
// C3D20 local node order: mid node 8 + k lies on the edge of corners kEdge[k]
__constant__ int8_t kEdge[12][2] = {{0, 1}, {1, 2}, {2, 3}, {3, 0}, {4, 5}, {5, 6},
                                    {6, 7}, {7, 4}, {0, 4}, {1, 5}, {2, 6}, {3, 7}};
// and corner a is on the edges kCornerEdge[a] (k of the mid nodes 8 + k)
__constant__ int8_t kCornerEdge[8][3] = {{0, 3, 8}, {0, 1, 9}, {1, 2, 10}, {2, 3, 11},
                                         {4, 7, 8}, {4, 5, 9}, {5, 6, 10}, {6, 7, 11}};

unsigned grid_for(int64_t n, int t = 256) { return (unsigned)((n + t - 1) / t); }

template <typename Op>
void cub_call(Op op, DBuf<uint8_t>& tmp, cudaStream_t s) {
    size_t bytes = 0;
    FX_CUDA_CHECK(op(nullptr, bytes));
    if (tmp.n < bytes) tmp.alloc(bytes, s);
    FX_CUDA_CHECK(op(tmp.ptr, bytes));
}

// flag[node] = 1 for element corners
__global__ void k_flag_corners(int n4, const int32_t* __restrict__ conn4, int n20, const int32_t* __restrict__ conn20,
                               int32_t* __restrict__ flag) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t m4 = 4 * (int64_t)n4, m8 = 8 * (int64_t)n20;
    if (t < m4) flag[conn4[t]] = 1;
    else if (t < m4 + m8) flag[conn20[20 * ((t - m4) / 8) + (t - m4) % 8]] = 1;
}

// every element's mid nodes: the smaller and larger corner of the edge, the least pair per node
// (any order of the elements gives the same); a mid node that is a corner elsewhere counts as bad
__global__ void k_mid_pairs(int n20, const int32_t* __restrict__ conn20, const int32_t* __restrict__ flag,
                            unsigned long long* __restrict__ pair, int* __restrict__ bad) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= 12 * (int64_t)n20) return;
    const int32_t* c = conn20 + 20 * (t / 12);
    const int k = (int)(t % 12), m = c[8 + k], a = c[kEdge[k][0]], b = c[kEdge[k][1]];
    if (flag[m] || a == b) atomicOr(bad, 1);
    atomicMin(pair + m, ((unsigned long long)min(a, b) << 32) | (unsigned)max(a, b));
}

// a mid node that lies on different edges in different elements counts as bad
__global__ void k_mid_check(int n20, const int32_t* __restrict__ conn20, const unsigned long long* __restrict__ pair,
                            int* __restrict__ bad) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= 12 * (int64_t)n20) return;
    const int32_t* c = conn20 + 20 * (t / 12);
    const int k = (int)(t % 12), a = c[kEdge[k][0]], b = c[kEdge[k][1]];
    if (pair[c[8 + k]] != (((unsigned long long)min(a, b) << 32) | (unsigned)max(a, b))) atomicOr(bad, 1);
}

__global__ void k_corner_index(int n, const int32_t* __restrict__ flag, const int32_t* __restrict__ rank,
                               int32_t* __restrict__ corner_of, int32_t* __restrict__ fine_of) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    corner_of[i] = flag[i] ? rank[i] - 1 : -1;
    if (flag[i]) fine_of[rank[i] - 1] = i;
}

// parents of every mid node and its two child items (key = corner, or nc for nodes that have none)
__global__ void k_parents(int n, int nc, const int32_t* __restrict__ corner_of,
                          const unsigned long long* __restrict__ pair, int2* __restrict__ par,
                          int32_t* __restrict__ key, int32_t* __restrict__ item) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int2 p = make_int2(-1, -1);
    if (corner_of[i] < 0 && pair[i] != ~0ull)
        p = make_int2(corner_of[(int)(pair[i] >> 32)], corner_of[(int)(pair[i] & 0xffffffffu)]);
    par[i] = p;
    key[2 * (int64_t)i] = p.x >= 0 ? p.x : nc;
    key[2 * (int64_t)i + 1] = p.y >= 0 ? p.y : nc;
    item[2 * (int64_t)i] = 2 * i;
    item[2 * (int64_t)i + 1] = 2 * i + 1;
}

// ptr[r] = first of the n ascending keys that is >= r, r = 0 .. rows
__global__ void k_bounds(int64_t n, int rows, const int32_t* __restrict__ key, int32_t* __restrict__ ptr) {
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e > n) return;
    const int lo = e == 0 ? 0 : key[e - 1] + 1, hi = e == n ? rows : min(key[e], rows);
    for (int r = lo; r <= hi; ++r) ptr[r] = (int32_t)e;
}

__global__ void k_corner_conn(int n4, const int32_t* __restrict__ conn4, int n20, const int32_t* __restrict__ conn20,
                              const int32_t* __restrict__ corner_of, int32_t* __restrict__ out4,
                              int32_t* __restrict__ out8) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t m4 = 4 * (int64_t)n4, m8 = 8 * (int64_t)n20;
    if (t < m4) out4[t] = corner_of[conn4[t]];
    else if (t < m4 + m8) out8[t - m4] = corner_of[conn20[20 * ((t - m4) / 8) + (t - m4) % 8]];
}

__global__ void k_weights(int n, const int2* __restrict__ par, const int32_t* __restrict__ fine_of,
                          const double* __restrict__ x, double* __restrict__ wgt) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int2 p = par[i];
    double o[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    if (p.x >= 0) {
        const double *a = x + 3 * (int64_t)fine_of[p.x], *b = x + 3 * (int64_t)fine_of[p.y], *m = x + 3 * (int64_t)i;
        double e[3], d[3], l2 = 0.0, ed = 0.0;
        for (int k = 0; k < 3; ++k) {
            e[k] = b[k] - a[k];
            d[k] = m[k] - 0.5 * (a[k] + b[k]);
            l2 += e[k] * e[k];
            ed += e[k] * d[k];
        }
        if (l2 > 0.0) {
            o[0] = ed / l2;
            for (int k = 0; k < 3; ++k) {
                o[1 + k] = e[k] / l2;
                o[4 + k] = d[k] - o[0] * e[k];
            }
        }
    }
    for (int k = 0; k < 8; ++k) wgt[8 * (int64_t)i + k] = o[k];
}

__global__ void k_corner_xyz(int n, const int32_t* __restrict__ fine_of, const double* __restrict__ x,
                             double* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    for (int k = 0; k < 3; ++k) out[3 * (int64_t)i + k] = x[3 * (int64_t)fine_of[i] + k];
}

// Element Galerkin matrices P_e^T K_e P_e (36 node-pair blocks of the 8 corners) from the 210 blocks
// of K_e. CTA per element: K_e is staged in shared memory by asynchronous 16-byte copies (15 kB, read once:
// the floor is that traffic), T = K_e P_e (160 blocks: C = I/2 +- (t I - f d^T) of a mid node applied from
// the right acts on rows alone, so 16 threads per corner take a block row at a time) is formed beside it,
// then P_e^T T by a thread per block column. 32k elements: 255 us, bound by shared memory; 404 with
// copies through registers, 445 with a warp per element and a lane per block.
constexpr int kThreadsG = 128;
__global__ void __launch_bounds__(kThreadsG) k_corner_elements(const int32_t* __restrict__ conn,
                                                               const int32_t* __restrict__ corner_of,
                                                               const int2* __restrict__ par,
                                                               const double* __restrict__ wgt,
                                                               const double* __restrict__ ebuf,
                                                               double* __restrict__ out) {
    __shared__ __align__(16) double K[kPairs20 * 9];
    __shared__ double T[160 * 9];
    __shared__ double W[12 * 8];  // per mid node {t, f, d, sign of its first local corner}
    const int tid = threadIdx.x;
    const int64_t e = blockIdx.x;
    const double* src = ebuf + e * (kPairs20 * 9);
    // (K_e starts on a multiple of 16 bytes: 15,120 per C3D20 element after 720 per C3D4)
    for (int i = tid; i < kPairs20 * 9 / 2; i += kThreadsG) __pipeline_memcpy_async(K + 2 * i, src + 2 * i, 16);
    __pipeline_commit();
    if (tid < 96) {
        const int k = tid >> 3, node = conn[20 * e + 8 + k];
        if ((tid & 7) < 7) W[tid] = wgt[8 * (int64_t)node + (tid & 7)];
        else W[tid] = corner_of[conn[20 * e + kEdge[k][0]]] == par[node].x ? -1.0 : 1.0;
    }
    __pipeline_wait_prior(0);
    __syncthreads();
    auto sign = [&](int k, int a) { return kEdge[k][0] == a ? W[8 * k + 7] : -W[8 * k + 7]; };
    {  // rows of T_ib = K_ib + sum over b's mid nodes m of K_im C_mb: 16 threads per corner b, with its weights
        const int b = tid >> 4;
        int m[3];
        double w0[3], f[3][3], d[3][3];
#pragma unroll
        for (int u = 0; u < 3; ++u) {
            const int k = kCornerEdge[b][u];
            const double* w = W + 8 * k;
            const double sg = sign(k, b);
            m[u] = 8 + k;
            w0[u] = 0.5 + sg * w[0];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                f[u][c] = w[1 + c];
                d[u][c] = sg * w[4 + c];
            }
        }
        for (int t = tid & 15; t < 60; t += 16) {
            const int i = t / 3, r = t - 3 * i;
            auto row = [&](int j, double y[3]) {  // of K_ij
                const double* blk = K + 9 * pair_index(20, min(i, j), max(i, j)) + (i <= j ? 3 * r : r);
                const int st = i <= j ? 1 : 3;
#pragma unroll
                for (int c = 0; c < 3; ++c) y[c] = blk[c * st];
            };
            double o[3], y[3];
            row(b, o);
#pragma unroll
            for (int u = 0; u < 3; ++u) {
                row(m[u], y);
                const double yf = y[0] * f[u][0] + y[1] * f[u][1] + y[2] * f[u][2];
#pragma unroll
                for (int c = 0; c < 3; ++c) o[c] += w0[u] * y[c] - yf * d[u][c];
            }
#pragma unroll
            for (int c = 0; c < 3; ++c) T[180 * b + 3 * t + c] = o[c];  // block (b, i): at 20 b + i
        }
    }
    __syncthreads();
    if (tid < kPairs8 * 3) {  // column c of block q = (a, b): T_ab + sum over a's mid nodes m of C_ma^T T_mb
        const int q = tid / 3, c = tid - 3 * q;
        int a = 0, at = q;
        while (at >= 8 - a) at -= 8 - a++;
        const int b = a + at;
        double o[3];
#pragma unroll
        for (int r = 0; r < 3; ++r) o[r] = T[9 * (20 * b + a) + 3 * r + c];
#pragma unroll
        for (int u = 0; u < 3; ++u) {
            const int k = kCornerEdge[a][u];
            const double* w = W + 8 * k;
            const double* y = T + 9 * (20 * b + 8 + k) + c;
            const double sg = sign(k, a);
            const double fy = w[1] * y[0] + w[2] * y[3] + w[3] * y[6];
#pragma unroll
            for (int r = 0; r < 3; ++r) o[r] += (0.5 + sg * w[0]) * y[3 * r] - sg * w[4 + r] * fy;
        }
#pragma unroll
        for (int r = 0; r < 3; ++r) K[9 * q + 3 * r + c] = o[r];  // (K_e is not read any more)
    }
    __syncthreads();
    for (int i = tid; i < kPairs8 * 9; i += kThreadsG) out[e * (kPairs8 * 9) + i] = K[i];
}
static_assert(kThreadsG == 128 && kPairs8 * 3 <= kThreadsG, "16 threads per corner; a thread per block column");

// C = I / 2 +- M of a mid node towards one corner: y (3x3, row-major) -> y C (right) or C^T y (left)
__device__ __forceinline__ void mul_right(const double y[9], const MidWeight& w, double sg, double o[9]) {
#pragma unroll
    for (int r = 0; r < 3; ++r) {  // row r of y (I/2 + sg (t I - f d^T))
        const double yf = y[3 * r] * w.f[0] + y[3 * r + 1] * w.f[1] + y[3 * r + 2] * w.f[2];
#pragma unroll
        for (int c = 0; c < 3; ++c) o[3 * r + c] += (0.5 + sg * w.t) * y[3 * r + c] - sg * yf * w.d[c];
    }
}
__device__ __forceinline__ void mul_left(const double y[9], const MidWeight& w, double sg, double o[9]) {
#pragma unroll
    for (int c = 0; c < 3; ++c) {  // column c of (I/2 + sg (t I - d f^T)) y
        const double fy = w.f[0] * y[c] + w.f[1] * y[3 + c] + w.f[2] * y[6 + c];
#pragma unroll
        for (int r = 0; r < 3; ++r) o[3 * r + c] += (0.5 + sg * w.t) * y[3 * r + c] - sg * w.d[r] * fy;
    }
}

__global__ void k_bc_counts(int n, const int32_t* __restrict__ dof, const double* __restrict__ cnt,
                            double* __restrict__ out) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m < n) out[dof[m]] = cnt[m];
}

// P^T D P of the penalty's diagonal D, added to the level's matrix. A thread owns a block row: its
// corner's own DOFs and the constrained mid nodes among its children, in order.
__global__ void k_corner_penalty(CornerView V, const double* __restrict__ bc_cnt,
                                 const unsigned long long* __restrict__ maxdiag, const int32_t* __restrict__ row_ptr,
                                 const int32_t* __restrict__ goff, const int32_t* __restrict__ cols,
                                 double* __restrict__ vals) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= V.n) return;
    const double md = __longlong_as_double((long long)*maxdiag);
    if (!(md > 0.0)) return;
    const double pen = md * 1.0e6;
    const int64_t g0 = goff[i], ng = goff[i + 1] - g0;
    const int cnt = row_ptr[i + 1] - row_ptr[i];
    auto add = [&](int col, const double x[9]) {
        for (int k = 0; k < cnt; ++k)
            if (cols[4 * g0 + k] == col) {
                for (int e = 0; e < 9; ++e) vals[(g0 * 9 + e * ng + k / 4) * 4 + (k & 3)] += pen * x[e];
                return;
            }
    };
    {
        const double* c = bc_cnt + 3 * (int64_t)V.fine_of[i];
        if (c[0] != 0.0 || c[1] != 0.0 || c[2] != 0.0) {
            const double x[9] = {c[0], 0, 0, 0, c[1], 0, 0, 0, c[2]};
            add(i, x);
        }
    }
    for (int e = V.ch_ptr[i]; e < V.ch_ptr[i + 1]; ++e) {
        const int item = V.ch[e], node = item >> 1;
        const double* c = bc_cnt + 3 * (int64_t)node;
        if (c[0] == 0.0 && c[1] == 0.0 && c[2] == 0.0) continue;
        const MidWeight w = mid_weight(V.wgt, node);
        const int2 p = V.par[node];
        const double sg = (item & 1) ? 1.0 : -1.0;
        const double D[9] = {c[0], 0, 0, 0, c[1], 0, 0, 0, c[2]};
        double L[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0}, X[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0}, Y[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
        mul_left(D, w, sg, L);  // C^T D
        mul_right(L, w, sg, X);
        mul_right(L, w, -sg, Y);
        add(i, X);
        add((item & 1) ? p.x : p.y, Y);
    }
}

}  // namespace

CornerView corner_view(const CornerLevel& c) {
    return CornerView{c.n, c.n_fine, c.corner_of.ptr, c.fine_of.ptr, c.ch_ptr.ptr, c.ch.ptr, c.par.ptr, c.wgt.ptr};
}

void build_corner_level(const ElemView& g4, const ElemView& g20, int n_nodes, uint64_t id, CornerLevel& c,
                        cudaStream_t s) {
    c.built_for = id;
    c.usable = false;
    c.n_fine = n_nodes;
    if (!g20.n) return;
    const int64_t ends = 4 * (int64_t)g4.n + 8 * (int64_t)g20.n;
    const unsigned ge = grid_for(ends), gm = grid_for(12 * (int64_t)g20.n);
    DBuf<int32_t> flag, rank, key, key_s, item;
    DBuf<unsigned long long> pair;
    DBuf<int> bad;
    DBuf<uint8_t> tmp;
    flag.alloc(n_nodes, s);
    flag.zero(s);
    rank.alloc(n_nodes, s);
    pair.alloc(n_nodes, s);
    FX_CUDA_CHECK(cudaMemsetAsync(pair.ptr, 0xff, pair.bytes(), s));
    bad.alloc(1, s);
    bad.zero(s);
    FX_LAUNCH(k_flag_corners, ge, 256, 0, s, g4.n, g4.conn, g20.n, g20.conn, flag.ptr);
    FX_LAUNCH(k_mid_pairs, gm, 256, 0, s, g20.n, g20.conn, flag.ptr, pair.ptr, bad.ptr);
    FX_LAUNCH(k_mid_check, gm, 256, 0, s, g20.n, g20.conn, pair.ptr, bad.ptr);
    cub_call([&](void* t, size_t& b) {
        return cub::DeviceScan::InclusiveSum(t, b, flag.ptr, rank.ptr, n_nodes, s);
    }, tmp, s);
    int h[2] = {0, 0};
    FX_CUDA_CHECK(cudaMemcpyAsync(h, rank.ptr + n_nodes - 1, sizeof(int), cudaMemcpyDeviceToHost, s));
    FX_CUDA_CHECK(cudaMemcpyAsync(h + 1, bad.ptr, sizeof(int), cudaMemcpyDeviceToHost, s));
    stream_wait(s, "corner level");
    c.n = h[0];
    if (h[1] || c.n > 0.6 * n_nodes) return;
    c.usable = true;
    c.corner_of.alloc(n_nodes, s);
    c.fine_of.alloc(c.n, s);
    c.par.alloc(n_nodes, s);
    FX_LAUNCH(k_corner_index, grid_for(n_nodes), 256, 0, s, n_nodes, flag.ptr, rank.ptr, c.corner_of.ptr,
              c.fine_of.ptr);
    const int64_t items = 2 * (int64_t)n_nodes;
    key.alloc(items, s);
    key_s.alloc(items, s);
    item.alloc(items, s);
    c.ch.alloc(items, s);
    c.ch_ptr.alloc(c.n + 1, s);
    FX_LAUNCH(k_parents, grid_for(n_nodes), 256, 0, s, n_nodes, c.n, c.corner_of.ptr, pair.ptr, c.par.ptr, key.ptr,
              item.ptr);
    int bits = 1;
    while ((int64_t(1) << bits) < c.n + 1) ++bits;
    cub_call([&](void* t, size_t& b) {
        return cub::DeviceRadixSort::SortPairs(t, b, key.ptr, key_s.ptr, item.ptr, c.ch.ptr, items, 0, bits, s);
    }, tmp, s);
    FX_LAUNCH(k_bounds, grid_for(items + 1), 256, 0, s, items, c.n, key_s.ptr, c.ch_ptr.ptr);
    c.conn4.alloc(4 * (size_t)g4.n, s);
    c.conn8.alloc(8 * (size_t)g20.n, s);
    FX_LAUNCH(k_corner_conn, ge, 256, 0, s, g4.n, g4.conn, g20.n, g20.conn, c.corner_of.ptr, c.conn4.ptr, c.conn8.ptr);
    build_bsr_structure(ElemView{g4.n, c.conn4.ptr, nullptr}, ElemView{g20.n, c.conn8.ptr, nullptr}, c.n, c.S, s, 8);
}

void corner_weights(CornerLevel& c, const double* xyz, cudaStream_t s) {
    c.wgt.alloc(8 * (size_t)c.n_fine, s);
    c.xyz.alloc(3 * (size_t)c.n, s);
    FX_LAUNCH(k_weights, grid_for(c.n_fine), 256, 0, s, c.n_fine, c.par.ptr, c.fine_of.ptr, xyz, c.wgt.ptr);
    FX_LAUNCH(k_corner_xyz, grid_for(c.n), 256, 0, s, c.n, c.fine_of.ptr, xyz, c.xyz.ptr);
}

void corner_matrix(CornerLevel& c, const ElemView& g4, const ElemView& g20, const double* ebuf, const BcView& bc,
                   const unsigned long long* maxdiag, cudaStream_t s) {
    const size_t v4 = (size_t)g4.n * kPairs4 * 9;
    c.ebuf.alloc(v4 + (size_t)g20.n * kPairs8 * 9 + 9, s);
    if (v4) FX_CUDA_CHECK(cudaMemcpyAsync(c.ebuf.ptr, ebuf, v4 * sizeof(double), cudaMemcpyDeviceToDevice, s));
    if (g20.n)
        FX_LAUNCH(k_corner_elements, (unsigned)g20.n, kThreadsG, 0, s, g20.conn, c.corner_of.ptr, c.par.ptr, c.wgt.ptr,
                  ebuf + v4, c.ebuf.ptr + v4);
    c.vals.alloc((size_t)c.S.n_groups * 36, s);
    launch_bsr_gather<double>(c.S, c.ebuf.ptr, c.vals.ptr, s);
    if (bc.n) {
        c.bc_cnt.alloc(3 * (size_t)c.n_fine, s);
        c.bc_cnt.zero(s);
        FX_LAUNCH(k_bc_counts, grid_for(bc.n), 256, 0, s, bc.n, bc.dof, bc.cnt, c.bc_cnt.ptr);
        FX_LAUNCH(k_corner_penalty, grid_for(c.n), 256, 0, s, corner_view(c), c.bc_cnt.ptr, maxdiag, c.S.row_ptr.ptr,
                  c.S.goff.ptr, c.S.cols.ptr, c.vals.ptr);
    }
    c.minv.alloc((size_t)c.n * 9, s);
    launch_block_jacobi<double>(c.S, c.vals.ptr, c.minv.ptr, s);
}

// A kernel of this file's module (preload_kernels() loads all of the module's kernels).
const void* kernels_anchor_corner() { return reinterpret_cast<const void*>(&k_bounds); }

}  // namespace fx

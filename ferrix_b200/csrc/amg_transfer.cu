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

bool build_transfer(const FineView& F, int na, const int32_t* agg, const double* Q, const double* dinv, double omega,
                    Transfer& t, DBuf<int32_t>& c_ptr, DBuf<int32_t>& c_cols, int64_t* ncb, DBuf<uint8_t>& tmp,
                    cudaStream_t s) {
    const int n = F.n, bs = F.bs;
    const int abits = bits_for(na > 1 ? na : 2), nbits = bits_for(n > 1 ? n : 2);
    t.n = n;
    t.na = na;
    t.bs = bs;
    DBuf<int64_t> cnt, end;
    DBuf<int32_t> w_ptr;
    bool smooth = F.nblocks > 0;
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
    // ---- entries by aggregate (a stable sort: ascending fine row within one)
    {
        DBuf<int32_t> ids, col_s, t_ent;
        ids.alloc(p.n, s);
        col_s.alloc(p.n, s);
        t_ent.alloc(p.n, s);
        t.t_row.alloc(p.n, s);
        t.t_ptr.alloc(na + 1, s);
        FX_LAUNCH(k_iota, grid_for(p.n), 256, 0, s, p.n, ids.ptr);
        cub_call([&](void* q, size_t& b) {
            return cub::DeviceRadixSort::SortPairs(q, b, p.col.ptr, col_s.ptr, ids.ptr, t_ent.ptr, (int)p.n, 0,
                                                   abits, s);
        }, tmp, s);
        FX_LAUNCH(k_row_bounds, grid_for(p.n + 1), 256, 0, s, p.n, na, col_s.ptr, t.t_ptr.ptr);
        FX_LAUNCH(k_pick, grid_for(p.n), 256, 0, s, p.n, t_ent.ptr, p.row.ptr, t.t_row.ptr);
        const int64_t n32 = bs == 3 ? p32_size<3>(p.n) : p32_size<6>(p.n);
        t.val32.alloc(n32, s);
        t.t_val32.alloc(n32, s);
        if (bs == 3) {
            FX_LAUNCH(k_interleave<3>, grid_for(n32), 256, 0, s, p.n, nullptr, t.val.ptr, t.val32.ptr);
            FX_LAUNCH(k_interleave<3>, grid_for(n32), 256, 0, s, p.n, t_ent.ptr, t.val.ptr, t.t_val32.ptr);
        } else {
            FX_LAUNCH(k_interleave<6>, grid_for(n32), 256, 0, s, p.n, nullptr, t.val.ptr, t.val32.ptr);
            FX_LAUNCH(k_interleave<6>, grid_for(n32), 256, 0, s, p.n, t_ent.ptr, t.val.ptr, t.t_val32.ptr);
        }
    }
    // ---- W = A P
    if (F.nblocks > 0) {
        compress(total, nbits + abits, abits, t.w, tmp, s, [&](auto* keys, uint64_t* vals) {
            using KT = std::remove_pointer_t<decltype(keys)>;
            FX_LAUNCH(k_items_w<KT>, grid_for(F.nblocks), 256, 0, s, F, t.ptr.ptr, p.col.ptr, end.ptr, abits, keys, vals);
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
            FX_LAUNCH(k_items_c<KT>, grid_for(p.n), 256, 0, s, p.n, p.row.ptr, p.col.ptr, w_ptr.ptr, t.w.col.ptr,
                      end.ptr, abits, keys, vals);
        });
    }
    *ncb = t.c.n;
    c_ptr.alloc(na + 1, s);
    c_cols = std::move(t.c.col);
    if (t.c.n) FX_LAUNCH(k_row_bounds, grid_for(t.c.n + 1), 256, 0, s, t.c.n, na, t.c.row.ptr, c_ptr.ptr);
    else c_ptr.zero(s);
    t.w.col.release();
    t.col = std::move(p.col);
    return smooth;
}

void galerkin_product(const FineView& F, const Transfer& t, double* c_vals, cudaStream_t s) {
    if (!t.c.n) return;
    DBuf<double> W;
    W.alloc((size_t)t.w.n * t.bs * 6, s);
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

// A kernel of this file's module (preload_kernels() loads all of the module's kernels).
const void* kernels_anchor_amg_transfer() { return reinterpret_cast<const void*>(&k_iota); }

}  // namespace fx

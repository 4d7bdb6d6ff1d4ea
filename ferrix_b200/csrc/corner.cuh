// Transfer between the nodes of a C3D20 mesh and its corners (corner.hpp), shared by the per-step
// kernels and the persistent solve.
#pragma once

#include "corner.hpp"
#include "device.cuh"

namespace fx {

struct MidWeight {
    double t, f[3], d[3];
};

__device__ __forceinline__ MidWeight mid_weight(const double* __restrict__ wgt, int node) {
    const double2* w = reinterpret_cast<const double2*>(wgt + 8 * (int64_t)node);
    const double2 a = __ldg(w), b = __ldg(w + 1), c = __ldg(w + 2), e = __ldg(w + 3);
    return MidWeight{a.x, {a.y, b.x, b.y}, {c.x, c.y, e.x}};
}

constexpr int kCornerLanes = 8;  // lanes per corner of the restriction: one round of loads for its ~6 mid nodes

// (P^T r) of corner i by a group of kCornerLanes lanes (sub: lane within it), the lanes' sums
// added by an xor tree; every lane of the warp takes part, with i < 0 for a group without a corner.
// wait: called in every lane before r is read, with the list's ends and the corner's node at hand.
template <bool CG, typename Wait = NoWait>
__device__ __forceinline__ void corner_restrict_row(const CornerView& V, const double* r, int i, int sub,
                                                    double (&t)[3], Wait wait = Wait()) {
    auto ld = [&](int64_t k) { return CG ? __ldcg(r + k) : r[k]; };
    t[0] = t[1] = t[2] = 0.0;
    const int e0 = i >= 0 ? __ldg(V.ch_ptr + i) : 0, e1 = i >= 0 ? __ldg(V.ch_ptr + i + 1) : 0;
    const int64_t o = i >= 0 && sub == 0 ? 3 * (int64_t)__ldg(V.fine_of + i) : 0;
    wait();
    if (i >= 0) {
        if (sub == 0)
            for (int k = 0; k < 3; ++k) t[k] = ld(o + k);
        for (int e = e0 + sub; e < e1; e += kCornerLanes) {
            const int item = __ldg(V.ch + e), node = item >> 1;
            const MidWeight w = mid_weight(V.wgt, node);
            const double r0 = ld(3 * (int64_t)node), r1 = ld(3 * (int64_t)node + 1), r2 = ld(3 * (int64_t)node + 2);
            const double fr = w.f[0] * r0 + w.f[1] * r1 + w.f[2] * r2;
            const double sg = (item & 1) ? 1.0 : -1.0;  // I / 2 -+ M^T
            t[0] += 0.5 * r0 + sg * (w.t * r0 - w.d[0] * fr);
            t[1] += 0.5 * r1 + sg * (w.t * r1 - w.d[1] * fr);
            t[2] += 0.5 * r2 + sg * (w.t * r2 - w.d[2] * fr);
        }
    }
#pragma unroll
    for (int s = kCornerLanes / 2; s > 0; s >>= 1)
#pragma unroll
        for (int k = 0; k < 3; ++k) t[k] += __shfl_xor_sync(0xffffffffu, t[k], s);
}

// (P x_c) of fine node j
// wait: called before xc is read, with the node's parents at hand.
template <bool CG, typename Wait = NoWait>
__device__ __forceinline__ void corner_prolong_node(const CornerView& V, const double* xc, int j, double (&u)[3],
                                                    Wait wait = Wait()) {
    auto ld = [&](int64_t k) { return CG ? __ldcg(xc + k) : xc[k]; };
    const int i = __ldg(V.corner_of + j);
    const int2 p = __ldg(V.par + j);
    wait();
    u[0] = u[1] = u[2] = 0.0;
    if (i >= 0) {
        for (int k = 0; k < 3; ++k) u[k] = ld(3 * (int64_t)i + k);
    } else if (p.x >= 0) {
        const MidWeight w = mid_weight(V.wgt, j);
        double a[3], b[3], e[3];
        for (int k = 0; k < 3; ++k) {
            a[k] = ld(3 * (int64_t)p.x + k);
            b[k] = ld(3 * (int64_t)p.y + k);
        }
        for (int k = 0; k < 3; ++k) e[k] = b[k] - a[k];
        const double de = w.d[0] * e[0] + w.d[1] * e[1] + w.d[2] * e[2];
        for (int k = 0; k < 3; ++k) u[k] = 0.5 * (a[k] + b[k]) + w.t * e[k] - w.f[k] * de;
    }
}

}  // namespace fx

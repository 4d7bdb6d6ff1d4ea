// Corner level of C3D20 meshes: the multigrid's first coarse level holds the element corners only
// (three DOFs per node, trilinear functions), about a quarter of the nodes.
//
// A mid-edge node interpolates from its edge's two corners; where it lies off the edge's middle
// (offset d = t e + d', e the edge, d' normal to it) the part along the edge moves the
// weights and the normal part turns with the edge:
//   u = (u1 + u2) / 2 + M (u2 - u1),  M = t I - f d'^T,  f = e / |e|^2,
// so that rigid motions of a distorted mesh stay close to the coarse space (a 3 x 4 x 60 jittered
// box: 36 CG iterations against 49 with plain averages).
// The Galerkin matrix P^T K P is formed per element (P only couples nodes of one element) and
// gathered into a BSR3 matrix of its own, so the fine-level smoother kernels run on it as they are.
#pragma once

#include <cstdint>

#include "kernels.hpp"

namespace fx {

struct CornerLevel {
    uint64_t built_for = 0;  // BsrStructure::id of the mesh structure this was built for (0: none)
    bool usable = false;     // the mesh has mid nodes and every one lies on one edge
    int n = 0, n_fine = 0;   // corners, nodes of the mesh
    DBuf<int32_t> corner_of;  // per fine node: its corner index, -1 for the others
    DBuf<int32_t> fine_of;    // per corner: its fine node
    DBuf<int2> par;           // per fine node: corner indices of a mid node's edge, else (-1, -1)
    DBuf<int32_t> ch_ptr, ch;  // per corner: its mid nodes, 2 * node + (1 when it is the edge's second corner)
    DBuf<int32_t> conn4, conn8;  // elements over corner indices
    BsrStructure S;
    DBuf<double> wgt;  // per fine node {t, f, d', 0}
    DBuf<double> ebuf, vals, minv, xyz, bc_cnt;
};

// Builds the level's structure for the mesh (once per mesh); c.usable tells whether it pays: at
// least 40 % of the nodes are mid nodes, and no node is a corner of one element and a mid node of
// another or lies on two different edges.
void build_corner_level(const ElemView& g4, const ElemView& g20, int n_nodes, uint64_t id, CornerLevel& c,
                        cudaStream_t s);
// interpolation weights and corner coordinates of the configuration xyz
void corner_weights(CornerLevel& c, const double* xyz, cudaStream_t s);
// c.vals = P^T K P of the element buffer's matrix with the penalty of the constrained DOFs, and
// c.minv, its 3x3 block inverses
void corner_matrix(CornerLevel& c, const ElemView& g4, const ElemView& g20, const double* ebuf, const BcView& bc,
                   const unsigned long long* maxdiag, cudaStream_t s);

// What the transfer kernels read (also from the persistent solve).
struct CornerView {
    int n = 0, n_fine = 0;
    const int32_t *corner_of = nullptr, *fine_of = nullptr, *ch_ptr = nullptr, *ch = nullptr;
    const int2* par = nullptr;
    const double* wgt = nullptr;
};
CornerView corner_view(const CornerLevel& c);

}  // namespace fx

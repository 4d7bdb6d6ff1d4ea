// Aggregation multigrid preconditioner for the stiffness systems (3 DOF per
// node), used inside PCG in place of the 3x3 block-Jacobi preconditioner.
//
// Hierarchy (setup, all on the GPU, deterministic):
//   * C3D20 meshes: the first coarse level is the corner level (corner.hpp), a planar BSR3
//     matrix like the fine one (417k-DOF box to 1e-10: 116 CG iterations without it and with
//     unsmoothed aggregation, 36 with both, 59.2 -> 25.4 ms a solve);
//   * aggregation by spatial binning of the level's points (nodes, then
//     aggregate centroids) into the cells of a
//     grid that cuts their bounding box into equal parts per direction;
//   * tentative prolongator from the six rigid-body modes (three translations,
//     three rotations about the aggregate centroid): per aggregate a QR of the
//     stacked near-null-space rows (one warp per aggregate, modified
//     Gram-Schmidt applied twice); Q gives the tentative rows, R the next
//     level's near-null-space (Vanek, Mandel & Brezina 1996);
//   * smoothed prolongator P = (I - omega D^-1 A) Q and Galerkin coarse matrix
//     A_c = P^T A P (amg_transfer.hpp). Without the smoothing step the CG needs about twice
//     the iterations (C3D4, 205k DOF to 1e-10: 64 against 36, 14.3 -> 13.8 ms a solve);
//   * Chebyshev smoothing of degree 2 on D^-1 A (D = block diagonal) with the
//     largest eigenvalue from power iteration; dense inverse at the coarsest
//     level.
//   * a last planar level that is small enough itself (kDensePlanarDof) takes the dense inverse
//     and ends the hierarchy: the corner level of small C3D20 meshes, or a small C3D4 system whole.
// Application: one V-cycle per PCG iteration.
#pragma once

#include <cuda_fp16.h>

#include <vector>

#include "amg_transfer.hpp"
#include "corner.hpp"
#include "kernels.hpp"
#include "pcg.hpp"

namespace fx {

// State of the software grid barrier of the cooperative coarse-cycle launch (zeroed
// before a solve; a wait that ran out leaves it inconsistent until then).
struct GridBarState {
    unsigned int count, gen;
};

struct ClInst;

struct AmgLevel {
    int n = 0;   // block rows (nodes at level 0, aggregates above)
    int bs = 3;  // block size
    // planar levels (the fine system, and the corner level of C3D20 meshes): BSR3 matrix, 3x3 block
    // inverses of its diagonal, and the smoother's copies of the values: FP32, or FP16 of the
    // scaled matrix S A S (S = diag(a_ii)^-1/2) with sqrt(a_ii) per node (null: FP64 smoothing)
    const BsrStructure* S0 = nullptr;
    const double* vals0 = nullptr;
    const double* dinv0 = nullptr;
    const float* vals32 = nullptr;
    const __half* vals16 = nullptr;
    const float4* sq4 = nullptr;
    // coarse levels: row-major block CSR, blocks of bs x bs
    DBuf<int32_t> row_ptr, cols;
    DBuf<double> vals, dinv;
    DBuf<double2> pvals;  // the cycle's copy of vals (coarse_row6)
    int64_t nblocks = 0;
    double lmax = 0.0;
    // transfer to the next level (its pair lists are kept for refresh) and the scale of its
    // coarse corrections relative to Amg::overcorrect()
    Transfer tr;
    double pscale = 1.0;
    bool corner_next = false;  // the next level is the corner level (transfer corner.hpp instead of tr)
    // work vectors (n * bs); xs: at 6x6 levels the pre-smoothed iterate (the cycle's result goes to
    // x), at the corner level the cycle's result
    DBuf<double> x, b, r, d, t, xs;
    const double* result() const { return S0 ? xs.ptr : x.ptr; }
    // planar levels with FP32 smoother values: directions and the iterate as float4 per node
    DBuf<float> d4a, d4b, x4;
    // coarsest level: dense inverse (n*bs)^2
    bool coarsest = false;
    DBuf<double> dense_inv;
    // K-cycle work vectors (first coarse level): z1, v1, r, z2, v2 and scalars
    DBuf<double> kc[5], kcs;
    DBuf<int32_t> blk_row;  // levels > 0: the row of every block
    // last power-iteration vector of the eigenvalue estimate (start of the next refresh's)
    DBuf<double> ev;
    const double* dinv_ptr() const { return S0 ? dinv0 : dinv.ptr; }
};

struct AmgStats {
    int levels = 0;
    std::vector<int> sizes;   // DOF per level
    double setup_ms = 0.0;
};

// A planar level's matrix as setup() and refresh() take it (AmgLevel's fields of the same names).
struct PlanarIn {
    const BsrStructure* S = nullptr;
    const double *vals = nullptr, *dinv = nullptr;
    const float* vals32 = nullptr;
    const __half* vals16 = nullptr;
    const float4* sq4 = nullptr;
};

// First smoothing step of a coarse level, done by the restriction kernel into it.
struct CoarseStart {
    const double* dinv;  // 6x6 block inverses of the coarse level
    double *r, *d, *xs;
    double c2;
};

class Amg {
   public:
    // in: the fine matrix and, with a corner level (corner != null), that level's. xyz: FP64
    // coordinates (device, 3 per node) of the last planar level's nodes. cell0: edge of the first
    // aggregates' cells, 0 = chosen from the mesh (pick_cell; node_volume: volume per such node).
    // dense: the last planar level may be the coarsest (dense_planar()); not with a cell0 of the caller's.
    void setup(const PlanarIn* in, const CornerLevel* corner, const double* xyz, double cell0, double node_volume,
               bool dense, cudaStream_t s, AmgStats* st);
    // New matrix values on the structure of the last setup: aggregates, prolongators (values
    // included) and coarse patterns are kept; coarse values, block inverses, eigenvalue
    // estimates and the coarsest inverse are recomputed.
    void refresh(const PlanarIn* in, cudaStream_t s, AmgStats* st);
    // New fine matrix values only: the smoother works on them, everything below and the eigenvalue
    // estimates stay as they are.
    void keep(const PlanarIn& fine, AmgStats* st);
    int planar() const { return planar_; }  // planar levels: 1, or 2 with a corner level
    uint64_t built_for = 0;  // BsrStructure::id of the last setup (0: none)
    // Chebyshev degree (1..8)
    void set_degree(int degree) { degree_ = degree; }
    // every transfer of the next setup tentative, and no planar level the coarsest (PcgOptions)
    void set_tentative(bool on) { tentative_ = on; }
    // FP16 smoother directions: where the V-cycle started from x = 0 finds r.D^-1 r of its
    // right-hand side (rdr) and the two floats where each V-cycle publishes its power-of-two
    // scale of the stored directions (hs); null: unscaled
    void set_smoother_scale(const double* rdr, float* hs) {
        rdr_ = rdr;
        hs_ = hs;
    }
    // K-cycle at the first coarse level (true) or V-cycles throughout.
    void set_cycle(bool kcycle) { kcycle_ = kcycle; }
    // Chebyshev smoother: 0 = first kind on [lmax/30, lmax], 1 = fourth kind
    void set_smoother_kind(int kind) { cheb_kind_ = kind; }
    // coarse corrections x += alpha P e; first-kind Chebyshev interval [lmax / ratio, lmax]
    // scale of coarse corrections; all: of every one (PcgOptions), else of a level's times its pscale
    void set_overcorrect(double alpha, bool all) {
        alpha_ = alpha;
        alpha_all_ = all;
    }
    double pscale(const AmgLevel& l) const { return alpha_all_ ? 1.0 : l.pscale; }
    void set_cheb_ratio(double ratio) { cheb_ratio_ = ratio; }
    bool kcycle() const { return kcycle_; }
    // z = cycle(r), FP64 vectors of 3 * n_nodes. With part != null the last smoothing step also
    // leaves partial sums of (r.z, r.zold) (zold null: 0; for the flexible CG), two doubles for each
    // of its apply_grid() CTAs.
    // started: the level-0 start (r0 = b, x = d = c2 D^-1 b) was done by the caller, into start0()
    void apply(const double* r, double* z, double* part, const double* zold, cudaStream_t s, bool started = false);
    unsigned apply_grid() const;
    // slots of the `part` buffer apply() writes
    void set_part_slots(int64_t n) { part_slots_ = n; }
    // where the level-0 start writes: the smoother's residual, iterate and first direction
    // (FP32 float4 per node when the smoother is FP32, else FP64), and its coefficient
    struct Start0 {
        double *r, *x, *d;
        float4* d4;
        double c2;
        const float4* sq4;  // FP16 smoother: the float4 direction is written scaled by sqrt(a_ii)
        float* hs;          // FP16 directions: where the start publishes the V-cycle's scale (else null)
    };
    Start0 start0() const;
    // the hierarchy, smoother coefficients and work vectors, for the persistent solve
    void describe(ClInst& out) const;
    // The coarse part of each V-cycle as one cooperative launch (on: after every setup /
    // refresh the hierarchy's descriptor is uploaded; flag = where a barrier timeout is
    // reported) or as one launch per coarse-level step (off).
    void set_fused_coarse(bool on, double* flag) {
        fused_coarse_ = on;
        gflag_ = flag;
    }
    void upload_descriptor(cudaStream_t s);
    int degree() const { return degree_; }
    double overcorrect() const { return alpha_; }
    std::vector<AmgLevel> L;

   private:
    // started: the restriction into this level already did the first smoothing step
    void cycle(int l, const double* b, double* x, cudaStream_t s, bool started = false);
    // the start that the restriction into level m does (dinv null: none)
    CoarseStart coarse_start(int m) const;
    void coarse(int m, cudaStream_t s);
    void coarsest_inverse(AmgLevel& l, cudaStream_t s);
    // V-cycle from planar level m (whose smoother values are VT)
    template <typename VT>
    void vcycle_of(int m, const double* b, double* z, double* part, const double* zold, cudaStream_t s, bool started);
    void vcycle(int m, const double* b, double* z, double* part, const double* zold, cudaStream_t s, bool started);
    void first_coarse(cudaStream_t s);  // from the last planar level's residual into its iterate
    int planar_ = 1;
    CornerView corner_;
    bool kcycle_ = false;
    int64_t part_slots_ = 0;
    int cheb_kind_ = 0;
    double alpha_ = 1.0, cheb_ratio_ = 30.0;
    bool alpha_all_ = false;
    int degree_ = 2;
    bool tentative_ = false;
    const double* rdr_ = nullptr;
    float* hs_ = nullptr;
    float* h16_scale_slot() const;
    bool fused_coarse_ = false;
    double* gflag_ = nullptr;
    DBuf<ClInst> desc_;
    DBuf<GridBarState> gbar_;
    DBuf<uint8_t> tmp_;
    DBuf<double> red_;  // reduction scratch
};

// ---- persistent solve of small systems (amg_cluster.cu)
// The whole multigrid-preconditioned CG of one system runs inside one thread-block
// cluster: every CG step and V-cycle phase is a loop over the cluster's threads,
// phases are separated by hardware cluster barriers, dot products are summed per
// CTA and across the cluster through distributed shared memory in a fixed order.
// One launch advances any number of systems (one cluster each); a system's
// arithmetic does not depend on the others, so it is the same alone and in a batch.
constexpr int kClMaxLevels = 8;

struct ClTransfer {  // transfer.cuh
    int na = 0;
    const int32_t *ptr = nullptr, *col = nullptr, *t_ptr = nullptr, *t_row = nullptr;
    const double2 *val = nullptr, *t_val = nullptr;
    double pscale = 1.0;
};

struct ClLevel {  // coarse level m >= 1 (6x6 blocks) and its transfer to level m + 1
    int n = 0, coarsest = 0;
    const int32_t *row_ptr = nullptr, *cols = nullptr;
    const double2* vals = nullptr;
    const double *dinv = nullptr, *dense_inv = nullptr;
    ClTransfer tr;
    double *x = nullptr, *b = nullptr, *r = nullptr, *d = nullptr, *t = nullptr, *xs = nullptr;
    double c2_start = 0.0, c1[8] = {}, c2[8] = {};
};

// A planar level: BSR3 (FP64 values; FP32 copy for the smoother or null), 3x3 block inverses
struct ClPlanar {
    int n = 0;
    const int32_t *goff = nullptr, *cols = nullptr;
    const double* vals64 = nullptr;
    const float* vals32 = nullptr;
    const double* dinv0 = nullptr;
    const float4* sq4 = nullptr;  // FP16 smoother: the FP32 iterate copy is scaled by sqrt(a_ii)
    double *lr = nullptr, *lx = nullptr, *ld = nullptr, *lt = nullptr;
    double *b = nullptr, *z = nullptr;  // the corner level's right-hand side and result
    const double* dense_inv = nullptr;  // the corner level as the coarsest
    float *d4a = nullptr, *d4b = nullptr, *x4 = nullptr;
    double c2_start = 0.0, c1[8] = {}, c2[8] = {};
};

struct ClInst {
    int n = 0, levels = 0, planar = 1;  // lev[m] is used from m = planar on
    ClPlanar pl[2];
    CornerView corner;     // with two planar levels: the transfer between them
    double corner_scale = 1.0;  // of its corrections, relative to the overcorrection factor
    ClTransfer tr;         // last planar level to the first 6x6 level
    // the CG: right-hand side, iterate and work vectors (3n each)
    const double* b = nullptr;
    double *x = nullptr, *r = nullptr, *z = nullptr, *p = nullptr, *q = nullptr;
    ClLevel lev[kClMaxLevels];
};

struct ClResult {
    long long iterations;
    int status;  // FX_OK, FX_NUMERICAL (breakdown), FX_CONVERGENCE (max_iter)
    int pad;
    double rzd, bd;  // r.D^-1 r at the end and b.D^-1 b
};

// Launches the persistent solve of `n` systems (descriptors and results in device
// memory); fp32: level-0 smoothing with the FP32 values. Smoother degree 1..8,
// coarse corrections scaled by alpha.
void launch_amg_cluster(const ClInst* insts, ClResult* res, int n, bool fp32, double rtol, int max_iter, int degree,
                        double alpha, cudaStream_t s);
// The coarse part of one V-cycle (restriction from the level-0 residual, coarse
// levels, prolongation into the level-0 iterate) of the system `inst` describes,
// as one cooperative launch over all SMs; *flag = 1 when a barrier wait ran out.
void launch_coarse_grid(const ClInst* inst, GridBarState* st, double* flag, bool fp32, int degree, double alpha,
                        cudaStream_t s);
// Systems of at most this many DOF are solved by the persistent launch by default, alone
// or in a batch. Alone, a cluster is slower than the multi-launch path from about 3,600 DOF
// on (3.9 ms against 3.3 ms there, 17 ms against 7 ms at 15k DOF); in a batch of 64 C3D4
// decks of 2k-60k DOF spread over four worker streams, one persistent launch per worker
// took 243-324 ms against 183 ms for the multi-launch path on every stream (B200).
constexpr int64_t kClDefaultMaxDof = 2000;

// A last planar level of at most this many DOF is inverted as it is: 3 DOF per row, so the inverse of
// 1,200 DOF (~0.6 ms) replaces the transfer's setup (~0.4 ms) and a smaller inverse, and the CG needs 20 %
// fewer iterations of fewer launches.
constexpr int kDensePlanarDof = 1200;
inline bool dense_planar(int64_t rows) { return 3 * rows <= kDensePlanarDof; }

// The default of the option amg_aggregate_nodes: with it the hierarchy chooses its cells (pick_cell).
constexpr int kAmgAggregateNodes = 40;

// CUDA-event time (ms per launch) of the fused fine-level Chebyshev step (SpMV +
// smoother update) on the given FP64 system, with FP32 values when fp32; bytes =
// compulsory traffic of one launch.
double profile_smoother_op(const BsrStructure& S, const double* vals64, const double* dinv64, bool fp32, bool fp16,
                           int reps,
                           cudaStream_t s, double* bytes);

// CG on the FP64 BSR3 system preconditioned by one V-cycle per iteration.
class AmgPcg {
   public:
    AmgPcg() = default;
    AmgPcg(const AmgPcg&) = delete;
    AmgPcg& operator=(const AmgPcg&) = delete;
    ~AmgPcg() { drop_graph(); }
    // Whether the next solve on this structure keeps the hierarchy below the fine level as it is
    // (reuse: the caller allows it, the matrix being a later Newton tangent of the same increment).
    // A V-cycle with a lagged coarse operator is symmetric, and positive definite as long as the fine level's kept
    // eigenvalue estimate bounds the new tangent's (the smoother's Chebyshev polynomial of the default interval and
    // degree exceeds 1 from 13/12 of it on); the CG tests the true system. So a solve on the kept
    // hierarchy may take longer, and can fail: once one takes a quarter (and more than 4 iterations) longer than
    // the first did, the next recomputes the hierarchy; one that fails, finds a negative r.z or takes twice the
    // first's iterations and 50 ends, to be done over on a recomputed one (kept(), outdate()). (NLGEOM beam, 16k DOF:
    // setups 80 of 215 ms with every tangent's recomputed.)
    bool keeps(const BsrStructure& S, bool reuse) const {
        return reuse && amg.built_for == S.id && !amg.L.empty() && amg.L[0].n == S.n_rows && !stale_;
    }
    bool kept() const { return kept_; }  // the last solve was on the kept hierarchy
    void outdate() { stale_ = true; }    // the next one recomputes it
    // iterations of the solve that prepare() was called for (solve() calls it itself)
    void solved(long long iterations) {
        if (fresh_) first_iters_ = iterations;
        else if (iterations > first_iters_ + first_iters_ / 4 + 4) stale_ = true;
        fresh_ = false;
    }
    // For the persistent solve: set up (or refresh) the hierarchy for the system and
    // allocate the CG vectors, without iterating; then describe it for the kernel.
    // corner: the corner level with its matrix, or null; cell0, node_volume: Amg::setup
    // persistent: for the persistent solve (which has no dense fine level)
    void prepare(const BsrStructure& S, const double* vals64, const double* dinv64, const double* xyz,
                 const CornerLevel* corner, double cell0, double node_volume, const PcgOptions& opt, cudaStream_t s,
                 AmgStats* st, bool reuse, bool persistent = false);
    ClInst describe(const double* b, double* x) const;
    // ||b - A x||_D / ||b||_D of the assembled FP64 system after a persistent solve
    double true_relres(const double* b, const double* x, cudaStream_t s);
    // reuse: keep the hierarchy (keeps()), or else at least its aggregates, prolongators and coarse
    // patterns when the last setup was on the same structure S (the values are refreshed)
    int solve(const BsrStructure& S, const double* vals64, const double* dinv64, const double* xyz,
              const CornerLevel* corner, double cell0, double node_volume, const double* b, double* x, const PcgOptions& opt, cudaStream_t s, int64_t* launches, long long* iters,
              double* relres, AmgStats* st, bool reuse = false);
    Amg amg;

   private:
    const BsrStructure* S_ = nullptr;
    const double* vals64_ = nullptr;
    const double* dinv64_ = nullptr;
    DBuf<double> r_, z_, z2_, p_, q_, part_, rd_part_, sc_;
    DBuf<float> vals32_;
    DBuf<__half> vals16_;
    DBuf<float4> sq4_;
    DBuf<float> hs_;  // FP16 smoother directions: the current V-cycle's {2^k, 2^-k}
    bool kept_ = false;
    bool no16_ = false;  // FP16 smoothing was given up on this hierarchy (kTry16)
    bool fresh_ = false, stale_ = false;  // the hierarchy was (re)computed for this solve; should be for the next
    long long first_iters_ = 0;
    // the captured iterations, kept while the hierarchy is: what they were captured with
    void drop_graph();
    const float* fine_fp32(const BsrStructure& S, const double* vals64, cudaStream_t s);  // into vals32_
    cudaGraphExec_t gexec_ = nullptr;
    int64_t graph_launches_ = 0;
    const void* graph_key_[4] = {nullptr, nullptr, nullptr, nullptr};
};

}  // namespace fx

// Internal declarations of the aggregation multigrid preconditioner (amg.cu).
#pragma once

#include <cuda_bf16.h>

#include <cstdint>
#include <vector>

#include "internal.cuh"

namespace bartels {

struct FactorPattern;
struct PcgState;

// One level of the hierarchy. Level 0 is the plan's Hessian (3x3 blocks in the
// plan's value layout, pinned vertices excluded); coarse levels hold 6x6 blocks
// (3 translations + 3 rotations per aggregate), row-major, in block-CSR order.
struct MgLevel {
  int n = 0;       // nodes (level 0: the plan's vertices)
  int bs = 0;      // DOFs per node: 3 on level 0, 6 on coarse levels
  int64_t nnzb = 0;
  int *rp = nullptr, *ci = nullptr, *dpos = nullptr;  // coarse levels: block pattern, diagonal positions
  float *val = nullptr;                               // coarse levels: 36 floats per block
  // coarse levels: BF16 copy (A + A^T) / 2 of val, exactly symmetric, read by
  // the smoothing, residual and power-iteration kernels; rev = position of
  // the transposed block
  __nv_bfloat16 *val16 = nullptr;
  int *rev = nullptr;
  float *dinv = nullptr;                              // coarse levels: 36 floats per node (inverse diagonal block)
  // transfer to the next coarser level (none on the coarsest)
  int nc = 0;                         // nodes of the next level
  int *agg = nullptr;                 // n: aggregate of each node, -1 outside the system (pinned)
  int *mptr = nullptr, *midx = nullptr;  // members of each aggregate, ascending
  float *Q = nullptr;                 // n x bs x 6 (row-major): the tentative prolongator block of each node
  int *gptr = nullptr;                // next level's nnzb + 1: Galerkin contributions per coarse block
  int2 *gent = nullptr;               // (fine row, fine block index) of each contribution, in summation order
  // work vectors (bs * n floats)
  float *b = nullptr, *x = nullptr, *x2 = nullptr, *r = nullptr, *d = nullptr, *d2 = nullptr;
  int deg = 1;  // Chebyshev degree of the smoother on this level
};

constexpr int kMgMaxLevels = 12;
constexpr int kMgCoef = 16;  // per level: 1/theta, then (c1, c2) per further Chebyshev step
constexpr int kMgClusterMax = 16;  // CTAs of the coarse-cycle cluster

constexpr int kMgClusterLevels = 8;

// One level as the coarse-cycle kernel sees it: its nodes split into
// contiguous ranges, one per CTA of the cluster (split: first node, bsplit:
// first block, msplit: first member-list entry of each range). The o_* are
// byte offsets of the level's areas in a CTA's shared memory, sized for the
// largest range; g* are the level's vectors in global memory, for the entries
// that other CTAs read.
struct MgClLevel {
  int deg = 1;
  int split[kMgClusterMax + 1] = {}, bsplit[kMgClusterMax + 1] = {}, msplit[kMgClusterMax + 1] = {};
  const int *rp = nullptr, *ci = nullptr;
  const int *mptr = nullptr, *midx = nullptr;  // members (finer nodes) of each node, none on the first level
  const int *agg = nullptr;                    // aggregate of each node (none on the last level)
  const __nv_bfloat16 *val16 = nullptr;
  const float *dinv = nullptr, *Q = nullptr;
  float *gb = nullptr, *gx = nullptr, *gd = nullptr, *gd2 = nullptr, *gres = nullptr;
  int o_val = 0, o_ci = 0, o_rp = 0, o_dinv = 0, o_Q = 0, o_agg = 0, o_mptr = 0, o_mem = 0;
  int o_b = 0, o_x = 0, o_r = 0, o_d = 0;
};
enum { kMgLastDense = 0, kMgLastExact = 1, kMgLastCheb = 2 };
struct MgClArgs {
  int nlev = 0, first = 0, ctas = 0, last_mode = 0, nd = 0, smem = 0;
  int o_db = 0;  // the coarsest right-hand side gathered by every CTA (dense)
  const float *ainv = nullptr, *coef = nullptr;
  MgClLevel lv[kMgClusterLevels];  // lv[0] is hierarchy level `first`
};

struct MgHierarchy {
  std::vector<MgLevel> lv;
  int dense = 0;          // the coarsest level is solved with its dense inverse
  int nd = 0;             // dense size (6 x nodes of the coarsest level)
  int coarse_blockdiag = 0;  // coarsest level is block diagonal: its block-Jacobi solve is exact
  float *ainv = nullptr;  // nd x nd
  float *panel = nullptr; // 2 x 6 x nd: pivot rows of the dense inversion
  float *coef = nullptr;  // kMgMaxLevels x kMgCoef Chebyshev coefficients (device)
  double *norms = nullptr;  // 2 per level: squared norms of the last two power iterates
  double *part = nullptr;   // reduction partials
  int nparts = 0;
  int pinned_gen = -1;    // plan->pinned_gen the hierarchy was built for
  int64_t coarse_nnz = 0; // stored entries of all coarse levels (operator complexity)
  PcgState *st_once = nullptr;  // state for a single application outside PCG
  double *segn = nullptr;       // per-segment norms of the finest level's last two power iterates
  int segn_n = 0;
  // BF16 copy of the finest level's values in the sliced-ELL layout, made exactly
  // symmetric, for the V-cycle's own SpMVs (nullptr: the FP32 values are used)
  uint2 *a16 = nullptr;
  // levels first .. last as one kernel of one thread-block cluster (ctas == 0: not used)
  MgClArgs cl;
  std::vector<void *> allocs;
  ~MgHierarchy();
};

// Smoother of level 0: block-Jacobi (minv, 6 floats per vertex) or the learned
// factor M = G^T G (gl / gu in the factor pattern fp).
struct MgSmoother {
  const float *minv = nullptr;
  const __nv_bfloat16 *gl = nullptr, *gu = nullptr;
  const FactorPattern *fp = nullptr;
  const uint2 *lsell = nullptr, *usell = nullptr;  // the factor in the plan's sliced-ELL layouts, on large meshes
};

// Build (or keep) the hierarchy for the plan's pattern and pinned set.
int mg_prepare(bartels_ctx ctx, bartels_mesh_plan plan);
void mg_destroy(MgHierarchy *mg);
// Galerkin products, inverse diagonal blocks, the coarsest inverse and the
// smoothers' eigenvalue bounds for the Hessian values (plan layout).
int mg_setup_numeric(bartels_ctx ctx, bartels_mesh_plan plan, const float *values, const MgSmoother &sm);
// z = B r (one V-cycle) for the PCG loop: every kernel is a no-op once st->done;
// the last one also forms r.z, beta = r.z / r.z_old and stores r.z in st.
// pre_done: the level-0 pre-smoothing was taken by mg_enqueue_update (block-
// Jacobi smoother only).
int mg_enqueue_apply(bartels_ctx ctx, bartels_mesh_plan plan, const float *values, const MgSmoother &sm,
                     const float *r, float *z, float *y, double *part, PcgState *st, bool pre_done);
// The PCG update (x += alpha p, r -= alpha Ap, r.r, iteration count and
// convergence test) fused with the level-0 block-Jacobi pre-smoothing of the
// next V-cycle.
int mg_enqueue_update(bartels_ctx ctx, bartels_mesh_plan plan, const MgSmoother &sm, const float *pa,
                      const float *pb, const float *ap, float *x, float *r, double *part, PcgState *st);
// z = B r once (no PCG state), for tests of the preconditioner itself.
int mg_apply_once(bartels_ctx ctx, bartels_mesh_plan plan, const float *values, const MgSmoother &sm, const float *r,
                  float *z);

}  // namespace bartels

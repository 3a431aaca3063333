// Aggregation multigrid preconditioner for the Newton systems.
//
// No counterpart in the reference, whose search direction factors the Hessian
// with Eigen::SparseLU (src/search_direction_newton_sparse.cpp:12-18). Block-
// Jacobi PCG needs O(1/h) iterations on these systems (1,759 per Newton
// iteration on the 96^3-cell cube); a multigrid V-cycle bounds them
// independently of the mesh size.
//
// Hierarchy (built once per plan pattern and pinned set, on the host):
//   * aggregates: greedy aggregation of the free vertices over the Hessian's
//     block graph in index order (pass 1: a node whose neighbourhood is still
//     free roots an aggregate of that neighbourhood; pass 2: the rest join the
//     lowest-numbered neighbouring aggregate; pass 3: leftovers group with their
//     free neighbours), the scheme of Vanek, Mandel & Brezina (1996);
//   * tentative prolongator: per aggregate, the six rigid-body modes of
//     elasticity (translations, rotations about the mesh centroid) restricted
//     to its members, orthonormalised (modified Gram-Schmidt, twice); the
//     triangular factor R carries the modes to the next level. A mode that an
//     aggregate cannot represent (collinear members) becomes an exactly-zero
//     column, i.e. a coarse DOF with a zero row and column ("dead"), which the
//     block inverses treat as absent;
//   * coarse patterns and, per coarse block, the ordered list of fine blocks
//     whose Galerkin products P_v^T A_vw P_w sum into it (deterministic sums).
// Levels are added until the coarsest has at most kDenseNodes nodes (solved
// by its dense inverse) or aggregation stops reducing (all nodes isolated,
// e.g. packed meshes: the coarsest is then block diagonal and its block-
// Jacobi solve is exact).
//
// Per Newton system (device): Galerkin products level by level, inverses of
// the 6x6 diagonal blocks, the coarsest dense inverse, and the largest
// eigenvalue of M A on every smoothed level by power iteration (M the level's
// smoother), from which the Chebyshev coefficients follow.
//
// V-cycle (the PCG preconditioner, symmetric): on level 0 one Chebyshev step
// of the smoother before and after the coarse correction; on coarse levels
// `deg` steps (by default 1 on level 1, 2 where it is in the cluster launch, 5
// below). The smoother of level 0 is block-Jacobi or the learned factor
// M = G^T G (the network's output on the Hessian's lower block pattern). The
// smoothing passes read exactly symmetric BF16 copies of the operators (the
// fine one in the sliced-ELL layout); the Galerkin products use the FP32 values. The
// levels that fit the shared memory of one thread-block cluster run as one
// kernel (k_mgc_cluster). Every kernel becomes a no-op once the PCG's
// convergence flag is set, so fixed-length CUDA graphs of PCG iterations can
// contain it.
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <memory>

#include "amg_internal.cuh"
#include "lpcg_internal.cuh"
#include "pcg_common.cuh"
#include "sell.cuh"

namespace bartels {

int reduce_sum(bartels_ctx ctx, const double *in, int n, double *out);
int launch_minv_blk(bartels_ctx ctx, bartels_mesh_plan plan, const float *values, float *minv);
int plan_lanes_spmv(bartels_ctx ctx, bartels_mesh_plan plan);
int plan_lanes_tri(bartels_ctx ctx, bartels_mesh_plan plan);

namespace {

constexpr int kDenseNodes = 64;   // coarsest level solved densely up to 64 nodes (384 DOFs)
constexpr int kPowerIters = 10;   // power iterations for each smoother's largest eigenvalue
constexpr int kCoarsestDeg = 6;   // Chebyshev steps on a coarsest level that is neither dense nor block diagonal

int env_int(const char *name, int dflt, int lo, int hi) {
  const char *s = std::getenv(name);
  if (!s || !*s) return dflt;
  const int v = std::atoi(s);
  return std::min(hi, std::max(lo, v));
}

// ------------------------------------------------------------ host set-up ---
struct HostLevel {
  int n = 0, bs = 0;
  std::vector<int> rp, ci;       // block pattern
  std::vector<char> active;      // node takes part in the system
  std::vector<double> B;         // n x bs x 6 near-null space (row-major per node)
  // transfer to the next level
  std::vector<int> agg, mptr, midx, gptr;
  std::vector<int2> gent;
  std::vector<float> Q;          // n x bs x 6
  int nc = 0;
};

// Greedy aggregation over the active nodes of a level, in index order.
int aggregate(const HostLevel &L, std::vector<int> &agg) {
  const int n = L.n;
  agg.assign(n, -1);
  int na = 0;
  for (int v = 0; v < n; ++v) {  // pass 1: roots with an entirely free neighbourhood
    if (!L.active[v] || agg[v] >= 0) continue;
    bool free_nb = true;
    for (int k = L.rp[v]; k < L.rp[v + 1] && free_nb; ++k) {
      const int w = L.ci[k];
      if (L.active[w] && agg[w] >= 0) free_nb = false;
    }
    if (!free_nb) continue;
    for (int k = L.rp[v]; k < L.rp[v + 1]; ++k) {
      const int w = L.ci[k];
      if (L.active[w]) agg[w] = na;
    }
    agg[v] = na++;
  }
  std::vector<int> join(n, -1);
  for (int v = 0; v < n; ++v) {  // pass 2: join the lowest-numbered neighbouring aggregate of pass 1
    if (!L.active[v] || agg[v] >= 0) continue;
    int best = INT_MAX;
    for (int k = L.rp[v]; k < L.rp[v + 1]; ++k) {
      const int w = L.ci[k];
      if (L.active[w] && agg[w] >= 0) best = std::min(best, agg[w]);
    }
    if (best != INT_MAX) join[v] = best;
  }
  for (int v = 0; v < n; ++v)
    if (join[v] >= 0) agg[v] = join[v];
  for (int v = 0; v < n; ++v) {  // pass 3: leftovers group with their free neighbours
    if (!L.active[v] || agg[v] >= 0) continue;
    for (int k = L.rp[v]; k < L.rp[v + 1]; ++k) {
      const int w = L.ci[k];
      if (L.active[w] && agg[w] < 0) agg[w] = na;
    }
    agg[v] = na++;
  }
  return na;
}

// Orthonormalise the m x 6 block Bm (row-major) of one aggregate in place:
// Bm = Qm R, modified Gram-Schmidt applied twice per column. A column whose
// remainder is below 1e-9 of the block's largest column norm is dead: its Q
// column and R row are zero.
void mgs_qr(double *Bm, int m, double R[36]) {
  for (int i = 0; i < 36; ++i) R[i] = 0.0;
  double scale = 0.0;
  for (int c = 0; c < 6; ++c) {
    double s = 0.0;
    for (int i = 0; i < m; ++i) s += Bm[6 * i + c] * Bm[6 * i + c];
    scale = std::max(scale, std::sqrt(s));
  }
  bool alive[6];
  for (int c = 0; c < 6; ++c) {
    for (int pass = 0; pass < 2; ++pass)
      for (int j = 0; j < c; ++j) {
        if (!alive[j]) continue;
        double h = 0.0;
        for (int i = 0; i < m; ++i) h += Bm[6 * i + j] * Bm[6 * i + c];
        for (int i = 0; i < m; ++i) Bm[6 * i + c] -= h * Bm[6 * i + j];
        R[6 * j + c] += h;
      }
    double s = 0.0;
    for (int i = 0; i < m; ++i) s += Bm[6 * i + c] * Bm[6 * i + c];
    s = std::sqrt(s);
    alive[c] = s > 1e-9 * scale;
    if (alive[c]) {
      for (int i = 0; i < m; ++i) Bm[6 * i + c] /= s;
      R[6 * c + c] = s;
    } else {
      for (int i = 0; i < m; ++i) Bm[6 * i + c] = 0.0;
      for (int j = 0; j < 6; ++j) R[6 * c + j] = 0.0;
    }
  }
}

// Transfer operators from level L to a new level C (nodes = aggregates).
void build_transfer(HostLevel &L, HostLevel &C) {
  const int n = L.n, bs = L.bs;
  const int na = L.nc;
  // members of each aggregate, ascending
  L.mptr.assign(na + 1, 0);
  for (int v = 0; v < n; ++v)
    if (L.agg[v] >= 0) L.mptr[L.agg[v] + 1]++;
  for (int a = 0; a < na; ++a) L.mptr[a + 1] += L.mptr[a];
  L.midx.assign(L.mptr[na], 0);
  {
    std::vector<int> fill(L.mptr.begin(), L.mptr.end() - 1);
    for (int v = 0; v < n; ++v)
      if (L.agg[v] >= 0) L.midx[fill[L.agg[v]]++] = v;
  }
  // tentative prolongator blocks and the coarse near-null space
  L.Q.assign((size_t)n * bs * 6, 0.f);
  C.n = na;
  C.bs = 6;
  C.B.assign((size_t)na * 36, 0.0);
  C.active.assign(na, 1);
  std::vector<double> Bm;
  for (int a = 0; a < na; ++a) {
    const int m0 = L.mptr[a], m1 = L.mptr[a + 1];
    const int rows = (m1 - m0) * bs;
    Bm.assign((size_t)rows * 6, 0.0);
    for (int i = m0; i < m1; ++i) {
      const int v = L.midx[i];
      std::memcpy(&Bm[(size_t)(i - m0) * bs * 6], &L.B[(size_t)v * bs * 6], sizeof(double) * bs * 6);
    }
    double R[36];
    mgs_qr(Bm.data(), rows, R);
    for (int i = m0; i < m1; ++i) {
      const int v = L.midx[i];
      for (int e = 0; e < bs * 6; ++e) L.Q[(size_t)v * bs * 6 + e] = (float)Bm[(size_t)(i - m0) * bs * 6 + e];
    }
    std::memcpy(&C.B[(size_t)a * 36], R, sizeof(R));
  }
  // coarse pattern: aggregates connected by a fine block between active nodes
  C.rp.assign(na + 1, 0);
  C.ci.clear();
  std::vector<int> mark(na, -1), cols;
  for (int a = 0; a < na; ++a) {
    cols.clear();
    for (int i = L.mptr[a]; i < L.mptr[a + 1]; ++i) {
      const int v = L.midx[i];
      for (int k = L.rp[v]; k < L.rp[v + 1]; ++k) {
        const int w = L.ci[k];
        if (!L.active[w]) continue;
        const int b = L.agg[w];
        if (mark[b] != a) {
          mark[b] = a;
          cols.push_back(b);
        }
      }
    }
    std::sort(cols.begin(), cols.end());
    C.ci.insert(C.ci.end(), cols.begin(), cols.end());
    C.rp[a + 1] = (int)C.ci.size();
  }
  // Galerkin contributions per coarse block: members ascending, their blocks ascending
  const int64_t ncb = C.rp[na];
  L.gptr.assign(ncb + 1, 0);
  auto coarse_pos = [&](int a, int b) {
    return (int)(std::lower_bound(C.ci.begin() + C.rp[a], C.ci.begin() + C.rp[a + 1], b) - C.ci.begin());
  };
  for (int a = 0; a < na; ++a)
    for (int i = L.mptr[a]; i < L.mptr[a + 1]; ++i) {
      const int v = L.midx[i];
      for (int k = L.rp[v]; k < L.rp[v + 1]; ++k) {
        const int w = L.ci[k];
        if (L.active[w]) L.gptr[coarse_pos(a, L.agg[w]) + 1]++;
      }
    }
  for (int64_t b = 0; b < ncb; ++b) L.gptr[b + 1] += L.gptr[b];
  L.gent.assign(L.gptr[ncb], int2{0, 0});
  std::vector<int> fill(L.gptr.begin(), L.gptr.end() - 1);
  for (int a = 0; a < na; ++a)
    for (int i = L.mptr[a]; i < L.mptr[a + 1]; ++i) {
      const int v = L.midx[i];
      for (int k = L.rp[v]; k < L.rp[v + 1]; ++k) {
        const int w = L.ci[k];
        if (L.active[w]) L.gent[fill[coarse_pos(a, L.agg[w])]++] = int2{v, k};
      }
    }
}

template <class T>
int upload(MgHierarchy *mg, T **dst, const std::vector<T> &src) {
  *dst = nullptr;
  if (src.empty()) return BARTELS_OK;
  void *p = nullptr;
  BT_CUDA(dev_malloc(&p, sizeof(T) * src.size()));
  mg->allocs.push_back(p);
  BT_CUDA(cudaMemcpy(p, src.data(), sizeof(T) * src.size(), cudaMemcpyHostToDevice));
  *dst = static_cast<T *>(p);
  return BARTELS_OK;
}

int dalloc(MgHierarchy *mg, void **dst, size_t bytes) {
  *dst = nullptr;
  if (bytes == 0) return BARTELS_OK;
  BT_CUDA(dev_malloc(dst, (bytes + 255) & ~size_t(255)));
  mg->allocs.push_back(*dst);
  return BARTELS_OK;
}

template <class T>
int dalloc_n(MgHierarchy *mg, T **dst, size_t count) {
  void *p = nullptr;
  BT_CHECK(dalloc(mg, &p, sizeof(T) * count));
  *dst = static_cast<T *>(p);
  return BARTELS_OK;
}

}  // namespace

constexpr int kClThreads = 512;  // threads per CTA of the coarse-cycle cluster
__global__ void k_mgc_cluster(const __grid_constant__ MgClArgs a, const PcgState *__restrict__ st);

namespace {

// launch configuration of one cluster of `ctas` CTAs
cudaLaunchConfig_t cluster_config(bartels_ctx ctx, int ctas, int threads, int smem, cudaLaunchAttribute *at) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ctas);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = ctx->stream;
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = ctas;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cfg;
}

// Node ranges of a level for `ctas` CTAs, balanced by stored blocks (a dense
// level: by nodes, so that 4 CTAs hold the inverse of kDenseNodes nodes).
void cluster_split(const HostLevel &h, bool dense, int ctas, int *split) {
  if (dense) {
    const int per = (h.n + ctas - 1) / ctas;
    for (int q = 0; q <= ctas; ++q) split[q] = std::min(h.n, q * per);
    return;
  }
  const int64_t total = h.rp[h.n];
  for (int q = 0; q <= ctas; ++q) {
    const int64_t want = total * q / ctas;
    split[q] = (int)(std::lower_bound(h.rp.begin(), h.rp.end(), want) - h.rp.begin());
  }
  split[0] = 0;
  split[ctas] = h.n;
}

// Shared-memory layout of levels first .. last for a cluster of a.ctas CTAs;
// returns the bytes each CTA needs.
int64_t cluster_layout(MgClArgs &a) {
  int64_t off = 0;
  auto take = [&](int64_t bytes) {
    const int64_t o = off;
    off += (bytes + 15) & ~int64_t(15);
    return (int)std::min<int64_t>(o, INT_MAX);
  };
  for (int l = 0; l < a.nlev; ++l) {
    MgClLevel &L = a.lv[l];
    const bool last = l + 1 == a.nlev, dense = last && a.last_mode == kMgLastDense;
    int64_t rows = 0, blocks = 0, mems = 0;
    for (int q = 0; q < a.ctas; ++q) {
      rows = std::max<int64_t>(rows, L.split[q + 1] - L.split[q]);
      blocks = std::max<int64_t>(blocks, L.bsplit[q + 1] - L.bsplit[q]);
      mems = std::max<int64_t>(mems, L.msplit[q + 1] - L.msplit[q]);
    }
    if (dense) {
      L.o_val = take(sizeof(float) * 6 * rows * a.nd);
    } else {
      L.o_val = take(72 * blocks);
      L.o_ci = take(4 * blocks);
      L.o_rp = take(4 * (rows + 1));
      L.o_dinv = take(144 * rows);
    }
    if (!last) {
      L.o_Q = take(144 * rows);
      L.o_agg = take(4 * rows);
    }
    if (l > 0) {
      L.o_mptr = take(4 * (rows + 1));
      L.o_mem = take(4 * mems);
    }
    if (!dense) {
      L.o_b = take(24 * rows);
      L.o_x = take(24 * rows);
      L.o_r = take(24 * rows);
      L.o_d = take(24 * rows);
    }
  }
  if (a.last_mode == kMgLastDense) a.o_db = take(sizeof(float) * a.nd);
  return off;
}

// The coarse part of the hierarchy as one cluster launch (k_mgc_cluster):
// levels from the finest one that fits the cluster's shared memory down to the
// coarsest, on 16 CTAs or, where the device cannot host so many as one cluster,
// 8 or 4. Leaves cl.ctas = 0 (the per-level launches) when not even the coarsest
// level fits or no cluster can be hosted.
int build_cluster(bartels_ctx ctx, MgHierarchy *mg, const std::vector<HostLevel> &H) {
  constexpr int kSmem = 220 * 1024;
  const int L = (int)H.size();
  int want = env_int("BARTELS_MG_CLUSTER", kMgClusterMax, 0, kMgClusterMax);
  mg->cl = MgClArgs();
  if (want == 0) return BARTELS_OK;
  want = std::max(want, 4);
  BT_CUDA(cudaFuncSetAttribute(k_mgc_cluster, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem));
  BT_CUDA(cudaFuncSetAttribute(k_mgc_cluster, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  for (int ctas : {want, 8, 4}) {
    if (ctas > want) continue;
    for (int first = std::max(1, L - kMgClusterLevels); first < L; ++first) {
      MgClArgs a;
      a.first = first;
      a.nlev = L - first;
      a.last_mode = mg->dense ? kMgLastDense : (mg->coarse_blockdiag ? kMgLastExact : kMgLastCheb);
      a.nd = mg->nd;
      a.ainv = mg->ainv;
      a.coef = mg->coef;
      a.ctas = ctas;
      for (int l = 0; l < a.nlev; ++l) {
        const HostLevel &h = H[first + l];
        MgClLevel &c = a.lv[l];
        cluster_split(h, mg->dense && l + 1 == a.nlev, a.ctas, c.split);
        for (int q = 0; q <= a.ctas; ++q) {
          c.bsplit[q] = h.rp[c.split[q]];
          c.msplit[q] = l > 0 ? H[first + l - 1].mptr[c.split[q]] : 0;
        }
      }
      const int64_t smem = cluster_layout(a);
      if (smem > kSmem) continue;
      a.smem = (int)smem;
      cudaLaunchAttribute at[1];
      const cudaLaunchConfig_t cfg = cluster_config(ctx, a.ctas, kClThreads, a.smem, at);
      int fit = 0;
      if (cudaOccupancyMaxActiveClusters(&fit, k_mgc_cluster, &cfg) != cudaSuccess) {
        cudaGetLastError();
        fit = 0;
      }
      if (fit < 1) continue;
      for (int l = 0; l < a.nlev; ++l) {
        const MgLevel &d = mg->lv[first + l];
        MgClLevel &c = a.lv[l];
        c.deg = d.deg;
        c.rp = d.rp;
        c.ci = d.ci;
        c.agg = d.agg;
        c.val16 = d.val16;
        c.dinv = d.dinv;
        c.Q = d.Q;
        c.gb = d.b;
        c.gx = d.x;
        c.gd = d.d;
        c.gd2 = d.d2;
        c.gres = l + 1 < a.nlev ? d.x2 : d.x;  // as level_result
        if (l > 0) {
          c.mptr = mg->lv[first + l - 1].mptr;
          c.midx = mg->lv[first + l - 1].midx;
        }
      }
      mg->cl = a;
      return BARTELS_OK;
    }
  }
  return BARTELS_OK;
}

}  // namespace

MgHierarchy::~MgHierarchy() {
  for (void *p : allocs) cudaFree(p);
}

// Build the hierarchy of the plan's pattern for its current pinned set (kept
// while the pinned set is unchanged).
int mg_prepare(bartels_ctx ctx, bartels_mesh_plan plan) {
  if (plan->mg && plan->mg->pinned_gen == plan->pinned_gen) return BARTELS_OK;
  delete plan->mg;
  plan->mg = nullptr;
  BT_CUDA(cudaStreamSynchronize(ctx->stream));
  const int nV = plan->nV;
  std::vector<unsigned char> pinned(nV, 0);
  if (plan->pinned) BT_CUDA(cudaMemcpy(pinned.data(), plan->pinned, nV, cudaMemcpyDeviceToHost));
  std::vector<double> X(3 * (size_t)nV);
  BT_CUDA(cudaMemcpy(X.data(), plan->X, sizeof(double) * X.size(), cudaMemcpyDeviceToHost));

  std::vector<HostLevel> H(1);
  HostLevel &L0 = H[0];
  L0.n = nV;
  L0.bs = 3;
  L0.rp = plan->h_brp;
  L0.ci = plan->h_bcol;
  L0.active.assign(nV, 1);
  int nfree = 0;
  double cx = 0, cy = 0, cz = 0;
  for (int v = 0; v < nV; ++v) {
    L0.active[v] = pinned[v] ? 0 : 1;
    if (L0.active[v]) {
      nfree++;
      cx += X[3 * v];
      cy += X[3 * v + 1];
      cz += X[3 * v + 2];
    }
  }
  if (nfree == 0) return fail(BARTELS_E_UNSUPPORTED, "multigrid: every vertex is pinned");
  cx /= nfree;
  cy /= nfree;
  cz /= nfree;
  // rigid-body modes of level 0: translations and rotations about the centroid
  // (theta x (x - c) = -[x - c]_x theta)
  L0.B.assign((size_t)nV * 18, 0.0);
  for (int v = 0; v < nV; ++v) {
    const double dx = X[3 * v] - cx, dy = X[3 * v + 1] - cy, dz = X[3 * v + 2] - cz;
    double *b = &L0.B[(size_t)v * 18];
    b[0] = 1; b[7] = 1; b[14] = 1;                 // translations
    b[3] = 0;   b[4] = dz;  b[5] = -dy;            // row x: (theta x d)_x = ty dz - tz dy
    b[9] = -dz; b[10] = 0;  b[11] = dx;            // row y
    b[15] = dy; b[16] = -dx; b[17] = 0;            // row z
  }
  int coarse_blockdiag = 0, dense = 0;
  for (int l = 0; l + 1 < kMgMaxLevels; ++l) {
    HostLevel &L = H[l];
    int nact = 0;
    for (int v = 0; v < L.n; ++v) nact += L.active[v];
    if (l > 0 && nact <= kDenseNodes) {
      dense = 1;
      break;
    }
    std::vector<int> agg;
    const int na = aggregate(L, agg);
    if (na >= nact) {  // no reduction: every node is isolated (block-diagonal level)
      coarse_blockdiag = 1;
      for (int v = 0; v < L.n && coarse_blockdiag; ++v)
        for (int k = L.rp[v]; k < L.rp[v + 1]; ++k)
          if (L.ci[k] != v && L.active[L.ci[k]]) {
            coarse_blockdiag = 0;
            break;
          }
      break;
    }
    L.agg = std::move(agg);
    L.nc = na;
    H.emplace_back();
    build_transfer(H[l], H[l + 1]);
  }
  if (H.size() < 2) return fail(BARTELS_E_UNSUPPORTED, "multigrid: the system is too small for a coarse level");

  std::unique_ptr<MgHierarchy> own(new MgHierarchy());  // the plan's once it is complete
  MgHierarchy *mg = own.get();
  mg->pinned_gen = plan->pinned_gen;
  mg->dense = dense;
  mg->coarse_blockdiag = dense ? 0 : coarse_blockdiag;
  const int deg0 = env_int("BARTELS_MG_DEG0", 1, 1, 1);
  // Chebyshev degrees: level 1 (the largest coarse level; its one step is
  // fused into the restriction) and the levels below it, whose steps are
  // cheap and cut the PCG iterations. n = 96, a multigrid solve to 1e-9: level
  // 1 at 1 with 3 / 4 / 5 / 6 below gives 59.8 / 57.6 / 56.4 / 55.7 ms (n = 48,
  // learned smoother: 14.0 / 13.7 / 13.7 / 13.9), level 1 at 2 with 4 / 5 below
  // 59.4 / 58.5.
  const int degc = env_int("BARTELS_MG_DEGC", 1, 1, (kMgCoef - 1) / 2 + 1);
  // level 1 inside the cluster launch, where a step is cheap (24^3 Newton step:
  // 1 / 2 / 3 / 4 / 5 give 12.5 / 11.6 / 11.4 / 11.5 / 11.8 ms, smaller solves
  // are best at 2)
  const char *set = std::getenv("BARTELS_MG_DEGC");  // chosen by the user: wherever level 1 runs
  const int degcl = env_int("BARTELS_MG_DEGCL", set && *set ? degc : 2, 1, (kMgCoef - 1) / 2 + 1);
  const int degc2 = env_int("BARTELS_MG_DEGC2", 5, 1, (kMgCoef - 1) / 2 + 1);
  mg->lv.resize(H.size());
  for (size_t l = 0; l < H.size(); ++l) {
    HostLevel &h = H[l];
    MgLevel &d = mg->lv[l];
    d.n = h.n;
    d.bs = h.bs;
    d.deg = l == 0 ? deg0 : (l + 1 == H.size() ? kCoarsestDeg : (l == 1 ? degc : degc2));
    d.nc = h.nc;
    if (l > 0) {
      d.nnzb = h.rp[h.n];
      mg->coarse_nnz += 36 * d.nnzb;
      std::vector<int> dpos(h.n, -1);
      for (int v = 0; v < h.n; ++v)
        for (int k = h.rp[v]; k < h.rp[v + 1]; ++k)
          if (h.ci[k] == v) dpos[v] = k;
      for (int v = 0; v < h.n; ++v)
        if (dpos[v] < 0) return fail(BARTELS_E_DEVICE, "multigrid: coarse level without a diagonal block");
      BT_CHECK(upload(mg, &d.rp, h.rp));
      BT_CHECK(upload(mg, &d.ci, h.ci));
      BT_CHECK(upload(mg, &d.dpos, dpos));
      BT_CHECK(dalloc_n(mg, &d.val, 36 * (size_t)d.nnzb));
      BT_CHECK(dalloc_n(mg, &d.val16, 36 * (size_t)d.nnzb));
      BT_CHECK(dalloc_n(mg, &d.dinv, 36 * (size_t)d.n));
      // position of block (J, I) for each block (I, J) (Galerkin patterns are symmetric)
      std::vector<int> rev(d.nnzb, -1);
      for (int v = 0; v < h.n; ++v)
        for (int k = h.rp[v]; k < h.rp[v + 1]; ++k) {
          const int w = h.ci[k];
          const int *b = h.ci.data() + h.rp[w], *e = h.ci.data() + h.rp[w + 1];
          const int *f = std::lower_bound(b, e, v);
          if (f == e || *f != v) return fail(BARTELS_E_DEVICE, "multigrid: coarse pattern is not symmetric");
          rev[k] = (int)(f - h.ci.data());
        }
      BT_CHECK(upload(mg, &d.rev, rev));
    } else {
      d.nnzb = plan->nnzb;
    }
    if (l + 1 < H.size()) {
      BT_CHECK(upload(mg, &d.agg, h.agg));
      BT_CHECK(upload(mg, &d.mptr, h.mptr));
      BT_CHECK(upload(mg, &d.midx, h.midx));
      BT_CHECK(upload(mg, &d.Q, h.Q));
      BT_CHECK(upload(mg, &d.gptr, h.gptr));
      BT_CHECK(upload(mg, &d.gent, h.gent));
    }
    const size_t nv = (size_t)d.bs * d.n;
    if (l > 0) BT_CHECK(dalloc_n(mg, &d.b, nv));
    BT_CHECK(dalloc_n(mg, &d.x, nv));
    BT_CHECK(dalloc_n(mg, &d.x2, nv));
    BT_CHECK(dalloc_n(mg, &d.r, nv));
    BT_CHECK(dalloc_n(mg, &d.d, nv));
    if (l > 0) BT_CHECK(dalloc_n(mg, &d.d2, nv));
  }
  if (env_int("BARTELS_MG_FINE_BF16", 1, 0, 1)) {
    SellPattern *sp;
    BT_CHECK(plan_sell(plan, &sp));
    BT_CHECK(dalloc_n(mg, &mg->a16, 288 * (size_t)std::max<int64_t>(sp->groups, 1)));
  }
  if (mg->dense) {
    mg->nd = 6 * mg->lv.back().n;
    BT_CHECK(dalloc_n(mg, &mg->ainv, (size_t)mg->nd * mg->nd));
    BT_CHECK(dalloc_n(mg, &mg->panel, 2 * 6 * (size_t)mg->nd));
  }
  BT_CHECK(dalloc_n(mg, &mg->coef, (size_t)kMgMaxLevels * kMgCoef));
  BT_CHECK(dalloc_n(mg, &mg->norms, 2 * (size_t)kMgMaxLevels));
  mg->nparts = 4096;
  BT_CHECK(dalloc_n(mg, &mg->part, (size_t)mg->nparts));
  BT_CUDA(cudaMemset(mg->coef, 0, sizeof(float) * kMgMaxLevels * kMgCoef));
  BT_CHECK(build_cluster(ctx, mg, H));
  if (mg->cl.ctas && mg->cl.first == 1 && H.size() > 2) mg->lv[1].deg = mg->cl.lv[0].deg = degcl;
  plan->mg = own.release();
  return BARTELS_OK;
}

// ===================================================== numeric set-up ======
// Galerkin kernels: a group of kGalLanes consecutive lanes per coarse block;
// lane l of the group takes the block's contributions l, l + kGalLanes, ...
// in list order, and the group's partial sums are combined by a fixed
// butterfly, so each coarse entry is summed in the same order on every run.
// The heavy blocks (a diagonal block sums every pair of its aggregate's
// members, ~400 contributions at n = 96) no longer hold up a whole warp.
constexpr int kGalLanes = 8;
#define GAL_GROUP_LOOP_BEGIN                                                                       \
  const int gl = threadIdx.x % kGalLanes;                                                          \
  const int64_t gid = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / kGalLanes;                \
  const int64_t ngroups = ((int64_t)gridDim.x * blockDim.x) / kGalLanes;                           \
  for (int64_t b0 = gid - gid % (32 / kGalLanes); b0 < ncb; b0 += ngroups) {                        \
    const int64_t b = b0 + gid % (32 / kGalLanes);                                                 \
    const bool active = b < ncb;
#define GAL_GROUP_LOOP_END }

// butterfly sum over the group (every lane of the warp takes part), then the
// group's lanes store the block's 9 float4s round-robin
__device__ __forceinline__ void gal_group_store(float C[36], bool active, int gl, float *__restrict__ out) {
#pragma unroll
  for (int o = kGalLanes / 2; o > 0; o >>= 1)
#pragma unroll
    for (int i = 0; i < 36; ++i) C[i] += __shfl_xor_sync(0xffffffffu, C[i], o);
  if (active) {
    float4 *o4 = reinterpret_cast<float4 *>(out);
#pragma unroll
    for (int i = 0; i < 9; ++i)
      if (i % kGalLanes == gl) o4[i] = make_float4(C[4 * i], C[4 * i + 1], C[4 * i + 2], C[4 * i + 3]);
  }
}

// Galerkin product level 0 -> 1: C_IJ = sum over the block's contributions
// (v, k) of Q_v^T A_vw Q_w, A_vw read from the plan's value layout (row 3v+a
// of block row v holds its blocks' columns contiguously). One thread per
// coarse block, contributions summed in list order.
__global__ void __launch_bounds__(128)
k_mg_gal0(int64_t ncb, const int *__restrict__ gptr, const int2 *__restrict__ gent, const int *__restrict__ brp,
          const int *__restrict__ bcol, const float *__restrict__ val, const float *__restrict__ Q,
          float *__restrict__ cval) {
  GAL_GROUP_LOOP_BEGIN
    float C[36];
#pragma unroll
    for (int i = 0; i < 36; ++i) C[i] = 0.f;
    const int e1 = active ? gptr[b + 1] : 0;
    for (int e = (active ? gptr[b] : 0) + gl; e < e1; e += kGalLanes) {
      const int2 g = __ldg(gent + e);
      const int v = g.x, k = g.y;
      const int rb = __ldg(brp + v), rs = 3 * (__ldg(brp + v + 1) - rb);
      const int w = __ldg(bcol + k);
      const float *a0 = val + 9ll * rb + 3 * (k - rb);
      float A[9];
#pragma unroll
      for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int c = 0; c < 3; ++c) A[3 * a + c] = __ldg(a0 + a * rs + c);
      const float *qw = Q + 18ll * w;
      float T[18];  // A Q_w (3 x 6)
#pragma unroll
      for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int c = 0; c < 6; ++c)
          T[6 * a + c] = A[3 * a] * __ldg(qw + c) + A[3 * a + 1] * __ldg(qw + 6 + c) + A[3 * a + 2] * __ldg(qw + 12 + c);
      const float *qv = Q + 18ll * v;
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        float q[6];
#pragma unroll
        for (int c = 0; c < 6; ++c) q[c] = __ldg(qv + 6 * a + c);
#pragma unroll
        for (int c = 0; c < 6; ++c)
#pragma unroll
          for (int d = 0; d < 6; ++d) C[6 * c + d] += q[c] * T[6 * a + d];
      }
    }
    gal_group_store(C, active, gl, cval + 36 * b);
  GAL_GROUP_LOOP_END
}

// Galerkin product between coarse levels (6x6 blocks, 6x6 prolongator blocks).
__global__ void __launch_bounds__(128)
k_mg_galc(int64_t ncb, const int *__restrict__ gptr, const int2 *__restrict__ gent, const int *__restrict__ ci,
          const float *__restrict__ val, const float *__restrict__ Q, float *__restrict__ cval) {
  GAL_GROUP_LOOP_BEGIN
    float C[36];
#pragma unroll
    for (int i = 0; i < 36; ++i) C[i] = 0.f;
    const int e1 = active ? gptr[b + 1] : 0;
    for (int e = (active ? gptr[b] : 0) + gl; e < e1; e += kGalLanes) {
      const int2 g = __ldg(gent + e);
      const int v = g.x, k = g.y;
      const int w = __ldg(ci + k);
      const float *A = val + 36ll * k;
      const float *qw = Q + 36ll * w;
      float T[36];  // A Q_w
#pragma unroll
      for (int a = 0; a < 6; ++a) {
        float ar[6];
#pragma unroll
        for (int c = 0; c < 6; ++c) ar[c] = __ldg(A + 6 * a + c);
#pragma unroll
        for (int d = 0; d < 6; ++d) {
          float s = 0.f;
#pragma unroll
          for (int c = 0; c < 6; ++c) s += ar[c] * __ldg(qw + 6 * c + d);
          T[6 * a + d] = s;
        }
      }
      const float *qv = Q + 36ll * v;
#pragma unroll
      for (int a = 0; a < 6; ++a) {
        float q[6];
#pragma unroll
        for (int c = 0; c < 6; ++c) q[c] = __ldg(qv + 6 * a + c);
#pragma unroll
        for (int c = 0; c < 6; ++c)
#pragma unroll
          for (int d = 0; d < 6; ++d) C[6 * c + d] += q[c] * T[6 * a + d];
      }
    }
    gal_group_store(C, active, gl, cval + 36 * b);
  GAL_GROUP_LOOP_END
}

// Inverse of each node's 6x6 diagonal block (symmetrised, FP64 Gauss-Jordan,
// FP32 storage). Dead DOFs (a zero diagonal entry: a mode the aggregate cannot
// represent) get zero rows and columns in the inverse. A block that is not
// positive definite falls back to the inverse of its diagonal.
__global__ void k_mg_inv6(int n, const int *__restrict__ dpos, const float *__restrict__ val, float *__restrict__ dinv) {
  for (int I = blockIdx.x * blockDim.x + threadIdx.x; I < n; I += gridDim.x * blockDim.x) {
    const float *a = val + 36ll * dpos[I];
    double A[36];
    bool dead[6];
    for (int i = 0; i < 6; ++i)
      for (int j = 0; j < 6; ++j) A[6 * i + j] = 0.5 * ((double)a[6 * i + j] + (double)a[6 * j + i]);
    for (int i = 0; i < 6; ++i) {
      dead[i] = !(A[7 * i] != 0.0);
      if (dead[i]) {
        for (int j = 0; j < 6; ++j) A[6 * i + j] = A[6 * j + i] = 0.0;
        A[7 * i] = 1.0;
      }
    }
    double D[36];
    for (int i = 0; i < 36; ++i) D[i] = A[i];
    bool ok = true;
    for (int k = 0; k < 6 && ok; ++k) {
      const double piv = A[7 * k];
      if (!(piv > 0.0) || !isfinite(piv)) {
        ok = false;
        break;
      }
      const double p = 1.0 / piv;
      for (int j = 0; j < 6; ++j)
        if (j != k) A[6 * k + j] *= p;
      for (int i = 0; i < 6; ++i) {
        if (i == k) continue;
        const double f = A[6 * i + k];
        for (int j = 0; j < 6; ++j)
          if (j != k) A[6 * i + j] -= f * A[6 * k + j];
      }
      for (int i = 0; i < 6; ++i)
        if (i != k) A[6 * i + k] *= -p;
      A[7 * k] = p;
    }
    float *o = dinv + 36ll * I;
    for (int i = 0; i < 6; ++i)
      for (int j = 0; j < 6; ++j) {
        double vv;
        if (ok) vv = A[6 * i + j];
        else vv = (i == j && D[7 * i] > 0.0) ? 1.0 / D[7 * i] : 0.0;
        if (dead[i] || dead[j]) vv = 0.0;
        o[6 * i + j] = (float)vv;
      }
  }
}

__device__ __forceinline__ unsigned cl_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cl_barrier() {
  __syncwarp();  // the aligned form wants the warp's lanes together
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Dense inverse of the coarsest level (nd = 6 x nodes <= 384, symmetrised) by
// in-place block Gauss-Jordan without pivoting (the matrix is SPD). Dead DOFs
// as in k_mg_inv6. One thread-block cluster; each CTA keeps the rows of its
// own nodes (split) in shared memory. Per node K: the owner inverts the 6x6 pivot
// block, scales the node's 6 rows with it and publishes them (panel, double-
// buffered), then every CTA updates its other rows. One cluster barrier per node: 64 nodes take
// 320 us (406 with the pivot block inverted by one thread); a single CTA with a barrier
// per scalar pivot took 58 us for 8 nodes and 552 us for 18.
struct MgInvArgs {
  int nodes = 0, split[kMgClusterMax + 1] = {};
  const int *rp = nullptr, *ci = nullptr, *rev = nullptr, *dpos = nullptr;
  const float *val = nullptr;
  float *panel = nullptr, *ainv = nullptr;
};
constexpr int kInvThreads = 512, kInvCtas = 8;
// own rows and the panel of the largest dense level
constexpr int kInvSmem = (int)sizeof(float) * (6 * ((kDenseNodes + kInvCtas - 1) / kInvCtas) + 6) * 6 * kDenseNodes;
__global__ void __launch_bounds__(kInvThreads, 1)
k_mg_dense_inv(const __grid_constant__ MgInvArgs a) {
  extern __shared__ __align__(16) float sA[];  // own rows (6 x own nodes) x nd, then the panel 6 x nd
  __shared__ unsigned char dead[6 * kDenseNodes];
  __shared__ float sPiv[36];
  const int rank = cl_rank(), n0 = a.split[rank], n1 = a.split[rank + 1], rows = 6 * (n1 - n0), nd = 6 * a.nodes;
  float *sP = sA + rows * nd;
  for (int i = threadIdx.x; i < nd; i += blockDim.x) dead[i] = !(a.val[36ll * a.dpos[i / 6] + 7 * (i % 6)] != 0.f);
  for (int e = threadIdx.x; e < rows * nd; e += blockDim.x) sA[e] = 0.f;
  __syncthreads();
  for (int I = n0; I < n1; ++I)
    for (int e = threadIdx.x; e < 36 * (a.rp[I + 1] - a.rp[I]); e += blockDim.x) {
      const int k = a.rp[I] + e / 36, r = (e % 36) / 6, c = e % 6, i = 6 * I + r, j = 6 * a.ci[k] + c;
      const float t = 0.5f * (a.val[36ll * k + 6 * r + c] + a.val[36ll * a.rev[k] + 6 * c + r]);
      sA[(i - 6 * n0) * nd + j] = (dead[i] || dead[j]) ? 0.f : t;
    }
  __syncthreads();
  for (int i = threadIdx.x; i < rows; i += blockDim.x)
    if (dead[6 * n0 + i]) sA[i * nd + 6 * n0 + i] = 1.f;
  __syncthreads();
  for (int K = 0; K < a.nodes; ++K) {
    float *pan = a.panel + (K & 1) * 6 * nd;
    if (K >= n0 && K < n1) {
      float *R = sA + 6 * (K - n0) * nd;  // the node's 6 rows
      if (threadIdx.x < 32) {
        // P = inverse of the 6x6 pivot block: lane r < 6 holds its row r
        const int r = min((int)threadIdx.x, 5);
        float w[6];
#pragma unroll
        for (int c = 0; c < 6; ++c) w[c] = R[r * nd + 6 * K + c];
#pragma unroll
        for (int k = 0; k < 6; ++k) {
          const float piv = __shfl_sync(0xffffffffu, w[k], k), p = piv > 0.f ? 1.f / piv : 0.f, f = w[k];
#pragma unroll
          for (int c = 0; c < 6; ++c) {
            const float t = (c == k ? 1.f : __shfl_sync(0xffffffffu, w[c], k)) * p;
            w[c] = r == k ? t : (c == k ? -f * t : w[c] - f * t);
          }
        }
        if (threadIdx.x < 6)
#pragma unroll
          for (int c = 0; c < 6; ++c) sPiv[6 * r + c] = w[c];
      }
      __syncthreads();
      for (int j = threadIdx.x; j < nd; j += blockDim.x) {
        float v[6];
        const int jj = j - 6 * K;
#pragma unroll
        for (int c = 0; c < 6; ++c) v[c] = jj >= 0 && jj < 6 ? (c == jj ? 1.f : 0.f) : R[c * nd + j];
#pragma unroll
        for (int r = 0; r < 6; ++r) {
          float t = 0.f;
#pragma unroll
          for (int c = 0; c < 6; ++c) t += sPiv[6 * r + c] * v[c];
          R[r * nd + j] = t;
          pan[r * nd + j] = t;
        }
      }
    }
    cl_barrier();
    for (int e = threadIdx.x; e < 6 * nd; e += blockDim.x) sP[e] = __ldcg(pan + e);
    __syncthreads();
    // one warp per row: row -= f . panel, f the row's entries in the node's columns
    for (int i = threadIdx.x >> 5; i < rows; i += blockDim.x >> 5) {
      if (n0 + i / 6 == K) continue;
      float *row = sA + i * nd, f[6];
#pragma unroll
      for (int k = 0; k < 6; ++k) f[k] = row[6 * K + k];
      __syncwarp();
      for (int j = threadIdx.x & 31; j < nd; j += 32) {
        float s = 0.f;
#pragma unroll
        for (int k = 0; k < 6; ++k) s += f[k] * sP[k * nd + j];
        row[j] = (j >= 6 * K && j < 6 * K + 6) ? -s : row[j] - s;
      }
    }
    __syncthreads();
  }
  for (int e = threadIdx.x; e < rows * nd; e += blockDim.x) {
    const int i = 6 * n0 + e / nd, j = e % nd;
    a.ainv[6ll * n0 * nd + e] = (dead[i] || dead[j]) ? 0.f : sA[e];
  }
}

__device__ __forceinline__ void apply_dinv6(const float *__restrict__ dinv, int I, const float r[6], float z[6]) {
  const float4 *m4 = reinterpret_cast<const float4 *>(dinv + 36ll * I);
  float m[36];
#pragma unroll
  for (int q = 0; q < 9; ++q) {
    const float4 t = __ldg(m4 + q);
    m[4 * q] = t.x; m[4 * q + 1] = t.y; m[4 * q + 2] = t.z; m[4 * q + 3] = t.w;
  }
#pragma unroll
  for (int a = 0; a < 6; ++a) {
    float s = 0.f;
#pragma unroll
    for (int c = 0; c < 6; ++c) s += m[6 * a + c] * r[c];
    z[a] = s;
  }
}

// ============================================================= transfers ===
// b_c[I] = sum over members v of Q_v^T r_v: L lanes per aggregate (members
// strided over the lanes, fixed shuffle tree).
// With cdinv set it also takes the coarse level's first smoothing step from
// x = 0 (x = c Dinv b, r = b, d = x; c = ccoef[0], or 1 without ccoef).
template <int BSF, int L>
__global__ void __launch_bounds__(256)
k_mg_restrict(int nc, const int *__restrict__ mptr, const int *__restrict__ midx, const float *__restrict__ Q,
              const float *__restrict__ r, float *__restrict__ bc, const float *__restrict__ cdinv,
              float *__restrict__ cx, float *__restrict__ cr, float *__restrict__ cd, const float *__restrict__ ccoef,
              const PcgState *__restrict__ st) {
  pdl_wait();
  pdl_trigger();
  if (st && st->done) return;
  const int lane = threadIdx.x & 31, sl = lane % L, g = lane / L;
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  for (int I0 = warp * (32 / L); I0 < nc; I0 += nwarps * (32 / L)) {
    const int I = I0 + g;
    float acc[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (I < nc) {
      const int m1 = __ldg(mptr + I + 1);
      for (int m = __ldg(mptr + I) + sl; m < m1; m += L) {
        const int v = __ldg(midx + m);
        const float *q = Q + (int64_t)BSF * 6 * v;
#pragma unroll
        for (int a = 0; a < BSF; ++a) {
          const float rv = __ldcg(r + (int64_t)BSF * v + a);
#pragma unroll
          for (int c = 0; c < 6; ++c) acc[c] += __ldg(q + 6 * a + c) * rv;
        }
      }
    }
#pragma unroll
    for (int o = L / 2; o > 0; o >>= 1)
#pragma unroll
      for (int c = 0; c < 6; ++c) acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], o);
    if (I < nc && sl == 0) {
#pragma unroll
      for (int c = 0; c < 6; ++c) bc[6 * I + c] = acc[c];
      if (cdinv) {
        const float cf = ccoef ? ccoef[0] : 1.f;
        float z[6];
        apply_dinv6(cdinv, I, acc, z);
#pragma unroll
        for (int c = 0; c < 6; ++c) {
          const float xv = cf * z[c];
          cx[6 * I + c] = xv;
          if (cr) cr[6 * I + c] = acc[c];
          if (cd) cd[6 * I + c] = xv;
        }
      }
    }
  }
}

// x_v += Q_v x_c[agg v] (nodes outside the system keep their value)
template <int BSF>
__global__ void __launch_bounds__(256)
k_mg_prolong(int n, const int *__restrict__ agg, const float *__restrict__ Q, const float *__restrict__ xc,
             float *__restrict__ x, const PcgState *__restrict__ st) {
  pdl_wait();
  pdl_trigger();
  if (st && st->done) return;
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
    const int I = __ldg(agg + v);
    if (I < 0) continue;
    float c[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) c[k] = __ldcg(xc + 6 * I + k);
    const float *q = Q + (int64_t)BSF * 6 * v;
#pragma unroll
    for (int a = 0; a < BSF; ++a) {
      float s = 0.f;
#pragma unroll
      for (int k = 0; k < 6; ++k) s += __ldg(q + 6 * a + k) * c[k];
      x[(int64_t)BSF * v + a] += s;
    }
  }
}

// ================================================= level-0 (plan layout) ===
// x = c Dinv r with the 3x3 block-Jacobi inverse (c = coef[0], or 1 without coef)
__global__ void __launch_bounds__(256)
k_mg0_bj(int nV, const float *__restrict__ minv, const float *__restrict__ r, float *__restrict__ x,
         const float *__restrict__ coef, const PcgState *__restrict__ st) {
  pdl_wait();
  pdl_trigger();
  if (st && st->done) return;
  const float c = coef ? coef[0] : 1.f;
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < nV; v += gridDim.x * blockDim.x) {
    float rv[3], zv[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) rv[k] = __ldcg(r + 3 * v + k);
    apply_minv(minv, v, rv, zv);
#pragma unroll
    for (int k = 0; k < 3; ++k) x[3 * v + k] = c * zv[k];
  }
}

// The PCG update fused with the level-0 pre-smoothing of the block-Jacobi
// V-cycle: x += alpha p; r -= alpha Ap; x0 = c Dinv r (c = coef[0]); partial
// sums of r.r. The last block stores r.r, advances the iteration count and
// applies the convergence test, as k_pcg_update_f does.
__global__ void __launch_bounds__(256)
k_mg0_update(int nV, const float *__restrict__ pa, const float *__restrict__ pb, const float *__restrict__ ap,
             float *__restrict__ x, float *__restrict__ r, const float *__restrict__ minv, float *__restrict__ x0,
             const float *__restrict__ coef, double *__restrict__ part, PcgState *__restrict__ st) {
  pdl_wait();
  pdl_trigger();
  if (st->done) return;
  const int it = st->it;
  const float *p = (it & 1) ? pb : pa;
  const float alpha = st->alpha, c = coef[0];
  float arr = 0.f;
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < nV; v += gridDim.x * blockDim.x) {
    float rv[3], zv[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const int i = 3 * v + k;
      x[i] += alpha * __ldcg(p + i);
      rv[k] = r[i] - alpha * __ldcg(ap + i);
      r[i] = rv[k];
      arr += rv[k] * rv[k];
    }
    apply_minv(minv, v, rv, zv);
#pragma unroll
    for (int k = 0; k < 3; ++k) x0[3 * v + k] = c * zv[k];
  }
  double s = cta_sum_f(arr);
  if (threadIdx.x == 0) part[blockIdx.x] = s;
  if (last_block(&st->count)) {
    const double rr = sum_partials(part, gridDim.x);
    if (threadIdx.x == 0) {
      st->rr = rr;
      st->it = it + 1;
      if (rr <= st->tol2 || it + 1 >= st->max_it || !(rr == rr)) st->done = 1;
      st->count = 0;
    }
  }
}

// out = b - A x, or A x without b (rows of pinned vertices give 0)
__device__ __forceinline__ void mg0_resid_row(int v, const float *s, const float *b, float *out,
                                              const unsigned char *pinned) {
  const bool pin = pinned && pinned[v];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const float t = b ? __ldcg(b + 3 * v + k) - s[k] : s[k];
    out[3 * v + k] = pin ? 0.f : t;
  }
}

// over the values' own layout, G lanes per row
template <int G>
__global__ void __launch_bounds__(256)
k_mg0_resid(int nV, const int *__restrict__ brp, const int *__restrict__ bcol, const float *__restrict__ val,
            const float *__restrict__ b, const float *__restrict__ x, float *__restrict__ out,
            const unsigned char *__restrict__ pinned, const PcgState *__restrict__ st) {
  pdl_wait();
  pdl_trigger();
  if (st && st->done) return;
  BT_ROW_LOOP_BEGIN(G)
  float s[3] = {0.f, 0.f, 0.f};
  if (active) spmv_row_acc<G>(v, sl, brp, bcol, val, [&](int c) { return __ldcg(x + c); }, s[0], s[1], s[2]);
  group_reduce<G>(s[0], s[1], s[2]);
  if (active && sl == 0) mg0_resid_row(v, s, b, out, pinned);
  BT_ROW_LOOP_END
}

// over the sliced-ELL BF16 copy (bound by HBM: 18 B of values and 4 B of column per block)
template <int S>
__global__ void __launch_bounds__(256)
k_mg0_resid_sell(SellView sv, const uint2 *__restrict__ val, const float *__restrict__ b, const float *x,
                 float *__restrict__ out, const unsigned char *__restrict__ pinned, const PcgState *__restrict__ st) {
  pdl_wait();
  pdl_trigger();
  if (st && st->done) return;
  sell_pass<S>(sv, val, x, [&](int v, float *s) { mg0_resid_row(v, s, b, out, pinned); });
}

// Final step of the V-cycle with the block-Jacobi smoother:
// z = x + c Dinv (b - A x), partial sums of b.z; the last block stores r.z
// and beta = r.z / r.z_old in the PCG state.
__device__ __forceinline__ float mg0_post_row(int v, const float *s, const float *minv, const float *b, const float *x,
                                              float *z, const unsigned char *pinned, float c) {
  float bv[3], rv[3], zv[3], acc = 0.f;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    bv[k] = __ldcg(b + 3 * v + k);
    rv[k] = bv[k] - s[k];
  }
  apply_minv(minv, v, rv, zv);
  const bool pin = pinned && pinned[v];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const float zk = pin ? 0.f : __ldcg(x + 3 * v + k) + c * zv[k];
    z[3 * v + k] = zk;
    acc += bv[k] * zk;
  }
  return acc;
}
__device__ __forceinline__ void finish_rz(float acc, double *__restrict__ part, PcgState *__restrict__ st) {
  double s = cta_sum_f(acc);
  if (threadIdx.x == 0) part[blockIdx.x] = s;
  if (last_block(&st->count)) {
    const double rz = sum_partials(part, gridDim.x);
    if (threadIdx.x == 0) {
      st->beta = (float)(rz / st->rz);
      st->rz = rz;
      st->count = 0;
    }
  }
}
template <int G>
__global__ void __launch_bounds__(256)
k_mg0_post_bj(int nV, const int *__restrict__ brp, const int *__restrict__ bcol, const float *__restrict__ val,
              const float *__restrict__ minv, const float *__restrict__ b, const float *__restrict__ x,
              float *__restrict__ z, const unsigned char *__restrict__ pinned, const float *__restrict__ coef,
              double *__restrict__ part, PcgState *__restrict__ st) {
  pdl_wait();
  pdl_trigger();
  if (st->done) return;
  const float c = coef[0];
  float acc = 0.f;
  BT_ROW_LOOP_BEGIN(G)
  float s[3] = {0.f, 0.f, 0.f};
  if (active) spmv_row_acc<G>(v, sl, brp, bcol, val, [&](int cc) { return __ldcg(x + cc); }, s[0], s[1], s[2]);
  group_reduce<G>(s[0], s[1], s[2]);
  if (active && sl == 0) acc += mg0_post_row(v, s, minv, b, x, z, pinned, c);
  BT_ROW_LOOP_END
  finish_rz(acc, part, st);
}
template <int S>
__global__ void __launch_bounds__(256)
k_mg0_post_bj_sell(SellView sv, const uint2 *__restrict__ val, const float *__restrict__ minv,
                   const float *__restrict__ b, const float *x, float *__restrict__ z,
                   const unsigned char *__restrict__ pinned, const float *__restrict__ coef,
                   double *__restrict__ part, PcgState *__restrict__ st) {
  pdl_wait();
  pdl_trigger();
  if (st->done) return;
  const float c = coef[0];
  float acc = 0.f;
  sell_pass<S>(sv, val, x, [&](int v, float *s) { acc += mg0_post_row(v, s, minv, b, x, z, pinned, c); });
  finish_rz(acc, part, st);
}

// y = G r (learned factor, lower rows; pinned rows give 0)
template <int G>
__global__ void __launch_bounds__(256)
k_mg0_fac_lower(int nV, const int4 *__restrict__ meta, const int *__restrict__ bcol,
                const __nv_bfloat16 *__restrict__ gl, const float *__restrict__ r, float *__restrict__ y,
                const unsigned char *__restrict__ pinned, const PcgState *__restrict__ st) {
  pdl_wait();
  pdl_trigger();
  if (st && st->done) return;
  BT_ROW_LOOP_BEGIN(G)
  float s0 = 0.f, s1 = 0.f, s2 = 0.f;
  if (active) {
    const int4 m = __ldg(meta + v);
    const int nl = (m.w & 0xFFFF) + 1;
    tri_row_acc4<G>(sl, bcol + m.x, gl + m.y, 3 * nl, padded_row(nl), [&](int c) { return __ldcg(r + c); }, s0, s1,
                    s2);
  }
  group_reduce<G>(s0, s1, s2);
  if (active && sl == 0) {
    if (pinned && pinned[v]) s0 = s1 = s2 = 0.f;
    y[3 * v] = s0;
    y[3 * v + 1] = s1;
    y[3 * v + 2] = s2;
  }
  BT_ROW_LOOP_END
}

// out = (xin, or 0) + c G^T y (upper rows), c = coef[0] (1 without coef). With
// b and part (the final V-cycle step) also r.z = b.out and beta in the state.
template <int G>
__global__ void __launch_bounds__(256)
k_mg0_fac_upper(int nV, const int4 *__restrict__ meta, const int *__restrict__ bcol,
                const __nv_bfloat16 *__restrict__ gu, const float *__restrict__ y, const float *__restrict__ xin,
                float *__restrict__ out, const unsigned char *__restrict__ pinned, const float *__restrict__ coef,
                const float *__restrict__ b, double *__restrict__ part, PcgState *__restrict__ st) {
  pdl_wait();
  pdl_trigger();
  if (st && st->done) return;
  const float c = coef ? coef[0] : 1.f;
  float acc = 0.f;
  BT_ROW_LOOP_BEGIN(G)
  float s0 = 0.f, s1 = 0.f, s2 = 0.f;
  if (active) {
    const int4 m = __ldg(meta + v);
    const int d = m.w & 0xFFFF, nu = (m.w >> 16) - d;
    tri_row_acc4<G>(sl, bcol + m.x + d, gu + m.z, 3 * nu, padded_row(nu), [&](int cc) { return __ldcg(y + cc); }, s0,
                    s1, s2);
  }
  group_reduce<G>(s0, s1, s2);
  if (active && sl == 0) {
    const bool pin = pinned && pinned[v];
    float o[3] = {c * s0, c * s1, c * s2};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      if (xin) o[k] += __ldcg(xin + 3 * v + k);
      if (pin) o[k] = 0.f;
      out[3 * v + k] = o[k];
      if (b) acc += __ldcg(b + 3 * v + k) * o[k];
    }
  }
  BT_ROW_LOOP_END
  if (part) finish_rz(acc, part, st);
}

// The same passes over the factor's sliced-ELL copies, where one warp per slice fills
// the GPU (2,432 slices on 152 SMs): whole solves on 117k vertices 12.6 -> 11.8 ms, on
// 531k 42.8 -> 38.8; on 15.6k vertices the lane form is faster (4.26 ms, 4.44).
__global__ void __launch_bounds__(256)
k_mg0_fac_lower_sell(SellView sv, const uint2 *__restrict__ val, const float *r, float *__restrict__ y,
                     const unsigned char *__restrict__ pinned, const PcgState *__restrict__ st) {
  pdl_wait();
  pdl_trigger();
  if (st && st->done) return;
  sell_pass<1>(sv, val, r, [&](int v, float *s) {
    const bool pin = pinned && pinned[v];
#pragma unroll
    for (int k = 0; k < 3; ++k) y[3 * v + k] = pin ? 0.f : s[k];
  });
}

__global__ void __launch_bounds__(256)
k_mg0_fac_upper_sell(SellView sv, const uint2 *__restrict__ val, const float *y, const float *__restrict__ xin,
                     float *__restrict__ out, const unsigned char *__restrict__ pinned,
                     const float *__restrict__ coef, const float *__restrict__ b, double *__restrict__ part,
                     PcgState *__restrict__ st) {
  pdl_wait();
  pdl_trigger();
  if (st && st->done) return;
  const float c = coef ? coef[0] : 1.f;
  float acc = 0.f;
  sell_pass<1>(sv, val, y, [&](int v, float *s) {
    const bool pin = pinned && pinned[v];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      float o = c * s[k];
      if (xin) o += __ldcg(xin + 3 * v + k);
      if (pin) o = 0.f;
      out[3 * v + k] = o;
      if (b) acc += __ldcg(b + 3 * v + k) * o;
    }
  });
  if (part) finish_rz(acc, part, st);
}

// BF16 copy of a coarse level, exactly symmetric: block k gets
// (C_k + C_rev(k)^T) / 2, rounded once (C_k and C_rev(k) come from separate
// Galerkin sums and may differ in their last bits).
__global__ void __launch_bounds__(256)
k_mgc_to_bf16(int64_t nnzb, const int *__restrict__ rev, const float *__restrict__ val,
              __nv_bfloat16 *__restrict__ val16) {
  for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < nnzb; k += (int64_t)gridDim.x * blockDim.x) {
    const float *a = val + 36 * k, *t = val + 36ll * __ldg(rev + k);
    __nv_bfloat16 *o = val16 + 36 * k;
#pragma unroll
    for (int r = 0; r < 6; ++r)
#pragma unroll
      for (int c = 0; c < 6; ++c)
        o[6 * r + c] = __float2bfloat16_rn(0.5f * (__ldg(a + 6 * r + c) + __ldg(t + 6 * c + r)));
  }
}

// ======================================================== coarse levels ===
// Row I of a 6x6-block level: G lanes stride the row's blocks; s = A_I. x
template <int G, class XV>
__device__ __forceinline__ void crow_acc(int I, int sl, const int *__restrict__ rp, const int *__restrict__ ci,
                                         const __nv_bfloat16 *__restrict__ val, XV &&xv, float s[6]) {
  const int k1 = __ldg(rp + I + 1);
  for (int k = __ldg(rp + I) + sl; k < k1; k += G) {
    const int J = __ldg(ci + k);
    float xj[6];
#pragma unroll
    for (int c = 0; c < 6; ++c) xj[c] = xv(6 * J + c);
    // 36 BF16 values = 9 x 8 bytes
    const uint2 *a2 = reinterpret_cast<const uint2 *>(val + 36ll * k);
    float a[36];
#pragma unroll
    for (int q = 0; q < 9; ++q) {
      const uint2 t = __ldg(a2 + q);
      a[4 * q] = __uint_as_float(t.x << 16);
      a[4 * q + 1] = __uint_as_float(t.x & 0xFFFF0000u);
      a[4 * q + 2] = __uint_as_float(t.y << 16);
      a[4 * q + 3] = __uint_as_float(t.y & 0xFFFF0000u);
    }
#pragma unroll
    for (int r = 0; r < 6; ++r)
#pragma unroll
      for (int c = 0; c < 6; ++c) s[r] += a[6 * r + c] * xj[c];
  }
}

template <int G>
__device__ __forceinline__ void group_reduce6(float s[6]) {
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1)
#pragma unroll
    for (int r = 0; r < 6; ++r) s[r] += __shfl_xor_sync(0xffffffffu, s[r], o);
}


#define BT_CROW_LOOP_BEGIN(G)                                                   \
  const int lane_ = threadIdx.x & 31, sl = lane_ % (G), gw_ = lane_ / (G);     \
  const int warp_ = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;              \
  const int nwarps_ = (gridDim.x * blockDim.x) >> 5;                           \
  for (int ib_ = warp_ * (32 / (G)); ib_ < n; ib_ += nwarps_ * (32 / (G))) {   \
    const int I = ib_ + gw_;                                                    \
    const bool active = I < n;
#define BT_CROW_LOOP_END }

// first smoothing step from x = 0: x = d = c0 Dinv b, r = b (x = Dinv b when exact)
__global__ void __launch_bounds__(256)
k_mgc_first(int n, const float *__restrict__ dinv, const float *__restrict__ b, float *__restrict__ x,
            float *__restrict__ r, float *__restrict__ d, const float *__restrict__ coef,
            const PcgState *__restrict__ st) {
  pdl_wait();
  pdl_trigger();
  if (st && st->done) return;
  const float c = coef ? coef[0] : 1.f;
  for (int I = blockIdx.x * blockDim.x + threadIdx.x; I < n; I += gridDim.x * blockDim.x) {
    float bv[6], z[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) bv[k] = __ldcg(b + 6 * I + k);
    apply_dinv6(dinv, I, bv, z);
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      const float xv = c * z[k];
      x[6 * I + k] = xv;
      if (r) r[6 * I + k] = bv[k];
      if (d) d[6 * I + k] = xv;
    }
  }
}

// Chebyshev step j >= 1: r -= A d_in; d_out = c1 d_in + c2 Dinv r; x += d_out
template <int G>
__global__ void __launch_bounds__(256)
k_mgc_cheb(int n, const int *__restrict__ rp, const int *__restrict__ ci, const __nv_bfloat16 *__restrict__ val,
           const float *__restrict__ dinv, const float *__restrict__ d_in, float *__restrict__ d_out,
           float *__restrict__ r, float *__restrict__ x, const float *__restrict__ coef, int j,
           const PcgState *__restrict__ st) {
  pdl_wait();
  pdl_trigger();
  if (st && st->done) return;
  const float c1 = coef[2 * j - 1], c2 = coef[2 * j];
  BT_CROW_LOOP_BEGIN(G)
  float s[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (active) crow_acc<G>(I, sl, rp, ci, val, [&](int c) { return __ldcg(d_in + c); }, s);
  group_reduce6<G>(s);
  if (active && sl == 0) {
    float rv[6], z[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      rv[k] = r[6 * I + k] - s[k];
      r[6 * I + k] = rv[k];
    }
    apply_dinv6(dinv, I, rv, z);
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      const float dk = c1 * __ldcg(d_in + 6 * I + k) + c2 * z[k];
      d_out[6 * I + k] = dk;
      x[6 * I + k] += dk;
    }
  }
  BT_CROW_LOOP_END
}

// r = b - A x
template <int G>
__global__ void __launch_bounds__(256)
k_mgc_resid(int n, const int *__restrict__ rp, const int *__restrict__ ci, const __nv_bfloat16 *__restrict__ val,
            const float *__restrict__ b, const float *__restrict__ x, float *__restrict__ r,
            const PcgState *__restrict__ st) {
  pdl_wait();
  pdl_trigger();
  if (st && st->done) return;
  BT_CROW_LOOP_BEGIN(G)
  float s[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (active) crow_acc<G>(I, sl, rp, ci, val, [&](int c) { return __ldcg(x + c); }, s);
  group_reduce6<G>(s);
  if (active && sl == 0)
#pragma unroll
    for (int k = 0; k < 6; ++k) r[6 * I + k] = __ldcg(b + 6 * I + k) - s[k];
  BT_CROW_LOOP_END
}

// first post-smoothing step: r = b - A x; d = c0 Dinv r; x_out = x + d
template <int G>
__global__ void __launch_bounds__(256)
k_mgc_post_first(int n, const int *__restrict__ rp, const int *__restrict__ ci, const __nv_bfloat16 *__restrict__ val,
                 const float *__restrict__ dinv, const float *__restrict__ b, const float *__restrict__ x,
                 float *__restrict__ x_out, float *__restrict__ r, float *__restrict__ d,
                 const float *__restrict__ coef, const PcgState *__restrict__ st) {
  pdl_wait();
  pdl_trigger();
  if (st && st->done) return;
  const float c0 = coef[0];
  BT_CROW_LOOP_BEGIN(G)
  float s[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (active) crow_acc<G>(I, sl, rp, ci, val, [&](int c) { return __ldcg(x + c); }, s);
  group_reduce6<G>(s);
  if (active && sl == 0) {
    float rv[6], z[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      rv[k] = __ldcg(b + 6 * I + k) - s[k];
      r[6 * I + k] = rv[k];
    }
    apply_dinv6(dinv, I, rv, z);
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      const float dk = c0 * z[k];
      d[6 * I + k] = dk;
      x_out[6 * I + k] = __ldcg(x + 6 * I + k) + dk;
    }
  }
  BT_CROW_LOOP_END
}

// y = Dinv (A x) (power iteration on a coarse level)
template <int G>
__global__ void __launch_bounds__(256)
k_mgc_MA(int n, const int *__restrict__ rp, const int *__restrict__ ci, const __nv_bfloat16 *__restrict__ val,
         const float *__restrict__ dinv, const float *__restrict__ x, float *__restrict__ y) {
  BT_CROW_LOOP_BEGIN(G)
  float s[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (active) crow_acc<G>(I, sl, rp, ci, val, [&](int c) { return __ldcg(x + c); }, s);
  group_reduce6<G>(s);
  if (active && sl == 0) {
    float z[6];
    apply_dinv6(dinv, I, s, z);
#pragma unroll
    for (int k = 0; k < 6; ++k) y[6 * I + k] = z[k];
  }
  BT_CROW_LOOP_END
}

// coarsest level, dense, outside the cluster launch: x = Ainv b, a warp per row
__global__ void __launch_bounds__(256)
k_mg_dense_apply(int nd, const float *__restrict__ ainv, const float *__restrict__ b, float *__restrict__ x,
                 const PcgState *__restrict__ st) {
  pdl_wait();
  pdl_trigger();
  if (st && st->done) return;
  const int lane = threadIdx.x & 31, i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (i >= nd) return;
  float s = 0.f;
  for (int j = lane; j < nd; j += 32) s += __ldg(ainv + (int64_t)i * nd + j) * __ldcg(b + j);
  s = warp_sumf(s);
  if (lane == 0) x[i] = s;
}

// ==================================== coarse levels in one cluster launch ===
// The coarse part of the V-cycle (every level from cl.first down to the
// coarsest and back) as one kernel of one thread-block cluster. Each CTA owns
// a contiguous range of every level's nodes and keeps their BF16 blocks,
// inverse diagonal blocks, transfer blocks and own vector entries in shared
// memory. A step gathers its neighbours' vector entries through L2 and ends in
// one hardware cluster barrier.
//
// Why: as launches these levels are 27 dependent kernels of 1 - 42 CTAs per
// V-cycle, each bound by its launch and by a chain of three L2 latencies (row
// pointer -> column -> vector), 4 - 9 us apiece. Here a step is one barrier
// (~500 cycles, plus the flush of the step's stores) and one L2 latency (~460);
// measured after its wait, the coarse part takes 42 us on the 96^3-cell cube
// (1,331 + 64 nodes; ~150 us as launches) and 12 us at 24^3 (670 + 27). The
// operators are staged before the wait on the previous kernel, i.e. while that
// one is still running. 16 CTAs beat 8 (12.5 against 13.0 ms for a 24^3 Newton
// step, 56.5 against 60.4 ms for a 96^3 solve): a step's row products are
// bound by the shared-memory and issue rate of the CTAs that hold the level. Gathering
// through distributed shared memory instead was measured and is slower: a
// single load takes ~500 cycles, and scattered 24-byte entries from 1024
// threads ~8,000.
__device__ __forceinline__ void ldcg6(const float *v, int node, float x[6]) {
  const float2 *p = reinterpret_cast<const float2 *>(v + 6 * node);
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    const float2 t = __ldcg(p + q);
    x[2 * q] = t.x;
    x[2 * q + 1] = t.y;
  }
}

// d = a * b + c on two packed FP32 values
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;"
      : "=l"(d)
      : "l"(*reinterpret_cast<unsigned long long *>(&a)), "l"(*reinterpret_cast<unsigned long long *>(&b)),
        "l"(*reinterpret_cast<unsigned long long *>(&c)));
  return *reinterpret_cast<float2 *>(&d);
}

// s = (A v)_i of the CTA's own row i, over a group of G lanes (all lanes end with the sum)
template <int G>
__device__ __forceinline__ void cl_row(const char *sm, const MgClLevel &L, const float *v, int i, bool active, int sl,
                                       float s[6]) {
  float2 s2[6];
#pragma unroll
  for (int c = 0; c < 6; ++c) s2[c] = make_float2(0.f, 0.f);
  if (active) {
    const int *rp = reinterpret_cast<const int *>(sm + L.o_rp);
    const int *ci = reinterpret_cast<const int *>(sm + L.o_ci);
    const int k0 = rp[0], k1 = rp[i + 1] - k0;
#pragma unroll 2
    for (int k = rp[i] - k0 + sl; k < k1; k += G) {
      float2 x[3];
      const float2 *xp = reinterpret_cast<const float2 *>(v) + 3 * ci[k];
#pragma unroll
      for (int q = 0; q < 3; ++q) x[q] = __ldcg(xp + q);
      const uint2 *a2 = reinterpret_cast<const uint2 *>(sm + L.o_val) + 9 * k;
#pragma unroll
      for (int q = 0; q < 9; ++q) {
        const uint2 t = a2[q];  // entries 4q .. 4q + 3 of the row-major block: pairs 2q and 2q + 1 of its 18
        s2[(2 * q) / 3] = fma2(make_float2(__uint_as_float(t.x << 16), __uint_as_float(t.x & 0xFFFF0000u)),
                               x[(2 * q) % 3], s2[(2 * q) / 3]);
        s2[(2 * q + 1) / 3] = fma2(make_float2(__uint_as_float(t.y << 16), __uint_as_float(t.y & 0xFFFF0000u)),
                                   x[(2 * q + 1) % 3], s2[(2 * q + 1) / 3]);
      }
    }
  }
#pragma unroll
  for (int c = 0; c < 6; ++c) s[c] = s2[c].x + s2[c].y;
  group_reduce6<G>(s);
}

// One smoothing step of the CTA's own rows: r -= A v (kStepPost: r = b - A v,
// v = x), then with z = Dinv r
//   kStepCheb:  d = c1 d + c2 z, acc += d
//   kStepPost:  d = c2 z, acc = x + d  (acc is the b area: b is read for the last time here)
//   kStepResid: d = Q^T r, the node's share of the restriction
// and out = d for the other CTAs, or acc on the level's final step. A row's
// group holds the whole sum in every lane; its lanes share the components of
// the 6x6 product.
enum { kStepCheb = 0, kStepPost = 1, kStepResid = 2 };
template <int G>
__device__ __forceinline__ void cl_step_g(char *sm, const MgClLevel &L, int r0, int rows, int mode, const float *v,
                                          float *out, int o_acc, bool final, float c1, float c2) {
  const int sl = threadIdx.x % G, g = threadIdx.x / G;
  const float *rr = reinterpret_cast<const float *>(sm + (mode == kStepPost ? L.o_b : L.o_r));
  float *rw = reinterpret_cast<float *>(sm + L.o_r), *d = reinterpret_cast<float *>(sm + L.o_d);
  float *x = reinterpret_cast<float *>(sm + L.o_x), *acc = reinterpret_cast<float *>(sm + o_acc);
  const float *M = reinterpret_cast<const float *>(sm + (mode == kStepResid ? L.o_Q : L.o_dinv));
  for (int i0 = 0; i0 < rows; i0 += blockDim.x / G) {
    const int i = i0 + g;
    const bool active = i < rows;
    float s[6];
    cl_row<G>(sm, L, v, i, active, sl, s);
    float rn[6];
    if (active)
#pragma unroll
      for (int c = 0; c < 6; ++c) rn[c] = rr[6 * i + c] - s[c];
    __syncwarp();
    if (active)
#pragma unroll
    for (int a = sl; a < 6; a += G) {
      const float *m = M + 36 * i + (mode == kStepResid ? a : 6 * a);  // column a of Q, row a of Dinv
      const int st = mode == kStepResid ? 6 : 1;
      float z = 0.f, mine = rn[0];
#pragma unroll
      for (int c = 0; c < 6; ++c) z += m[st * c] * rn[c];
#pragma unroll
      for (int c = 1; c < 6; ++c) mine = a == c ? rn[c] : mine;
      const int e = 6 * i + a;
      float o = z;
      if (mode != kStepResid) {
        rw[e] = mine;
        const float dk = mode == kStepCheb ? c1 * d[e] + c2 * z : c2 * z;
        const float ak = (mode == kStepCheb ? acc[e] : x[e]) + dk;
        d[e] = dk;
        acc[e] = ak;
        o = final ? ak : dk;
      }
      out[6 * r0 + e] = o;
    }
  }
}
__device__ __forceinline__ void cl_step(char *sm, const MgClLevel &L, int r0, int rows, int mode, const float *v,
                                        float *out, int o_acc, bool final, float c1, float c2) {
  // as many lanes per row as keep the CTA's threads busy in one pass
  if (rows <= kClThreads / 16) cl_step_g<16>(sm, L, r0, rows, mode, v, out, o_acc, final, c1, c2);
  else if (rows <= kClThreads / 8) cl_step_g<8>(sm, L, r0, rows, mode, v, out, o_acc, final, c1, c2);
  else cl_step_g<4>(sm, L, r0, rows, mode, v, out, o_acc, final, c1, c2);
}

// asynchronous global -> shared copies of n 4-byte words (8: n even, both ends 8-byte aligned)
__device__ __forceinline__ void cl_stage8(unsigned dst, const void *src, int n) {
  const char *s = static_cast<const char *>(src);
  for (int i = threadIdx.x; i < n / 2; i += blockDim.x)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst + 8 * i), "l"(s + 8ll * i) : "memory");
}
__device__ __forceinline__ void cl_stage4(unsigned dst, const void *src, int n) {
  const char *s = static_cast<const char *>(src);
  for (int i = threadIdx.x; i < n; i += blockDim.x)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst + 4 * i), "l"(s + 4ll * i) : "memory");
}

__global__ void __launch_bounds__(kClThreads, 1)
k_mgc_cluster(const __grid_constant__ MgClArgs a, const PcgState *__restrict__ st) {
  extern __shared__ __align__(16) char sm[];
  __shared__ float s_coef[kMgClusterLevels * kMgCoef];
  const unsigned rank = cl_rank();
  const unsigned smb = (unsigned)__cvta_generic_to_shared(sm);
  const int last = a.nlev - 1;
  // Stage the operators. They were written by the set-up launches, which are
  // complete: this kernel starts at the earliest when its predecessor's own
  // wait has returned.
  for (int i = threadIdx.x; i < a.nlev * kMgCoef; i += blockDim.x) s_coef[i] = a.coef[kMgCoef * a.first + i];
  for (int l = 0; l < a.nlev; ++l) {
    const MgClLevel &L = a.lv[l];
    const int r0 = L.split[rank], nr = L.split[rank + 1] - r0, k0 = L.bsplit[rank], nk = L.bsplit[rank + 1] - k0;
    if (l == last && a.last_mode == kMgLastDense) {
      cl_stage8(smb + L.o_val, a.ainv + 6ll * r0 * a.nd, 6 * nr * a.nd);
    } else {
      cl_stage8(smb + L.o_val, L.val16 + 36ll * k0, 18 * nk);
      cl_stage8(smb + L.o_dinv, L.dinv + 36ll * r0, 36 * nr);
      cl_stage4(smb + L.o_ci, L.ci + k0, nk);
      cl_stage4(smb + L.o_rp, L.rp + r0, nr + 1);
    }
    if (l < last) {
      cl_stage8(smb + L.o_Q, L.Q + 36ll * r0, 36 * nr);
      cl_stage4(smb + L.o_agg, L.agg + r0, nr);
    }
    if (l > 0) {
      const int m0 = L.msplit[rank];
      cl_stage4(smb + L.o_mptr, L.mptr + r0, nr + 1);
      cl_stage4(smb + L.o_mem, L.midx + m0, L.msplit[rank + 1] - m0);
    }
  }
  asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  pdl_wait();
  pdl_trigger();
  if (st && st->done) return;  // the same for every CTA: nothing writes the flag while this kernel runs

  auto F = [&](int o) { return reinterpret_cast<float *>(sm + o); };
  const int lane = threadIdx.x & 31;
  // ---- down
  const float *t_fine = nullptr;  // the finer level's shares of the restriction
  for (int l = 0; l <= last; ++l) {
    const MgClLevel &L = a.lv[l];
    const int r0 = L.split[rank], rows = L.split[rank + 1] - r0;
    const bool dense = l == last && a.last_mode == kMgLastDense;
    const bool exact = l == last && a.last_mode == kMgLastExact;
    const float *cf = s_coef + kMgCoef * l;
    // right-hand side and first step from x = 0: x = d = c0 Dinv b, r = b. One warp per node.
    for (int i = threadIdx.x >> 5; i < rows; i += blockDim.x >> 5) {
      const int c = lane & 7;
      float bv = 0.f;
      if (l == 0) {
        if (c < 6) bv = __ldcg(L.gb + 6 * (r0 + i) + c);
      } else {
        const int *mp = reinterpret_cast<const int *>(sm + L.o_mptr);
        const int *mem = reinterpret_cast<const int *>(sm + L.o_mem);
        if (c < 6)
#pragma unroll 4
          for (int m = mp[i] - mp[0] + (lane >> 3); m < mp[i + 1] - mp[0]; m += 4)
            bv += __ldcg(t_fine + 6 * mem[m] + c);
        bv += __shfl_xor_sync(0xffffffffu, bv, 8);
        bv += __shfl_xor_sync(0xffffffffu, bv, 16);
      }
      float bb[6];
#pragma unroll
      for (int k = 0; k < 6; ++k) bb[k] = __shfl_sync(0xffffffffu, bv, k);
      if (lane < 6) {
        const int e = 6 * i + lane;
        if (dense) {
          L.gb[6 * r0 + e] = bv;
        } else {
          const float *m = F(L.o_dinv) + 36 * i + 6 * lane;
          float z = 0.f;
#pragma unroll
          for (int k = 0; k < 6; ++k) z += m[k] * bb[k];
          const float xv = exact ? z : cf[0] * z;
          F(L.o_b)[e] = bv;
          F(L.o_x)[e] = xv;
          F(L.o_r)[e] = bv;
          F(L.o_d)[e] = xv;
          (l == last && (exact || L.deg == 1) ? L.gres : L.gd)[6 * r0 + e] = xv;
        }
      }
    }
    cl_barrier();
    if (dense) {
      // x = Ainv b: every CTA gathers b, then one warp per row of its own nodes
      float *db = F(a.o_db);
      for (int j = threadIdx.x; j < a.nd; j += blockDim.x) db[j] = __ldcg(L.gb + j);
      __syncthreads();
      for (int i = threadIdx.x >> 5; i < 6 * rows; i += blockDim.x >> 5) {
        const float *m = F(L.o_val) + i * a.nd;
        float s = 0.f;
        for (int j = lane; j < a.nd; j += 32) s += m[j] * db[j];
        s = warp_sumf(s);
        if (lane == 0) L.gres[6 * r0 + i] = s;
      }
      cl_barrier();
      break;
    }
    if (exact) break;
    float *din = L.gd, *dout = L.gd2;
    for (int j = 1; j < L.deg; ++j) {
      const bool fin = l == last && j + 1 == L.deg;
      cl_step(sm, L, r0, rows, kStepCheb, din, fin ? L.gres : dout, L.o_x, fin, cf[2 * j - 1], cf[2 * j]);
      cl_barrier();
      float *t = din;
      din = dout;
      dout = t;
    }
    if (l < last) {
      cl_step(sm, L, r0, rows, kStepResid, din, dout, L.o_x, false, 0.f, 0.f);
      t_fine = dout;
      cl_barrier();
    }
  }
  // ---- up
  for (int l = last - 1; l >= 0; --l) {
    const MgClLevel &L = a.lv[l];
    const int r0 = L.split[rank], rows = L.split[rank + 1] - r0;
    const float *cf = s_coef + kMgCoef * l;
    const int *agg = reinterpret_cast<const int *>(sm + L.o_agg);
    const float *xc = a.lv[l + 1].gres;
    for (int e = threadIdx.x; e < 6 * rows; e += blockDim.x) {  // x += Q x_c
      float c[6];
      ldcg6(xc, agg[e / 6], c);
      const float *q = F(L.o_Q) + 6 * e;
      float s = 0.f;
#pragma unroll
      for (int k = 0; k < 6; ++k) s += q[k] * c[k];
      s += F(L.o_x)[e];
      F(L.o_x)[e] = s;
      L.gx[6 * r0 + e] = s;
    }
    cl_barrier();
    cl_step(sm, L, r0, rows, kStepPost, L.gx, L.deg == 1 ? L.gres : L.gd, L.o_b, L.deg == 1, 0.f, cf[0]);
    float *din = L.gd, *dout = L.gd2;
    for (int j = 1; j < L.deg; ++j) {
      cl_barrier();
      const bool fin = j + 1 == L.deg;
      cl_step(sm, L, r0, rows, kStepCheb, din, fin ? L.gres : dout, L.o_b, fin, cf[2 * j - 1], cf[2 * j]);
      float *t = din;
      din = dout;
      dout = t;
    }
    if (l > 0) cl_barrier();
  }
}

// ==================================================== eigenvalue bounds ===
// deterministic start vector in [-1, 1] (integer hash of the index)
__global__ void k_mg_hash_fill(int64_t n, float *__restrict__ v, unsigned seed) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    unsigned h = (unsigned)i * 2654435761u ^ seed;
    h ^= h >> 16;
    h *= 2246822519u;
    h ^= h >> 13;
    h *= 3266489917u;
    h ^= h >> 16;
    v[i] = (float)(h & 0xFFFFFF) * (2.f / 16777215.f) - 1.f;
  }
}

__global__ void __launch_bounds__(256) k_mg_sumsq(int64_t n, const float *__restrict__ v, double *__restrict__ part) {
  float acc = 0.f;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const float t = v[i];
    acc += t * t;
  }
  double s = cta_sum_f(acc);
  if (threadIdx.x == 0) part[blockIdx.x] = s;
}

// Packed meshes: squared norms of v over each segment's DOFs (one CTA per
// segment, fixed order)
__global__ void __launch_bounds__(256)
k_mg_seg_sumsq(const int *__restrict__ voff, const float *__restrict__ v, double *__restrict__ out) {
  const int s = blockIdx.x;
  float acc = 0.f;
  for (int i = 3 * voff[s] + threadIdx.x; i < 3 * voff[s + 1]; i += blockDim.x) {
    const float t = v[i];
    acc += t * t;
  }
  const double r = cta_sum_f(acc);
  if (threadIdx.x == 0) out[s] = r;
}

// The power iteration of a block-diagonal operator runs independently in each
// block, so the per-segment norm ratios estimate every segment's own largest
// eigenvalue; their maximum bounds all of them (a ratio over the whole vector
// is dominated by the largest segments and can miss a small stiff one).
// Written as norms (1, max ratio) for k_mg_coef.
__global__ void k_mg_seg_lmax(int nseg, const double *__restrict__ prev, const double *__restrict__ last,
                              double *__restrict__ norms) {
  double m = 0.0;
  for (int s = threadIdx.x; s < nseg; s += blockDim.x)
    if (prev[s] > 0.0 && last[s] > 0.0 && isfinite(last[s])) m = fmax(m, last[s] / prev[s]);
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  if (threadIdx.x == 0) {
    norms[0] = 1.0;
    norms[1] = m > 0.0 ? m : 1.0;
  }
}

struct MgDegrees {
  int deg[kMgMaxLevels];
  int nlev;
};

// Chebyshev coefficients of each smoothed level from its power-iteration
// norms: lambda_max = 1.1 |y_K| / |y_{K-1}|, interval [lambda_max / 10,
// lambda_max]; coef = {1/theta, (c1_j, c2_j) for j = 1 .. deg-1} with
// rho_0 = delta/theta, rho_j = 1/(2 sigma - rho_{j-1}), c1_j = rho_j rho_{j-1},
// c2_j = 2 rho_j / delta (the Chebyshev semi-iteration, Saad 2003, Alg. 12.1).
__global__ void k_mg_coef(MgDegrees dg, const double *__restrict__ norms, float *__restrict__ coef) {
  const int l = threadIdx.x;
  if (l >= dg.nlev) return;
  const double a = norms[2 * l], b = norms[2 * l + 1];
  double lmax = (a > 0.0 && b > 0.0 && isfinite(a) && isfinite(b)) ? 1.1 * sqrt(b / a) : 1.0;
  const double lmin = lmax / 10.0;
  const double theta = 0.5 * (lmax + lmin), delta = 0.5 * (lmax - lmin), sigma = theta / delta;
  float *c = coef + kMgCoef * l;
  c[0] = (float)(1.0 / theta);
  double rho = 1.0 / sigma;
  for (int j = 1; j < dg.deg[l] && 2 * j < kMgCoef; ++j) {
    const double rn = 1.0 / (2.0 * sigma - rho);
    c[2 * j - 1] = (float)(rn * rho);
    c[2 * j] = (float)(2.0 * rn / delta);
    rho = rn;
  }
}

// ================================================================= host ====
namespace {

constexpr int kGc = 8;  // lanes per row on coarse levels

int grid_n(bartels_ctx ctx, int64_t n, int per_block = 256) {
  const int64_t g = (n + per_block - 1) / per_block;
  return (int)std::max<int64_t>(1, std::min<int64_t>(g, (int64_t)ctx->num_sms * 8));
}
// rows walked by groups of G lanes, 8 warps per 256-thread block
int grid_rows(bartels_ctx ctx, int64_t rows, int G) {
  const int64_t warps = (rows * G + 31) / 32;
  const int64_t g = (warps + 7) / 8;
  return (int)std::max<int64_t>(1, std::min<int64_t>(g, (int64_t)ctx->num_sms * 8));
}

// result vector of a level after its part of the V-cycle
float *level_result(const MgHierarchy *mg, int l) {
  const bool coarsest = l + 1 == (int)mg->lv.size();
  return coarsest ? mg->lv[l].x : mg->lv[l].x2;
}

// Chebyshev smoothing of a coarse level from x = 0 (deg steps): x, r, d. The
// first step is skipped when the restriction into the level has taken it.
int cheb_from_zero(bartels_ctx ctx, const MgLevel &c, const float *coef, bool first_done, const PcgState *st) {
  const int gr = grid_rows(ctx, c.n, kGc);
  if (!first_done)
    BT_LAUNCH_PDL(ctx, k_mgc_first, grid_n(ctx, c.n), 256, 0, c.n, c.dinv, c.b, c.x, c.r, c.d, coef, st);
  float *dc = c.d, *dn = c.d2;
  for (int j = 1; j < c.deg; ++j) {
    BT_LAUNCH_PDL(ctx, k_mgc_cheb<kGc>, gr, 256, 0, c.n, c.rp, c.ci, c.val16, c.dinv, dc, dn, c.r, c.x, coef, j, st);
    std::swap(dc, dn);
  }
  return BARTELS_OK;
}

// Restriction into level l (from level l - 1's residual r with its transfer
// blocks), taking level l's first smoothing step in the same kernel where that
// step is local (every level but a dense coarsest). Returns whether it did.
template <int BSF>
int restrict_into(bartels_ctx ctx, MgHierarchy *mg, const MgLevel &f, const float *r, int l, const PcgState *st,
                  bool *first_done) {
  MgLevel &c = mg->lv[l];
  const bool last = l + 1 == (int)mg->lv.size();
  // the cluster kernel takes the first step itself
  const bool fuse = !(mg->cl.ctas && l == mg->cl.first) && !(last && mg->dense);
  const bool exact = last && mg->coarse_blockdiag;  // x = Dinv b
  const float *coef = exact ? nullptr : mg->coef + kMgCoef * l;
  const float *dinv = fuse ? (const float *)c.dinv : nullptr;
  float *cx = fuse ? c.x : nullptr, *cr = fuse && !exact ? c.r : nullptr, *cd = fuse && !exact ? c.d : nullptr;
  const float *cf = fuse ? coef : nullptr;
  // A warp per aggregate while one per SM sub-partition's eight warps is enough for
  // all: its ~25 members then are one round of loads (solve on 117k vertices, 4.6k
  // aggregates: 13.4 -> 13.0 ms). With 34.8k aggregates eight lanes are faster
  // (48.4 ms, 16 or 32 lanes 49.1).
#define BT_RL(L)                                                                                              \
  BT_LAUNCH_PDL(ctx, (k_mg_restrict<BSF, L>), grid_rows(ctx, (c.n + 32 / L - 1) / (32 / L), 32), 256, 0, c.n, \
                f.mptr, f.midx, f.Q, r, c.b, dinv, cx, cr, cd, cf, st)
  if (c.n <= 32 * ctx->num_sms) BT_RL(32);
  else BT_RL(8);
#undef BT_RL
  *first_done = fuse;
  return BARTELS_OK;
}

int launch_cluster(bartels_ctx ctx, MgHierarchy *mg, const PcgState *st) {
  const MgClArgs &a = mg->cl;
  cudaLaunchAttribute at[2];
  cudaLaunchConfig_t cfg = cluster_config(ctx, a.ctas, kClThreads, a.smem, at);
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.numAttrs = 2;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, k_mgc_cluster, a, st);
  ctx->launches++;
  if (e != cudaSuccess) return fail(BARTELS_E_DEVICE, std::string("launch k_mgc_cluster: ") + cudaGetErrorString(e));
  return BARTELS_OK;
}

int enqueue_coarse(bartels_ctx ctx, MgHierarchy *mg, int l, bool first_done, const PcgState *st) {
  if (mg->cl.ctas && l == mg->cl.first) return launch_cluster(ctx, mg, st);
  MgLevel &c = mg->lv[l];
  const float *coef = mg->coef + kMgCoef * l;
  const int last = (int)mg->lv.size() - 1;
  if (l == last) {
    if (mg->dense) {
      BT_LAUNCH_PDL(ctx, k_mg_dense_apply, (mg->nd + 7) / 8, 256, 0, mg->nd, mg->ainv, c.b, c.x, st);
    } else if (mg->coarse_blockdiag) {
      if (!first_done)
        BT_LAUNCH_PDL(ctx, k_mgc_first, grid_n(ctx, c.n), 256, 0, c.n, c.dinv, c.b, c.x, (float *)nullptr,
                  (float *)nullptr, (const float *)nullptr, st);
    } else {
      BT_CHECK(cheb_from_zero(ctx, c, coef, first_done, st));
    }
    return BARTELS_OK;
  }
  const int gr = grid_rows(ctx, c.n, kGc);
  BT_CHECK(cheb_from_zero(ctx, c, coef, first_done, st));
  BT_LAUNCH_PDL(ctx, k_mgc_resid<kGc>, gr, 256, 0, c.n, c.rp, c.ci, c.val16, c.b, c.x, c.r, st);
  bool next_first = false;
  BT_CHECK(restrict_into<6>(ctx, mg, c, c.r, l + 1, st, &next_first));
  BT_CHECK(enqueue_coarse(ctx, mg, l + 1, next_first, st));
  BT_LAUNCH_PDL(ctx, k_mg_prolong<6>, grid_n(ctx, c.n), 256, 0, c.n, c.agg, c.Q, level_result(mg, l + 1), c.x, st);
  BT_LAUNCH_PDL(ctx, k_mgc_post_first<kGc>, gr, 256, 0, c.n, c.rp, c.ci, c.val16, c.dinv, c.b, c.x, c.x2, c.r, c.d, coef,
            st);
  float *dc = c.d, *dn = c.d2;
  for (int j = 1; j < c.deg; ++j) {
    BT_LAUNCH_PDL(ctx, k_mgc_cheb<kGc>, gr, 256, 0, c.n, c.rp, c.ci, c.val16, c.dinv, dc, dn, c.r, c.x2, coef, j, st);
    std::swap(dc, dn);
  }
  return BARTELS_OK;
}

// level-0 launches for the plan's SpMV lane count (4, 8 or 16) or factor lane count (4 or 8)
#define BT_MG_G(G_, ...)                \
  do {                                  \
    if ((G_) == 4) {                    \
      constexpr int GL = 4;             \
      __VA_ARGS__;                      \
    } else if ((G_) == 16) {            \
      constexpr int GL = 16;            \
      __VA_ARGS__;                      \
    } else {                            \
      constexpr int GL = 8;             \
      __VA_ARGS__;                      \
    }                                   \
  } while (0)

int fac_lower(bartels_ctx ctx, bartels_mesh_plan plan, const MgSmoother &sm, const float *in, float *out,
              const PcgState *st) {
  if (sm.lsell) {
    const SellView sv = plan->sell_factor[0]->view();
    BT_LAUNCH_PDL(ctx, k_mg0_fac_lower_sell, sell_grid(ctx, sv.nslices, 1), 256, 0, sv, sm.lsell, in, out, plan->pinned,
                  st);
    return BARTELS_OK;
  }
  const int GT = plan_lanes_tri(ctx, plan) == 8 ? 8 : 4;
  const int g = grid_rows(ctx, plan->nV, GT);
  BT_MG_G(GT, BT_LAUNCH_PDL(ctx, k_mg0_fac_lower<GL>, g, 256, 0, plan->nV, sm.fp->meta, plan->bcol, sm.gl, in, out,
                        plan->pinned, st));
  return BARTELS_OK;
}

int fac_upper(bartels_ctx ctx, bartels_mesh_plan plan, const MgSmoother &sm, const float *y, const float *xin,
              float *out, const float *coef, const float *b, double *part, PcgState *st) {
  if (sm.usell) {
    const SellView sv = plan->sell_factor[1]->view();
    BT_LAUNCH_PDL(ctx, k_mg0_fac_upper_sell, sell_grid(ctx, sv.nslices, 1), 256, 0, sv, sm.usell, y, xin, out,
                  plan->pinned, coef, b, part, st);
    return BARTELS_OK;
  }
  const int GT = plan_lanes_tri(ctx, plan) == 8 ? 8 : 4;
  const int g = grid_rows(ctx, plan->nV, GT);
  BT_MG_G(GT, BT_LAUNCH_PDL(ctx, k_mg0_fac_upper<GL>, g, 256, 0, plan->nV, sm.fp->meta, plan->bcol, sm.gu, y, xin, out,
                        plan->pinned, coef, b, part, st));
  return BARTELS_OK;
}

// out = b - A x on the finest level, with the V-cycle's BF16 copy of A when it has one
int resid0(bartels_ctx ctx, bartels_mesh_plan plan, const float *values, const float *b, const float *x, float *out,
           const PcgState *st) {
  const uint2 *a16 = plan->mg ? plan->mg->a16 : nullptr;
  if (a16) {
    const SellView sv = plan->sell->view();
    const int S = sell_split(ctx, sv.nslices), g = sell_grid(ctx, sv.nslices, S);
    if (S == 1) BT_LAUNCH_PDL(ctx, k_mg0_resid_sell<1>, g, 256, 0, sv, a16, b, x, out, plan->pinned, st);
    else if (S == 2) BT_LAUNCH_PDL(ctx, k_mg0_resid_sell<2>, g, 256, 0, sv, a16, b, x, out, plan->pinned, st);
    else BT_LAUNCH_PDL(ctx, k_mg0_resid_sell<4>, g, 256, 0, sv, a16, b, x, out, plan->pinned, st);
  } else {
    const int G = plan_lanes_spmv(ctx, plan);
    const int g = grid_rows(ctx, plan->nV, G);
    BT_MG_G(G, BT_LAUNCH_PDL(ctx, k_mg0_resid<GL>, g, 256, 0, plan->nV, plan->brp, plan->bcol, values, b, x, out,
                             plan->pinned, st));
  }
  return BARTELS_OK;
}

int sumsq_into(bartels_ctx ctx, MgHierarchy *mg, int64_t n, const float *v, double *out) {
  const int g = std::min(grid_n(ctx, n), mg->nparts);
  BT_LAUNCH(ctx, k_mg_sumsq, g, 256, 0, n, v, mg->part);
  return reduce_sum(ctx, mg->part, g, out);
}

}  // namespace

void mg_destroy(MgHierarchy *mg) { delete mg; }

int mg_setup_numeric(bartels_ctx ctx, bartels_mesh_plan plan, const float *values, const MgSmoother &sm) {
  MgHierarchy *mg = plan->mg;
  if (!mg) return fail(BARTELS_E_INVALID_ARG, "multigrid: no hierarchy");
  const int L = (int)mg->lv.size();
  if (mg->a16) {
    FactorPattern *fp = nullptr;
    BT_CHECK(plan_factor_pattern(plan, &fp));
    BT_CHECK(sell_fill_bf16(ctx, plan, values, fp->rev, mg->a16));
  }
  for (int l = 0; l + 1 < L; ++l) {
    MgLevel &f = mg->lv[l], &c = mg->lv[l + 1];
    const int g = grid_n(ctx, c.nnzb * kGalLanes, 128);  // kGalLanes lanes per coarse block
    if (l == 0)
      BT_LAUNCH(ctx, k_mg_gal0, g, 128, 0, c.nnzb, f.gptr, f.gent, plan->brp, plan->bcol, values, f.Q, c.val);
    else
      BT_LAUNCH(ctx, k_mg_galc, g, 128, 0, c.nnzb, f.gptr, f.gent, f.ci, f.val, f.Q, c.val);
    BT_LAUNCH(ctx, k_mg_inv6, grid_n(ctx, c.n, 128), 128, 0, c.n, c.dpos, c.val, c.dinv);
    BT_LAUNCH(ctx, k_mgc_to_bf16, grid_n(ctx, c.nnzb), 256, 0, c.nnzb, (const int *)c.rev, (const float *)c.val,
              c.val16);
  }
  if (mg->dense) {
    const MgLevel &c = mg->lv[L - 1];
    MgInvArgs ia;
    ia.nodes = c.n;
    ia.rp = c.rp;
    ia.ci = c.ci;
    ia.rev = c.rev;
    ia.dpos = c.dpos;
    ia.val = c.val;
    ia.panel = mg->panel;
    ia.ainv = mg->ainv;
    const int ctas = std::min(c.n, kInvCtas), per = (c.n + ctas - 1) / ctas;
    for (int q = 0; q <= kMgClusterMax; ++q) ia.split[q] = std::min(c.n, q * per);
    const int smem = (int)sizeof(float) * (6 * per + 6) * mg->nd;
    // the same value from every thread: a smaller one would take another context's launch its memory
    BT_CUDA(cudaFuncSetAttribute(k_mg_dense_inv, cudaFuncAttributeMaxDynamicSharedMemorySize, kInvSmem));
    cudaLaunchAttribute at[1];
    cudaLaunchConfig_t cfg = cluster_config(ctx, ctas, kInvThreads, smem, at);
    const cudaError_t e = cudaLaunchKernelEx(&cfg, k_mg_dense_inv, ia);
    ctx->launches++;
    if (e != cudaSuccess) return fail(BARTELS_E_DEVICE, std::string("launch k_mg_dense_inv: ") + cudaGetErrorString(e));
  }
  // largest eigenvalue of M A on every smoothed level (power iteration; per
  // segment on the finest level of a packed plan)
  const int nseg = (plan->seg && plan->seg->nseg > 0) ? plan->seg->nseg : 0;
  if (nseg > mg->segn_n) {
    mg->segn_n = 0;
    BT_CHECK(dalloc_n(mg, &mg->segn, 2 * (size_t)nseg));
    mg->segn_n = nseg;
  }
  MgDegrees dg{};
  dg.nlev = L;
  for (int l = 0; l < L; ++l) {
    MgLevel &c = mg->lv[l];
    dg.deg[l] = c.deg;
    const bool smoothed = l + 1 < L || (!mg->dense && !mg->coarse_blockdiag);
    if (!smoothed) continue;
    const int64_t n = (int64_t)c.bs * c.n;
    float *x = c.x, *y = c.x2;
    BT_LAUNCH(ctx, k_mg_hash_fill, grid_n(ctx, n), 256, 0, n, x, 0x9e3779b9u + 7919u * (unsigned)l);
    for (int it = 0; it < kPowerIters; ++it) {
      if (l == 0) {
        BT_CHECK(resid0(ctx, plan, values, nullptr, x, c.r, nullptr));
        if (sm.gl) {
          BT_CHECK(fac_lower(ctx, plan, sm, c.r, c.d, nullptr));
          BT_CHECK(fac_upper(ctx, plan, sm, c.d, nullptr, y, nullptr, nullptr, nullptr, nullptr));
        } else {
          BT_LAUNCH_PDL(ctx, k_mg0_bj, grid_n(ctx, plan->nV), 256, 0, plan->nV, sm.minv, c.r, y, (const float *)nullptr,
                    (const PcgState *)nullptr);
        }
      } else {
        BT_LAUNCH(ctx, k_mgc_MA<kGc>, grid_rows(ctx, c.n, kGc), 256, 0, c.n, c.rp, c.ci, c.val16, c.dinv, x, y);
      }
      if (it == kPowerIters - 2) BT_CHECK(sumsq_into(ctx, mg, n, y, mg->norms + 2 * l));
      if (it == kPowerIters - 1) BT_CHECK(sumsq_into(ctx, mg, n, y, mg->norms + 2 * l + 1));
      if (l == 0 && nseg > 0 && it >= kPowerIters - 2)
        BT_LAUNCH(ctx, k_mg_seg_sumsq, nseg, 256, 0, plan->seg->voff, y,
                  mg->segn + (it == kPowerIters - 1 ? nseg : 0));
      std::swap(x, y);
    }
    if (l == 0 && nseg > 0)
      BT_LAUNCH(ctx, k_mg_seg_lmax, 1, 32, 0, nseg, (const double *)mg->segn, (const double *)(mg->segn + nseg),
                mg->norms);
  }
  BT_LAUNCH(ctx, k_mg_coef, 1, 32, 0, dg, mg->norms, mg->coef);
  return BARTELS_OK;
}

int mg_enqueue_update(bartels_ctx ctx, bartels_mesh_plan plan, const MgSmoother &sm, const float *pa,
                      const float *pb, const float *ap, float *x, float *r, double *part, PcgState *st) {
  MgHierarchy *mg = plan->mg;
  BT_LAUNCH_PDL(ctx, k_mg0_update, grid_n(ctx, plan->nV), 256, 0, plan->nV, pa, pb, ap, x, r, sm.minv, mg->lv[0].x,
            (const float *)mg->coef, part, st);
  return BARTELS_OK;
}

int mg_enqueue_apply(bartels_ctx ctx, bartels_mesh_plan plan, const float *values, const MgSmoother &sm,
                     const float *r, float *z, float *y, double *part, PcgState *st, bool pre_done) {
  MgHierarchy *mg = plan->mg;
  MgLevel &l0 = mg->lv[0];
  const float *c0 = mg->coef;
  const int nV = plan->nV;
  if (sm.gl) {
    BT_CHECK(fac_lower(ctx, plan, sm, r, y, st));
    BT_CHECK(fac_upper(ctx, plan, sm, y, nullptr, l0.x, c0, nullptr, nullptr, st));
  } else if (!pre_done) {
    BT_LAUNCH_PDL(ctx, k_mg0_bj, grid_n(ctx, nV), 256, 0, nV, sm.minv, r, l0.x, c0, st);
  }
  BT_CHECK(resid0(ctx, plan, values, r, l0.x, l0.r, st));
  bool first_done = false;
  BT_CHECK(restrict_into<3>(ctx, mg, l0, l0.r, 1, st, &first_done));
  BT_CHECK(enqueue_coarse(ctx, mg, 1, first_done, st));
  BT_LAUNCH_PDL(ctx, k_mg_prolong<3>, grid_n(ctx, nV), 256, 0, nV, l0.agg, l0.Q, level_result(mg, 1), l0.x, st);
  if (sm.gl) {
    BT_CHECK(resid0(ctx, plan, values, r, l0.x, l0.r, st));
    BT_CHECK(fac_lower(ctx, plan, sm, l0.r, y, st));
    BT_CHECK(fac_upper(ctx, plan, sm, y, l0.x, z, c0, r, part, st));
  } else {
    if (mg->a16) {
      const SellView sv = plan->sell->view();
      const int S = sell_split(ctx, sv.nslices), g = sell_grid(ctx, sv.nslices, S);
      const uint2 *a16 = mg->a16;
      if (S == 1)
        BT_LAUNCH_PDL(ctx, k_mg0_post_bj_sell<1>, g, 256, 0, sv, a16, sm.minv, r, l0.x, z, plan->pinned, c0, part, st);
      else if (S == 2)
        BT_LAUNCH_PDL(ctx, k_mg0_post_bj_sell<2>, g, 256, 0, sv, a16, sm.minv, r, l0.x, z, plan->pinned, c0, part, st);
      else
        BT_LAUNCH_PDL(ctx, k_mg0_post_bj_sell<4>, g, 256, 0, sv, a16, sm.minv, r, l0.x, z, plan->pinned, c0, part, st);
    } else {
      const int G = plan_lanes_spmv(ctx, plan);
      const int g = grid_rows(ctx, nV, G);
      BT_MG_G(G, BT_LAUNCH_PDL(ctx, k_mg0_post_bj<GL>, g, 256, 0, nV, plan->brp, plan->bcol, values, sm.minv, r, l0.x, z,
                               plan->pinned, c0, part, st));
    }
  }
  return BARTELS_OK;
}

int mg_apply_once(bartels_ctx ctx, bartels_mesh_plan plan, const float *values, const MgSmoother &sm, const float *r,
                  float *z) {
  MgHierarchy *mg = plan->mg;
  if (!mg->st_once) {
    BT_CHECK(dalloc_n(mg, &mg->st_once, 1));
    BT_CUDA(cudaMemsetAsync(mg->st_once, 0, sizeof(PcgState), ctx->stream));
  }
  BT_CHECK(mg_enqueue_apply(ctx, plan, values, sm, r, z, mg->lv[0].d, mg->part, mg->st_once, false));
  BT_CUDA(cudaStreamSynchronize(ctx->stream));
  return BARTELS_OK;
}

}  // namespace bartels

// Block-Jacobi PCG of a small system as one thread-block cluster launch.
//
// On a system of ten thousand unknowns an iteration of the general loop is three
// dependent kernels of 4 - 40 CTAs, ~19 us of launches and cross-kernel
// latencies around ~1 us of work. Here a whole inner solve is one kernel of a
// 16-CTA cluster: the matrix, the direction and the CTA's own vectors stay in
// shared memory, and an iteration costs three cluster barriers (direction
// published, p.Ap reduced, r.z and r.r reduced) and one pass over shared memory.
//
// Layout: groups of 32 consecutive rows, entry j of the group's rows stored
// together ([group][j][lane], padded to the group's longest row), one lane per
// row. Consecutive rows of a mesh's matrix have neighbouring columns, so the
// lanes' gathers from the staged direction hit different banks. Entries past the
// jcap that fit shared memory are read from L2, also contiguously.
#include <algorithm>
#include <climits>
#include <vector>

#include "pcg_small.cuh"

namespace bartels {

namespace {
constexpr int kCtas = 16, kMaxThreads = 1024;
constexpr int kMaxN = kSmallMaxN;
constexpr int64_t kMaxEntries = 2 << 20;    // past this the cluster's L2 bandwidth loses to the whole GPU
constexpr int kSmemBytes = 225 * 1024;       // beside the static arrays
}  // namespace

bool pcg_small_plan(int n, const int *row_ptr, PcgSmall &s, std::vector<int> &off) {
  s = PcgSmall();
  if (n < 1 || n > kMaxN) return false;
  s.n = n;
  // rows per CTA: whole groups (32) of whole vertices (3)
  const int per = (n + kCtas - 1) / kCtas;
  s.rows = (per + 95) / 96 * 96;
  s.groups = (n + 31) / 32;
  off.assign(s.groups + 1, 0);
  int longest = 0;
  for (int g = 0; g < s.groups; ++g) {
    int len = 0;
    for (int i = 32 * g; i < std::min(n, 32 * g + 32); ++i) len = std::max(len, row_ptr[i + 1] - row_ptr[i]);
    longest = std::max(longest, len);
    const int64_t next = (int64_t)off[g] + len;
    if (32 * next > kMaxEntries) return false;
    off[g + 1] = (int)next;
  }
  s.entries = 32ll * off[s.groups];
  const int fixed = 4 * ((n + 3) & ~3) + s.rows * 28;  // p; x, r, z, p, Ap and the inverse blocks of the own rows
  s.jcap = std::min(longest, (kSmemBytes - fixed) / (6 * s.rows));
  if (s.jcap < 0) return false;
  s.smem = fixed + 6 * s.rows * s.jcap;
  return true;
}

static size_t up256(size_t b) { return (b + 255) & ~size_t(255); }
size_t pcg_small_bytes(const PcgSmall &s) {
  return up256(4 * ((size_t)s.groups + 1)) + up256(4 * (size_t)s.entries + 4) + up256(2 * (size_t)s.entries + 4);
}

// one warp per group, one lane per row
__global__ void __launch_bounds__(256)
k_small_fill(int n, int groups, const int *__restrict__ off, const int *__restrict__ rp, const int *__restrict__ ci,
             const float *__restrict__ val, const unsigned char *__restrict__ pinned, float *__restrict__ oval,
             unsigned short *__restrict__ ocol) {
  const int lane = threadIdx.x & 31;
  for (int g = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; g < groups; g += (gridDim.x * blockDim.x) >> 5) {
    const int i = 32 * g + lane;
    int k = 0, k1 = 0;
    if (i < n && !(pinned && pinned[i / 3])) {
      k = rp[i];
      k1 = rp[i + 1];
    }
    for (int j = off[g]; j < off[g + 1]; ++j, ++k) {
      oval[32ll * j + lane] = k < k1 ? val[k] : 0.f;
      ocol[32ll * j + lane] = (unsigned short)(k < k1 ? ci[k] : min(i, n - 1));
    }
  }
}

__device__ __forceinline__ unsigned small_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// (the aligned forms want the warp's lanes together, which a loop before may have parted)
__device__ __forceinline__ void small_arrive() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void small_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ void small_barrier() {
  small_arrive();
  small_wait();
}

// Sums across warps and CTAs are unevaluated float pairs h + l (Knuth's two-sum,
// with the low parts added up): off by ~2^-46 of the sum, or by the spacing of the
// smallest floats (1.4e-45 a step), where the FP32 partials that they add are off by
// 2^-24; at a fraction of the latency of this GPU's FP64 adds (a tree of nine took
// ~2,500 cycles). That holds while the sums stay well inside the float range; r.z
// and p.Ap scale with the matrix too, so the solve watches them: one that leaves the
// range ends as kSmallRange, for the general loop, whose sums are FP64.
__device__ __forceinline__ float2 pair_add(float2 a, float2 b) {
  const float s = __fadd_rn(a.x, b.x), t = __fsub_rn(s, a.x);
  const float e = __fadd_rn(__fsub_rn(a.x, __fsub_rn(s, t)), __fsub_rn(b.x, t));
  const float l = __fadd_rn(__fadd_rn(a.y, b.y), e);
  const float h = __fadd_rn(s, l);
  return make_float2(h, __fadd_rn(__fsub_rn(s, h), l));
}
template <int N>
__device__ __forceinline__ float2 pair_reduce(float2 v) {
#pragma unroll
  for (int o = N / 2; o > 0; o >>= 1) {
    // the lower lane's value first, so that both lanes form the same sum
    const float2 w = make_float2(__shfl_xor_sync(0xffffffffu, v.x, o), __shfl_xor_sync(0xffffffffu, v.y, o));
    v = (threadIdx.x & o) ? pair_add(w, v) : pair_add(v, w);
  }
  return v;
}
// ~40 steps of 1.4e-45 stay below 2^-24 of the sum, and no partial sum overflows; NaN is out
__device__ __forceinline__ bool small_in_range(float2 a) { return fabsf(a.x) > 1e-36f && fabsf(a.x) < 1e36f; }
__device__ __forceinline__ double pair_value(float2 a) { return (double)a.x + (double)a.y; }
// a / b rounded to FP32 (one correction of the FP32 quotient)
__device__ __forceinline__ float pair_div(float2 a, float2 b) {
  const float q = a.x / b.x;
  const float r = __fadd_rn(__fmaf_rn(-q, b.x, a.x), __fmaf_rn(-q, b.y, a.y));
  const float c = r / b.x;
  return isfinite(c) ? q + c : q;
}

// Sum over the cluster of one FP32 partial per thread (two with W = 2): FP32
// within a warp, float pairs across warps and CTAs, in a fixed order, the same
// bits in every CTA. slot: W x kCtas pairs. Ends in a cluster barrier; the sums
// are left to warp 0's lanes.
template <int W>
__device__ __forceinline__ void small_reduce(float a, float b, float (*warps)[32], float2 *slot, unsigned rank,
                                             float2 out[W]) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  a = warp_sumf(a);
  if (W > 1) b = warp_sumf(b);
  if (lane == 0) {
    warps[0][w] = a;
    if (W > 1) warps[1][w] = b;
  }
  __syncthreads();
  if (w == 0) {
#pragma unroll
    for (int q = 0; q < W; ++q) {
      const float2 s = pair_reduce<32>(make_float2(32 * lane < blockDim.x ? warps[q][lane] : 0.f, 0.f));
      if (lane < kCtas) {
        unsigned ad;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
                     : "=r"(ad)
                     : "r"((unsigned)__cvta_generic_to_shared(slot + q * kCtas + rank)), "r"(lane));
        asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(ad), "f"(s.x), "f"(s.y) : "memory");
      }
    }
  }
  small_barrier();
  if (w == 0) {
#pragma unroll
    for (int q = 0; q < W; ++q) out[q] = pair_reduce<kCtas>(slot[q * kCtas + (lane & (kCtas - 1))]);
  }
}

__global__ void __launch_bounds__(kMaxThreads, 1)
k_pcg_small(PcgSmall m, const float *__restrict__ rres, const float *__restrict__ minv, float *__restrict__ x,
            float *__restrict__ p, PcgState *__restrict__ st, double inner_rel2, double abs_tol2, int max_it, int cont) {
  extern __shared__ __align__(16) char sm[];
  __shared__ float s_warps[2][32];
  __shared__ __align__(8) float2 s_pap[kCtas], s_rz[2 * kCtas];
  // A CTA's shared memory may be written by the others only once it is known to
  // run: all arrive here and wait before the first reduction. Staging lies between.
  small_arrive();
  const unsigned rank = small_rank();
  const int n = m.n, r0 = rank * m.rows, nr = max(0, min(m.rows, n - r0)), nv = (nr + 2) / 3;
  float *sp = reinterpret_cast<float *>(sm);           // the whole direction
  float *xs = sp + ((n + 3) & ~3), *rs = xs + m.rows, *zs = rs + m.rows, *ps = zs + m.rows, *as = ps + m.rows;
  float *mi = as + m.rows;                             // 6 per vertex: 2 per row
  float *sv = mi + 2 * m.rows;                         // staged values, then columns
  unsigned short *sc = reinterpret_cast<unsigned short *>(sv + (size_t)m.jcap * m.rows);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const int g0 = r0 / 32, ng = (nr + 31) / 32;
  __shared__ int s_off[kMaxN / kCtas / 32 + 8];
  for (int g = threadIdx.x; g <= ng; g += blockDim.x) s_off[g] = m.off[min(g0 + g, m.groups)];
  // stage the matrix (a group's entries are contiguous), the inverse blocks and the own rows
  __syncthreads();
  for (int g = warp; g < ng; g += nwarps) {
    const int o = s_off[g], len = min(s_off[g + 1] - o, m.jcap);
    const unsigned dv = (unsigned)__cvta_generic_to_shared(sv + g * m.jcap * 32),
                   dc = (unsigned)__cvta_generic_to_shared(sc + g * m.jcap * 32);
    const char *pv = reinterpret_cast<const char *>(m.val + 32ll * o);
    const char *pc = reinterpret_cast<const char *>(m.col + 32ll * o);
    for (int e = lane; e < 8 * len; e += 32)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dv + 16 * e), "l"(pv + 16ll * e) : "memory");
    for (int e = lane; e < 4 * len; e += 32)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dc + 16 * e), "l"(pc + 16ll * e) : "memory");
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
  for (int i = threadIdx.x; i < 6 * nv; i += blockDim.x) mi[i] = __ldcg(minv + 2ll * r0 + i);
  for (int i = threadIdx.x; i < nr; i += blockDim.x) {
    rs[i] = __ldcg(rres + r0 + i);
    xs[i] = 0.f;
    ps[i] = cont ? __ldcg(p + r0 + i) : 0.f;
    as[i] = 0.f;
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  small_wait();
  // x += alpha p, r -= alpha Ap and z = M^-1 r of the own vertices (a last vertex may have fewer than 3
  // rows), partials of r.z and r.r
  auto update = [&](float alpha, float &arz, float &arr) {
    arz = arr = 0.f;
    for (int v = threadIdx.x; v < nv; v += blockDim.x) {
      float rv[3], zv[3];
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const int i = 3 * v + k;
        rv[k] = 0.f;
        if (i < nr) {
          xs[i] += alpha * ps[i];
          rv[k] = rs[i] - alpha * as[i];
          rs[i] = rv[k];
        }
      }
      apply_minv(mi, v, rv, zv);
#pragma unroll
      for (int k = 0; k < 3; ++k)
        if (3 * v + k < nr) {
          zs[3 * v + k] = zv[k];
          arz += rv[k] * zv[k];
          arr += rv[k] * rv[k];
        }
    }
  };
  // Scalars: the sums live in warp 0 (the same bits in every CTA), the ones
  // that all threads use in shared memory.
  __shared__ float s_alpha, s_beta;
  __shared__ int s_done;
  float arz, arr;
  update(0.f, arz, arr);
  float2 d2[2], rz = make_float2(0.f, 0.f), pap = rz;
  double rr = 0.0, rr0 = 0.0, tol2 = 0.0;
  const double st_rz = st->rz;
  const float st_beta = st->beta;
  int it = cont ? st->it : 0;
  const int last = it + max_it;
  small_reduce<2>(arz, arr, s_warps, s_rz, rank, d2);
  if (warp == 0) {
    // as k_pcg_init: beta against the replaced residual when the direction continues
    const double rz_old = (cont && st_beta > 0.f) ? st_rz / (double)st_beta : 0.0;
    rz = d2[0];
    rr = rr0 = pair_value(d2[1]);
    tol2 = fmax(inner_rel2 * rr, abs_tol2);
    if (lane == 0) {
      s_alpha = 0.f;
      s_beta = (rz_old > 0.0 && rz_old < HUGE_VAL) ? (float)(pair_value(rz) / rz_old) : 0.f;
      s_done = rr <= tol2 || max_it <= 0 ? 1 : small_in_range(d2[0]) && small_in_range(d2[1]) ? 0 : kSmallRange;
    }
  }
  __syncthreads();
  // every CTA holds the same scalars, bit for bit, so all leave the loop together
  while (!s_done) {
    const float beta = s_beta;
    for (int i = threadIdx.x; i < nr; i += blockDim.x) {
      const float t = zs[i] + beta * ps[i];
      ps[i] = t;
      p[r0 + i] = t;
    }
    small_barrier();
    for (int i = threadIdx.x; i < n / 4; i += blockDim.x)
      reinterpret_cast<float4 *>(sp)[i] = __ldcg(reinterpret_cast<const float4 *>(p) + i);
    for (int i = n / 4 * 4 + threadIdx.x; i < n; i += blockDim.x) sp[i] = __ldcg(p + i);
    __syncthreads();
    float acc = 0.f;
    for (int g = warp; g < ng; g += nwarps) {
      const int o = s_off[g], len = s_off[g + 1] - o, ls = min(len, m.jcap);
      float s = 0.f;
      const float *v = sv + g * m.jcap * 32 + lane;
      const unsigned short *c = sc + g * m.jcap * 32 + lane;
#pragma unroll 5
      for (int j = 0; j < ls; ++j) s += v[32 * j] * sp[c[32 * j]];
#pragma unroll 4
      for (int j = ls; j < len; ++j)
        s += __ldg(m.val + 32ll * (o + j) + lane) * sp[__ldg(m.col + 32ll * (o + j) + lane)];
      const int i = 32 * g + lane;
      if (i < nr) {
        as[i] = s;
        acc += ps[i] * s;
      }
    }
    float2 d1[1];
    small_reduce<1>(acc, 0.f, s_warps, s_pap, rank, d1);
    if (warp == 0) {
      pap = d1[0];
      if (lane == 0) {
        s_alpha = pair_div(rz, pap);
        if (!small_in_range(pap)) s_done = kSmallRange;
      }
    }
    __syncthreads();
    update(s_alpha, arz, arr);
    small_reduce<2>(arz, arr, s_warps, s_rz, rank, d2);
    ++it;
    if (warp == 0) {
      rr = pair_value(d2[1]);
      if (lane == 0) {
        s_beta = pair_div(d2[0], rz);
        if (!s_done)
          s_done = rr <= tol2 || it >= last ? 1 : small_in_range(d2[0]) && small_in_range(d2[1]) ? 0 : kSmallRange;
      }
      rz = d2[0];
    }
    __syncthreads();
  }
  const float alpha = s_alpha, beta = s_beta;
  for (int i = threadIdx.x; i < nr; i += blockDim.x) x[r0 + i] = xs[i];
  if (rank == 0 && threadIdx.x == 0) {
    st->rz = pair_value(rz);
    st->rr = rr;
    st->rr0 = rr0;
    st->tol2 = tol2;
    st->pap = pair_value(pap);
    st->alpha = alpha;
    st->beta = beta;
    st->it = it;
    st->max_it = last;
    st->done = s_done;
  }
}

int pcg_small_fill(bartels_ctx ctx, PcgSmall &s, char *base, const std::vector<int> &off, const int *rp, const int *ci,
                   const float *val, const unsigned char *pinned) {
  s.off = reinterpret_cast<int *>(base);
  base += up256(4 * ((size_t)s.groups + 1));
  s.val = reinterpret_cast<float *>(base);
  base += up256(4 * (size_t)s.entries + 4);
  s.col = reinterpret_cast<unsigned short *>(base);
  BT_CUDA(cudaMemcpyAsync(s.off, off.data(), sizeof(int) * off.size(), cudaMemcpyHostToDevice, ctx->stream));
  BT_LAUNCH(ctx, k_small_fill, (s.groups + 7) / 8, 256, 0, s.n, s.groups, (const int *)s.off, rp, ci, val, pinned,
            s.val, s.col);
  return BARTELS_OK;
}

// launch configuration of one solve's cluster
static cudaLaunchConfig_t small_config(bartels_ctx ctx, int threads, int smem, cudaLaunchAttribute *at) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(kCtas);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = ctx->stream;
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = kCtas;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cfg;
}

bool pcg_small_hosted(bartels_ctx ctx) {
  if (ctx->small_hosted < 0) {
    cudaLaunchAttribute at[1];
    const cudaLaunchConfig_t cfg = small_config(ctx, kMaxThreads, kSmemBytes, at);
    int fit = 0;
    const bool ok = cudaFuncSetAttribute(k_pcg_small, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes) ==
                        cudaSuccess &&
                    cudaFuncSetAttribute(k_pcg_small, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) ==
                        cudaSuccess &&
                    cudaOccupancyMaxActiveClusters(&fit, k_pcg_small, &cfg) == cudaSuccess;
    if (!ok) cudaGetLastError();
    ctx->small_hosted = ok && fit >= 1;
  }
  return ctx->small_hosted != 0;
}

int pcg_small_run(bartels_ctx ctx, const PcgSmall &s, const float *rres, const float *minv, float *x, float *p,
                  PcgState *st, double inner_rel2, double abs_tol2, int max_it, int cont) {
  cudaLaunchAttribute at[1];
  // a warp per group of the CTA's rows: barriers cost less with fewer threads
  const cudaLaunchConfig_t cfg = small_config(ctx, std::min(kMaxThreads, std::max(256, s.rows)), s.smem, at);
  const cudaError_t e = cudaLaunchKernelEx(&cfg, k_pcg_small, s, rres, minv, x, p, st, inner_rel2, abs_tol2, max_it, cont);
  ctx->launches++;
  if (e != cudaSuccess) return fail(BARTELS_E_DEVICE, std::string("launch k_pcg_small: ") + cudaGetErrorString(e));
  return BARTELS_OK;
}

}  // namespace bartels

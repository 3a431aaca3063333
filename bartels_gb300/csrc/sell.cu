// Building and filling the sliced-ELL layout (sell.cuh).
#include <algorithm>
#include <memory>
#include <vector>

#include "lpcg_internal.cuh"
#include "sell.cuh"

namespace bartels {

constexpr int kSellWindow = 256;  // rows ordered by length within windows of this many

// start and number of row v's blocks in a layout
__device__ __forceinline__ int2 sell_range(int part, const int *brp, const int *diag_pos, int v) {
  const int rb = brp[v], nb = brp[v + 1] - rb;
  if (part == kSellFull) return make_int2(rb, nb);
  const int d = diag_pos[v];
  return part == kSellLower ? make_int2(rb, d + 1) : make_int2(rb + d, nb - d);
}

// One CTA per window: rank of each row by descending block count (ties keep
// the vertex order), and the groups of the window's slices.
__global__ void __launch_bounds__(kSellWindow)
k_sell_order(int nV, int part, const int *__restrict__ brp, const int *__restrict__ diag_pos, int *__restrict__ row,
             int *__restrict__ groups) {
  __shared__ int cnt[kSellWindow];
  const int v = blockIdx.x * kSellWindow + threadIdx.x;
  const int c = v < nV ? sell_range(part, brp, diag_pos, v).y : -1;
  cnt[threadIdx.x] = c;
  __syncthreads();
  int rank = 0;
  for (int t = 0; t < kSellWindow; ++t) rank += cnt[t] > c || (cnt[t] == c && t < (int)threadIdx.x);
  row[blockIdx.x * kSellWindow + rank] = v < nV ? v : -1;
  if (rank % 32 == 0) groups[(blockIdx.x * kSellWindow + rank) / 32] = c > 0 ? (c + 3) / 4 : 0;
}

__global__ void __launch_bounds__(256)
k_sell_cols(SellView sv, int part, const int *__restrict__ brp, const int *__restrict__ diag_pos,
            const int *__restrict__ bcol, int4 *__restrict__ col) {
  const int lane = threadIdx.x & 31, nw = (gridDim.x * blockDim.x) >> 5;
  for (int s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; s < sv.nslices; s += nw) {
    const int v = sv.row[32 * s + lane];
    const int2 rg = v >= 0 ? sell_range(part, brp, diag_pos, v) : make_int2(0, 0);
    const int rb = rg.x, nb = rg.y, own = v >= 0 ? 3 * v : 0;
    for (int g = sv.off[s]; g < sv.off[s + 1]; ++g) {
      const int j = 4 * (g - sv.off[s]);
      int c[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) c[q] = j + q < nb ? 3 * bcol[rb + j + q] : own;
      col[32ll * g + lane] = make_int4(c[0], c[1], c[2], c[3]);
    }
  }
}

// Fill: one CTA of 4 warps per slice, 4 groups (16 blocks) at a time. The rows'
// entries are staged in shared memory with contiguous loads (a row's scalar
// rows lie one after the other), then each warp writes one group.
constexpr int kFillBlocks = 16, kFillStride = 9 * kFillBlocks + 1;
template <bool BF16>
__global__ void __launch_bounds__(128)
k_sell_fill(SellView sv, const int *__restrict__ brp, const int *__restrict__ bcol, const float *__restrict__ val,
            const int *__restrict__ rev, void *__restrict__ out) {
  __shared__ float sh[32 * kFillStride];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int s = blockIdx.x; s < sv.nslices; s += gridDim.x) {
    const int g0 = sv.off[s], ng = sv.off[s + 1] - g0;
    const int v = sv.row[32 * s + lane];
    const int rb = v >= 0 ? brp[v] : 0, nb = v >= 0 ? brp[v + 1] - rb : 0;
    for (int c = 0; c < ng; c += kFillBlocks / 4) {
      __syncthreads();
      for (int i = warp; i < 32; i += 4) {
        const int rbi = __shfl_sync(0xffffffffu, rb, i), nbi = __shfl_sync(0xffffffffu, nb, i);
        const int e0 = 12 * c, e1 = min(3 * nbi, e0 + 3 * kFillBlocks);  // scalar columns of this chunk
        for (int r = 0; r < 3; ++r)
          for (int e = e0 + lane; e < e1; e += 32)
            sh[i * kFillStride + 3 * kFillBlocks * r + e - e0] = __ldg(val + 9ll * rbi + 3ll * r * nbi + e);
      }
      __syncthreads();
      const int g = c + warp;
      if (g < ng) {
        float a[9][4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int j = 4 * g + q;
#pragma unroll
          for (int r = 0; r < 3; ++r)
#pragma unroll
            for (int k = 0; k < 3; ++k)
              a[3 * r + k][q] = j < nb ? sh[lane * kFillStride + 3 * kFillBlocks * r + 3 * (j - 4 * c) + k] : 0.f;
          if (BF16 && j < nb) {
            const int w = __ldg(bcol + rb + j);
            if (w < v) {
              const int rbw = __ldg(brp + w), nbw = __ldg(brp + w + 1) - rbw;
              const float *t = val + 9ll * rbw + 3 * (__ldg(rev + rb + j) - rbw);
#pragma unroll
              for (int r = 0; r < 3; ++r)
#pragma unroll
                for (int k = 0; k < 3; ++k) a[3 * r + k][q] = __ldg(t + 3ll * k * nbw + r);
            } else if (w == v) {
              const float o1 = 0.5f * (a[1][q] + a[3][q]), o2 = 0.5f * (a[2][q] + a[6][q]),
                          o5 = 0.5f * (a[5][q] + a[7][q]);
              a[1][q] = a[3][q] = o1;
              a[2][q] = a[6][q] = o2;
              a[5][q] = a[7][q] = o5;
            }
          }
        }
        const int64_t o = 288ll * (g0 + g) + lane;
#pragma unroll
        for (int e = 0; e < 9; ++e) {
          if (BF16) {
            const __nv_bfloat162 lo = __floats2bfloat162_rn(a[e][0], a[e][1]),
                                 hi = __floats2bfloat162_rn(a[e][2], a[e][3]);
            static_cast<uint2 *>(out)[o + 32 * e] =
                make_uint2(*reinterpret_cast<const unsigned *>(&lo), *reinterpret_cast<const unsigned *>(&hi));
          } else {
            static_cast<float4 *>(out)[o + 32 * e] = make_float4(a[e][0], a[e][1], a[e][2], a[e][3]);
          }
        }
      }
    }
  }
}

// A warp per slice: lane l copies its row's groups, three 8-byte loads per scalar row.
__global__ void __launch_bounds__(256)
k_sell_fill_factor(SellView sv, int part, const int *__restrict__ brp, const int *__restrict__ diag_pos,
                   const int4 *__restrict__ meta, const __nv_bfloat16 *__restrict__ g, uint2 *__restrict__ out) {
  const int lane = threadIdx.x & 31, nw = (gridDim.x * blockDim.x) >> 5;
  for (int s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; s < sv.nslices; s += nw) {
    const int v = sv.row[32 * s + lane];
    const int nb = v >= 0 ? sell_range(part, brp, diag_pos, v).y : 0, rsp = padded_row(nb);
    const int4 m = v >= 0 ? __ldg(meta + v) : make_int4(0, 0, 0, 0);
    const __nv_bfloat16 *row = g + (part == kSellLower ? m.y : m.z);
    const int g0 = sv.off[s], ng = sv.off[s + 1] - g0;
    for (int c = 0; c < ng; ++c) {
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        unsigned w[6];  // 12 entries: blocks 4c .. 4c + 3, three columns each
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          const int e = 12 * c + 4 * q;
          const uint2 t = e < rsp ? __ldg(reinterpret_cast<const uint2 *>(row + (int64_t)r * rsp + e)) : make_uint2(0, 0);
          w[2 * q] = t.x;
          w[2 * q + 1] = t.y;
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          unsigned h[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int e = 3 * j + k;
            h[j] = 4 * c + j < nb ? (w[e / 2] >> (16 * (e & 1))) & 0xFFFFu : 0u;
          }
          out[288ll * (g0 + c) + 32 * (3 * r + k) + lane] = make_uint2(h[0] | h[1] << 16, h[2] | h[3] << 16);
        }
      }
    }
  }
}

SellPattern::~SellPattern() {
  if (off) cudaFree(off);
  if (row) cudaFree(row);
  if (col) cudaFree(col);
}

int plan_sell(bartels_mesh_plan plan, SellPattern **out, int part) {
  SellPattern *&slot = part == kSellFull ? plan->sell : plan->sell_factor[part - 1];
  if (!slot) {
    bartels_ctx ctx = plan->ctx;
    std::unique_ptr<SellPattern> p(new SellPattern());  // the plan's once it is complete
    p->part = part;
    const int nwin = (plan->nV + kSellWindow - 1) / kSellWindow;
    p->nslices = nwin * (kSellWindow / 32);
    BT_CUDA(dev_malloc(&p->row, sizeof(int) * 32 * (size_t)p->nslices));
    BT_CUDA(dev_malloc(&p->off, sizeof(int) * ((size_t)p->nslices + 1)));
    BT_LAUNCH(ctx, k_sell_order, nwin, kSellWindow, 0, plan->nV, part, plan->brp, plan->diag_pos, p->row,
              p->off);
    std::vector<int> g(p->nslices + 1, 0);
    StreamWait wait{ctx->stream};  // the copies below read and write g
    BT_CUDA(cudaMemcpyAsync(g.data() + 1, p->off, sizeof(int) * p->nslices, cudaMemcpyDeviceToHost, ctx->stream));
    BT_CUDA(cudaStreamSynchronize(ctx->stream));
    for (int s = 0; s < p->nslices; ++s) g[s + 1] += g[s];
    while (p->nslices > 0 && g[p->nslices] == g[p->nslices - 1]) p->nslices--;  // slices past the last vertex
    p->groups = g[p->nslices];
    BT_CUDA(cudaMemcpyAsync(p->off, g.data(), sizeof(int) * (p->nslices + 1), cudaMemcpyHostToDevice, ctx->stream));
    BT_CUDA(dev_malloc(&p->col, sizeof(int4) * 32 * (size_t)std::max<int64_t>(p->groups, 1)));
    BT_LAUNCH(ctx, k_sell_cols, sell_grid(ctx, p->nslices, 1), 256, 0, p->view(), part, plan->brp,
              plan->diag_pos, plan->bcol, p->col);
    BT_CUDA(cudaStreamSynchronize(ctx->stream));
    wait.armed = false;
    slot = p.release();
  }
  *out = slot;
  return BARTELS_OK;
}

int sell_fill_f32(bartels_ctx ctx, bartels_mesh_plan plan, const float *values, float4 *out) {
  const SellView sv = plan->sell->view();
  const int g = std::max(1, std::min(sv.nslices, ctx->num_sms * 16));
  BT_LAUNCH(ctx, k_sell_fill<false>, g, 128, 0, sv, plan->brp, plan->bcol, values, (const int *)nullptr, (void *)out);
  return BARTELS_OK;
}

int sell_fill_bf16(bartels_ctx ctx, bartels_mesh_plan plan, const float *values, const int *rev, uint2 *out) {
  const SellView sv = plan->sell->view();
  const int g = std::max(1, std::min(sv.nslices, ctx->num_sms * 16));
  BT_LAUNCH(ctx, k_sell_fill<true>, g, 128, 0, sv, plan->brp, plan->bcol, values, rev, (void *)out);
  return BARTELS_OK;
}

int sell_fill_factor(bartels_ctx ctx, bartels_mesh_plan plan, int part, const int4 *meta, const __nv_bfloat16 *g,
                     uint2 *out) {
  const SellView sv = plan->sell_factor[part - 1]->view();
  BT_LAUNCH(ctx, k_sell_fill_factor, sell_grid(ctx, sv.nslices, 1), 256, 0, sv, part, plan->brp, plan->diag_pos, meta,
            g, out);
  return BARTELS_OK;
}

// Warps per slice: one while there are two rounds of warps or so, else two or four,
// so that every SM has enough loads in flight. Whole solves with 1 / 2 / 4: 489
// slices (Newton, 15.6k vertices) 12.7 / 11.7 / 11.0 ms, 1,583 slices 7.6 / 7.1 / 7.3,
// 2,154 slices (block-Jacobi) 23.6 / 21.5 / 26.9, 3,677 slices 10.2 / 11.2 / 10.9.
int sell_split(bartels_ctx ctx, int nslices) {
  return nslices >= ctx->num_sms * 16 ? 1 : nslices >= ctx->num_sms * 8 ? 2 : 4;
}

// Five CTAs per SM are what the SpMV's 48 registers let reside: more came in a
// second, thinner round (n = 96 multigrid solve 48.1 ms with eight, 46.2 with five,
// 51.0 with six; n = 80 30.3 / 28.8 / 30.8).
int sell_grid(bartels_ctx ctx, int nslices, int split) {
  const int per = 8 / split;
  return std::max(1, std::min((nslices + per - 1) / per, ctx->num_sms * 5));
}

}  // namespace bartels

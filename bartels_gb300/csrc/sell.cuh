// Sliced-ELL layout of a plan's block rows for the passes that read the whole
// matrix: the PCG SpMV (FP32) and the fine level of the V-cycle (BF16).
//
// A slice is 32 vertex rows, one per lane of a warp; every row holds as many
// 3x3 blocks as the slice's longest, rounded up to whole groups of 4. Rows are
// ordered by length within windows of 256, so that a slice's rows are about
// equally long on any numbering. Per group and lane: the 4 blocks' columns
// (one 16-byte load) and, for each of a block's 9 entries, the 4 blocks' values
// (one 16-byte load in FP32, 8-byte in BF16), so every load of a warp is
// contiguous and a row needs no shuffle. Padding blocks hold zeros and point at
// the row's own vertex.
//
// The rows' scalar-CSR order needs several lanes per row, unaligned values, a
// division per entry and a butterfly per row: at n = 96 the padded-row SpMV
// took 107 us in the PCG loop and the BF16 passes 84 - 94 us, issue-bound at
// 0.77 / 0.60 of the copy bandwidth on their bytes.
#pragma once

#include <cuda_bf16.h>

#include <cstdint>

#include "internal.cuh"
#include "pcg_common.cuh"

namespace bartels {

struct SellView {
  int nslices = 0;
  const int *off = nullptr;   // nslices + 1, in groups
  const int *row = nullptr;   // 32 per slice: vertex, or -1
  const int4 *col = nullptr;  // 32 per group: 3 x the column vertices of the lane's 4 blocks
};

// The blocks of a row that a layout holds: all of them, or the learned factor's lower
// part (columns up to the diagonal) or upper part (from the diagonal on).
enum SellPart { kSellFull = 0, kSellLower = 1, kSellUpper = 2 };

// Storage of one layout, built on first use.
struct SellPattern {
  int part = kSellFull;
  int nslices = 0;
  int64_t groups = 0;
  int *off = nullptr, *row = nullptr;
  int4 *col = nullptr;
  ~SellPattern();
  SellView view() const { return {nslices, off, row, col}; }
};
int plan_sell(bartels_mesh_plan plan, SellPattern **out, int part = kSellFull);
// values (scalar-CSR) into the layout: FP32 (9 groups x 32 float4) as they are
int sell_fill_f32(bartels_ctx ctx, bartels_mesh_plan plan, const float *values, float4 *out);
// BF16, exactly symmetric: block (v, w), w < v, takes the transpose of (w, v), the
// diagonal block its symmetric part; rev[p] is the position of block p's transpose
int sell_fill_bf16(bartels_ctx ctx, bartels_mesh_plan plan, const float *values, const int *rev, uint2 *out);
// the factor's BF16 storage of that part (rows of three scalar rows padded to 4
// entries; off[v].y / .z is a row's offset in the lower / upper storage)
int sell_fill_factor(bartels_ctx ctx, bartels_mesh_plan plan, int part, const int4 *meta, const __nv_bfloat16 *g,
                     uint2 *out);

// Warps per slice: one where the slices fill the GPU; four (each takes every
// fourth group) on small meshes, where a pass is bound by its chain of loads.
int sell_split(bartels_ctx ctx, int nslices);
// CTAs of 256 threads for a pass (8 / split slices each, grid-stride)
int sell_grid(bartels_ctx ctx, int nslices, int split);

__device__ __forceinline__ void sell_values(const float4 *p, float a[4]) {
  const float4 t = __ldcs(p);
  a[0] = t.x; a[1] = t.y; a[2] = t.z; a[3] = t.w;
}
__device__ __forceinline__ void sell_values(const uint2 *p, float a[4]) {
  const uint2 t = __ldcs(p);
  a[0] = __uint_as_float(t.x << 16);
  a[1] = __uint_as_float(t.x & 0xFFFF0000u);
  a[2] = __uint_as_float(t.y << 16);
  a[3] = __uint_as_float(t.y & 0xFFFF0000u);
}

// (A x) of the lane's row of `slice` over the groups part, part + S, ...
// x is read through L2: the previous kernel may have written it while this one
// was already resident (2% slower at n = 96 than letting L1 keep its lines).
template <int S, class VT>
__device__ __forceinline__ void sell_row(const SellView &sv, const VT *__restrict__ val, int slice, int part,
                                         const float *x, float s[3]) {
  const int lane = threadIdx.x & 31;
  s[0] = s[1] = s[2] = 0.f;
  const int g1 = __ldg(sv.off + slice + 1);
#pragma unroll 2
  for (int g = __ldg(sv.off + slice) + part; g < g1; g += S) {
    const int4 c = __ldcs(sv.col + 32ll * g + lane);
    const VT *v = val + 288ll * g + lane;
    const int cc[4] = {c.x, c.y, c.z, c.w};
    float xv[4][3];
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int k = 0; k < 3; ++k) xv[j][k] = __ldcg(x + cc[j] + k);
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        float a[4];
        sell_values(v + 32 * (3 * r + k), a);
#pragma unroll
        for (int j = 0; j < 4; ++j) s[r] += a[j] * xv[j][k];
      }
  }
}

// Loop over the slices of a pass for a CTA of 256 threads (8 warps, S per
// slice). fn(v, s) runs once per row v (>= 0) with the row's product s.
template <int S, class VT, class Fn>
__device__ __forceinline__ void sell_pass(const SellView &sv, const VT *__restrict__ val, const float *x, Fn &&fn) {
  constexpr int kPer = 8 / S;  // slices per CTA step
  __shared__ float red[S > 1 ? 8 * 32 * 3 : 1];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, part = warp % S;
  for (int s0 = blockIdx.x * kPer; s0 < sv.nslices; s0 += gridDim.x * kPer) {
    const int slice = s0 + warp / S;
    float s[3] = {0.f, 0.f, 0.f};
    if (slice < sv.nslices) sell_row<S>(sv, val, slice, part, x, s);
    if constexpr (S > 1) {
#pragma unroll
      for (int k = 0; k < 3; ++k) red[(3 * warp + k) * 32 + lane] = s[k];
      __syncthreads();
      if (part == 0)
#pragma unroll
        for (int q = 1; q < S; ++q)
#pragma unroll
          for (int k = 0; k < 3; ++k) s[k] += red[(3 * (warp + q) + k) * 32 + lane];
    }
    if (slice < sv.nslices && part == 0) {
      const int v = __ldg(sv.row + 32ll * slice + lane);
      if (v >= 0) fn(v, s);
    }
    if constexpr (S > 1) __syncthreads();
  }
}

}  // namespace bartels

// split_tiles.cuh -- the BF16 split of one unit of rows or one tile, shared by
// the single-problem (split.cu) and grouped (grouped.cu) pre-pass kernels.
#pragma once
#include "split.cuh"
#include "split_device.cuh"

namespace cucosma {

// Loads v[0..7] = src[c .. c+7] (zero past cols); c % 8 == 0 and src rows
// 16-byte aligned, so the full case is two 16-byte loads.
__device__ __forceinline__ void load8(const float* __restrict__ src, int c, int cols, float (&v)[8]) {
  if (c + 8 <= cols) {
    const float4 a = *reinterpret_cast<const float4*>(src + c);
    const float4 b = *reinterpret_cast<const float4*>(src + c + 4);
    v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
  } else {
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] = c + e < cols ? src[c + e] : 0.f;
  }
}

// NT planes of 8 values: one 16-byte store each.
template <int NT>
__device__ __forceinline__ void store_planes8(__nv_bfloat16* dst, int64_t plane, const float (&v)[8]) {
  uint32_t pk[4][NT];
#pragma unroll
  for (int e = 0; e < 4; ++e) split_bf16x2_n<NT>(v[2 * e], v[2 * e + 1], pk[e]);
#pragma unroll
  for (int i = 0; i < NT; ++i)
    *reinterpret_cast<uint4*>(dst + i * plane) = make_uint4(pk[0][i], pk[1][i], pk[2][i], pk[3][i]);
}

__device__ __forceinline__ float xform_rt(int mode, float v, float y, float scale) {
  switch (mode) {
    case kXformScale: return xform<kXformScale>(v, y, scale);
    case kXformSigmoidGrad: return xform<kXformSigmoidGrad>(v, y, scale);
    case kXformReluGrad: return xform<kXformReluGrad>(v, y, scale);
    default: return v;
  }
}

// Row planes [NT][rows][kpad] of a source in its own layout: one warp per
// unit of up to 2048 columns of a row, lanes over 8-column groups (two
// 16-byte loads, one 16-byte store per plane), two groups in flight.
// Columns cols .. kpad-1 are written as 0 (kpad % 8 == 0).
constexpr int kRowUnit = 256;  // 8-column groups per warp
template <int NT>
__device__ __forceinline__ void split_rows_unit(const SplitJob& j, int64_t unit) {
  const int lane = threadIdx.x & 31;
  const int ng = (int)(j.kpad_r / 8), upr = (ng + kRowUnit - 1) / kRowUnit;
  const int64_t r = unit / upr;
  if (r >= j.rows) return;
  const int g0 = (int)(unit - r * upr) * kRowUnit, g1 = min(ng, g0 + kRowUnit);
  const float* srow = j.src + r * j.ld;
  const float* yrow = j.Y + r * j.ldy;
  __nv_bfloat16* drow = j.out_r + r * j.kpad_r;
  const int64_t plane = (int64_t)j.rows * j.kpad_r;
  constexpr int U = 2;
  for (int g = g0 + lane; g < g1; g += 32 * U) {
    float v[U][8];
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (g + 32 * u < g1) load8(srow, (g + 32 * u) * 8, j.cols, v[u]);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (g + 32 * u >= g1) break;
      const int c = (g + 32 * u) * 8;
      if (j.mode != kXformNone) {
        float y[8];
        if (j.Y != nullptr) {
          load8(yrow, c, j.cols, y);
        } else {
#pragma unroll
          for (int e = 0; e < 8; ++e) y[e] = 0.f;
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) v[u][e] = xform_rt(j.mode, v[u][e], y[e], j.scale);
      }
      store_planes8<NT>(drow + c, plane, v[u]);
    }
  }
}

// One 64 (source rows) x 64 (columns) tile of a source to transposed planes
// [NT][cols][kpad_c] and, for out_r, to row planes as well (the backward
// pass's G, needed in both layouts, is read and formed once).  Loads: 16 lanes
// cover a 256-byte row (float4 each) and write it to shared memory with the
// 16-byte chunk c of row k at c ^ (k / 8); then a lane converts 8 consecutive
// k of one column (8 lanes x 4 columns a warp: no bank conflicts, 128
// contiguous bytes per column and plane).
template <int NT>
__device__ __forceinline__ void split_cols_tile(const SplitJob& j, int tk, int tn, float* tile) {
  const int k0 = tk * 64, n0 = tn * 64;
  const int t = threadIdx.x, tx = t & 15, ty = t >> 4;
  // columns n .. n + 3 of a row (n % 4 == 0, 16-byte rows), zero past cols
  auto load4 = [&](const float* row, int n) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (n + 4 <= j.cols) {
      v = *reinterpret_cast<const float4*>(row + n);
    } else {
      if (n < j.cols) v.x = row[n];
      if (n + 1 < j.cols) v.y = row[n + 1];
      if (n + 2 < j.cols) v.z = row[n + 2];
    }
    return v;
  };
  const int n = n0 + 4 * tx;
  const bool use_y = j.mode != kXformNone && j.Y != nullptr;
  float4 q[4], y[4];
#pragma unroll
  for (int p = 0; p < 4; ++p) {  // every load of the tile in flight at once
    const int k = k0 + ty + 16 * p;
    q[p] = k < j.rows ? load4(j.src + (int64_t)k * j.ld, n) : make_float4(0.f, 0.f, 0.f, 0.f);
    y[p] = use_y && k < j.rows ? load4(j.Y + (int64_t)k * j.ldy, n) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    const int k = k0 + ty + 16 * p;
    if (j.mode != kXformNone) {
      q[p].x = xform_rt(j.mode, q[p].x, y[p].x, j.scale);
      q[p].y = xform_rt(j.mode, q[p].y, y[p].y, j.scale);
      q[p].z = xform_rt(j.mode, q[p].z, y[p].z, j.scale);
      q[p].w = xform_rt(j.mode, q[p].w, y[p].w, j.scale);
    }
    const int i = ty + 16 * p;
    *reinterpret_cast<float4*>(tile + i * 64 + ((tx ^ (i >> 3)) << 2)) = q[p];
    if (j.out_r != nullptr && k < j.rows && n < j.kpad_r) {  // kpad_r % 8 == 0: n + 3 < kpad_r as well
      uint32_t lo[NT], hi[NT];
      split_bf16x2_n<NT>(q[p].x, q[p].y, lo);
      split_bf16x2_n<NT>(q[p].z, q[p].w, hi);
      __nv_bfloat16* dst = j.out_r + (int64_t)k * j.kpad_r + n;
      const int64_t plane = (int64_t)j.rows * j.kpad_r;
#pragma unroll
      for (int i2 = 0; i2 < NT; ++i2) *reinterpret_cast<uint2*>(dst + i2 * plane) = make_uint2(lo[i2], hi[i2]);
    }
  }
  __syncthreads();
  const int lane = t & 31, kq = lane & 7;
  const int64_t plane = (int64_t)j.cols * j.kpad_c;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int nl = (t >> 5) * 8 + h * 4 + (lane >> 3), k = k0 + 8 * kq;
    if (n0 + nl < j.cols && k < j.kpad_c) {  // kpad_c % 8 == 0: k + 7 < kpad_c as well
      float v[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) v[e] = tile[(8 * kq + e) * 64 + (((nl >> 2) ^ kq) << 2) + (nl & 3)];
      store_planes8<NT>(j.out_c + (int64_t)(n0 + nl) * j.kpad_c + k, plane, v);
    }
  }
}

// Tiles tk0 .. tk1 - 1 (64 source rows each) of one 64-column strip to
// transposed planes, as split_cols_tile without a transform: the next tile's
// loads are in flight while one is converted.  For the grouped pre-pass, whose
// blocks first have to find their problem.
template <int NT>
__device__ __forceinline__ void split_cols_strip(const SplitJob& j, int tk0, int tk1, int tn, float* tile) {
  const int n0 = tn * 64, t = threadIdx.x, tx = t & 15, ty = t >> 4, n = n0 + 4 * tx;
  const int lane = t & 31, kq = lane & 7;
  const int64_t plane = (int64_t)j.cols * j.kpad_c;
  float4 q[4];
  auto load = [&](int tk) {
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      const int k = tk * 64 + ty + 16 * p;
      q[p] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (k >= j.rows) continue;
      const float* row = j.src + (int64_t)k * j.ld;
      if (n + 4 <= j.cols) {
        q[p] = *reinterpret_cast<const float4*>(row + n);  // n % 4 == 0, 16-byte rows
      } else {
        if (n < j.cols) q[p].x = row[n];
        if (n + 1 < j.cols) q[p].y = row[n + 1];
        if (n + 2 < j.cols) q[p].z = row[n + 2];
      }
    }
  };
  load(tk0);
  for (int tk = tk0; tk < tk1; ++tk) {
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      const int i = ty + 16 * p;
      *reinterpret_cast<float4*>(tile + i * 64 + ((tx ^ (i >> 3)) << 2)) = q[p];
    }
    __syncthreads();
    if (tk + 1 < tk1) load(tk + 1);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int nl = (t >> 5) * 8 + h * 4 + (lane >> 3), k = tk * 64 + 8 * kq;
      if (n0 + nl < j.cols && k < j.kpad_c) {  // kpad_c % 8 == 0: k + 7 < kpad_c as well
        float v[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) v[e] = tile[(8 * kq + e) * 64 + (((nl >> 2) ^ kq) << 2) + (nl & 3)];
        store_planes8<NT>(j.out_c + (int64_t)(n0 + nl) * j.kpad_c + k, plane, v);
      }
    }
    __syncthreads();  // the next tile overwrites the shared one
  }
}

}  // namespace cucosma

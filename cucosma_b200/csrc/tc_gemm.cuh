// tc_gemm.cuh -- parameters of the tcgen05 precision-path kernel.
#pragma once
#include <cstdint>

#include "common.cuh"

namespace cucosma {

constexpr int kOzakiDefaultSlices = 8;

// Ozaki tile geometry for S slices (stacked form, see tc_kernel.cuh): the B
// slices of a sub-tile of ozaki_sub(S) output columns are stacked along N, so
// one MMA of N = (S - p) * sub columns covers every diagonal that A slice p
// feeds; S * sub <= 256 (the largest MMA N).  ozaki_nsub(S) sub-tiles fill
// the 512 TMEM columns; the tile is 128 x ozaki_bn(S).
constexpr int ozaki_sub(int s) { return s <= 4 ? 64 : (s == 5 ? 48 : (s <= 8 ? 32 : 16)); }
constexpr int ozaki_nsub(int s) { return 512 / (s * ozaki_sub(s)); }
constexpr int ozaki_bn(int s) { return ozaki_nsub(s) * ozaki_sub(s); }

namespace tc {

// One problem of a grouped launch, stored in the workspace.  The tensor maps
// describe this problem's operand planes (they live in global memory; the
// TMA unit reads them there).
struct alignas(64) GroupEntry {
  CUtensorMap tmA, tmB;
  void* C;
  int64_t ldc;
  const int32_t* ea;  // Ozaki exponents of this problem (null for BF16)
  const int32_t* eb;
  int m, n, k, kblocks;
  int tiles_m, tiles_n;
  // operand pre-pass: sources, destination planes, first pre-pass block of
  // this problem for the A rows / B tiles / exponent passes
  const void* A;
  const void* B;
  int64_t lda, ldb, kpad;
  void* planes_a;
  void* planes_b;
  int pre_a_start, pre_b_start, exp_a_start, exp_b_start;
};

struct TcParams {
  // FP32 output C through TMA (not split-K partials, not grouped launches).
  // tmc (tma_out = 1): 32 x 32 boxes, 128-byte swizzle, for the kernels with
  // one staging block a warp; needs N % 4 == 0, since a box store clips the
  // columns past N only to the 16-byte granule.
  CUtensorMap tmc;
  // C with 64-column boxes (no swizzle), for L2 prefetches only: 256-byte row
  // requests (128-byte ones cap a stream near 4.6 TB/s on B200).
  CUtensorMap tmc_pf;
  // tmc3 (tma_wide = 1): C as {32 columns, N / 32 whole column chunks, M rows}
  // with [32 rows][2 chunks][32] boxes (128-byte swizzle per 128-byte line),
  // so the epilogue's loads and stores are 256-byte row requests; the last
  // N % 32 columns are outside the map.
  CUtensorMap tmc3;
  int tma_out, tma_wide;
  int m, n, k;
  int tiles_m, tiles_n;
  int kblocks;       // k-blocks of the whole K
  int kb_per_split;  // k-blocks per split-K unit
  int splits;
  int band;          // raster band height (tiles of M visited together)
  int epilogue;
  int partial;       // 1: raw partial sums into the workspace (split-K)
  double alpha, beta;
  void* out;
  int64_t ldo;
  int64_t ws_split_stride;
  const int32_t* ea;  // Ozaki row exponents of A
  const int32_t* eb;  // Ozaki column exponents of B
  // K-split last wave of an otherwise unsplit problem: the raster's tiles from
  // tail_tile0 on run as tail_splits units each, of tail_kb k-blocks, whose raw
  // partial tiles go to tail_ws as [split][tile][TILE_M][BN] for
  // tail_reduce_kernel.  tail_splits 1: none (tail_tile0 is the tile count).
  int tail_tile0, tail_splits, tail_kb;
  float* tail_ws;
  WaitCtl ctl;
  int skip_stage;  // test hook: ring position whose loads the producer omits (-1: none)
  // Grouped launch: when ngroups > 0 the problems come from groups[] (all
  // other per-problem fields above are ignored).
  const GroupEntry* groups;
  // Work list: position i * slots + s is the i-th unit of CTA (pair) s, as
  // {problem, tile of the problem}; problem -1 where a slot has no more.
  const int2* unit_list;
  int ngroups, total_tiles;  // total_tiles: positions
  // Optional device-side gate: the kernel runs only if *gate == gate_value
  // (the adaptive Ozaki call's slice count, chosen on the device).
  const int* gate;
  int gate_value;
  // Ozaki: slices per k-block in the stacked B layout (0: the kernel's own count).
  int b_layout_slices;
};

// Where a work unit's result goes (from TcParams, or from a GroupEntry).
struct OutCtx {
  int m, n, epilogue, partial;
  double alpha, beta;
  void* out;
  int64_t ldo, ws_split_stride;
  const int32_t* ea;
  const int32_t* eb;
  const CUtensorMap* tmc;     // non-null: 32 x 32 boxes of C (one staging block a warp)
  const CUtensorMap* tmc_pf;  // non-null: 64-column boxes for L2 prefetches of C
  const CUtensorMap* tmc3;    // non-null: 64-column 3-D boxes of C's whole chunks (two staging blocks)
  uint64_t* tbar;             // this epilogue warp's barriers for its C loads
  WaitCtl ctl;
};

// Operands of tail_reduce_kernel: tiles tile0 .. tile0 + count - 1 of the raster.
struct TailReduce {
  const float* ws;
  float* C;
  int64_t ldc;
  int m, n, tiles_m, tiles_n, band, tile_m, bn, tile0, count, splits;
  float alpha, beta;
  int epilogue;
};

// A resolved work unit: operand descriptors, tile coordinates, K range.
struct Unit {
  const CUtensorMap* ta;
  const CUtensorMap* tb;
  int tm, tn, z, kb0, kb1;
  int group;  // -1 when not grouped; -2 - i: the i-th K-split tile of the last wave (TcParams::tail_splits)
};

}  // namespace tc
}  // namespace cucosma

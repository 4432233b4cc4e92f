// tc_gemm.cu -- planning and host entry points of the tensor-core precision
// paths (BF16x3, BF16x6, Ozaki); the kernel template is in tc_kernel.cuh.
#include "simt_gemm.cuh"
#include "split.cuh"
#include "tc_fused.cuh"
#include <cstdlib>
#include "tc_kernel.cuh"

namespace cucosma {
namespace tc {

// Split-K reduction of the Ozaki path: tot = sum_z ws[z] (z ascending),
// C = epi(alpha * ldexp(tot, ea + eb) + beta * C).  With a gate it runs only
// for the slice count chosen on the device.
__global__ void ozaki_reduce_kernel(const double* __restrict__ ws, int64_t split_stride, int64_t ldw, int splits,
                                    double* C, int64_t ldc, int m, int n, const int32_t* __restrict__ ea,
                                    const int32_t* __restrict__ eb, double alpha, double beta, int epi,
                                    const int* gate, int gate_value) {
  pdl_wait();
  if (gate != nullptr && *gate != gate_value) return;
  const int64_t total = (int64_t)m * n;
  for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = idx / n;
    const int c = (int)(idx - r * n);
    const double* w = ws + r * ldw + c;
    double tot = w[0];
    for (int zz = 1; zz < splits; ++zz) tot = tot + w[zz * split_stride];
    const double v = ldexp(tot, ea[r] + eb[c]);
    double* po = C + r * ldc + c;
    const double o = beta == 0.0 ? alpha * v : fma(alpha, v, beta * *po);
    *po = apply_epi(o, epi);
  }
}

// C = epi(alpha * sum of a tile's partials + beta * C) for the tiles of a
// K-split last wave (TcParams::tail_ws), splits in ascending order; four
// columns a thread.  The partials lie in L2: bound by it and by launch latency.
__global__ void __launch_bounds__(256) tail_reduce_kernel(const __grid_constant__ TailReduce t) {
  pdl_wait();
  const int per_tile = t.tile_m * t.bn / 4, vpr = t.bn / 4;
  const int64_t split_stride = (int64_t)t.count * t.tile_m * t.bn;
  for (int64_t idx = (int64_t)blockIdx.x * 256 + threadIdx.x; idx < (int64_t)t.count * per_tile;
       idx += (int64_t)gridDim.x * 256) {
    const int i = (int)(idx / per_tile), v = (int)(idx - (int64_t)i * per_tile);
    int z, tm, tn;
    unit_coords(t.tile0 + i, t.tiles_m * t.tiles_n, t.tiles_m, t.tiles_n, t.band, z, tm, tn);
    const int r = tm * t.tile_m + v / vpr, c = tn * t.bn + (v % vpr) * 4;
    if (r >= t.m || c >= t.n) continue;
    const float* w = t.ws + idx * 4;
    float4 s = *reinterpret_cast<const float4*>(w);  // (columns past n: read, never used)
    for (int q = 1; q < t.splits; ++q) {
      const float4 a = *reinterpret_cast<const float4*>(w + q * split_stride);
      s.x += a.x, s.y += a.y, s.z += a.z, s.w += a.w;
    }
    float* o = t.C + (int64_t)r * t.ldc + c;
    const float acc[4] = {s.x, s.y, s.z, s.w};
    if (c + 4 <= t.n) {  // c % 4 == 0, 16-byte rows
      float4 cv = make_float4(0.f, 0.f, 0.f, 0.f);
      if (t.beta != 0.f) cv = *reinterpret_cast<const float4*>(o);
      cv.x = apply_epi(combine(acc[0], t.alpha, t.beta, &cv.x), t.epilogue);
      cv.y = apply_epi(combine(acc[1], t.alpha, t.beta, &cv.y), t.epilogue);
      cv.z = apply_epi(combine(acc[2], t.alpha, t.beta, &cv.z), t.epilogue);
      cv.w = apply_epi(combine(acc[3], t.alpha, t.beta, &cv.w), t.epilogue);
      *reinterpret_cast<float4*>(o) = cv;
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (c + e < t.n) o[e] = apply_epi(combine(acc[e], t.alpha, t.beta, o + e), t.epilogue);
    }
  }
}

// ------------------------------------------------------------ planning
// BF16 kernel variants (the descriptor's tile id selects one; 0 = auto).
enum Variant : int {
  kV3Promoted = 0,   // BF16x3 128 x 256, promoted (tile id 3)
  kV3Wide = 1,       // BF16x3 128 x 256, whole K in TMEM (tile id 1)
  kV3Small = 2,      // BF16x3 128 x 128, promoted, two accumulators (tile id 2)
  kV3Pair = 3,       // BF16x3 256 x 256 CTA pair (tile id 4)
  kV6Single = 4,     // BF16x6 128 x 128 (tile id 1)
  kV6Pair = 5,       // BF16x6 256 x 128 CTA pair, two double-buffered accumulators (tile id 2)
  kV6PairWide = 6,   // BF16x6 256 x 256 CTA pair, two accumulators, split release (tile id 3)
  kVOzaki = 7,
  kV3Fused = 10,     // BF16x3 256 x 128 pair, split fused into the kernel (tile id 5)
  kV6Fused = 11,     // BF16x6 256 x 128 pair, split fused into the kernel (tile id 4)
};

// Tiling of one kernel: tiles, K blocks and splits, raster band; tiles from
// tail_tile0 on (the last wave) run as tail_splits K splits (1: none).
struct Tiling {
  int slices, bn, tiles_m, tiles_n, kblocks, kb_per_split, splits, band;
  int tail_tile0, tail_splits, tail_kb;
};

struct Plan {
  int kind;  // 0 bf16x3, 1 bf16x6, 2 ozaki
  int variant, pair, tile_m, bn_local, bk;
  int fused;         // BF16 split done inside the GEMM kernel (no planes in the workspace)
  Tiling t;          // the kernel (Ozaki adaptive: the 8-slice candidate)
  int adaptive;      // Ozaki with the slice count chosen on the device
  int layout_slices; // Ozaki slices per k-block in the workspace
  Tiling t9;         // adaptive Ozaki: the 9-slice candidate
  NativePlan native; // adaptive Ozaki: the native FP64 fallback
  int64_t kpad;
  // Workspace: operand B first (its planes / slices, exponents and
  // magnitude sums depend on N and K only, so row blocks of one problem can
  // share them), then A, then the split-K partials of whichever kernel runs.
  size_t off_b, off_eb, off_colsum, off_stats, off_a, off_ea, off_rowsum, off_part, bytes;
  int64_t ldw;
};

static size_t al256(size_t x) { return (x + 255) & ~size_t(255); }

// split_k: 0 = chosen here, >= 1 as given (by the caller or the time model).
static Tiling make_tiling(const Plan& pl, int slices, int bn, const cucosma_gemm_desc* d, int64_t split_k,
                          const DeviceInfo* di) {
  Tiling t{};
  const int64_t M = d->m, N = d->n, K = d->k;
  t.slices = slices;
  t.bn = bn;
  t.tiles_m = (int)ceil_div(M, pl.tile_m);
  t.tiles_n = (int)ceil_div(N, bn);
  t.kblocks = (int)ceil_div(K, pl.bk);
  const int64_t tiles = std::max<int64_t>(1, (int64_t)t.tiles_m * t.tiles_n);  // (plans of empty problems are queried)
  // Work slots: one per SM, or one per SM pair for pair tiles.
  const int slots = pl.pair ? di->sms / 2 : di->sms;
  int64_t min_splits = 1, kbmax = INT32_MAX;
  if (pl.kind == 2) {
    // Exact INT32 diagonals: slices * kchunk * 127^2 < 2^31.
    kbmax = ((int64_t)2147483647 / ((int64_t)slices * 127 * 127)) / pl.bk;
    min_splits = ceil_div(t.kblocks, kbmax);
  }
  int64_t splits = split_k > 0 ? split_k : 1;
  if (split_k <= 0 && tiles < slots) splits = std::max<int64_t>(1, std::min<int64_t>(slots / tiles, t.kblocks / 16));
  splits = std::max(splits, min_splits);
  // More splits than one wave of units (the Ozaki exactness bound on long
  // K): as many splits as the same number of waves holds, so that the last
  // wave is full and every unit is shorter (256 x 256 x 1,048,576 at 8
  // slices: 64 splits x 8 tiles = 3.5 waves of 148; 74 splits fill 4).
  if (split_k <= 0 && splits > 1 && tiles * splits > slots) {
    const int64_t waves = ceil_div(tiles * splits, (int64_t)slots);
    splits = std::max(splits, waves * slots / tiles);
  }
  const int64_t kblocks = std::max(1, t.kblocks);
  splits = std::min(splits, kblocks);
  t.kb_per_split = (int)std::min<int64_t>(ceil_div(kblocks, splits), kbmax);
  t.splits = (int)ceil_div(kblocks, t.kb_per_split);
  // Raster band (tiles of M visited together): measured best at 8192^3 and
  // 16384^3 -- 16 for the BF16 paths (128 x 256 tiles), 4 for Ozaki; pair
  // tiles keep the same band height in rows (8 tiles of 256).
  t.band = d->swizzle > 0 ? d->swizzle : (pl.kind == 2 ? 4 : (pl.pair ? 8 : 16));
  return t;
}

// Operands beyond L2: the fused split pays off when the separate pre-pass (read the FP32
// operands, write nt BF16 planes) would take more than a quarter of the
// GEMM's own bound (tensor time at nt products of BF16, or the HBM time of
// reading the planes and writing -- with beta, also reading -- C): operands
// read only a few times, as in the large-K and large-N families (measured on
// B200, beta 0.5, BF16x3 / BF16x6: 256 x 256 x 1,048,576 0.58 / 0.88 ms fused
// against about 1.2 / 2.6 ms; 256 x 1,048,576 x 256 0.85 / 1.06 against 1.23
// / 1.19 ms), and not where operands are re-read by many tiles.
static bool fused_pays(const cucosma_gemm_desc* d, int nt) {
  const double M = (double)d->m, N = (double)d->n, K = (double)d->k;
  const double hbm = 6.5e12, bf16 = 1.6e15;
  const double products = nt == 2 ? 3.0 : 6.0;
  const double c_bytes = M * N * 4.0 * (d->beta != 0.0 ? 2.0 : 1.0);
  const double t_pre = (M * K + K * N) * (4.0 + 2.0 * nt) / hbm;
  const double t_mma = 2.0 * M * N * K * products / bf16;
  const double t_mem = ((M * K + K * N) * 2.0 * nt + c_bytes) / hbm;
  return t_pre > 0.25 * std::max(t_mma, t_mem);
}

// Modelled time (us) of one BF16 call: a tile per variant with
//   f + (u * k-blocks of a unit + e) * waves   (waves: rho of the whole waves
//   the units make on the CTAs or pairs, the rest of their plain ratio, since
//   the last wave runs with less contention; single-CTA tiles lose a tenth
//   more when they need several waves)
//   + the pre-pass at 5.5 TB/s, C at 11 TB/s of stores (and loads) beside the
//   MMAs, and per split-K call 3.1 us and the partials at 13.8 TB/s (L2).
// Least squares over 2281 measured calls on B200 (60 shapes, 64 to 8192 a
// side, operands that fit L2; every tile, 1 to 24 splits; CUDA graphs): rms
// error 5 to 10 %.  On those shapes the model's choice takes 1.017 of the best
// measured time (geometric mean) and 1/1.24 of the time of the rule it
// replaced, which took the largest tile, split only below one wave with 16
// k-blocks left, and fused from 32 MB (1234 x 1111 x 777 BF16x6: 38 us with 25
// of 74 pairs at work, 25.5 on 128 x 128 tiles; 2048^3 BF16x3: 89 us fused, 48
// with the pre-pass).
struct TileModel {
  int variant, tile_m, bn, fused;
  double f, u, e, rho;
};
constexpr TileModel kModelV3[] = {{kV3Small, 128, 128, 0, 6.5, 0.41, 2.2, 0.8},
                                  {kV3Pair, 256, 256, 0, 5.8, 0.43, 8.5, 0.76},
                                  {kV3Fused, 256, 128, 1, 5.6, 0.60, 2.5, 0.9}};
constexpr TileModel kModelV3Direct = {kV3Pair, 256, 256, 0, 9.3, 0.40, 2.6, 1.0};  // one accumulator chunk
constexpr TileModel kModelV6[] = {{kV6Single, 128, 128, 0, 7.2, 0.64, 1.8, 0.8},
                                  {kV6Pair, 256, 128, 0, 7.6, 0.60, 1.7, 0.8},
                                  {kV6PairWide, 256, 256, 0, 8.1, 1.01, 3.6, 0.92},
                                  {kV6Fused, 256, 128, 1, 5.8, 0.90, 2.1, 0.92}};

// us a k-block of a 256 x 256 pair takes in a thin last wave (BF16x3, BF16x6)
constexpr double kTailUnitUs[2] = {0.33, 0.93};

// The last wave of `tiles` unsplit units on `slots` CTAs or pairs, when it is
// partial: its K in `splits` parts of kb k-blocks, so that most slots have work
// for a shorter time.  unit_us: the modelled time of one k-block of a unit.
// Returns the modelled time saved: the k-blocks a slot no longer walks, less
// the reduction (a launch, and every partial tile out of and back into the SMs
// through L2); 0 (leave it whole) below 5.5 % of the units' time, where B200
// showed no gain beyond the runs' differences (BF16x6 8192^3, 62 tiles left,
// modelled 0.4 %; 2600^3 4.8 %; 4700 x 6100 x 520 2.7 %).  Above it, back to
// back: 1900 x 2500 x 4000 (a few tiles more than one wave) BF16x3 153..177 ->
// 122..127 us, BF16x6 325 -> 246; 4096^3 (half a wave left) BF16x3 325 -> 318,
// BF16x6 877..915 -> 762..829; 3000 x 5000 x 2000 BF16x3 162 -> 157; 5000^3
// BF16x3 734 -> 706.  kb is a whole number of promotion chunks, so a part's
// sums are the chunk sums of the whole.
struct Tail {
  int splits, kb;
  double saved;
};
static Tail plan_tail(int64_t tiles, int64_t slots, int64_t kblocks, double unit_us, double tile_elems) {
  Tail best{1, 0, 0.0};
  const int64_t r = tiles % slots;
  if (tiles < slots || r == 0) return best;
  const double least = 0.055 * (double)(ceil_div(tiles, slots) * kblocks) * unit_us;
  for (int64_t s = 2; s <= 8; ++s) {
    const int64_t kb = round_up(ceil_div(kblocks, s), kPromoteChunk);
    if (ceil_div(kblocks, kb) != s) continue;
    const double saved = ((double)kblocks - (double)(ceil_div(r * s, slots) * kb)) * unit_us -
                         (4.0 + (double)(r * s) * tile_elems * 8.0 / 13.8e6);
    if (saved > least && saved > best.saved * 1.02) best = {(int)s, (int)kb, saved};
  }
  return best;
}

// C's taller than the time model's calls with K of at most 12 k-blocks, whose
// operands, planes and C pass L2: the model counts the pre-pass and C at the
// rates of data in L2.  Fused where fused_pays says so: 72,739 x 200 x 161 BF16x3
// 67.6 us by the model, 49.1 fused, 28,640 x 892 x 371, beta 0.5, 140 / 109,
// 107,248 x 252 x 56 75.8 / 51.8; but within L2 33,722 x 452 x 207 45.8 / 53.3,
// wide 352 x 105,992 x 91 75.9 / 100.6, and rows not ending on 16 bytes 81,451 x
// 530 x 201 131 / 158.  68 tall calls: 0.95 of the time of the model alone.
static bool tall_short_k(const cucosma_gemm_desc* d, int slices, const DeviceInfo* di) {
  const double M = (double)d->m, N = (double)d->n, K = (double)d->k;
  return d->split_k <= 0 && d->m > 8192 && d->k <= 12 * 32 && d->n % 4 == 0 &&
         (M * K + K * N) * (4.0 + 2.0 * slices) + M * N * 4.0 > 0.95 * (double)di->l2_bytes && fused_pays(d, slices);
}

// The (tile, splits) with the smallest modelled time; forced > 0 fixes the splits.
static void choose_bf16(const cucosma_gemm_desc* d, int kind, const DeviceInfo* di, bool allow_fused, int& variant,
                        int64_t& splits) {
  const double M = (double)d->m, N = (double)d->n, K = (double)d->k;
  const int64_t kblocks = ceil_div(d->k, 32);
  const TileModel* tm = kind == 1 ? kModelV6 : kModelV3;
  const int count = kind == 1 ? 4 : 3;
  const double t_pre = (M * K + K * N) * (kind == 1 ? 10.0 : 8.0) / 5.5e6;
  const double t_c = M * N * 4.0 * (d->beta != 0.0 ? 2.0 : 1.0) / 11.4e6;
  double best = 1e300;
  for (int i = 0; i < count; ++i) {
    if (tm[i].fused && !allow_fused) continue;
    const bool pair = tm[i].tile_m == 256;
    const int64_t tiles = std::max<int64_t>(1, ceil_div(d->m, tm[i].tile_m) * ceil_div(d->n, tm[i].bn));
    const int64_t slots = pair ? di->sms / 2 : di->sms;
    auto consider = [&](int64_t s) {
      const TileModel& v = tm[i].variant == kV3Pair && s == 1 && kblocks <= kPromoteChunk ? kModelV3Direct : tm[i];
      const double ratio = (double)(tiles * s) / (double)slots, waves = (double)ceil_div(tiles * s, slots);
      double w = v.rho * waves + (1.0 - v.rho) * std::max(ratio, 1.0);
      double t = v.f + (v.u * (double)ceil_div(kblocks, s) + v.e) * w * (!pair && waves > 1.0 ? 1.1 : 1.0);
      if (!v.fused) t += t_pre;
      if (s > 1) t += 3.1 + (double)s * M * N * 8.0 / 13.8e6;
      if (s == 1 && d->split_k <= 0 && d->flags == 0 && (v.variant == kV3Pair || v.variant == kV6PairWide))
        t -= plan_tail(tiles, slots, kblocks, kTailUnitUs[kind], 256.0 * v.bn).saved;
      if (t + t_c < best) {
        best = t + t_c;
        variant = v.variant;
        splits = s;
      }
    };
    if (d->split_k > 0) {
      consider(std::min<int64_t>(d->split_k, kblocks));
      continue;
    }
    consider(1);
    // at least 4 k-blocks a split, at most two waves of units
    const int64_t smax = std::min(kblocks / 4, 2 * slots / tiles);
    for (int64_t s = 2; s <= smax; s += s < 8 ? 1 : s / 4) consider(s);
    const int64_t full = std::min(smax, slots / tiles);  // one whole wave
    if (full > 1) consider(full);
  }
}

static Plan make_plan(const cucosma_gemm_desc* d, const DeviceInfo* di, bool allow_fused = true) {
  Plan pl{};
  allow_fused = allow_fused && d->flags == 0;  // the test hooks run the pre-pass path (as does its workspace query)
  const int64_t M = d->m, N = d->n, K = d->k;
  int slices = 0, bn = 0;
  int64_t splits = d->split_k;
  pl.bk = 32;
  if (d->precision == CUCOSMA_PRECISION_OZAKI) {
    pl.kind = 2;
    pl.variant = kVOzaki;
    pl.adaptive = d->slices == 0;
    slices = pl.adaptive ? 8 : d->slices;
    pl.layout_slices = pl.adaptive ? kOzakiLayoutAdaptive : slices;
    bn = ozaki_bn(slices);
    pl.kpad = round_up(K, 32);
  } else {
    pl.kind = d->precision == CUCOSMA_PRECISION_BF16X6 ? 1 : 0;
    slices = pl.kind == 1 ? 3 : 2;
    pl.layout_slices = slices;
    switch (d->tile) {
      case 1: pl.variant = pl.kind == 0 ? kV3Wide : kV6Single; break;
      case 2: pl.variant = pl.kind == 0 ? kV3Small : kV6Pair; break;
      case 3: pl.variant = pl.kind == 0 ? kV3Promoted : kV6PairWide; break;
      case 4: pl.variant = pl.kind == 0 ? kV3Pair : allow_fused ? kV6Fused : kV6Pair; break;
      case 5:
        if (pl.kind == 0) {
          pl.variant = allow_fused ? kV3Fused : kV3Pair;
          break;
        }
        [[fallthrough]];
      default:
        // Auto.  Operands that fit L2: the time model, but for C's longer than
        // its calls had (8192) with K short enough that moving C decides
        // (long_short_k).  Larger ones: pair
        // tiles (unless there is a single 128-row block), fused where the
        // pre-pass's HBM traffic would show, splits by make_tiling.
        if (((double)M * K + (double)K * N) * 4.0 <= (double)di->l2_bytes &&
            !(allow_fused && tall_short_k(d, slices, di)))
          choose_bf16(d, pl.kind, di, allow_fused, pl.variant, splits);
        else if (M <= 128)
          pl.variant = pl.kind == 0 ? kV3Promoted : kV6Single;
        else if (allow_fused && fused_pays(d, slices))
          pl.variant = pl.kind == 0 ? kV3Fused : kV6Fused;
        else
          pl.variant = pl.kind == 0 ? kV3Pair : kV6PairWide;
    }
    bn = (pl.variant == kV3Small || pl.variant == kV6Single || pl.variant == kV6Pair || pl.variant == kV6Fused ||
          pl.variant == kV3Fused)
             ? 128
             : 256;
    pl.fused = pl.variant == kV3Fused || pl.variant == kV6Fused;
    pl.kpad = round_up(K, 8);
  }
  pl.pair = (pl.variant == kV3Pair || pl.variant == kV6Pair || pl.variant == kV6PairWide || pl.fused) ? 1 : 0;
  pl.tile_m = pl.pair ? 256 : 128;
  pl.bn_local = pl.pair ? bn / 2 : bn;
  pl.t = make_tiling(pl, slices, bn, d, splits, di);
  pl.t.tail_tile0 = pl.t.tiles_m * pl.t.tiles_n;
  pl.t.tail_splits = 1;
  // Automatic calls (a given tile or split count is run as given; the test
  // hooks too) on pair tiles: a partial last wave is split along K.
  if (pl.kind != 2 && d->tile == 0 && d->split_k <= 0 && d->flags == 0 && pl.t.splits == 1 &&
      (pl.variant == kV3Pair || pl.variant == kV6PairWide)) {
    const int slots =
        pl.variant == kV3Pair ? max_pair_clusters<Bf16x3Pair>(di->sms) : max_pair_clusters<Bf16x6PairWide>(di->sms);
    const Tail tail = plan_tail(pl.t.tail_tile0, slots, pl.t.kblocks, kTailUnitUs[pl.kind],
                                (double)pl.tile_m * bn);
    if (tail.splits > 1) {
      pl.t.tail_tile0 -= pl.t.tail_tile0 % slots;
      pl.t.tail_splits = tail.splits;
      pl.t.tail_kb = tail.kb;
    }
  }
  if (pl.adaptive) {
    pl.t9 = make_tiling(pl, 9, ozaki_bn(9), d, splits, di);
    cucosma_gemm_desc nd = *d;
    nd.precision = CUCOSMA_PRECISION_NATIVE;
    nd.slices = 0;
    nd.tile = 1;  // the 128 x 128 kernel: the fallback equals a native call with that tile bit for bit
    pl.native = plan_native(&nd, di->sms);
  }
  const int es_in = pl.kind == 2 ? 1 : 2;
  const int es_out = pl.kind == 2 ? 8 : 4;
  const size_t ls = pl.fused ? 0 : (size_t)pl.layout_slices;  // the fused kernel keeps no planes
  size_t off = 0;
  pl.off_b = off;
  off = al256(off + ls * N * pl.kpad * es_in);
  pl.off_eb = pl.off_colsum = pl.off_stats = off;
  if (pl.kind == 2) {
    off = al256(off + (size_t)N * 4);
    pl.off_colsum = pl.off_stats = off;
    if (pl.adaptive) {
      off = al256(off + (size_t)N * 8);
      pl.off_stats = off;
      off = al256(off + sizeof(OzakiStats));
    }
  }
  pl.off_a = off;
  off = al256(off + ls * M * pl.kpad * es_in);
  pl.off_ea = pl.off_rowsum = off;
  if (pl.kind == 2) {
    off = al256(off + (size_t)M * 4);
    pl.off_rowsum = off;
    if (pl.adaptive) off = al256(off + (size_t)M * 8);
  }
  pl.ldw = round_up(N, 4);
  pl.off_part = off;
  size_t part = pl.t.splits > 1 ? (size_t)pl.t.splits * M * pl.ldw * es_out : 0;
  if (pl.t.tail_splits > 1)
    part = (size_t)pl.t.tail_splits * (pl.t.tiles_m * pl.t.tiles_n - pl.t.tail_tile0) * pl.tile_m * bn * es_out;
  if (pl.adaptive) {
    if (pl.t9.splits > 1) part = std::max(part, (size_t)pl.t9.splits * M * pl.ldw * es_out);
    part = std::max(part, pl.native.ws_bytes);
  }
  if (part) off = al256(off + part);
  pl.bytes = off;
  return pl;
}

// Every unit's K fits one promotion chunk: the kernels whose epilogue reads
// TMEM directly.
static bool one_chunk(const Tiling& t) { return t.splits == 1 && t.kblocks <= kPromoteChunk; }

// BF16x6 128 x 128 tiles: eight epilogue warps, or four and a deeper ring with
// the same sums.  Four where the MMAs wait for operands that come from HBM, as
// they and their planes (10 bytes an element) exceed L2, and units are long
// enough for that to outweigh their epilogue.  B200, eight / four: 26 x 6656 x
// 23052 510 / 492 us, 128 x 18944 x 1024 70.8 / 68.4, 128 x 60000 x 256 64.7 /
// 61.3; but from L2 512 x 512 x 4096 29.2 / 31.2, 128 x 6656 x 1024 30.0 / 31.9,
// and 4 k-blocks a unit, beta 0.5, 128 x 100000 x 128 60.0 / 68.0.
static bool deep_ring(const cucosma_gemm_desc* d, const Tiling& t, const DeviceInfo* di) {
  const double elems = (double)d->m * (double)d->k + (double)d->k * (double)d->n;
  return elems * 10.0 > (double)di->l2_bytes && t.kb_per_split >= 8;
}

// Fused tiles, C-heavy: whether the epilogue outlasts a unit's conversions and
// MMAs, so that its two staging blocks are worth a pipeline stage.  Lines
// between K of 48 and 800, 128 to 1500 rows or columns by 20,000 to 150,000, on
// B200; us with two blocks / one at 150,000 x 200 x K: BF16x3, beta 0.5, K = 256
// 126 / 135, 400 205 / 171; BF16x6, beta 0.5, 160 129 / 135, 256 168 / 150; beta
// 0 BF16x6 64 72 / 70, 256 142 / 132; sigmoid at beta 0.5 BF16x3 640 254 / 260,
// 800 317 / 309.  With two blocks the last N % 32 columns leave by rows, which
// beside a whole chunk in the same 64 columns is slower than one block's boxes
// where C is not read (60,000 x 500 x 128 BF16x3 sigmoid 100 / 80, 30,000 x 1000
// x 250 121 / 94; few such tiles in a wide C).  With one block rows that do not
// end on 16 bytes leave one by one: two blocks there.
static bool epilogue_bound(const cucosma_gemm_desc* d, const Plan& pl) {
  // most k-blocks of a unit: [precision][C read][sigmoid]
  constexpr int kMost[2][2][2] = {{{4, 8}, {8, 20}}, {{3, 5}, {5, 14}}};
  if (d->n % 4 != 0 || pl.t.splits > 1) return true;
  if (d->beta == 0.0 && d->n % 64 > 32 && d->n < 4096) return false;
  return pl.t.kblocks <= kMost[pl.kind][d->beta != 0.0][d->epilogue == CUCOSMA_EPILOGUE_SIGMOID];
}

static int plan_launches(const Plan& pl) {
  if (pl.fused) return 1 + (pl.t.splits > 1 ? 1 : 0);
  if (pl.kind != 2) return 2 + (pl.t.splits > 1 || pl.t.tail_splits > 1 ? 1 : 0);  // the split of A and B, the GEMM
  if (!pl.adaptive) return 4 + (pl.t.splits > 1 ? 1 : 0);
  // pre-pass (3), decision, the three gated kernels and their reductions
  return 7 + (pl.t.splits > 1) + (pl.t9.splits > 1) + (pl.native.splits > 1 && !pl.native.cluster);
}

}  // namespace tc

// ------------------------------------------------------------ host API
using namespace tc;

cucosma_status tc_workspace_size(const cucosma_gemm_desc* d, size_t* bytes, const DeviceInfo* di) {
  *bytes = make_plan(d, di).bytes;
  return CUCOSMA_STATUS_SUCCESS;
}

bool tc_plan_is_fused(const cucosma_gemm_desc* d, const DeviceInfo* di) { return make_plan(d, di).fused != 0; }

void tc_plan_info(const cucosma_gemm_desc* d, const DeviceInfo* di, cucosma_plan_info* info, bool allow_fused) {
  const Plan pl = make_plan(d, di, allow_fused);
  info->path = pl.kind + 1;
  info->tile_m = pl.tile_m;
  info->tile_n = pl.t.bn;
  info->tile_k = pl.bk;
  info->splits = pl.t.splits;
  info->band = pl.t.band;
  info->slices = pl.adaptive ? 0 : pl.t.slices;
  info->launches = plan_launches(pl);
  info->kchunk = (int64_t)pl.t.kb_per_split * pl.bk;
  info->kpad = pl.kpad;
  info->workspace_bytes = pl.bytes;
  info->off_a = pl.off_a;
  info->off_b = pl.off_b;
  info->off_ea = pl.off_ea;
  info->off_eb = pl.off_eb;
  info->off_part = pl.off_part;
  info->off_choice = pl.adaptive ? pl.off_stats + offsetof(OzakiStats, choice) : 0;
  info->layout_slices = pl.layout_slices;
  info->fused = pl.fused;
}

namespace {

// Kernel parameters of one tiling (shared fields of every precision path).
TcParams tc_params(const cucosma_gemm_desc* d, const Tiling& t, const Plan& pl, void* C, uint8_t* w,
                   const DeviceInfo* di, bool boxes2d = false) {
  TcParams p{};
  p.m = (int)d->m;
  p.n = (int)d->n;
  p.k = (int)d->k;
  p.tiles_m = t.tiles_m;
  p.tiles_n = t.tiles_n;
  p.kblocks = t.kblocks;
  p.kb_per_split = t.kb_per_split;
  p.splits = t.splits;
  p.tail_tile0 = t.tail_tile0;
  p.tail_splits = t.tail_splits;
  p.tail_kb = t.tail_kb;
  p.tail_ws = t.tail_splits > 1 ? reinterpret_cast<float*>(w + pl.off_part) : nullptr;
  p.band = t.band;
  p.epilogue = d->epilogue;
  p.alpha = d->alpha;
  p.beta = d->beta;
  wait_ctl(di, &p.ctl.status, &p.ctl.timeout_ns);
  p.skip_stage = (d->flags & CUCOSMA_FLAG_TEST_SKIP_STAGE) ? 0 : -1;
  if (t.splits > 1) {
    p.partial = 1;
    p.out = w + pl.off_part;
    p.ldo = pl.ldw;
    p.ws_split_stride = (int64_t)d->m * pl.ldw;
  } else {
    p.partial = 0;
    p.out = C;
    p.ldo = d->ldc;
    // FP32 results leave through TMA (validation made C's base and rows
    // 16-byte aligned): the kernels with two staging blocks a warp move whole
    // 32-column chunks by 3-D boxes and store the last N % 32 columns as rows;
    // those with one block (boxes2d) use 2-D boxes when rows end on a 16-byte
    // boundary (a box store clips the columns past N only to the 16-byte
    // granule: on B200 it wrote the rest of the last granule).
    // CUCOSMA_TMA_EPILOGUE=0 turns the TMA paths off.
    static const bool tma_epilogue = [] {
      const char* e = std::getenv("CUCOSMA_TMA_EPILOGUE");
      return !(e && e[0] == '0');
    }();
    if (tma_epilogue && pl.kind != 2) {
      const uint64_t N = (uint64_t)d->n, M = (uint64_t)d->m, ldc = (uint64_t)d->ldc;
      const CUtensorMapDataType f32 = CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
      if (boxes2d && N % 4 == 0)
        p.tma_out = encode_2d(&p.tmc, f32, 4, C, N, M, ldc, 32, 32, CU_TENSOR_MAP_SWIZZLE_128B) ? 1 : 0;
      if (!boxes2d && N >= 32)
        p.tma_wide = encode_3d(&p.tmc3, f32, 4, C, 32, N / 32, M, 32, ldc, 32, 2, 32, CU_TENSOR_MAP_SWIZZLE_128B) ? 1 : 0;
      // prefetches of C (beta != 0 only)
      if ((p.tma_out || p.tma_wide) && d->beta != 0.0 &&
          !encode_2d(&p.tmc_pf, f32, 4, C, N, M, ldc, 64, 32, CU_TENSOR_MAP_SWIZZLE_NONE))
        p.tma_out = p.tma_wide = 0;
    }
  }
  return p;
}

// One Ozaki GEMM (+ its split-K reduction) with t.slices slices read from a
// layout of pl.layout_slices slices per k-block; gated when gate != null.
cudaError_t run_ozaki(const cucosma_gemm_desc* d, const Plan& pl, const Tiling& t, void* C, uint8_t* w,
                      const DeviceInfo* di, cudaStream_t st, const int* gate, int& launches) {
  const int s = t.slices, ls = pl.layout_slices;
  const int m = (int)d->m, n = (int)d->n;
  int32_t* ea = reinterpret_cast<int32_t*>(w + pl.off_ea);
  int32_t* eb = reinterpret_cast<int32_t*>(w + pl.off_eb);
  TcParams p = tc_params(d, t, pl, C, w, di);
  p.ea = ea;
  p.eb = eb;
  p.gate = gate;
  p.gate_value = s;
  p.b_layout_slices = ls;
  // A slices (packed) as a 3-D byte tensor {32 ls (slices of one k-block), k-blocks, rows}: boxes of 128
  // bytes bring slices 4j .. 4j+3; B slices (stacked) as {32 bytes, columns, k-block * ls + slice}, one
  // box = slices 0 .. s-1 of a sub-tile.
  const uint64_t kbs = (uint64_t)pl.kpad / 32;
  CUtensorMap ta, tb;
  if (!encode_3d(&ta, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, w + pl.off_a, 32ull * ls, kbs, m, 32ull * ls,
                 (uint64_t)pl.kpad * ls, 128, 1, 128, CU_TENSOR_MAP_SWIZZLE_128B) ||
      !encode_3d(&tb, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, w + pl.off_b, 32, n, kbs * ls, 32, 32ull * n, 32, ozaki_sub(s),
                 s, CU_TENSOR_MAP_SWIZZLE_32B))
    return cudaErrorInvalidValue;
  const int grid = std::min(t.tiles_m * t.tiles_n * t.splits, di->sms);
  cudaError_t e;
  switch (s) {
    case 4: e = launch<Ozaki<4>>(ta, tb, p, grid, st); break;
    case 5: e = launch<Ozaki<5>>(ta, tb, p, grid, st); break;
    case 6: e = launch<Ozaki<6>>(ta, tb, p, grid, st); break;
    case 7: e = launch<Ozaki<7>>(ta, tb, p, grid, st); break;
    case 8: e = launch<Ozaki<8>>(ta, tb, p, grid, st); break;
    case 9: e = launch<Ozaki<9>>(ta, tb, p, grid, st); break;
    default: return cudaErrorInvalidValue;
  }
  launches += 1;
  if (e == cudaSuccess && t.splits > 1) {
    const int64_t work = (int64_t)m * n;
    const unsigned blocks = (unsigned)std::max<int64_t>(1, std::min<int64_t>(ceil_div(work, 256), di->sms * 8));
    e = launch_after(t.splits <= 8, ozaki_reduce_kernel, dim3(blocks), 256, 0, st, (const double*)p.out, p.ws_split_stride, pl.ldw,
                     t.splits, (double*)C, d->ldc, m, n, (const int32_t*)ea, (const int32_t*)eb, d->alpha, d->beta,
                     d->epilogue, gate, s);
    launches += 1;
  }
  return e;
}

}  // namespace

cucosma_status tc_gemm_ex(const cucosma_gemm_desc* d, const void* A, const void* B, void* C, void* ws,
                          size_t ws_bytes, const DeviceInfo* di, cudaStream_t st, int prep) {
  // Callers that supply prepared planes (prep without both operands) never
  // get the fused kernel, which reads the FP32 operands themselves.
  const bool allow_fused =
      (prep & (kPrepA | kPrepB)) == (kPrepA | kPrepB) && !(prep & kNoFused) && A != nullptr && B != nullptr;
  const Plan pl = make_plan(d, di, allow_fused);
  if (pl.bytes > 0 && (ws == nullptr || ws_bytes < pl.bytes)) return CUCOSMA_STATUS_WORKSPACE_TOO_SMALL;
  if (pl.kind == 2 && (pl.t.slices < 4 || pl.t.slices > 9)) return CUCOSMA_STATUS_NOT_SUPPORTED;
  uint8_t* w = static_cast<uint8_t*>(ws);
  const int m = (int)d->m, n = (int)d->n, k = (int)d->k;
  cudaError_t e = cudaSuccess;
  int launches = 0;
  if (pl.fused) {
    // FP32 operand tiles straight from the caller's buffers.  BF16x3 (in
    // place): A [128 rows][64 K] and B [64 K][64 columns] boxes, 256-byte
    // rows; BF16x6: A [128 rows][32 K] (128-byte swizzle) and B [32 K][64].
    const int kw = pl.kind == 0 ? 64 : 32;  // k-values per FP32 row of a stage
    CUtensorMap ta, tb;
    if (!encode_2d(&ta, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, A, k, m, d->lda, kw, 128,
                   pl.kind == 0 ? CU_TENSOR_MAP_SWIZZLE_NONE : CU_TENSOR_MAP_SWIZZLE_128B) ||
        !encode_2d(&tb, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, B, n, k, d->ldb, pl.bn_local, kw,
                   CU_TENSOR_MAP_SWIZZLE_NONE))
      return CUCOSMA_STATUS_LAUNCH_FAILED;
    // C-heavy shapes (C traffic above a quarter of the operands'): the
    // variant with two staging blocks per epilogue warp and three stages
    // (256 x 1,048,576 x 256, beta 0.5: 0.85 against 0.94 ms on B200)
    const double c_bytes = (double)d->m * d->n * 4.0 * (d->beta != 0.0 ? 2.0 : 1.0);
    const double ab_bytes = ((double)d->m * d->k + (double)d->k * d->n) * 4.0;
    const bool c_heavy = c_bytes > 0.25 * ab_bytes && epilogue_bound(d, pl);
    const TcParams p = tc_params(d, pl.t, pl, C, w, di, !c_heavy);
    prof_begin(st);
    // (BF16x3 that neither reads C nor takes the sigmoid has nothing to gain
    // from it: 256 x 200,001 x 64 84.4 us promoted, 88.3 direct)
    const bool direct = c_heavy && one_chunk(pl.t) &&
                        (pl.kind == 1 || d->beta != 0.0 || d->epilogue == CUCOSMA_EPILOGUE_SIGMOID);
    // C read by rows, not boxes: 512 x 8191 x 4096 BF16x3, beta 0.5, 168 us,
    // 199 with C read beside its stores, 182 on the two-block variant
    const bool rows_c = !c_heavy && !p.tma_out && !p.partial && d->beta != 0.0;
    if (pl.kind == 1)
      e = direct    ? launch_fused_inplace<Bf16x6Pair, 2, true>(ta, tb, p, di->sms, st)
          : c_heavy ? launch_fused_inplace<Bf16x6Pair, 2>(ta, tb, p, di->sms, st)
          : rows_c  ? launch_fused_inplace<Bf16x6Pair, 1, false, true>(ta, tb, p, di->sms, st)
                    : launch_fused_inplace<Bf16x6Pair, 1>(ta, tb, p, di->sms, st);
    else
      e = direct    ? launch_fused_inplace<Bf16x3Pair128, 2, true>(ta, tb, p, di->sms, st)
          : c_heavy ? launch_fused_inplace<Bf16x3Pair128, 2>(ta, tb, p, di->sms, st)
          : rows_c  ? launch_fused_inplace<Bf16x3Pair128, 1, false, true>(ta, tb, p, di->sms, st)
                    : launch_fused_inplace<Bf16x3Pair128, 1>(ta, tb, p, di->sms, st);
    prof_end(st);
    launches += 1;
    if (e == cudaSuccess && pl.t.splits > 1) {
      e = simt::launch_reduce<float>((const float*)p.out, p.ws_split_stride, pl.ldw, pl.t.splits, (float*)C, d->ldc, m,
                                     n, d->alpha, d->beta, d->epilogue, di->sms, st);
      launches += 1;
    }
  } else if (pl.kind != 2) {
    const int nt = pl.t.slices;
    SplitJobs jobs{};
    if (prep & kPrepA) jobs.rows((const float*)A, d->lda, m, k, w + pl.off_a, pl.kpad);
    if (prep & kPrepB) jobs.cols((const float*)B, d->ldb, k, n, w + pl.off_b, pl.kpad);
    if (jobs.count > 0) {
      e = launch_split_bf16(jobs, nt, st);
      launches += 1;
    }
    if (e != cudaSuccess) return CUCOSMA_STATUS_LAUNCH_FAILED;
    CUtensorMap ta, tb;
    if (!encode_3d(&ta, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, w + pl.off_a, k, m, nt, pl.kpad, (uint64_t)m * pl.kpad,
                   pl.bk, 128, nt, CU_TENSOR_MAP_SWIZZLE_64B) ||
        !encode_3d(&tb, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, w + pl.off_b, k, n, nt, pl.kpad, (uint64_t)n * pl.kpad,
                   pl.bk, pl.bn_local, nt, CU_TENSOR_MAP_SWIZZLE_64B))
      return CUCOSMA_STATUS_LAUNCH_FAILED;
    const TcParams p = tc_params(d, pl.t, pl, C, w, di, pl.variant == kV3Wide);
    const int tail_tiles = pl.t.tiles_m * pl.t.tiles_n - pl.t.tail_tile0;
    const int units = pl.t.tail_splits > 1 ? pl.t.tail_tile0 + tail_tiles * pl.t.tail_splits
                                           : pl.t.tiles_m * pl.t.tiles_n * pl.t.splits;
    const int grid = std::min(units, di->sms);
    auto pair_grid = [&](int clusters) { return 2 * std::max(1, std::min(units, clusters)); };
    prof_begin(st);
    switch (pl.variant) {
      case kV6Single:
        e = deep_ring(d, pl.t, di) ? launch<Bf16x6Deep>(ta, tb, p, grid, st) : launch<Bf16x6>(ta, tb, p, grid, st);
        break;
      case kV6Pair: e = launch<Bf16x6Pair>(ta, tb, p, pair_grid(max_pair_clusters<Bf16x6Pair>(di->sms)), st); break;
      case kV6PairWide:
        if (pl.t.tail_splits > 1)
          e = launch<WithTail<Bf16x6PairWide>>(ta, tb, p, pair_grid(max_pair_clusters<Bf16x6PairWide>(di->sms)), st);
        else
          e = launch<Bf16x6PairWide>(ta, tb, p, pair_grid(max_pair_clusters<Bf16x6PairWide>(di->sms)), st);
        break;
      case kV3Small: e = launch<Bf16x3Promoted>(ta, tb, p, grid, st); break;
      case kV3Wide: e = launch<Bf16x3Wide>(ta, tb, p, grid, st); break;
      case kV3Pair:
        if (one_chunk(pl.t))
          e = launch<Bf16x3PairDirect>(ta, tb, p, pair_grid(max_pair_clusters<Bf16x3PairDirect>(di->sms)), st);
        else if (pl.t.tail_splits > 1)
          e = launch<WithTail<Bf16x3Pair>>(ta, tb, p, pair_grid(max_pair_clusters<Bf16x3Pair>(di->sms)), st);
        else
          e = launch<Bf16x3Pair>(ta, tb, p, pair_grid(max_pair_clusters<Bf16x3Pair>(di->sms)), st);
        break;
      default: e = launch<Bf16x3>(ta, tb, p, grid, st);
    }
    prof_end(st);
    launches += 1;
    if (e == cudaSuccess && pl.t.splits > 1) {
      e = simt::launch_reduce<float>((const float*)p.out, p.ws_split_stride, pl.ldw, pl.t.splits, (float*)C, d->ldc, m,
                                     n, d->alpha, d->beta, d->epilogue, di->sms, st);
      launches += 1;
    }
    if (e == cudaSuccess && pl.t.tail_splits > 1) {
      const TailReduce t{p.tail_ws, static_cast<float*>(C), d->ldc, m, n, pl.t.tiles_m, pl.t.tiles_n, pl.t.band,
                         pl.tile_m, pl.t.bn, pl.t.tail_tile0, tail_tiles, pl.t.tail_splits, (float)d->alpha,
                         (float)d->beta, d->epilogue};
      const int64_t vecs = (int64_t)tail_tiles * pl.tile_m * pl.t.bn / 4;
      e = launch_after(true, tail_reduce_kernel, dim3((unsigned)std::min<int64_t>(ceil_div(vecs, 256), di->sms * 8)),
                       256, 0, st, t);
      launches += 1;
    }
  } else {
    const int ls = pl.layout_slices;
    int32_t* ea = reinterpret_cast<int32_t*>(w + pl.off_ea);
    int32_t* eb = reinterpret_cast<int32_t*>(w + pl.off_eb);
    OzakiStats* stats = pl.adaptive ? reinterpret_cast<OzakiStats*>(w + pl.off_stats) : nullptr;
    unsigned long long* colsum = pl.adaptive ? reinterpret_cast<unsigned long long*>(w + pl.off_colsum) : nullptr;
    unsigned long long* rowsum = pl.adaptive ? reinterpret_cast<unsigned long long*>(w + pl.off_rowsum) : nullptr;
    if (prep & (kPrepA | kPrepB)) {
      OzakiOperands o{};
      o.A = (const double*)A;
      o.lda = d->lda;
      o.B = (const double*)B;
      o.ldb = d->ldb;
      o.m = m;
      o.n = n;
      o.k = k;
      o.kpad = pl.kpad;
      o.ea = ea;
      o.eb = eb;
      o.sa = reinterpret_cast<int8_t*>(w + pl.off_a);
      o.sb = reinterpret_cast<int8_t*>(w + pl.off_b);
      o.rowsum = rowsum;
      o.colsum = colsum;
      e = launch_ozaki_prep(ls, o, (prep & kPrepA) != 0, (prep & kPrepB) != 0, stats, di->sms, st, &launches);
    }
    if (e == cudaSuccess && pl.adaptive) {
      e = launch_ozaki_decide(rowsum, m, colsum, n, k, stats, di->sms, st);
      launches += 1;
    }
    if (e != cudaSuccess) return CUCOSMA_STATUS_LAUNCH_FAILED;
    prof_begin(st);
    if (!pl.adaptive) {
      e = run_ozaki(d, pl, pl.t, C, w, di, st, nullptr, launches);
    } else {
      // Three kernels, each gated on the device's choice: 8 slices, 9
      // slices, or native FP64 (the two not chosen return at once).
      const int* gate = &stats->choice;
      e = run_ozaki(d, pl, pl.t, C, w, di, st, gate, launches);
      if (e == cudaSuccess) e = run_ozaki(d, pl, pl.t9, C, w, di, st, gate, launches);
      if (e == cudaSuccess) {
        cucosma_gemm_desc nd = *d;
        nd.precision = CUCOSMA_PRECISION_NATIVE;
        // (counts its own launches)
        if (native_gemm_gated(&nd, pl.native, A, B, C, w + pl.off_part, di, st, gate, 0) != CUCOSMA_STATUS_SUCCESS)
          e = cudaErrorLaunchFailure;
      }
    }
    prof_end(st);
  }
  note_launches(launches);
  return e == cudaSuccess ? CUCOSMA_STATUS_SUCCESS : CUCOSMA_STATUS_LAUNCH_FAILED;
}

}  // namespace cucosma

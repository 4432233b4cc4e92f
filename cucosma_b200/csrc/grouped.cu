// grouped.cu -- many uneven GEMMs in one persistent tcgen05 launch.
//
// The reference can only run one compile-time shape per build (config.h:9-31);
// a batch of 512 shapes would be 512 builds.  Here a plan lays every
// problem's operand planes out in the workspace, encodes one pair of TMA
// descriptors per problem, and uploads a table of GroupEntry records.  A
// launch is then:
//   BF16x3 / BF16x6: one table-driven split kernel for the A rows and the B
//                    tiles of every problem + the persistent GEMM kernel;
//   Ozaki:           exponents, slices (both table-driven) + the GEMM kernel.
// The tiles of all problems are dealt out to the GEMM's CTAs (or pairs) by the
// plan's work list (work_list below; tc_kernel.cuh, resolve_unit), so small
// problems no longer leave most of the GPU idle the way one launch per problem
// does.
#include <algorithm>
#include <cstring>
#include <new>
#include <vector>

#include "split_device.cuh"
#include "split_tiles.cuh"
#include "tc_kernel.cuh"

struct cucosma_grouped_plan_st {
  cucosma_gemm_desc desc;
  int count = 0, kind = 0, slices = 0, total_tiles = 0, grid = 0;
  int tile = 1, tile_m = 128, tile_n = 128, pair = 0, from_cache = 0;
  int pre_depth = 1, pre_a_blocks = 0, pre_b_blocks = 0, exp_a_blocks = 0, exp_b_blocks = 0;
  int device = 0;
  void* workspace = nullptr;
  cucosma::tc::GroupEntry* table = nullptr;  // device copy inside the workspace
  const int* starts = nullptr;      // [4][count]: pre-pass blocks (A, B), exponent blocks (A, B) before each problem
  const int2* unit_list = nullptr;  // the GEMM's work list (TcParams::unit_list)
};

namespace cucosma {
namespace tc {

// Problem owning pre-pass block b: the last one whose (ascending) start is <=
// b.  The block's 256 threads probe as many starts at a time -- one load
// latency for batches of up to 256 problems, two up to 65536; a binary search
// by every thread was nine in a row for 512, and counting all starts 256 at a
// time grew with the batch (20,000 problems of 8 to 32 a side, BF16x3: 1009 us,
// 877 by binary search).
__device__ __forceinline__ int find_entry(const int* __restrict__ starts, int count, int b) {
  int lo = 0, n = count;  // the owner is one of problems lo .. lo + n - 1
  while (n > 1) {
    const int step = (n + 255) / 256, at = (int)threadIdx.x * step;
    const int below = __syncthreads_count(at < n && starts[lo + at] <= b) - 1;
    lo += below * step;
    n = min(step, n - below * step);
  }
  return lo;
}

// BF16 split of every problem (NT terms).  Blocks [0, a_blocks): 8 * depth row
// units of some A; blocks after that: up to depth 64 x 64 tiles of one column
// strip of some B, transposed.  Large batches take kPreDepth of them a block,
// because each block first waits for its problem's table entry; batches whose
// blocks would not fill the SMs then (four a block's loads in series) one.
constexpr int kPreDepth = 4;
template <int NT>
__global__ void __launch_bounds__(256, 4)
    grouped_split_bf16_kernel(const GroupEntry* __restrict__ g, const int* __restrict__ starts, int count,
                              int a_blocks, int depth) {
  __shared__ __align__(16) float tile[64 * 64];
  int b = blockIdx.x;
  SplitJob j{};
  if (b < a_blocks) {
    const GroupEntry& e = g[find_entry(starts, count, b)];
    j.src = static_cast<const float*>(e.A);
    j.ld = e.lda;
    j.rows = e.m;
    j.cols = e.k;
    j.out_r = static_cast<__nv_bfloat16*>(e.planes_a);
    j.kpad_r = e.kpad;
    const int64_t u0 = (int64_t)(b - e.pre_a_start) * (8 * depth) + (threadIdx.x >> 5);
#pragma unroll 1
    for (int i = 0; i < 8 * depth; i += 8) split_rows_unit<NT>(j, u0 + i);
  } else {
    b -= a_blocks;
    const GroupEntry& e = g[find_entry(starts + count, count, b)];
    const int t = b - e.pre_b_start, tiles_n = (e.n + 63) / 64;
    j.src = static_cast<const float*>(e.B);
    j.ld = e.ldb;
    j.rows = e.k;
    j.cols = e.n;
    j.out_c = static_cast<__nv_bfloat16*>(e.planes_b);
    j.kpad_c = e.kpad;
    const int tk0 = t / tiles_n * depth, tk1 = min(tk0 + depth, (int)((e.kpad + 63) / 64));
    split_cols_strip<NT>(j, tk0, tk1, t % tiles_n, tile);
  }
}

// Ozaki exponents of every problem: blocks [0, a_blocks) take 8 rows of some
// A (warp per row); the rest take 32 columns of some B (8 thread rows
// striding over K).
__global__ void __launch_bounds__(256) grouped_ozaki_exp_kernel(const GroupEntry* __restrict__ g,
                                                                const int* __restrict__ starts, int count,
                                                                int a_blocks) {
  __shared__ double red[8][33];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  int b = blockIdx.x;
  if (b < a_blocks) {
    const GroupEntry& e = g[find_entry(starts + 2 * count, count, b)];
    const int r = (b - e.exp_a_start) * 8 + warp;
    if (r >= e.m) return;
    const double* src = static_cast<const double*>(e.A) + (int64_t)r * e.lda;
    double m = 0.0;
    for (int c = lane; c < e.k; c += 32) m = fmax(m, fabs(src[c]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (lane == 0) const_cast<int32_t*>(e.ea)[r] = exp_of(m);
    return;
  }
  b -= a_blocks;
  const GroupEntry& e = g[find_entry(starts + 3 * count, count, b)];
  const int n = (b - e.exp_b_start) * 32 + lane;
  const double* B = static_cast<const double*>(e.B);
  double m = 0.0;
  if (n < e.n)
    for (int k = warp; k < e.k; k += 8) m = fmax(m, fabs(B[(int64_t)k * e.ldb + n]));
  red[warp][lane] = m;
  __syncthreads();
  if (warp == 0 && n < e.n) {
    for (int i = 1; i < 8; ++i) m = fmax(m, red[i][lane]);
    const_cast<int32_t*>(e.eb)[n] = exp_of(m);
  }
}

// Ozaki slices of every problem (A packed, B stacked): blocks [0, a_blocks) take
// 8 rows of some A (warp per row, lanes over 4-column groups); the rest take
// one 32 (k) x 64 (n) tile of some B, transposed.
template <int S>
__global__ void __launch_bounds__(256) grouped_ozaki_slice_kernel(const GroupEntry* __restrict__ g,
                                                                  const int* __restrict__ starts, int count,
                                                                  int a_blocks) {
  __shared__ double tile[32][65];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  int b = blockIdx.x;
  if (b < a_blocks) {
    const GroupEntry& e = g[find_entry(starts, count, b)];
    const int r = (b - e.pre_a_start) * 8 + warp;
    if (r >= e.m) return;
    const double* src = static_cast<const double*>(e.A) + (int64_t)r * e.lda;
    int8_t* out = static_cast<int8_t*>(e.planes_a);
    const int ex = e.ea[r];
    const int nc4 = (int)(e.kpad / 4);
    for (int gi = lane; gi < nc4; gi += 32) {
      const int c = gi * 4;
      double v[4];
      if (c + 4 <= e.k) {
        const double2 v0 = *reinterpret_cast<const double2*>(src + c);  // 16-byte rows, c % 4 == 0
        const double2 v1 = *reinterpret_cast<const double2*>(src + c + 2);
        v[0] = v0.x, v[1] = v0.y, v[2] = v1.x, v[3] = v1.y;
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] = c + j < e.k ? src[c + j] : 0.0;
      }
      uint32_t w[S];
      slice4_packed<S>(v, ex, w);
#pragma unroll
      for (int t = 0; t < S; ++t) *reinterpret_cast<uint32_t*>(out + packed_index<S>(r, c, e.kpad, t)) = w[t];
    }
    return;
  }
  // one 32 (k) x 64 (n) tile of some B: 16 lanes load 64 doubles of a row; a
  // lane slices 4 consecutive k of one column (one 4-byte store per slice)
  b -= a_blocks;
  const GroupEntry& e = g[find_entry(starts + count, count, b)];
  const int t = b - e.pre_b_start;
  const int tiles_n64 = (e.n + 63) / 64;
  const int k0 = (t / tiles_n64) * 32, n0 = (t % tiles_n64) * 64;
  const double* B = static_cast<const double*>(e.B);
#pragma unroll
  for (int p = 0; p < 2; ++p) {
    const int i = p * 16 + tid / 16, c = (tid % 16) * 4;
    const int k = k0 + i, n = n0 + c;
    double v[4] = {0.0, 0.0, 0.0, 0.0};
    if (k < e.k) {
      const double* src = B + (int64_t)k * e.ldb + n;
      if (n + 4 <= e.n) {
        const double2 v0 = *reinterpret_cast<const double2*>(src);
        const double2 v1 = *reinterpret_cast<const double2*>(src + 2);
        v[0] = v0.x, v[1] = v0.y, v[2] = v1.x, v[3] = v1.y;
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] = n + j < e.n ? src[j] : 0.0;
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) tile[i][c + j] = v[j];
  }
  __syncthreads();
  int8_t* out = static_cast<int8_t*>(e.planes_b);
#pragma unroll
  for (int p = 0; p < 2; ++p) {
    const int item = p * 256 + tid, nl = item / 8, kq = item % 8;
    const int n = n0 + nl, k = k0 + kq * 4;
    if (n >= e.n) continue;
    const int ex = e.eb[n];
    const double v[4] = {tile[kq * 4][nl], tile[kq * 4 + 1][nl], tile[kq * 4 + 2][nl], tile[kq * 4 + 3][nl]};
    uint32_t w[S];
    slice4_packed<S>(v, ex, w);
#pragma unroll
    for (int s_ = 0; s_ < S; ++s_) *reinterpret_cast<uint32_t*>(out + stacked_index<S>(n, k, e.n, s_)) = w[s_];
  }
}

// ----------------------------------------------------------------- host
namespace {

size_t al256(size_t x) { return (x + 255) & ~size_t(255); }

// Tile of a grouped launch (descriptor tile id, 0 = the tuner's cached choice
// for this batch, else automatic_tile()):
//   BF16X3  1 = 128 x 128 promoted, 2 = 128 x 256 promoted, 3 = 256 x 256 CTA pair;
//           4 / 5 = 256 x 128 / 256 x 256 CTA pair, bit-identical to 1
//   BF16X6  1 = 128 x 128, 2 = 256 x 256 CTA pair (split release)
//   OZAKI   1 = 128 x ozaki_bn(slices)
struct GTile {
  int id, tile_m, bn, pair;
};
bool grouped_tile(int kind, int slices, int id, GTile& g) {
  if (kind == 0 && id >= 1 && id <= 5) {
    g = id == 1   ? GTile{1, 128, 128, 0}
        : id == 2 ? GTile{2, 128, 256, 0}
        : id == 3 ? GTile{3, 256, 256, 1}
        : id == 4 ? GTile{4, 256, 128, 1}
                  : GTile{5, 256, 256, 1};
    return true;
  }
  if (kind == 1 && id >= 1 && id <= 2) {
    g = id == 1 ? GTile{1, 128, 128, 0} : GTile{2, 256, 256, 1};
    return true;
  }
  if (kind == 2 && id == 1) {
    g = GTile{1, 128, ozaki_bn(slices), 0};
    return true;
  }
  return false;
}

struct Layout {
  int kind, slices, bn, tile_m, pair, tile;
  size_t table_bytes, total_bytes, off_starts, off_units;
  size_t most_table_bytes;  // table_bytes of the tile with the longest work list
  std::vector<GroupEntry> entries;  // pointers relative to the workspace base (offsets)
  std::vector<size_t> off_a, off_b, off_ea, off_eb;
  std::vector<int> order;   // table order of the problems
  int64_t positions;        // of the work list: whole rounds of one unit a slot
  int slots;                // CTAs (pairs) that walk it
  int pre_depth, pre_a, pre_b, exp_a, exp_b;
};

// Blocks of the BF16 split of one problem's A and B, depth units a block.
int64_t split_a_blocks(const cucosma_gemm_problem& q, int64_t kpad, int depth) {
  return ceil_div(q.m * ceil_div(kpad / 8, kRowUnit), 8 * depth);
}
int64_t split_b_blocks(const cucosma_gemm_problem& q, int64_t kpad, int depth) {
  return ceil_div(kpad, 64 * depth) * ceil_div(q.n, 64);
}

// Work list of a tile: the units (tiles of the problems, longest K first) in
// rounds of one per slot, each round's longest to the slot with the least work
// so far, work being k-blocks plus a constant for the epilogue.  Handing them
// out round-robin left the busiest slot a third above the mean on 64 problems
// of the benchmark's distribution (601 against 452 k-blocks of 32).  Loads less
// than one unit apart count as equal and keep the slots in order, so that
// neighbouring tiles of a problem still run on neighbouring SMs (sorted by the
// exact loads, the 512-problem batch lost 8 % to L2).  Returns the busiest
// slot's work.
constexpr int kUnitOverhead = 4;  // k-blocks
int64_t work_list(const cucosma_gemm_problem* pr, const std::vector<int>& order, int tile_m, int bn, int slots,
                  std::vector<int2>* list) {
  std::vector<int64_t> load(slots, 0);
  std::vector<std::pair<int64_t, int>> round(slots);  // (load in units, slot), least first
  int next = slots;                                   // slots of this round served so far
  for (int e = 0; e < (int)order.size(); ++e) {
    const cucosma_gemm_problem& p = pr[order[e]];
    const int64_t tiles = ceil_div(p.m, tile_m) * ceil_div(p.n, bn);
    const int64_t work = ceil_div(p.k, 32) + kUnitOverhead;
    for (int64_t t = 0; t < tiles; ++t) {
      if (next == slots) {
        const int64_t least = *std::min_element(load.begin(), load.end());
        for (int s = 0; s < slots; ++s) round[s] = {(load[s] - least) / work, s};
        std::sort(round.begin(), round.end());
        if (list) list->resize(list->size() + slots, int2{-1, 0});
        next = 0;
      }
      const int s = round[next++].second;
      load[s] += work;
      if (list) (*list)[list->size() - slots + s] = int2{e, (int)t};
    }
  }
  return *std::max_element(load.begin(), load.end());
}

// CTAs (pairs) of a grouped launch with `units` units.
int launch_slots(int64_t units, int pair, int sms) {
  return (int)std::max<int64_t>(1, std::min<int64_t>(units, pair ? max_pair_clusters<Bf16x3PairSmall>(sms) : sms));
}

// Tiles of all problems; their numbers and the work list's positions are ints,
// so batches of more are refused.
constexpr int64_t kMaxUnits = INT32_MAX - 4096;
int64_t unit_count(const cucosma_gemm_problem* pr, int count, int tile_m, int bn) {
  int64_t n = 0;
  for (int i = 0; i < count && n <= kMaxUnits; ++i) n += ceil_div(pr[i].m, tile_m) * ceil_div(pr[i].n, bn);
  return n;
}

// Work of the busiest slot.  Past kWalkUnits units a slot has thousands, whose
// spread no longer matters, and dealing them out would take the host longer
// than it saves: the mean and one unit more stand for it.
constexpr int64_t kWalkUnits = 1 << 20;
double busiest_slot(const cucosma_gemm_problem* pr, const std::vector<int>& order, int tile_m, int bn, int64_t units,
                    int slots) {
  if (units <= kWalkUnits) return (double)work_list(pr, order, tile_m, bn, slots, nullptr);
  double total = 0.0, most = 0.0;
  for (int e : order) {
    const double work = (double)(ceil_div(pr[e].k, 32) + kUnitOverhead);
    total += work * (double)(ceil_div(pr[e].m, tile_m) * ceil_div(pr[e].n, bn));
    most = std::max(most, work);
  }
  return total / slots + most;
}

// Automatic tile: of the tiles that give bit-identical results, the one whose
// busiest slot finishes first at these times per k-block of a slot (us, fitted
// to batches of 16, 64 and 512 of the benchmark's distribution on B200: GEMM
// kernel 2.69 ms on 128 x 128 tiles, 2.50 on 256 x 128 pairs, 2.39 on
// 256 x 256 for the 512; L2 feeds the SMs about 7 TB/s, which bounds the
// narrower tiles).  Batches of at most two waves keep the 128 x 128 tile.
int automatic_tile(int kind, const cucosma_gemm_problem* pr, const std::vector<int>& order, int sms) {
  struct Option {
    int id, tile_m, bn, pair;
    double us;
  };
  static constexpr Option kV3[] = {{1, 128, 128, 0, 0.60}, {4, 256, 128, 1, 0.50}, {5, 256, 256, 1, 0.83}};
  static constexpr Option kV6[] = {{1, 128, 128, 0, 0.90}, {2, 256, 256, 1, 1.30}};
  if (kind == 2) return 1;
  const int count = (int)order.size();
  if (unit_count(pr, count, 128, 128) <= 2 * (int64_t)sms) return 1;
  int best = 1;
  double t_best = 1e300;
  for (const Option* o = kind == 0 ? kV3 : kV6, *end = o + (kind == 0 ? 3 : 2); o != end; ++o) {
    const int64_t units = unit_count(pr, count, o->tile_m, o->bn);
    const int slots = launch_slots(units, o->pair, sms);
    const double t = o->us * busiest_slot(pr, order, o->tile_m, o->bn, units, slots);
    if (t < t_best) {
      t_best = t;
      best = o->id;
    }
  }
  return best;
}

cucosma_status layout(const cucosma_gemm_desc* d, const cucosma_gemm_problem* pr, int count, int sms, Layout& L,
                      int tile = -1) {
  if (!d || !pr || count <= 0) return CUCOSMA_STATUS_INVALID_VALUE;
  if (d->flags != 0 || d->epilogue < 0 || d->epilogue > CUCOSMA_EPILOGUE_RELU) return CUCOSMA_STATUS_INVALID_VALUE;
  if (d->precision == CUCOSMA_PRECISION_OZAKI) {
    if (d->dtype != CUCOSMA_R_64F) return CUCOSMA_STATUS_NOT_SUPPORTED;
    L.kind = 2;
    L.slices = d->slices ? d->slices : kOzakiDefaultSlices;
    if (L.slices < 4 || L.slices > 9) return CUCOSMA_STATUS_NOT_SUPPORTED;
  } else if (d->precision == CUCOSMA_PRECISION_BF16X3 || d->precision == CUCOSMA_PRECISION_BF16X6) {
    if (d->dtype != CUCOSMA_R_32F) return CUCOSMA_STATUS_NOT_SUPPORTED;
    L.kind = d->precision == CUCOSMA_PRECISION_BF16X6 ? 1 : 0;
    L.slices = L.kind == 1 ? 3 : 2;
  } else {
    return CUCOSMA_STATUS_NOT_SUPPORTED;  // the grouped launch is a tensor-core path
  }
  for (int i = 0; i < count; ++i) {
    const cucosma_gemm_problem& q = pr[i];
    if (q.m <= 0 || q.n <= 0 || q.k <= 0) return CUCOSMA_STATUS_INVALID_VALUE;
    if (q.m > INT32_MAX || q.n > INT32_MAX || q.k > INT32_MAX) return CUCOSMA_STATUS_INVALID_VALUE;
  }
  // Table order: K descending (stable): the long-K tiles are dealt out first
  // and the short ones even out the end.
  std::vector<int>& order = L.order;
  order.resize(count);
  for (int i = 0; i < count; ++i) order[i] = i;
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return pr[a].k > pr[b].k; });
  if (tile < 0) tile = d->tile;
  GTile g{};
  if (!grouped_tile(L.kind, L.slices, tile != 0 ? tile : 1, g)) return CUCOSMA_STATUS_NOT_SUPPORTED;
  if (unit_count(pr, count, g.tile_m, g.bn) > kMaxUnits) return CUCOSMA_STATUS_NOT_SUPPORTED;
  if (tile == 0) grouped_tile(L.kind, L.slices, automatic_tile(L.kind, pr, order, sms), g);
  L.bn = g.bn;
  L.tile_m = g.tile_m;
  L.pair = g.pair;
  L.tile = g.id;
  const int es_in = L.kind == 2 ? 8 : 4;
  const int es_pl = L.kind == 2 ? 1 : 2;
  const int64_t kmax_exact = ((int64_t)2147483647 / ((int64_t)L.slices * 127 * 127)) / 32 * 32;
  const int64_t units = unit_count(pr, count, L.tile_m, L.bn);
  auto list_length = [&](int64_t n, int slots) { return ceil_div(n, slots) * slots; };
  L.slots = launch_slots(units, L.pair, sms);
  L.positions = list_length(units, L.slots);
  L.off_starts = al256(sizeof(GroupEntry) * (size_t)count);
  L.off_units = L.off_starts + al256(sizeof(int) * 4 * (size_t)count);
  L.table_bytes = L.off_units + al256(sizeof(int2) * (size_t)L.positions);
  L.most_table_bytes = L.table_bytes;
  for (int id = 1; grouped_tile(L.kind, L.slices, id, g); ++id) {
    const int64_t n = unit_count(pr, count, g.tile_m, g.bn);
    if (n <= kMaxUnits)
      L.most_table_bytes = std::max(L.most_table_bytes, L.off_units + al256(sizeof(int2) * (size_t)list_length(n, launch_slots(n, g.pair, sms))));
  }
  size_t off = L.table_bytes;
  L.entries.assign(count, GroupEntry{});
  L.off_a.resize(count);
  L.off_b.resize(count);
  L.off_ea.resize(count);
  L.off_eb.resize(count);
  int64_t deep_blocks = 0;
  for (int i = 0; i < count; ++i)
    deep_blocks += split_a_blocks(pr[i], round_up(pr[i].k, 8), kPreDepth) + split_b_blocks(pr[i], round_up(pr[i].k, 8), kPreDepth);
  L.pre_depth = deep_blocks < 4 * (int64_t)sms ? 1 : kPreDepth;  // (four resident blocks an SM)
  int pa = 0, pb = 0, xa = 0, xb = 0;
  for (int i = 0; i < count; ++i) {
    const cucosma_gemm_problem& q = pr[order[i]];
    if (q.lda < q.k || q.ldb < q.n || q.ldc < q.n || !q.A || !q.B || !q.C) return CUCOSMA_STATUS_INVALID_VALUE;
    if ((reinterpret_cast<uintptr_t>(q.A) | reinterpret_cast<uintptr_t>(q.B) | reinterpret_cast<uintptr_t>(q.C)) & 15)
      return CUCOSMA_STATUS_MISALIGNED;
    if ((q.lda * es_in) % 16 || (q.ldb * es_in) % 16 || (q.ldc * es_in) % 16) return CUCOSMA_STATUS_MISALIGNED;
    if (L.kind == 2 && q.k > kmax_exact) return CUCOSMA_STATUS_NOT_SUPPORTED;  // no split-K in grouped launches
    GroupEntry& e = L.entries[i];
    e.m = (int)q.m;
    e.n = (int)q.n;
    e.k = (int)q.k;
    e.kpad = L.kind == 2 ? round_up(q.k, 32) : round_up(q.k, 8);
    e.kblocks = (int)ceil_div(q.k, 32);
    e.tiles_m = (int)ceil_div(q.m, L.tile_m);
    e.tiles_n = (int)ceil_div(q.n, L.bn);
    e.C = q.C;
    e.ldc = q.ldc;
    e.A = q.A;
    e.B = q.B;
    e.lda = q.lda;
    e.ldb = q.ldb;
    e.pre_a_start = pa;
    pa += (int)(L.kind == 2 ? ceil_div(q.m, 8) : split_a_blocks(q, e.kpad, L.pre_depth));
    e.pre_b_start = pb;
    pb += L.kind == 2 ? (int)(ceil_div(e.kpad, 32) * ceil_div(q.n, 64)) : (int)split_b_blocks(q, e.kpad, L.pre_depth);
    e.exp_a_start = xa;
    xa += (int)ceil_div(q.m, 8);
    e.exp_b_start = xb;
    xb += (int)ceil_div(q.n, 32);
    L.off_a[i] = off;
    off = al256(off + (size_t)L.slices * q.m * e.kpad * es_pl);
    L.off_b[i] = off;
    off = al256(off + (size_t)L.slices * q.n * e.kpad * es_pl);
    if (L.kind == 2) {
      L.off_ea[i] = off;
      off = al256(off + (size_t)q.m * 4);
      L.off_eb[i] = off;
      off = al256(off + (size_t)q.n * 4);
    }
  }
  L.pre_a = pa;
  L.pre_b = pb;
  L.exp_a = xa;
  L.exp_b = xb;
  L.total_bytes = off;
  return CUCOSMA_STATUS_SUCCESS;
}

}  // namespace
}  // namespace tc

size_t grouped_table_bytes(const cucosma_gemm_desc* d, const cucosma_gemm_problem* pr, int count,
                           const DeviceInfo* di) {
  tc::Layout L;
  return tc::layout(d, pr, count, di->sms, L, 1) == CUCOSMA_STATUS_SUCCESS ? L.most_table_bytes : 0;
}

int grouped_automatic_tile(const cucosma_gemm_desc* d, const cucosma_gemm_problem* pr, int count,
                           const DeviceInfo* di) {
  tc::Layout L;
  return tc::layout(d, pr, count, di->sms, L, 0) == CUCOSMA_STATUS_SUCCESS ? L.tile : 0;
}

}  // namespace cucosma

using namespace cucosma;
using namespace cucosma::tc;

static cucosma_status grouped_workspace_size(const cucosma_gemm_desc* d, const cucosma_gemm_problem* problems,
                                             int count, size_t* bytes) {
  const DeviceInfo* di = device_info();
  const int sms = di ? di->sms : 148;  // (sizes can be asked for without a device)
  Layout L;
  cucosma_status s = layout(d, problems, count, sms, L);
  if (s != CUCOSMA_STATUS_SUCCESS) return s;
  // tile 0: room for the list of any tile, so that the tuner can try them all
  // here and a plan made after it can take its choice
  *bytes = L.total_bytes + (d->tile == 0 ? L.most_table_bytes - L.table_bytes : 0);
  return CUCOSMA_STATUS_SUCCESS;
}

static cucosma_status grouped_plan_create(const cucosma_gemm_desc* d, const cucosma_gemm_problem* problems, int count,
                                          void* workspace, size_t workspace_bytes, cucosma_grouped_plan* plan) {
  const DeviceInfo* di = device_info();
  if (!di) return CUCOSMA_STATUS_LAUNCH_FAILED;
  if (di->cc_major != 10 || di->cc_minor != 0) return CUCOSMA_STATUS_ARCH_MISMATCH;
  // tile 0: the tuner's choice for this batch of shapes, when it has one
  int tile = d ? d->tile : 0, from_cache = 0;
  if (d && tile == 0) {
    tile = grouped_tuned_tile(d, problems, count, di);
    from_cache = tile > 0;
  }
  Layout L;
  cucosma_status s = layout(d, problems, count, di->sms, L, tile);
  if (s != CUCOSMA_STATUS_SUCCESS) return s;
  if (!workspace || workspace_bytes < L.total_bytes) return CUCOSMA_STATUS_WORKSPACE_TOO_SMALL;
  if (reinterpret_cast<uintptr_t>(workspace) & 255) return CUCOSMA_STATUS_MISALIGNED;
  uint8_t* w = static_cast<uint8_t*>(workspace);
  for (int i = 0; i < count; ++i) {
    GroupEntry& e = L.entries[i];
    e.planes_a = w + L.off_a[i];
    e.planes_b = w + L.off_b[i];
    const int s_ = L.slices;
    bool ok;
    if (L.kind == 2) {
      e.ea = reinterpret_cast<int32_t*>(w + L.off_ea[i]);
      e.eb = reinterpret_cast<int32_t*>(w + L.off_eb[i]);
      const uint64_t kbs = (uint64_t)e.kpad / 32;
      ok = encode_3d(&e.tmA, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, e.planes_a, 32ull * s_, kbs, e.m, 32ull * s_,
                     (uint64_t)e.kpad * s_, 128, 1, 128, CU_TENSOR_MAP_SWIZZLE_128B) &&
           encode_3d(&e.tmB, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, e.planes_b, 32, e.n, kbs * s_, 32, 32ull * e.n, 32,
                     ozaki_sub(s_), s_, CU_TENSOR_MAP_SWIZZLE_32B);
    } else {
      ok = encode_3d(&e.tmA, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, e.planes_a, e.k, e.m, s_, e.kpad,
                     (uint64_t)e.m * e.kpad, 32, 128, s_, CU_TENSOR_MAP_SWIZZLE_64B) &&
           encode_3d(&e.tmB, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, e.planes_b, e.k, e.n, s_, e.kpad,
                     (uint64_t)e.n * e.kpad, 32, L.pair ? L.bn / 2 : L.bn, s_, CU_TENSOR_MAP_SWIZZLE_64B);
    }
    if (!ok) return CUCOSMA_STATUS_LAUNCH_FAILED;
  }
  std::vector<uint8_t> image(L.table_bytes, 0);
  std::memcpy(image.data(), L.entries.data(), sizeof(GroupEntry) * (size_t)count);
  int* starts = reinterpret_cast<int*>(image.data() + L.off_starts);
  for (int i = 0; i < count; ++i) {
    const GroupEntry& e = L.entries[i];
    starts[i] = e.pre_a_start;
    starts[count + i] = e.pre_b_start;
    starts[2 * count + i] = e.exp_a_start;
    starts[3 * count + i] = e.exp_b_start;
  }
  std::vector<int2> units;
  units.reserve((size_t)L.positions);
  work_list(problems, L.order, L.tile_m, L.bn, L.slots, &units);
  std::memcpy(image.data() + L.off_units, units.data(), sizeof(int2) * units.size());
  if (cudaMemcpy(workspace, image.data(), L.table_bytes, cudaMemcpyHostToDevice) != cudaSuccess)
    return CUCOSMA_STATUS_LAUNCH_FAILED;
  auto* p = new cucosma_grouped_plan_st;
  p->desc = *d;
  p->count = count;
  p->kind = L.kind;
  p->slices = L.slices;
  p->total_tiles = (int)L.positions;
  p->grid = L.slots * (L.pair ? 2 : 1);
  p->tile = L.tile;
  p->tile_m = L.tile_m;
  p->tile_n = L.bn;
  p->pair = L.pair;
  p->from_cache = from_cache;
  p->pre_depth = L.pre_depth;
  p->pre_a_blocks = L.pre_a;
  p->pre_b_blocks = L.pre_b;
  p->exp_a_blocks = L.exp_a;
  p->exp_b_blocks = L.exp_b;
  cudaGetDevice(&p->device);
  p->workspace = workspace;
  p->table = reinterpret_cast<GroupEntry*>(workspace);
  p->starts = reinterpret_cast<const int*>(w + L.off_starts);
  p->unit_list = reinterpret_cast<const int2*>(w + L.off_units);
  *plan = p;
  return CUCOSMA_STATUS_SUCCESS;
}

extern "C" cucosma_status cucosma_grouped_plan_destroy(cucosma_grouped_plan plan) {
  delete plan;
  return CUCOSMA_STATUS_SUCCESS;
}

// The tables are built in host memory first; a batch too large for that is an error, not an exception.
extern "C" cucosma_status cucosma_grouped_workspace_size(const cucosma_gemm_desc* d,
                                                         const cucosma_gemm_problem* problems, int count,
                                                         size_t* bytes) {
  if (!bytes) return CUCOSMA_STATUS_INVALID_VALUE;
  try {
    return grouped_workspace_size(d, problems, count, bytes);
  } catch (const std::bad_alloc&) {
    return CUCOSMA_STATUS_ALLOC_FAILED;
  }
}

extern "C" cucosma_status cucosma_grouped_plan_create(const cucosma_gemm_desc* d,
                                                      const cucosma_gemm_problem* problems, int count,
                                                      void* workspace, size_t workspace_bytes,
                                                      cucosma_grouped_plan* plan) {
  if (!plan) return CUCOSMA_STATUS_INVALID_VALUE;
  *plan = nullptr;
  try {
    return grouped_plan_create(d, problems, count, workspace, workspace_bytes, plan);
  } catch (const std::bad_alloc&) {
    return CUCOSMA_STATUS_ALLOC_FAILED;
  }
}

extern "C" cucosma_status cucosma_grouped_plan_get_tile(cucosma_grouped_plan plan, int32_t* tile, int32_t* tile_m,
                                                       int32_t* tile_n, int32_t* from_cache) {
  if (!plan) return CUCOSMA_STATUS_INVALID_VALUE;
  if (tile) *tile = plan->tile;
  if (tile_m) *tile_m = plan->tile_m;
  if (tile_n) *tile_n = plan->tile_n;
  if (from_cache) *from_cache = plan->from_cache;
  return CUCOSMA_STATUS_SUCCESS;
}

template <int S>
static cudaError_t launch_ozaki_grouped(const cucosma_grouped_plan_st& pl, const TcParams& p, const CUtensorMap& dummy,
                                        int grid, cudaStream_t st) {
  grouped_ozaki_slice_kernel<S><<<pl.pre_a_blocks + pl.pre_b_blocks, 256, 0, st>>>(pl.table, pl.starts,
                                                                                   pl.count, pl.pre_a_blocks);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  prof_begin(st);
  e = launch<Ozaki<S>>(dummy, dummy, p, grid, st);
  prof_end(st);
  return e;
}

extern "C" cucosma_status cucosma_gemm_grouped(cucosma_grouped_plan plan, void* stream) {
  if (!plan) return CUCOSMA_STATUS_INVALID_VALUE;
  const DeviceInfo* di = device_info();
  if (!di) return CUCOSMA_STATUS_LAUNCH_FAILED;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  TcParams p{};
  p.skip_stage = -1;
  p.epilogue = plan->desc.epilogue;
  p.alpha = plan->desc.alpha;
  p.beta = plan->desc.beta;
  p.groups = plan->table;
  p.unit_list = plan->unit_list;
  p.ngroups = plan->count;
  p.total_tiles = plan->total_tiles;
  p.splits = 1;
  wait_ctl(di, &p.ctl.status, &p.ctl.timeout_ns);
  const int grid = plan->grid;  // the CTAs the work list was made for
  CUtensorMap dummy;
  std::memset(&dummy, 0, sizeof(dummy));
  cudaError_t e;
  if (plan->kind != 2) {
    const unsigned blocks = (unsigned)(plan->pre_a_blocks + plan->pre_b_blocks);
    if (plan->slices == 3)
      grouped_split_bf16_kernel<3><<<blocks, 256, 0, st>>>(plan->table, plan->starts, plan->count, plan->pre_a_blocks,
                                                           plan->pre_depth);
    else
      grouped_split_bf16_kernel<2><<<blocks, 256, 0, st>>>(plan->table, plan->starts, plan->count, plan->pre_a_blocks,
                                                           plan->pre_depth);
    e = cudaGetLastError();
    if (e != cudaSuccess) return CUCOSMA_STATUS_LAUNCH_FAILED;
    prof_begin(st);
    if (plan->kind == 1)
      e = plan->tile == 2
              ? launch<Bf16x6PairWide>(dummy, dummy, p, grid, st)
              : launch<Bf16x6>(dummy, dummy, p, grid, st);
    else
      e = plan->tile == 5
              ? launch<Bf16x3PairSplit>(dummy, dummy, p, grid, st)
          : plan->tile == 4
              ? launch<Bf16x3PairSmall>(dummy, dummy, p, grid, st)
          : plan->tile == 3 ? launch<Bf16x3Pair>(dummy, dummy, p, grid, st)
          : plan->tile == 2 ? launch<Bf16x3>(dummy, dummy, p, grid, st)
                            : launch<Bf16x3Promoted>(dummy, dummy, p, grid, st);
    prof_end(st);
    note_launches(2);
  } else {
    grouped_ozaki_exp_kernel<<<plan->exp_a_blocks + plan->exp_b_blocks, 256, 0, st>>>(plan->table, plan->starts,
                                                                                      plan->count, plan->exp_a_blocks);
    e = cudaGetLastError();
    if (e != cudaSuccess) return CUCOSMA_STATUS_LAUNCH_FAILED;
    switch (plan->slices) {
      case 4: e = launch_ozaki_grouped<4>(*plan, p, dummy, grid, st); break;
      case 5: e = launch_ozaki_grouped<5>(*plan, p, dummy, grid, st); break;
      case 6: e = launch_ozaki_grouped<6>(*plan, p, dummy, grid, st); break;
      case 7: e = launch_ozaki_grouped<7>(*plan, p, dummy, grid, st); break;
      case 8: e = launch_ozaki_grouped<8>(*plan, p, dummy, grid, st); break;
      case 9: e = launch_ozaki_grouped<9>(*plan, p, dummy, grid, st); break;
      default: return CUCOSMA_STATUS_NOT_SUPPORTED;
    }
    note_launches(3);
  }
  return e == cudaSuccess ? CUCOSMA_STATUS_SUCCESS : CUCOSMA_STATUS_LAUNCH_FAILED;
}

// skinny.cu -- native-precision GEMM for skinny shapes (see skinny.cuh).
//
// Kind 1, small K (K <= 16): the whole K fits one shared-memory tile; a CTA
// produces a 64-row x (64 * VEC)-column block of C (M <= 4: 4 x (256 * VEC),
// M <= 8: 8 x (128 * VEC) or 8 x (256 * VEC)), each thread 16 (4, 8) rows x VEC
// columns with one vector store per row.  The kernel is bound by writing C
// (and reading it when beta != 0), the form of 38416 x 38416 x 4 and
// 4 x 3,000,000 x 4 (B200: 21.7 -> 14.9 us, 6.4 TB/s, with 4 rows a thread,
// four B rows in flight and C's loads ahead; 4 x 2,000,000 x 6 FP64, beta 0.5,
// 62 -> 39 us; 8 x 1,000,000 x 16, beta 0.5, 27 -> 24 us; plan_skinny says when
// M of 5 to 8 takes which form).
//
// Kind 2, thin M or N (<= 8) with K > 16: a CTA owns an 8 x 8 output block and
// one K split; its 256 threads stride over K, each keeping the 64 partial
// products, then reduce across the CTA in a fixed order.  Splits write raw
// partials that a second kernel sums in a fixed order (the split-K reduction
// of simt_gemm.cu, or one warp per output when there are many splits and few
// outputs), so the result is deterministic.  The form of 4 x 8 x 3,000,000 (the
// reference's SPLIT_K = 320 row), HBM-bound on reading A and B once.
//
// Both accumulate each dot product with FMAs in ascending k and apply
// C = epi(alpha * acc + beta * C) like every other kernel here.
#include <algorithm>

#include "simt_gemm.cuh"
#include "skinny.cuh"

namespace cucosma {

// CTAS: resident CTAs an SM.  ROWS_B: rows of B whose loads are in flight when it
// comes straight from global memory.
template <typename T, int RG, int RPT, int CTAS, int ROWS_B>
__global__ void __launch_bounds__(256, CTAS)
    smallk_kernel(const T* __restrict__ A, int64_t lda, const T* __restrict__ B, int64_t ldb, T* C, int64_t ldc,
                  int m, int n, int k, T alpha, T beta, int epi, int tiles_n, int64_t tiles) {
  // RG row groups of RPT rows x (256 / RG) column groups of VEC columns.  With
  // one or two row groups every B element is used by one or two threads only,
  // so B is read straight from global memory; otherwise a K x BNS tile is shared
  // and A lies k-major, so that a k-step reads its rows as vectors (element by
  // element, 100000 x 64 x 16 FP32 took 44 us, now 42; FP64 43 and 40).
  constexpr int VEC = Vec<T>::n;
  using V = typename Vec<T>::type;
  constexpr int CG = 256 / RG, BMS = RG * RPT, BNS = CG * VEC;
  constexpr bool SHARE_B = RG > 2;
  __shared__ __align__(16) T As[SHARE_B ? skinny::kMaxSmallK : BMS][SHARE_B ? BMS + VEC : skinny::kMaxSmallK + 1];
  __shared__ __align__(16) T Bs[SHARE_B ? skinny::kMaxSmallK : 1][SHARE_B ? BNS : VEC];
  const int tid = threadIdx.x, cg = tid % CG, rg = tid / CG;
  int tm_loaded = -1;  // the row block As holds
  for (int64_t t = blockIdx.x; t < tiles; t += gridDim.x) {
    const int tm = (int)(t / tiles_n), tn = (int)(t - (int64_t)tm * tiles_n);
    const int m0 = tm * BMS, n0 = tn * BNS;
    if (SHARE_B || tm != tm_loaded) {
      __syncthreads();  // the previous block's reads of As / Bs are done
      for (int i = tid; i < BMS * k; i += 256) {
        const int r = i / k, kk = i - r * k;
        const T v = m0 + r < m ? A[(int64_t)(m0 + r) * lda + kk] : T(0);
        if constexpr (SHARE_B)
          As[kk][r] = v;
        else
          As[r][kk] = v;
      }
    }
    if constexpr (SHARE_B) {
      for (int i = tid; i < k * CG; i += 256) {
        const int kk = i / CG, c = (i - kk * CG) * VEC, col = n0 + c;
        const T* src = B + (int64_t)kk * ldb + col;
        V v;
        T* pv = reinterpret_cast<T*>(&v);
        if (col + VEC <= n) {
          v = *reinterpret_cast<const V*>(src);  // col % VEC == 0 and 16-byte rows
        } else {
#pragma unroll
          for (int e = 0; e < VEC; ++e) pv[e] = col + e < n ? src[e] : T(0);
        }
        *reinterpret_cast<V*>(&Bs[kk][c]) = v;
      }
    }
    if (SHARE_B || tm != tm_loaded) __syncthreads();
    tm_loaded = tm;
    const int col = n0 + cg * VEC;
    T acc[RPT][VEC];
#pragma unroll
    for (int r = 0; r < RPT; ++r)
#pragma unroll
      for (int e = 0; e < VEC; ++e) acc[r][e] = T(0);
    // four rows a thread: the tile's C loads go out first, beside those of B
    constexpr bool EARLY_C = !SHARE_B && RPT <= 4;
    V cold[EARLY_C ? RPT : 1];
    if (EARLY_C && beta != T(0) && col + VEC <= n) {
#pragma unroll
      for (int r = 0; r < RPT; ++r)
        if (m0 + rg * RPT + r < m)
          cold[r] = *reinterpret_cast<const V*>(C + (int64_t)(m0 + rg * RPT + r) * ldc + col);
    }
    if constexpr (SHARE_B) {
#pragma unroll 2
      for (int kk = 0; kk < k; ++kk) {
        const V bv = *reinterpret_cast<const V*>(&Bs[kk][cg * VEC]);
        const T* b = reinterpret_cast<const T*>(&bv);
#pragma unroll
        for (int r = 0; r < RPT; r += VEC) {
          const V av = *reinterpret_cast<const V*>(&As[kk][rg * RPT + r]);
          const T* a = reinterpret_cast<const T*>(&av);
#pragma unroll
          for (int q = 0; q < VEC; ++q)
#pragma unroll
            for (int e = 0; e < VEC; ++e) acc[r + q][e] = fma(a[q], b[e], acc[r + q][e]);
        }
      }
    } else {
      // B straight from global memory: ROWS_B rows' loads in flight at a time
      for (int k0 = 0; k0 < k; k0 += ROWS_B) {
        V bv[ROWS_B];
#pragma unroll
        for (int u = 0; u < ROWS_B; ++u) {
          const int kk = k0 + u;
          if (u > 0 && kk >= k) break;
          T* pb = reinterpret_cast<T*>(&bv[u]);
          const T* src = B + (int64_t)kk * ldb + col;
          if (col + VEC <= n) {
            bv[u] = *reinterpret_cast<const V*>(src);
          } else {
#pragma unroll
            for (int e = 0; e < VEC; ++e) pb[e] = col + e < n ? src[e] : T(0);
          }
        }
#pragma unroll
        for (int u = 0; u < ROWS_B; ++u) {
          if (ROWS_B > 1 && k0 + u >= k) break;
          const T* b = reinterpret_cast<const T*>(&bv[u]);
#pragma unroll
          for (int r = 0; r < RPT; ++r) {
            const T a = As[rg * RPT + r][k0 + u];
#pragma unroll
            for (int e = 0; e < VEC; ++e) acc[r][e] = fma(a, b[e], acc[r][e]);
          }
        }
      }
    }
    if (col >= n) continue;
    // four rows' C loads before their stores (a store could alias the next row's load, so it would wait for each);
    // row by row in the form of one row of B and four CTAs an SM, whose blocks are one wave and whose registers the
    // batch spilled (6 x 500,000 x 5 FP32, beta 0.5, 7.9 -> 7.4 us)
    constexpr int CB = !SHARE_B && ROWS_B == 1 ? 1 : 4;
#pragma unroll
    for (int r0 = 0; r0 < RPT; r0 += CB) {
      V cv[CB];
      if constexpr (EARLY_C) {
#pragma unroll
        for (int q = 0; q < CB; ++q) cv[q] = cold[r0 + q];
      } else if (beta != T(0) && col + VEC <= n) {
#pragma unroll
        for (int q = 0; q < CB; ++q) {
          const int row = m0 + rg * RPT + r0 + q;
          if (row < m) cv[q] = *reinterpret_cast<const V*>(C + (int64_t)row * ldc + col);
        }
      }
#pragma unroll
      for (int q = 0; q < CB; ++q) {
        const int r = r0 + q, row = m0 + rg * RPT + r;
        if (row >= m) break;
        T* o = C + (int64_t)row * ldc + col;
        if (col + VEC <= n) {
          V ov;
          const T* pc = reinterpret_cast<const T*>(&cv[q]);
          T* po = reinterpret_cast<T*>(&ov);
#pragma unroll
          for (int e = 0; e < VEC; ++e) po[e] = apply_epi(combine(acc[r][e], alpha, beta, pc + e), epi);
          *reinterpret_cast<V*>(o) = ov;
        } else {
#pragma unroll
          for (int e = 0; e < VEC; ++e)
            if (col + e < n) o[e] = apply_epi(combine(acc[r][e], alpha, beta, o + e), epi);
        }
      }
    }
  }
}

// The last steps of thin_kernel's reduction and the sum over its splits, where
// the sums are largest, round once: FP32 sums are added in 64 bits, FP64 ones
// with the rounding error of each addition carried along (D. E. Knuth, TAOCP 2,
// 4.2.2, theorem B).  The rms error is 0.5 to 0.9 of that of four CTAs an SM
// with four (FP64: two) consecutive k a lane, which this kernel replaced; 0.9
// to 1.6 without.  2 % of the time over 110 shapes on B200.
struct SumF64 {
  double hi, lo;
};
__device__ __forceinline__ double widen(float x) { return (double)x; }
__device__ __forceinline__ SumF64 widen(double x) { return SumF64{x, 0.0}; }
__device__ __forceinline__ double add(double a, double b) { return a + b; }
__device__ __forceinline__ SumF64 add(SumF64 a, SumF64 b) {
  const double s = a.hi + b.hi, t = s - a.hi;
  return SumF64{s, a.lo + b.lo + ((a.hi - (s - t)) + (b.hi - t))};
}
__device__ __forceinline__ double shfl_xor(double x, int off) { return __shfl_xor_sync(0xffffffffu, x, off); }
__device__ __forceinline__ SumF64 shfl_xor(SumF64 x, int off) {
  return SumF64{__shfl_xor_sync(0xffffffffu, x.hi, off), __shfl_xor_sync(0xffffffffu, x.lo, off)};
}
__device__ __forceinline__ float narrow(double x) { return (float)x; }
// (an infinite or NaN sum has no error term)
__device__ __forceinline__ double narrow(SumF64 x) { return isfinite(x.hi) ? x.hi + x.lo : x.hi; }

// Thin kernel: lanes take consecutive k, so a warp's load of a row of the A
// block is one contiguous line, and its loads of 32 rows of the B block
// (32-byte FP32 rows) contiguous too when B is as narrow as the block; KU
// steps of 256 k are loaded before the first product.  HBM-bound: 4 x 8 x
// 3,000,000 FP32 on B200 39.8 -> 23.8 us (6.1 TB/s); the form it
// replaced gave each lane four consecutive k, whose B loads lay 128 bytes
// apart, and was bound by L1 (82 % busy).
// RS x CS: the part of the 8 x 8 block that exists (4 or 8 rows and columns):
// fewer accumulators leave registers for loads in flight (4 x 8: 31 us with
// three CTAs an SM and spills, 28 with two steps in flight, 27 with four and
// two CTAs an SM, the reduction included).
template <typename T, int RS, int CS>
__global__ void __launch_bounds__(256, skinny::thin_ctas<T>(RS, CS))
    thin_kernel(const T* __restrict__ A, int64_t lda, const T* __restrict__ B, int64_t ldb, T* out, int64_t ldo,
                int m, int n, int k, int64_t kchunk, int groups_n, T alpha, T beta, int epi, int partial,
                int64_t split_stride) {
  constexpr int S = skinny::kThin;
  constexpr int VEC = Vec<T>::n;
  constexpr int KU = RS * CS * (int)sizeof(T) <= 128 ? 4 : 2;
  using V = typename Vec<T>::type;
  const int gm = blockIdx.x / groups_n, gn = blockIdx.x - gm * groups_n;
  const int m0 = gm * S, n0 = gn * S;
  const int rows = min(RS, m - m0), cols = min(CS, n - n0);
  const int64_t kb = (int64_t)blockIdx.y * kchunk, ke = min((int64_t)k, kb + kchunk);
  const T* a0 = A + (int64_t)m0 * lda;
  const T* b0 = B + n0;
  T acc[RS][CS];
#pragma unroll
  for (int i = 0; i < RS; ++i)
#pragma unroll
    for (int j = 0; j < CS; ++j) acc[i][j] = T(0);
  for (int64_t k0 = kb + threadIdx.x; k0 < ke; k0 += 256 * KU) {
    T a[KU][RS], b[KU][CS];
#pragma unroll
    for (int u = 0; u < KU; ++u) {
      const int64_t kk = k0 + 256 * u;
      const bool in = kk < ke;
#pragma unroll
      for (int i = 0; i < RS; ++i) a[u][i] = in && i < rows ? a0[(int64_t)i * lda + kk] : T(0);
      const T* brow = b0 + kk * ldb;
#pragma unroll
      for (int h = 0; h < CS / VEC; ++h) {
        if (in && (h + 1) * VEC <= cols) {  // n0 % 8 == 0 and 16-byte rows
          const V v = *reinterpret_cast<const V*>(brow + h * VEC);
          const T* pv = reinterpret_cast<const T*>(&v);
#pragma unroll
          for (int e = 0; e < VEC; ++e) b[u][h * VEC + e] = pv[e];
        } else {
#pragma unroll
          for (int e = 0; e < VEC; ++e) b[u][h * VEC + e] = in && h * VEC + e < cols ? brow[h * VEC + e] : T(0);
        }
      }
    }
#pragma unroll
    for (int u = 0; u < KU; ++u)
#pragma unroll
      for (int i = 0; i < RS; ++i)
#pragma unroll
        for (int j = 0; j < CS; ++j) acc[i][j] = fma(a[u][i], b[u][j], acc[i][j]);
  }
  // Fixed-order reduction: within each warp every step halves the outputs a
  // lane keeps (ending with one or two consecutive ones, or, for fewer outputs
  // than lanes, one that several lanes hold), then warps 0..7 in order.
  constexpr int OUT = RS * CS;
  using Wide = decltype(widen(T(0)));
  __shared__ Wide red[8][OUT];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  T v[OUT];
#pragma unroll
  for (int i = 0; i < OUT; ++i) v[i] = acc[i / CS][i % CS];
  int first = 0;  // the output v[0] (w[0]) is the sum of
#pragma unroll
  for (int off = 16, half = OUT / 2; off > 2; off >>= 1, half >>= 1) {
    const bool up = (lane & off) != 0;
    if (up) first += half;
#pragma unroll
    for (int i = 0; i < half; ++i) {
      const T keep = up ? v[i + half] : v[i], send = up ? v[i] : v[i + half];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
    }
  }
  Wide w[OUT / 8];
#pragma unroll
  for (int i = 0; i < OUT / 8; ++i) w[i] = widen(v[i]);
#pragma unroll
  for (int off = 2, half = OUT / 16; off > 0; off >>= 1, half >>= 1) {
    if (half > 0) {
      const bool up = (lane & off) != 0;
      if (up) first += half;
#pragma unroll
      for (int i = 0; i < half; ++i) {
        const Wide keep = up ? w[i + half] : w[i], send = up ? w[i] : w[i + half];
        w[i] = add(keep, shfl_xor(send, off));
      }
    } else {
      w[0] = add(w[0], shfl_xor(w[0], off));
    }
  }
  if constexpr (OUT == 64) red[warp][first + 1] = w[1];
  red[warp][first] = w[0];
  __syncthreads();
  if (threadIdx.x < OUT) {
    const int i = threadIdx.x / CS, j = threadIdx.x % CS;
    Wide sum = red[0][threadIdx.x];
#pragma unroll
    for (int q = 1; q < 8; ++q) sum = add(sum, red[q][threadIdx.x]);
    const T s = narrow(sum);
    if (i < rows && j < cols) {
      const int64_t r = m0 + i, c = n0 + j;
      if (partial) {
        out[(int64_t)blockIdx.y * split_stride + r * ldo + c] = s;
      } else {
        T* o = out + r * ldo + c;
        *o = apply_epi(combine(s, alpha, beta, o), epi);
      }
    }
  }
}

// Reduction of many splits for few outputs: one warp per output element,
// lanes sum splits lane, lane + 32, ... in order, then a fixed butterfly --
// deterministic, and not serialised on load latency like a sequential sum
// over hundreds of splits would be.
template <typename T>
__global__ void __launch_bounds__(256)
    thin_reduce_kernel(const T* __restrict__ ws, int64_t split_stride, int64_t ldw, int splits, T* C, int64_t ldc,
                       int m, int n, T alpha, T beta, int epi) {
  const int64_t o = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (o >= (int64_t)m * n) return;
  const int64_t r = o / n, c = o - r * n;
  const T* w = ws + r * ldw + c;
  auto sum = widen(T(0));
  int z = lane;
  for (; z + 32 * 7 < splits; z += 32 * 8) {  // loads of a batch issued before its adds (order kept)
    T v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = w[(int64_t)(z + 32 * j) * split_stride];
#pragma unroll
    for (int j = 0; j < 8; ++j) sum = add(sum, widen(v[j]));
  }
  for (; z < splits; z += 32) sum = add(sum, widen(w[(int64_t)z * split_stride]));
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) sum = add(sum, shfl_xor(sum, off));
  const T s = narrow(sum);
  if (lane == 0) {
    T* po = C + r * ldc + c;
    *po = apply_epi(combine(s, alpha, beta, po), epi);
  }
}

SkinnyPlan plan_skinny(int64_t m, int64_t n, int64_t k, int dtype_bytes, int split_k, int tile, double beta, int sms) {
  SkinnyPlan p{};
  if (tile == 1 || tile == 2 || m <= 0 || n <= 0 || k <= 0) return p;  // tile ids 1, 2: always the tile kernel
  const int vec = 16 / dtype_bytes;
  if (k <= skinny::kMaxSmallK) {
    p.kind = 1;
    p.splits = 1;
    // 4 x (256 vec) blocks when M <= 4, 8 x (128 vec) when M <= 8, else 64 x
    // (64 vec).  The second in two groups of four rows, which both read B and
    // are twice as many: once they exceed a wave, 8 rows a thread in blocks of
    // twice the columns (B200, beta 0: 5 x 361,026 x 2 FP32 5.7 us in groups,
    // 4.9 so; 5 x 361,026 x 13 FP64 12.8 and 10.2; 8 x 2,500,000 x 13 FP32 51.6
    // and 48.7).  FP32 that reads C has no registers left to load it ahead in
    // that form, so it takes it only while it saves a wave (5 x 600,000 x 13,
    // beta 0.5, 11.5 us in groups, 8 x 1,000,000 x 16 23.7 in groups and 27).
    p.tile_m = m <= skinny::kThin ? skinny::kThin : 64;
    const bool whole = m > 4 && m <= skinny::kThin && ceil_div(n, 128 * vec) > 4 * (int64_t)sms &&
                       (dtype_bytes == 8 || beta == 0.0 || ceil_div(n, 256 * vec) <= 4 * (int64_t)sms);
    p.tile_n = m <= 4 || whole ? 256 * vec : m <= skinny::kThin ? 128 * vec : 64 * vec;
    return p;
  }
  if (m > skinny::kThin && n > skinny::kThin) return p;
  p.kind = 2;
  p.tile_m = p.tile_n = skinny::kThin;
  const int64_t groups = ceil_div(m, skinny::kThin) * ceil_div(n, skinny::kThin);
  // One wave of resident CTAs; whole waves more, up to four CTAs an SM, while a
  // thread would add up more than 64 (FP64: 48) products in a row (8 x 16 x
  // 3,000,000 in one wave, 79 and 158: rms error 1.03 and 1.45 times that of
  // four CTAs an SM without the wider sums; 0.77 and 0.71 so).
  const int ctas = dtype_bytes == 4 ? skinny::thin_ctas<float>(skinny::thin_side(m), skinny::thin_side(n))
                                    : skinny::thin_ctas<double>(skinny::thin_side(m), skinny::thin_side(n));
  int64_t splits = split_k > 0 ? split_k : ceil_div(ctas * (int64_t)sms, groups);
  for (int waves = 2; split_k <= 0 && waves * ctas <= 4 && ceil_div(k, splits) > (dtype_bytes == 4 ? 64 : 48) * 256; waves *= 2)
    splits = ceil_div(waves * ctas * (int64_t)sms, groups);
  splits = std::max<int64_t>(1, std::min<int64_t>({splits, ceil_div(k, 256), 65535}));
  p.kchunk = round_up(ceil_div(k, splits), 32);  // whole 128-byte (FP64: 256) lines per split
  p.splits = (int)ceil_div(k, p.kchunk);
  p.ldw = round_up(n, vec);
  p.ws_bytes = p.splits > 1 ? (size_t)p.splits * (size_t)m * (size_t)p.ldw * dtype_bytes : 0;
  return p;
}

template <typename T>
cudaError_t launch_skinny(const SkinnyPlan& pl, const T* A, int64_t lda, const T* B, int64_t ldb, T* C, int64_t ldc,
                          int m, int n, int k, double alpha, double beta, int epi, void* ws, int sms,
                          cudaStream_t st) {
  if (pl.kind == 1) {
    const int tiles_n = (int)ceil_div(n, pl.tile_n);
    const int64_t tiles = ceil_div(m, pl.tile_m) * (int64_t)tiles_n;
    const int64_t grid = std::max<int64_t>(1, std::min<int64_t>(tiles, (int64_t)sms * 8));
    // 8 rows a thread: three rows of B in flight leave registers for three CTAs
    // an SM.  FP32 blocks that fit at once only as four, and those of several
    // waves, take four CTAs and one or two rows (5 x 600,000 x 13, beta 0.5, 9.7
    // us with one, 11.0 with two, 12.1 as three CTAs).
    constexpr bool kF32 = sizeof(T) == 4;
    const int64_t per_sm = ceil_div(tiles, (int64_t)sms);
    auto* kernel = pl.tile_m != skinny::kThin     ? smallk_kernel<T, 4, 16, 2, 1>
                   : m <= 4                       ? smallk_kernel<T, 1, 4, 4, 4>
                   : pl.tile_n == 128 * Vec<T>::n ? smallk_kernel<T, 2, 4, 4, 4>
                   : !kF32 || per_sm <= 3         ? smallk_kernel<T, 1, 8, 3, 3>
                   : per_sm <= 4                  ? smallk_kernel<T, 1, 8, kF32 ? 4 : 3, kF32 ? 1 : 3>
                                                  : smallk_kernel<T, 1, 8, kF32 ? 4 : 3, kF32 ? 2 : 3>;
    kernel<<<(unsigned)grid, 256, 0, st>>>(A, lda, B, ldb, C, ldc, m, n, k, (T)alpha, (T)beta, epi, tiles_n, tiles);
    return cudaGetLastError();
  }
  const int groups_n = (int)ceil_div(n, skinny::kThin);
  const int64_t groups = ceil_div(m, skinny::kThin) * (int64_t)groups_n;
  const dim3 grid((unsigned)groups, (unsigned)pl.splits);
  const int64_t stride = (int64_t)m * pl.ldw;
  const bool partial = pl.splits > 1;
  T* w = static_cast<T*>(ws);
  auto* kernel = m <= 4 ? (n <= 4 ? thin_kernel<T, 4, 4> : thin_kernel<T, 4, 8>)
                        : (n <= 4 ? thin_kernel<T, 8, 4> : thin_kernel<T, 8, 8>);
  kernel<<<grid, 256, 0, st>>>(A, lda, B, ldb, partial ? w : C, partial ? pl.ldw : ldc, m, n, k, pl.kchunk, groups_n,
                               (T)alpha, (T)beta, epi, partial ? 1 : 0, stride);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess || !partial) return e;
  if (pl.splits >= 32 && (int64_t)m * n <= (int64_t)sms * 64) {
    thin_reduce_kernel<T><<<(unsigned)ceil_div((int64_t)m * n, 8), 256, 0, st>>>(w, stride, pl.ldw, pl.splits, C, ldc,
                                                                                 m, n, (T)alpha, (T)beta, epi);
    return cudaGetLastError();
  }
  return simt::launch_reduce<T>(w, stride, pl.ldw, pl.splits, C, ldc, m, n, alpha, beta, epi, sms, st);
}

template cudaError_t launch_skinny<float>(const SkinnyPlan&, const float*, int64_t, const float*, int64_t, float*,
                                          int64_t, int, int, int, double, double, int, void*, int, cudaStream_t);
template cudaError_t launch_skinny<double>(const SkinnyPlan&, const double*, int64_t, const double*, int64_t, double*,
                                           int64_t, int, int, int, double, double, int, void*, int, cudaStream_t);

}  // namespace cucosma

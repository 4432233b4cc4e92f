// split.cu -- operand pre-passes of the tensor-core precision paths.
//
// BF16 split (BF16x3 / BF16x6 SGEMM): every FP32 entry x becomes terms
// t0 + t1 (+ t2) with t_i = RN_bf16(x - t0 - ... - t_{i-1}); each residual
// subtraction is exact in FP32.  A (M x K, row-major) keeps its layout;
// B (K x N, row-major) is written transposed (N x K) so that both operands
// are K-major for the tensor cores.  Planes: [nterms][rows][kpad].
//
// Ozaki slicing (INT8 DGEMM): per row of A / per column of B the exponent
// e with |x| < 2^e over the row / column; x * 2^-e is cut into s signed
// 7-bit integer slices q_t = trunc(r * 2^7), r <- r * 2^7 - q_t, exact in
// FP64.  Slices of A rows are stored packed (packed_index), those of B
// columns stacked (stacked_index); kpad = K rounded up to the 32-wide k-block.
//
// All pre-passes are HBM-bound elementwise / transpose kernels.
#include <cuda_bf16.h>

#include "split.cuh"
#include "split_device.cuh"
#include "split_tiles.cuh"

namespace cucosma {

// ------------------------------------------------------------------ BF16
// Every split a call needs in one launch (A and B of a GEMM; G, B and A of a
// backward pass): the blocks of the jobs follow one another.  HBM-bound at
// large sizes, launch-bound at small ones.  64 registers, so that four blocks
// an SM keep their loads in flight; a tile's loads (and Y's) are all issued
// before the first is used.  B200, against one launch per operand: 8192 x
// 8192 A and B to three planes 219 -> 208 us (6.4 TB/s), 4096 x 4096 to two
// 44.4 -> 40.5, 1234 x 777 and 777 x 1111 6.3 -> 4.2 and one launch less; the
// backward pass's four splits at 4096^3, two planes, sigmoid, 110 -> 84 us.
template <int NT>
__global__ void __launch_bounds__(256, 4) split_bf16_kernel(const __grid_constant__ SplitJobs jobs) {
  __shared__ __align__(16) float tile[64 * 64];
  pdl_trigger();
  int b = blockIdx.x, ji = 0;
  while (ji + 1 < jobs.count && b >= jobs.job[ji].blocks) b -= jobs.job[ji++].blocks;
  const SplitJob& j = jobs.job[ji];
  if (j.out_c == nullptr) {
    split_rows_unit<NT>(j, (int64_t)b * 8 + (threadIdx.x >> 5));
  } else {
    split_cols_tile<NT>(j, b / j.tiles_n, b % j.tiles_n, tile);
  }
}

// ----------------------------------------------------------------- Ozaki
// Exponents start at this sentinel; all-zero columns and long rows keep it
// until the slicing turns it into exp_of(0) = 0.
constexpr int32_t kExpSentinel = (int32_t)0x80808080;

// Column exponents of B (K x N): a block covers 64 rows of K and 512 columns
// (two per thread, 16-byte loads).  Each block's column maxima enter eb by
// atomicMax of their exponents -- exact, since the exponent of a maximum is
// the maximum of the exponents (frexp is monotonic in |x|); zero maxima stay
// out so that they cannot raise a column's exponent.
__device__ __forceinline__ void ozaki_col_exp_block(const double* __restrict__ B, int64_t ldb, int krows, int ncols,
                                                    int32_t* eb, int bx, int by) {
  const int c = (bx * 256 + threadIdx.x) * 2;
  const int k0 = by * 64, k1 = min(krows, k0 + 64);
  if (c >= ncols) return;
  double m0 = 0.0, m1 = 0.0;
  if (c + 1 < ncols) {
#pragma unroll 8
    for (int k = k0; k < k1; ++k) {
      const double2 v = *reinterpret_cast<const double2*>(B + (int64_t)k * ldb + c);  // c even, 16-byte rows
      m0 = fmax(m0, fabs(v.x));
      m1 = fmax(m1, fabs(v.y));
    }
  } else {
    for (int k = k0; k < k1; ++k) m0 = fmax(m0, fabs(B[(int64_t)k * ldb + c]));
  }
  if (m0 != 0.0) atomicMax(&eb[c], exp_of(m0));
  if (c + 1 < ncols && m1 != 0.0) atomicMax(&eb[c + 1], exp_of(m1));
}

// A rows of up to kRowRegK padded columns -> row exponents and packed
// slices: a 256-thread block per row.  The row is read once into registers
// (4 consecutive columns per thread and step, two 16-byte loads), the
// maximum is reduced across the block, and the slices are cut from the
// registers; a thread's 4 columns give one 4-byte store per slice.  With
// rowsum, also the row's magnitude sum sum_k floor(|a_rk| 2^(30 - e_r))
// (integer, so exact and order-free) into rowsum[r].  Longer rows take the
// chunked kernels below.
constexpr int kRowSteps = 8;                    // steps of 1024 columns held in registers
constexpr int kRowRegK = kRowSteps * 1024;
static_assert(kRowRegK == kOzakiRowChunk, "row chunk");

__device__ __forceinline__ void load4(const double* __restrict__ src, int c, int cols, double (&v)[4]) {
  if (c + 4 <= cols) {
    const double2 v0 = *reinterpret_cast<const double2*>(src + c);  // c % 4 == 0, 16-byte rows
    const double2 v1 = *reinterpret_cast<const double2*>(src + c + 2);
    v[0] = v0.x, v[1] = v0.y, v[2] = v1.x, v[3] = v1.y;
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = c + j < cols ? src[c + j] : 0.0;
  }
}

// Slices of 4 consecutive columns of row r (one 4-byte store per slice);
// returns their magnitude sum (see slice4_packed).
template <int S>
__device__ __forceinline__ unsigned long long store_slices4(int8_t* __restrict__ out, int64_t r, int c, int64_t kpad,
                                                            const double (&v)[4], int e) {
  uint32_t w[S];
  const unsigned long long mag = slice4_packed<S>(v, e, w);
#pragma unroll
  for (int t = 0; t < S; ++t) *reinterpret_cast<uint32_t*>(out + packed_index<S>(r, c, kpad, t)) = w[t];
  return mag;
}

template <int S>
__device__ __forceinline__ void ozaki_rows_block(const double* __restrict__ A, int64_t lda, int rows, int cols,
                                                 int64_t kpad, int32_t* __restrict__ ea, int8_t* __restrict__ out,
                                                 unsigned long long* __restrict__ rowsum, int b, int blocks) {
  const bool stats = rowsum != nullptr;
  __shared__ double red[8];
  __shared__ unsigned long long red_sum[8];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int r = b; r < rows; r += blocks) {
    const double* src = A + (int64_t)r * lda;
    double v[kRowSteps][4];
    double m = 0.0;
#pragma unroll
    for (int j = 0; j < kRowSteps; ++j) {
      const int c = (tid + 256 * j) * 4;
      if (c < kpad) {
        load4(src, c, cols, v[j]);
      } else {
#pragma unroll
        for (int q = 0; q < 4; ++q) v[j][q] = 0.0;
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) m = fmax(m, fabs(v[j][q]));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (lane == 0) red[warp] = m;
    __syncthreads();
    m = red[0];
#pragma unroll
    for (int w = 1; w < 8; ++w) m = fmax(m, red[w]);
    __syncthreads();  // red is reused by the next row
    const int e = exp_of(m);
    if (tid == 0) ea[r] = e;
    unsigned long long sum = 0;
#pragma unroll
    for (int j = 0; j < kRowSteps; ++j) {
      const int c = (tid + 256 * j) * 4;
      if (c < kpad) {
        const unsigned long long mg = store_slices4<S>(out, r, c, kpad, v[j], e);
        if (stats) sum += mg;
      }
    }
    if (stats) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      if (lane == 0) red_sum[warp] = sum;
      __syncthreads();
      if (tid == 0) {
        unsigned long long t = 0;
#pragma unroll
        for (int w = 0; w < 8; ++w) t += red_sum[w];
        rowsum[r] = t;
      }
      __syncthreads();  // red_sum is reused by the next row
    }
  }
}

// Rows longer than kRowRegK in chunks of kRowRegK columns (grid.x chunks,
// rows over grid.y), so that a few long rows still fill the GPU.  The first
// kernel takes each chunk's maximum into ea[r] by atomicMax of its exponent
// (ea starts at kExpSentinel; the exponent of a maximum is the maximum of
// the exponents, so this is exact); the second cuts the chunk's slices and
// adds its magnitude sum into rowsum[r] (integer atomics: exact and
// independent of the order of the blocks).  Rows that are all zero keep the
// sentinel until the second kernel's first chunk turns it into 0; every
// block reads the sentinel as 0.
__device__ __forceinline__ void ozaki_row_exp_block(const double* __restrict__ A, int64_t lda, int rows, int cols,
                                                    int32_t* __restrict__ ea, int chunk, int r0, int rstep) {
  __shared__ double red[8];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int c0 = chunk * kRowRegK;
  for (int r = r0; r < rows; r += rstep) {
    const double* src = A + (int64_t)r * lda;
    double m = 0.0;
#pragma unroll
    for (int j = 0; j < kRowSteps; ++j) {
      const int c = c0 + (tid + 256 * j) * 4;
      if (c < cols) {
        double w[4];
        load4(src, c, cols, w);
#pragma unroll
        for (int q = 0; q < 4; ++q) m = fmax(m, fabs(w[q]));
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (lane == 0) red[warp] = m;
    __syncthreads();
    m = red[0];
#pragma unroll
    for (int w = 1; w < 8; ++w) m = fmax(m, red[w]);
    __syncthreads();  // red is reused by the next row
    if (tid == 0 && m != 0.0) atomicMax(&ea[r], exp_of(m));
  }
}

template <int S>
__device__ __forceinline__ void ozaki_row_slice_block(const double* __restrict__ A, int64_t lda, int rows, int cols,
                                                      int64_t kpad, int32_t* __restrict__ ea, int8_t* __restrict__ out,
                                                      unsigned long long* __restrict__ rowsum, int chunk, int r0,
                                                      int rstep) {
  __shared__ unsigned long long red_sum[8];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int c0 = chunk * kRowRegK;
  for (int r = r0; r < rows; r += rstep) {
    const double* src = A + (int64_t)r * lda;
    int e = ea[r];
    if (e == kExpSentinel) {
      e = 0;
      if (chunk == 0 && tid == 0) ea[r] = 0;
    }
    unsigned long long sum = 0;
#pragma unroll
    for (int j = 0; j < kRowSteps; ++j) {
      const int c = c0 + (tid + 256 * j) * 4;
      if (c < kpad) {
        double w[4];
        load4(src, c, cols, w);
        const unsigned long long mg = store_slices4<S>(out, r, c, kpad, w, e);
        if (rowsum) sum += mg;
      }
    }
    if (rowsum) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      if (lane == 0) red_sum[warp] = sum;
      __syncthreads();
      if (tid == 0) {
        unsigned long long t = 0;
#pragma unroll
        for (int w = 0; w < 8; ++w) t += red_sum[w];
        if (t) atomicAdd(&rowsum[r], t);
      }
      __syncthreads();  // red_sum is reused by the next row
    }
  }
}

// B (K x N) -> stacked slices of its columns, through a 64 (k) x 64 (n)
// shared-memory tile (two 32-wide k-blocks: eight 16-byte loads per thread
// in flight before the barrier).  Loads: 16 lanes cover 64 doubles of a row
// of B.  Stores, per k-block: a lane slices 4 consecutive k of one column
// into one 4-byte store per slice; 8 lanes cover a column's 32 bytes and a
// warp 4 adjacent columns (128 contiguous bytes per slice).  The second
// k-block of the last tile may lie past kpad and is then skipped.
// Also finishes the column exponents (the blocks of the first k-tile turn
// the all-zero columns' sentinel into exp_of(0) = 0; every block reads the
// sentinel as 0) and, with colsum, adds each column's fixed-point magnitude
// sum sum_k floor(|b_kn| 2^(30 - e_n)) by integer atomics (exact, so the
// totals do not depend on the order of the blocks).
constexpr int kColTileK = 64;

template <int S>
__device__ __forceinline__ void ozaki_slice_cols_block(const double* __restrict__ B, int64_t ldb, int krows, int ncols,
                                                       int64_t kpad, int32_t* __restrict__ eb, int8_t* __restrict__ out,
                                                       unsigned long long* __restrict__ colsum, int bx, int by) {
  __shared__ double tile[kColTileK][65];
  const int k0 = by * kColTileK, n0 = bx * 64, t = threadIdx.x;
#pragma unroll
  for (int p = 0; p < kColTileK / 16; ++p) {
    const int i = p * 16 + t / 16, c = (t % 16) * 4;
    const int k = k0 + i, n = n0 + c;
    double v[4] = {0.0, 0.0, 0.0, 0.0};
    if (k < krows) {
      const double* src = B + (int64_t)k * ldb + n;
      if (n + 4 <= ncols) {
        const double2 v0 = *reinterpret_cast<const double2*>(src);
        const double2 v1 = *reinterpret_cast<const double2*>(src + 2);
        v[0] = v0.x, v[1] = v0.y, v[2] = v1.x, v[3] = v1.y;
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] = n + j < ncols ? src[j] : 0.0;
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) tile[i][c + j] = v[j];
  }
  __syncthreads();
#pragma unroll
  for (int p = 0; p < kColTileK / 16; ++p) {
    const int half = p >> 1;  // k-block of the tile
    const int item = (p & 1) * 256 + t, nl = item / 8, kq = item % 8;
    const int n = n0 + nl, kl = half * 32 + kq * 4, k = k0 + kl;
    if (k0 + half * 32 >= kpad) break;  // past the last k-block (uniform over the block)
    unsigned long long part = 0;
    if (n < ncols) {
      int e = eb[n];
      if (e == kExpSentinel) {
        e = 0;
        if (by == 0 && kl == 0) eb[n] = 0;
      }
      const double v[4] = {tile[kl][nl], tile[kl + 1][nl], tile[kl + 2][nl], tile[kl + 3][nl]};
      uint32_t w[S];
      const unsigned long long mg = slice4_packed<S>(v, e, w);
#pragma unroll
      for (int s_ = 0; s_ < S; ++s_) *reinterpret_cast<uint32_t*>(out + stacked_index<S>(n, k, ncols, s_)) = w[s_];
      if (colsum) part = mg;
    }
    if (colsum) {
      // the 8 lanes of a column are consecutive: reduce over them
#pragma unroll
      for (int o = 1; o < 8; o <<= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
      if (kq == 0 && n < ncols && part) atomicAdd(&colsum[n], part);
    }
  }
}

// The pre-pass of both operands in three launches (either operand can be left
// out: its block count is 0): the exponents and sums at their start values;
// B's column exponents beside A's rows (short rows complete, long rows'
// exponents); B's slices beside long rows' slices.  Replaces six memsets and
// four kernels in a row (B200, whole calls: 256^3 60 -> 46 us, 2624 x 511 x 395
// 113 -> 94, 2000^3 338 -> 308).  The slicing is bound by the integer ALUs, the
// exponents by HBM: B's exponents run beside A's rows.
struct OzakiPrep {
  const double* A;
  int64_t lda;
  int m;
  const double* B;
  int64_t ldb;
  int n, k;
  int64_t kpad;
  int32_t *ea, *eb;
  int8_t *sa, *sb;
  unsigned long long *rowsum, *colsum;  // null: no sums
  OzakiStats* stats;                    // null: not adaptive
  int a_chunks;                         // 0: short rows
  int b1, a1, b2, a2;                   // blocks of B and A in the second and third launch
  int tiles_exp, tiles_n;               // blocks across N of B's exponents and slices
  int do_a, do_b;
};

__global__ void __launch_bounds__(256) ozaki_init_kernel(const __grid_constant__ OzakiPrep p) {
  pdl_trigger();
  const int i0 = blockIdx.x * 256 + threadIdx.x, step = gridDim.x * 256;
  if (p.do_b)
    for (int i = i0; i < p.n; i += step) {
      p.eb[i] = kExpSentinel;
      if (p.colsum) p.colsum[i] = 0;
    }
  if (p.do_a)
    for (int i = i0; i < p.m; i += step) {
      p.ea[i] = kExpSentinel;
      if (p.rowsum) p.rowsum[i] = 0;
    }
  if (p.stats && i0 == 0) {
    if (p.do_b) p.stats->min_col = ~0ull;
    if (p.do_a) {  // min_row, done_blocks and choice restart for every A (min_col belongs to B)
      p.stats->min_row = ~0ull;
      p.stats->done_blocks = 0;
      p.stats->choice = -1;
    }
  }
}

template <int S>
__global__ void __launch_bounds__(256) ozaki_prep1_kernel(const __grid_constant__ OzakiPrep p) {
  pdl_trigger();
  pdl_wait();
  const int b = blockIdx.x;
  if (b < p.b1) {
    ozaki_col_exp_block(p.B, p.ldb, p.k, p.n, p.eb, b % p.tiles_exp, b / p.tiles_exp);
  } else if (p.a_chunks == 0) {
    ozaki_rows_block<S>(p.A, p.lda, p.m, p.k, p.kpad, p.ea, p.sa, p.rowsum, b - p.b1, p.a1);
  } else {
    const int i = b - p.b1;
    ozaki_row_exp_block(p.A, p.lda, p.m, p.k, p.ea, i % p.a_chunks, i / p.a_chunks, p.a1 / p.a_chunks);
  }
}

template <int S>
__global__ void __launch_bounds__(256) ozaki_prep2_kernel(const __grid_constant__ OzakiPrep p) {
  pdl_trigger();
  pdl_wait();
  const int b = blockIdx.x;
  if (b < p.b2) {
    ozaki_slice_cols_block<S>(p.B, p.ldb, p.k, p.n, p.kpad, p.eb, p.sb, p.colsum, b % p.tiles_n, b / p.tiles_n);
  } else {
    const int i = b - p.b2;
    ozaki_row_slice_block<S>(p.A, p.lda, p.m, p.k, p.kpad, p.ea, p.sa, p.rowsum, i % p.a_chunks, i / p.a_chunks,
                             p.a2 / p.a_chunks);
  }
}

// Minima of the row and column magnitude sums over the nonzero rows and
// columns into stats->min_row / min_col; the last block to finish then
// makes the path choice (see ozaki_choice) from both minima.
__device__ __forceinline__ unsigned long long block_min_nonzero(const unsigned long long* __restrict__ v, int count,
                                                                unsigned long long* red) {
  unsigned long long m = ~0ull;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
    const unsigned long long x = v[i];
    if (x != 0 && x < m) m = x;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long w = __shfl_xor_sync(0xffffffffu, m, o);
    m = w < m ? w : m;
  }
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
  __syncthreads();
  for (int w = 0; w < 8; ++w) m = red[w] < m ? red[w] : m;
  __syncthreads();  // red is reused
  return m;
}

__global__ void __launch_bounds__(256) ozaki_decide_kernel(const unsigned long long* __restrict__ rowsum, int nrows,
                                                           const unsigned long long* __restrict__ colsum, int ncols,
                                                           int64_t k, OzakiStats* stats) {
  pdl_wait();
  __shared__ unsigned long long red[8];
  const unsigned long long mrow = block_min_nonzero(rowsum, nrows, red);
  const unsigned long long m = block_min_nonzero(colsum, ncols, red);
  if (threadIdx.x == 0) {
    if (mrow != ~0ull) atomicMin(&stats->min_row, mrow);
    if (m != ~0ull) atomicMin(&stats->min_col, m);
    __threadfence();
    const unsigned prev = atomicAdd(&stats->done_blocks, 1u);
    if (prev == gridDim.x - 1) {
      __threadfence();
      const unsigned long long mr = atomicAdd(&stats->min_row, 0ull), mc = atomicAdd(&stats->min_col, 0ull);
      stats->choice = ozaki_choice(mr, mc, k);
    }
  }
}

// ---------------------------------------------------------------- launch
static unsigned grid_for(int64_t work, int threads, int sms) {
  int64_t b = ceil_div(work, threads);
  b = std::min<int64_t>(b, (int64_t)sms * 16);
  return (unsigned)std::max<int64_t>(b, 1);
}

cudaError_t launch_split_bf16(SplitJobs& jobs, int nterms, cudaStream_t st) {
  int64_t total = 0;
  for (int i = 0; i < jobs.count; ++i) {
    SplitJob& j = jobs.job[i];
    int64_t blocks;
    if (j.out_c == nullptr) {
      blocks = ceil_div((int64_t)j.rows * ceil_div(j.kpad_r / 8, kRowUnit), 8);
    } else {
      j.tiles_n = (int)ceil_div(j.cols, 64);
      blocks = ceil_div(j.kpad_c, 64) * j.tiles_n;
    }
    total += blocks;
    if (total > INT32_MAX) return cudaErrorInvalidValue;
    j.blocks = (int)blocks;
  }
  if (nterms == 3)
    split_bf16_kernel<3><<<(unsigned)total, 256, 0, st>>>(jobs);
  else
    split_bf16_kernel<2><<<(unsigned)total, 256, 0, st>>>(jobs);
  return cudaGetLastError();
}

template <int S>
static cudaError_t prep_s(const OzakiPrep& p, cudaStream_t st) {
  cudaError_t e = cudaSuccess;
  if (p.b1 + p.a1 > 0)
    e = launch_after(true, ozaki_prep1_kernel<S>, dim3((unsigned)(p.b1 + p.a1)), 256, 0, st, p);
  if (e == cudaSuccess && p.b2 + p.a2 > 0)
    e = launch_after(true, ozaki_prep2_kernel<S>, dim3((unsigned)(p.b2 + p.a2)), 256, 0, st, p);
  return e;
}

cudaError_t launch_ozaki_prep(int s, const OzakiOperands& o, bool do_a, bool do_b, OzakiStats* stats, int sms,
                              cudaStream_t st, int* launches) {
  OzakiPrep p{};
  p.A = o.A;
  p.lda = o.lda;
  p.m = o.m;
  p.B = o.B;
  p.ldb = o.ldb;
  p.n = o.n;
  p.k = o.k;
  p.kpad = o.kpad;
  p.ea = o.ea;
  p.eb = o.eb;
  p.sa = o.sa;
  p.sb = o.sb;
  p.rowsum = stats ? o.rowsum : nullptr;
  p.colsum = stats ? o.colsum : nullptr;
  p.stats = stats;
  p.do_a = do_a;
  p.do_b = do_b;
  int64_t b1 = 0, b2 = 0, a1 = 0, a2 = 0;
  if (do_b) {
    p.tiles_exp = (int)ceil_div(o.n, 512);
    p.tiles_n = (int)ceil_div(o.n, 64);
    b1 = p.tiles_exp * ceil_div(o.k, 64);
    b2 = p.tiles_n * ceil_div(o.kpad, kColTileK);
  }
  if (do_a) {
    if (o.kpad <= kRowRegK) {
      a1 = std::max<int64_t>(1, std::min<int64_t>(o.m, (int64_t)sms * 8));
    } else {
      p.a_chunks = (int)ceil_div(o.kpad, kRowRegK);
      // rows over as many blocks per chunk as one launch takes
      const int64_t rows = std::min<int64_t>(o.m, std::max<int64_t>(1, ((int64_t)1 << 30) / p.a_chunks));
      a1 = a2 = rows * p.a_chunks;
    }
  }
  if (b1 + a1 > INT32_MAX || b2 + a2 > INT32_MAX) return cudaErrorInvalidValue;
  p.b1 = (int)b1;
  p.b2 = (int)b2;
  p.a1 = (int)a1;
  p.a2 = (int)a2;
  const int cells = std::max(do_a ? o.m : 0, do_b ? o.n : 0);
  const unsigned init_blocks = (unsigned)std::max<int64_t>(1, std::min<int64_t>(ceil_div(cells, 256), (int64_t)sms * 2));
  ozaki_init_kernel<<<init_blocks, 256, 0, st>>>(p);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  switch (s) {
    case 4: e = prep_s<4>(p, st); break;
    case 5: e = prep_s<5>(p, st); break;
    case 6: e = prep_s<6>(p, st); break;
    case 7: e = prep_s<7>(p, st); break;
    case 8: e = prep_s<8>(p, st); break;
    case 9: e = prep_s<9>(p, st); break;
    default: return cudaErrorInvalidValue;
  }
  *launches += 1 + (p.b1 + p.a1 > 0) + (p.b2 + p.a2 > 0);
  return e;
}

cudaError_t launch_ozaki_decide(const unsigned long long* rowsum, int m, const unsigned long long* colsum, int n,
                                int64_t k, OzakiStats* stats, int sms, cudaStream_t st) {
  const unsigned blocks =
      (unsigned)std::max<int64_t>(1, std::min<int64_t>(ceil_div(std::max(m, n), 256), (int64_t)sms * 2));
  return launch_after(true, ozaki_decide_kernel, dim3(blocks), 256, 0, st, rowsum, m, colsum, n, k, stats);
}

}  // namespace cucosma

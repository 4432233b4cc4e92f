// backward.cu -- gradients of the fused forward Y = epi(alpha * A*B + beta*C0).
//
// No counterpart in the reference (forward only; its sigmoid epilogue is the
// commented block at cuCOSMAV100.cuh:2472-2476).  With G = alpha * dY (.)
// epi'(Z), epi' = Y(1-Y) for the sigmoid, [Y > 0] for ReLU, 1 for none:
//   dA = G * B^T   (m x k)        dB = A^T * G   (k x n)
// Both products run on the tcgen05 BF16 kernel of the forward precision.  The
// transposed operands are never materialised: the split pre-pass writes the
// K-major planes each product needs straight from the saved operands --
//   dA: A-planes = rows of G (computed from dY and Y inside the split),
//       B-planes = rows of B itself (B^T's K-major layout is B);
//   dB: A-planes = columns of A (A^T, transposing split),
//       B-planes = columns of G (G^T, transposing split).
// Three launches: every plane in one split kernel (G is formed once and
// written in both layouts), then the two GEMMs, each product with its own
// part of the caller's workspace.  A workspace that holds only the larger
// product (half of what the query asks for) runs one product after the
// other in it.
#include <algorithm>

#include "../../include/cucosma.h"
#include "api_internal.cuh"
#include "split.cuh"

namespace cucosma {
namespace {

bool al16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

void sub_desc(const cucosma_gemm_desc* f, int64_t m, int64_t n, int64_t k, int64_t ldc, cucosma_gemm_desc* d) {
  cucosma_gemm_desc_init(d);
  d->m = m;
  d->n = n;
  d->k = k;
  d->lda = k;  // operand strides unused: the planes are prepared here
  d->ldb = n;
  d->ldc = ldc;
  d->dtype = CUCOSMA_R_32F;
  d->precision = f->precision;
  d->tile = f->tile;
  d->split_k = 0;
  d->alpha = 1.0;
  d->beta = 0.0;
}

size_t part_bytes(size_t b) { return (b + 255) & ~size_t(255); }

int xform_of(int epilogue) {
  return epilogue == CUCOSMA_EPILOGUE_SIGMOID ? kXformSigmoidGrad
         : epilogue == CUCOSMA_EPILOGUE_RELU  ? kXformReluGrad
                                               : kXformScale;
}

cucosma_status check_bwd(const cucosma_gemm_desc* f) {
  if (!f) return CUCOSMA_STATUS_INVALID_VALUE;
  if (f->m <= 0 || f->n <= 0 || f->k <= 0 || f->m > INT32_MAX || f->n > INT32_MAX || f->k > INT32_MAX)
    return CUCOSMA_STATUS_INVALID_VALUE;
  if (f->dtype != CUCOSMA_R_32F) return CUCOSMA_STATUS_NOT_SUPPORTED;
  if (f->precision != CUCOSMA_PRECISION_BF16X3 && f->precision != CUCOSMA_PRECISION_BF16X6)
    return CUCOSMA_STATUS_NOT_SUPPORTED;
  if (f->epilogue < 0 || f->epilogue > CUCOSMA_EPILOGUE_RELU || f->flags) return CUCOSMA_STATUS_INVALID_VALUE;
  return CUCOSMA_STATUS_SUCCESS;
}

}  // namespace
}  // namespace cucosma

using namespace cucosma;

extern "C" cucosma_status cucosma_gemm_backward_workspace_size(const cucosma_gemm_desc* f, size_t* bytes) {
  if (!bytes) return CUCOSMA_STATUS_INVALID_VALUE;
  cucosma_status s = check_bwd(f);
  if (s != CUCOSMA_STATUS_SUCCESS) return s;
  const DeviceInfo* di = device_info();
  if (!di) return CUCOSMA_STATUS_LAUNCH_FAILED;
  // Each product's plan as the backward call builds it: tuned, and with its
  // planes prepared here (never the fused-split kernel, which keeps none).
  // The planes of both exist at once, one part after the other, unless they
  // would take more than an eighth of the GPU's memory: gradients that size fit
  // with the larger product's planes alone, and forming G twice is then less
  // than a hundredth of the products' time.
  auto need = [&](int64_t m, int64_t n, int64_t k, int64_t ldc) {
    cucosma_gemm_desc d0, tuned;
    cucosma_plan_info pi;
    sub_desc(f, m, n, k, ldc, &d0);
    tc_plan_info(apply_tuning(&d0, &tuned, di), di, &pi, false);
    return part_bytes(pi.workspace_bytes);
  };
  const size_t da = need(f->m, f->k, f->n, f->k), db = need(f->k, f->n, f->m, f->n);
  *bytes = da + db <= di->mem_bytes / 8 ? da + db : std::max(da, db);
  return CUCOSMA_STATUS_SUCCESS;
}

extern "C" cucosma_status cucosma_gemm_backward(const cucosma_gemm_desc* f, const void* A, const void* B,
                                                const void* Y, int64_t ldy, const void* dY, int64_t lddy, void* dA,
                                                int64_t ldda, void* dB, int64_t lddb, void* workspace,
                                                size_t workspace_bytes, void* stream) {
  cucosma_status s = check_bwd(f);
  if (s != CUCOSMA_STATUS_SUCCESS) return s;
  const int64_t m = f->m, n = f->n, k = f->k;
  if (!dY || (!dA && !dB)) return CUCOSMA_STATUS_INVALID_VALUE;
  if (f->epilogue != CUCOSMA_EPILOGUE_NONE && (!Y || ldy < n)) return CUCOSMA_STATUS_INVALID_VALUE;
  if (lddy < n || (dA && (!B || f->ldb < n || ldda < k)) || (dB && (!A || f->lda < k || lddb < n)))
    return CUCOSMA_STATUS_INVALID_VALUE;
  auto bad16 = [](const void* p, int64_t ld) { return p && (!al16(p) || (ld * 4) % 16); };
  if (bad16(dY, lddy) || (f->epilogue != CUCOSMA_EPILOGUE_NONE && bad16(Y, ldy)) || (dA && bad16(B, f->ldb)) ||
      (dB && bad16(A, f->lda)) || bad16(dA, ldda) || bad16(dB, lddb))
    return CUCOSMA_STATUS_MISALIGNED;
  const DeviceInfo* di = device_info();
  if (!di) return CUCOSMA_STATUS_LAUNCH_FAILED;
  if (di->cc_major != 10 || di->cc_minor != 0) return CUCOSMA_STATUS_ARCH_MISMATCH;
  if (!workspace) return CUCOSMA_STATUS_WORKSPACE_TOO_SMALL;
  if (!al16(workspace)) return CUCOSMA_STATUS_MISALIGNED;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  uint8_t* w = static_cast<uint8_t*>(workspace);
  const int nt = f->precision == CUCOSMA_PRECISION_BF16X6 ? 3 : 2;
  const int xf = xform_of(f->epilogue);
  const float scale = (float)f->alpha;
  const float* fY = static_cast<const float*>(Y);
  const float* fdY = static_cast<const float*>(dY);
  // Each product's descriptor is resolved against the tuning cache once and
  // that one descriptor gives both the plan (plane offsets, partials region)
  // and the launch, so the two cannot disagree; the plans must fit the
  // caller's workspace (the cache may have changed since it was sized).
  struct Product {
    cucosma_gemm_desc d0, tuned;
    const cucosma_gemm_desc* d = nullptr;
    cucosma_plan_info pi;
    uint8_t* w = nullptr;
    size_t bytes = 0;  // its part of the workspace
  } pa, pb;
  auto resolve = [&](Product& p, int64_t pm, int64_t pn, int64_t pk, int64_t ldc) {
    sub_desc(f, pm, pn, pk, ldc, &p.d0);
    p.d = apply_tuning(&p.d0, &p.tuned, di);
    tc_plan_info(p.d, di, &p.pi, false);  // the planes are prepared here: never the fused kernel
    p.w = w;
    p.bytes = part_bytes(p.pi.workspace_bytes);
  };
  resolve(pa, m, k, n, ldda);  // dA (m x k) = G (m x n) * B^T: K' = n
  resolve(pb, k, n, m, lddb);  // dB (k x n) = A^T (k x m) * G (m x n): K' = m
  // (both, whichever gradients are asked for, as the query does)
  if (std::max(pa.pi.workspace_bytes, pb.pi.workspace_bytes) > workspace_bytes) return CUCOSMA_STATUS_WORKSPACE_TOO_SMALL;
  auto run = [&](bool da, bool db) -> cucosma_status {
    SplitJobs jobs{};
    SplitJob& g = jobs.add(fdY, lddy, (int)m, (int)n, da ? pa.w + pa.pi.off_a : nullptr, da ? pa.pi.kpad : 0,
                           db ? pb.w + pb.pi.off_b : nullptr, db ? pb.pi.kpad : 0);
    g.mode = xf;
    g.scale = scale;
    g.Y = f->epilogue != CUCOSMA_EPILOGUE_NONE ? fY : nullptr;
    g.ldy = ldy;
    if (da) jobs.rows(static_cast<const float*>(B), f->ldb, (int)k, (int)n, pa.w + pa.pi.off_b, pa.pi.kpad);
    if (db) jobs.cols(static_cast<const float*>(A), f->lda, (int)m, (int)k, pb.w + pb.pi.off_a, pb.pi.kpad);
    if (launch_split_bf16(jobs, nt, st) != cudaSuccess) return CUCOSMA_STATUS_LAUNCH_FAILED;
    note_launches(1);
    cucosma_status e = CUCOSMA_STATUS_SUCCESS;
    if (da) e = tc_gemm_ex(pa.d, nullptr, nullptr, dA, pa.w, workspace_bytes - (size_t)(pa.w - w), di, st, 0);
    if (db && e == CUCOSMA_STATUS_SUCCESS)
      e = tc_gemm_ex(pb.d, nullptr, nullptr, dB, pb.w, workspace_bytes - (size_t)(pb.w - w), di, st, 0);
    return e;
  };
  if (dA && dB && pa.bytes + pb.pi.workspace_bytes > workspace_bytes) {
    if ((s = run(true, false)) != CUCOSMA_STATUS_SUCCESS) return s;
    return run(false, true);
  }
  if (dA && dB) pb.w = w + pa.bytes;
  return run(dA != nullptr, dB != nullptr);
}

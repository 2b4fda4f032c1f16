// A LoRA layer's launches, forward and backward, in one call each: what an eager training step pays per launch is the interpreter's
// 25 to 35 us, several times what these kernels take at a few thousand tokens. Eager step of 1537 tokens, 28 layers, on one
// host: 29.0 ms with single calls, 22.6 ms.
#include <algorithm>

#include "host_util.cuh"
#include "pmetal_b200.h"

namespace pm {
namespace {

// Ways to cut a reduction over tokens with `tiles` output tiles and `nk` k blocks: an SM streams its operands at a fixed rate, so the
// launch takes waves * (blocks per split + a fixed cost per CTA); an empty last split is not allowed. The rule of _splits_for
// (ops/native.py), which serves the single products.
int token_splits(int tiles, int nk) {
  const int sms = num_sms();
  int best = 1;
  long long best_cost = -1;
  for (int s = 1; s <= std::min(nk, 64); ++s) {
    const int per = (nk + s - 1) / s;
    if (static_cast<long long>(s - 1) * per >= nk) continue;
    const long long cost = ((static_cast<long long>(tiles) * s + sms - 1) / sms) * (per + 6);
    if (best_cost < 0 || cost < best_cost) {
      best = s;
      best_cost = cost;
    }
  }
  return best;
}

}  // namespace
}  // namespace pm

using namespace pm;

// t = scale x a^T [M, 64], y = x w^T + t[:, segment] b_segment^T (+ residual). x: [M, K] rows ldx apart, w: [N, K] rows ldw apart, a: [nseg r, K],
// b: [N, r], y: [M, N], residual (nullable) rows ldr apart. bn: tile width; M > 128.
extern "C" int pm_lora_linear_fwd(const void* x, int ldx, const void* w, int ldw, const void* a, const void* b, const void* residual, int ldr,
                                  void* t, void* y, int M, int N, int K, const int* seg_end, int nseg, int r, float scale, int bn,
                                  int* status, cudaStream_t st) {
  int rc = pm_lora_tall(x, ldx, a, K, 0, nseg * r, t, 64, M, K, nullptr, scale, 0, status, st);
  if (rc) return rc;
  const int mode = nseg > 1 ? 1 : 0;
  if (M >= 256 && bn >= 128)
    return pm_gemm_bf16_2sm(x, 0, ldx, M, w, 0, ldw, N, t, 0, 64, 64, b, 0, r, N, y, 0, N, residual, ldr, M, N, K, r, 0, 1.f, 1, mode,
                            mode ? seg_end : nullptr, r, 0, nullptr, 0, 0, status, st);
  return pm_gemm_bf16(x, 0, ldx, M, w, 0, ldw, N, t, 0, 64, 64, b, 0, r, N, y, 0, N, residual, ldr, M, N, K, r, 0, 1.f, bn, 1, mode,
                      mode ? seg_end : nullptr, r, 0, nullptr, 0, nullptr, 0, nullptr, 0, 0, status, st);
}

// dt = scale dy b [M, 64], dx = dy w + dt a (dx null: left out), ga [nseg r, K] += dt^T x, gb [N, r] += dy^T t, both fp32. w: [N, K] (w_t 0) or its
// transpose [K, N] (w_t 1), rows ldw apart; bn: tile width of dx.
extern "C" int pm_lora_linear_bwd(const void* dy, int ldd, const void* w, int w_t, int ldw, const void* a, const void* b, const void* x, int ldx,
                                  const void* t, void* dt, void* dx, float* ga, float* gb, int M, int N, int K, const int* seg_end, int nseg,
                                  int r, float scale, int bn, int* status, cudaStream_t st) {
  const int nr = nseg * r, nk = (M + 63) / 64;
  int rc = pm_lora_tall(dy, ldd, b, r, 1, r, dt, 64, M, N, nseg > 1 ? seg_end : nullptr, scale, 0, status, st);
  if (rc) return rc;
  if (dx) {
    rc = M >= 256 && bn >= 128
             ? pm_gemm_bf16_2sm(dy, 0, ldd, M, w, !w_t, ldw, K, dt, 0, 64, 64, a, 1, K, K, dx, 0, K, nullptr, 0, M, K, N, nr, 0, 1.f, 1, 0, nullptr,
                                0, 0, nullptr, 0, 0, status, st)
             : pm_gemm_bf16(dy, 0, ldd, M, w, !w_t, ldw, K, dt, 0, 64, 64, a, 1, K, K, dx, 0, K, nullptr, 0, M, K, N, nr, 0, 1.f, bn, 1, 0, nullptr,
                            0, 0, nullptr, 0, nullptr, 0, nullptr, 0, 0, status, st);
    if (rc) return rc;
  }
  if ((rc = pm_gemm_bf16(x, 1, ldx, K, dt, 1, 64, 64, nullptr, 0, 0, 0, nullptr, 0, 0, 0, ga, 3, K, nullptr, 0, K, 64, M, 0, nr, 1.f, 64,
                         token_splits((K + 127) / 128, nk), 0, nullptr, 0, 0, nullptr, 0, nullptr, 0, nullptr, 0, 0, status, st)))
    return rc;
  const int mode = nseg > 1 ? 2 : 0;
  return pm_gemm_bf16(dy, 1, ldd, N, t, 1, 64, 64, nullptr, 0, 0, 0, nullptr, 0, 0, 0, gb, 2, r, nullptr, 0, N, 64, M, 0, r, 1.f, 64,
                      token_splits((N + 127) / 128, nk), mode, mode ? seg_end : nullptr, r, 0, nullptr, 0, nullptr, 0, nullptr, 0, 0, status, st);
}

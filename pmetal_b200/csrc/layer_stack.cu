// The cached forward of all layers of a dense decoder in one call: the host side of a prompt or of a decode step.
//
// A layer is eight or nine launches (norm, q|k|v, head norm + rope + cache append, attention, output projection, norm, gate|up, its
// unit, down).
// Issued one by one through the interpreter they cost about 35 us of host time each, 12 ms for 28 layers, whatever the
// number of tokens; issued here a launch costs 2 to 4 us. Nothing is allocated and nothing is kept between calls: the
// caller passes the layer pointers, a scratch buffer and the step's metadata.
//
// Up to 128 tokens the linear layers run on gemm_skinny.cu, and the norms are part of them: the projection that writes the residual
// stream also writes it times the next norm's weight, with the rows' sums of squares, and the next projection multiplies its sums
// by 1 / rms. That leaves six kernels, each launched with programmatic stream serialization (pdl.cuh). A decode step of 28
// layers: one row 898 us with norm kernels, 838 us without; 64 rows 1803, 1791 us. Above 128 tokens the tile GEMMs run.
#include <stdint.h>

#include <algorithm>

#include "host_util.cuh"
#include "pdl.cuh"
#include "pmetal_b200.h"

namespace pm {
namespace {

constexpr int kSkinnyRows = 128;

struct Stack {
  int T;
  float eps;
  int* status;
  cudaStream_t st;
  // more than kSkinnyRows tokens
  int tile(const void* x, int K, const void* w, int N, void* y, const void* res) const {
    const int bn = N >= 256 ? 256 : N >= 128 ? 128 : N >= 64 ? 64 : 32;
    if (T >= 256 && bn >= 128)
      return pm_gemm_bf16_2sm(x, 0, K, T, w, 0, K, N, nullptr, 0, 0, 0, nullptr, 0, 0, 0, y, 0, N, res, res ? N : 0, T, N, K, 0, 0, 1.f, 1,
                              0, nullptr, 0, 0, nullptr, 0, 0, status, st);
    return pm_gemm_bf16(x, 0, K, T, w, 0, K, N, nullptr, 0, 0, 0, nullptr, 0, 0, 0, y, 0, N, res, res ? N : 0, T, N, K, 0, 0, 1.f, bn, 1, 0,
                        nullptr, 0, 0, nullptr, 0, nullptr, 0, nullptr, 0, 0, status, st);
  }
  // up to kSkinnyRows: reads the pair (rows * norm weight, sums of squares in `parts` parts)
  int normed(const void* xw, const float* ss, int parts, int K, const void* w, int N, void* y, int swiglu) const {
    return pm_linear_skinny_norm(xw, K, w, K, y, N, nullptr, 0, T, N, K, swiglu, 1.f, 0, 1, ss, parts, eps, nullptr, nullptr, nullptr, status,
                                 st);
  }
  // writes the residual stream and, where a norm follows (nw), the next pair
  int residual(const void* x, int K, const void* w, int N, void* y, const void* res, const void* nw, void* yw, float* ss) const {
    return pm_linear_skinny_norm(x, K, w, K, y, N, res, N, T, N, K, 0, 1.f, 0, 1, nullptr, 0, 0.f, nw, nw ? yw : nullptr, nw ? ss : nullptr,
                                 status, st);
  }
};

}  // namespace
}  // namespace pm

using namespace pm;

// Bytes of scratch that pm_layer_stack needs for T tokens.
extern "C" long long pm_layer_stack_scratch(int T, int H, int hq, int hkv, int I, int n_split) {
  const long long d = 128, t = T;
  long long n = 0;
  auto add = [&](long long b) { n += (b + 255) / 256 * 256; };
  add(2 * t * H); add(T <= kSkinnyRows ? 4ll * 128 * ((H + 127) / 128) : 4 * t); add(2 * t * (hq + 2 * hkv) * d); add(2 * t * hq * d); add(2 * t * hkv * d); add(2 * t * hq * d);
  add(2 * t * H); add(2 * t * H); add(T <= kSkinnyRows ? 0 : 4 * t * I); add(2 * t * I);
  if (n_split > 1) { add(4ll * n_split * t * hq * d); add(8ll * n_split * t * hq); }
  return n;
}

// layers: n_layers rows of 12 pointers on the host: input norm, q|k|v weight, q norm, k norm (0: none), output weight, post norm,
// gate|up weight, down weight, key cache, value cache, key scales, value scales (0: bf16 cache, else int8). x: [T, H]; out: [T, H].
// route: attention through 0 pm_paged_attn_ex with n_split, 1 pm_paged_attn_tc, 2 pm_paged_decode. Returns the first launcher's error.
extern "C" int pm_layer_stack(const long long* layers, int n_layers, const void* x, void* out, void* scratch, long long scratch_bytes,
                              int T, int H, int hq, int hkv, int I, float eps, float scale, const float* cs, const float* sn,
                              const long long* slots, const int* block_table, const int* seq_lens, const int* q_start,
                              const int* q_lens, int num_seqs, int max_blocks, int num_blocks, int max_q, int route, int n_split,
                              int* status, cudaStream_t st) {
  if (T <= 0 || n_layers <= 0 || H % 8 || I % 8 || hkv <= 0 || hq % hkv) return -1;
  if (scratch_bytes < pm_layer_stack_scratch(T, H, hq, hkv, I, n_split) || (reinterpret_cast<uintptr_t>(scratch) & 15)) return -2;
  const long long d = 128;
  const int ld = (hq + 2 * hkv) * 128;
  char* at = static_cast<char*>(scratch);
  auto buf = [&](long long bytes) {
    void* b = at;
    at += (bytes + 255) / 256 * 256;
    return b;
  };
  void* y = buf(2ll * T * H);
  const bool few = T <= kSkinnyRows;
  const int parts = (H + 127) / 128;
  float* rstd = static_cast<float*>(buf(few ? 4ll * 128 * parts : 4ll * T));   // few tokens: the sums of squares
  char* qkv = static_cast<char*>(buf(2ll * T * ld));
  void* q = buf(2ll * T * hq * d);
  void* k = buf(2ll * T * hkv * d);
  void* o = buf(2ll * T * hq * d);
  void* h = buf(2ll * T * H);
  void* xa = buf(2ll * T * H);
  void* gu = buf(T <= kSkinnyRows ? 0 : 4ll * T * I);
  void* act = buf(2ll * T * I);
  float* part_o = n_split > 1 ? static_cast<float*>(buf(4ll * n_split * T * hq * d)) : nullptr;
  float* part_ml = n_split > 1 ? static_cast<float*>(buf(8ll * n_split * T * hq)) : nullptr;
  const Stack s{T, eps, status, st};
  const PdlScope scope(few);
  int rc;
  if (few && (rc = pm_skinny_prep(x, reinterpret_cast<void*>(layers[0]), y, rstd, T, H, st))) return rc;
  for (int l = 0; l < n_layers; ++l) {
    const long long* p = layers + 12ll * l;
    auto ptr = [&](int i) { return reinterpret_cast<void*>(p[i]); };
    const bool q8 = p[10] != 0;
    if (few) {
      if ((rc = s.normed(y, rstd, l ? parts : 1, H, ptr(1), ld, qkv, 0))) return rc;
    } else {
      if ((rc = pm_rmsnorm_fwd(x, nullptr, ptr(0), y, nullptr, rstd, T, H, eps, st))) return rc;
      if ((rc = s.tile(y, H, ptr(1), ld, qkv, nullptr))) return rc;
    }
    if (q8) {
      void* v = qkv + (hq + hkv) * d * 2;
      if ((rc = pm_qknorm_rope_fwd(qkv, ld, ptr(2), ptr(3), cs, sn, q, k, T, hq, hkv, eps, st))) return rc;
      if ((rc = pm_kv_append_q8(k, hkv * d, v, ld, ptr(8), ptr(9), static_cast<float*>(ptr(10)), static_cast<float*>(ptr(11)), slots, T,
                                hkv, st)))
        return rc;
    } else if ((rc = pm_qknorm_rope_cache(qkv, ld, ptr(2), ptr(3), cs, sn, q, ptr(8), ptr(9), slots, T, hq, hkv, eps, st))) {
      return rc;
    }
    float *ksc = static_cast<float*>(ptr(10)), *vsc = static_cast<float*>(ptr(11));
    rc = route == 2 ? pm_paged_decode(q, ptr(8), ptr(9), ksc, vsc, o, block_table, seq_lens, q_start, q_lens, num_seqs, max_blocks, num_blocks,
                                      max_q, hq, hkv, scale, 0, status, st)
         : route == 1 ? pm_paged_attn_tc(q, ptr(8), ptr(9), o, block_table, seq_lens, q_start, q_lens, num_seqs, max_blocks, num_blocks, T,
                                         max_q, hq, hkv, scale, status, st)
                      : pm_paged_attn_ex(q, ptr(8), ptr(9), o, block_table, seq_lens, q_start, q_lens, part_o, part_ml, num_seqs,
                                         max_blocks, T, max_q, hq, hkv, n_split, scale, 0, 0, ksc, vsc, st);
    if (rc) return rc;
    void* to = l == n_layers - 1 ? out : xa;
    if (few) {
      const void* next = l == n_layers - 1 ? nullptr : reinterpret_cast<void*>(p[12]);      // the next layer's input norm
      if ((rc = s.residual(o, hq * 128, ptr(4), H, h, x, ptr(5), y, rstd))) return rc;
      if ((rc = s.normed(y, rstd, parts, H, ptr(6), I, act, 1))) return rc;
      if ((rc = s.residual(act, I, ptr(7), H, to, h, next, y, rstd))) return rc;
    } else {
      if ((rc = s.tile(o, hq * 128, ptr(4), H, h, x))) return rc;
      if ((rc = pm_rmsnorm_fwd(h, nullptr, ptr(5), y, nullptr, rstd, T, H, eps, st))) return rc;
      if ((rc = s.tile(y, H, ptr(6), 2 * I, gu, nullptr))) return rc;
      if ((rc = pm_swiglu_fwd(gu, act, T, I, st))) return rc;
      if ((rc = s.tile(act, I, ptr(7), H, to, h))) return rc;
    }
    x = to;
  }
  return 0;
}

// Linear layers on a few token rows (decode batches, short prompts): Y[M, N] = alpha * X[M, K] W[N, K]^T (+ residual), M <= 128, or
// SwiGLU over the (gate, up) halves of W, on tcgen05.
//
// The work is one pass over the weights, so the weight rows are the 128-row A operand of the MMA and the tokens are its
// columns (16, 32, 64 or 128 of them): no tensor-core row is spent on padding and X is small enough to be fetched by every CTA.
// A layer's matrix gives only 8 to 48 such tiles; K is therefore cut over the CTAs of a cluster, which add their partial
// tiles through distributed shared memory (fixed order: the result does not change from run to run) and share the output rows.
//
// What bounds it: the chain of launch, first bytes, MMA, sum and store, 3 to 4 us, where the bytes of a layer's matrix take
// 1 us. `chain` = 1 therefore launches with programmatic stream serialization: the weight tiles are requested before the
// wait for the previous kernel (the caller vouches that no kernel still running writes the weights), so their fetch runs
// under the previous kernel's tail. Measured in a captured chain over cold weights (4096 x 1024, 1024 x 2048, 2 x 3072 x 1024 with
// SwiGLU, 1024 x 3072), 64 rows: 6.1, 5.6, 7.0, 6.6 us (tile GEMM with K split through a workspace: 7.9, 9.6, 11, 10.5 us);
// 1 row: 4.3, 3.6, 4.9, 4.3 us (mat-vec of gemv.cu: 5.1, 4.3, 6.1, 5.9 us).
#include <algorithm>

#include "gemm_pair.cuh"
#include "pdl.cuh"
#include "pmetal_b200.h"

namespace pm {

struct FewRowParams {
  __nv_bfloat16* y;
  const __nv_bfloat16* res;
  long long ldy, ldr;
  int M, N, K;
  int nkb, per, splits, stages, swiglu;
  float alpha;
  int* status;
  // RMSNorm around the product (nullable). In: x holds rows times the norm's weight, ss_in [parts_in][128] partial sums of squares of
  // the rows themselves, so that a row's 1 / rms is a factor of its sums. Out: the same pair for the next norm, y2 = y * nw_out and
  // the sum of squares of every column tile, ss_out [tiles][128].
  const float* ss_in;
  int parts_in;
  float eps;
  const __nv_bfloat16* nw_out;
  __nv_bfloat16* y2;
  float* ss_out;
};

constexpr int kSkW = 128 * 64 * 2;        // one k block of a weight tile: 16 KB

// Sum over the cluster and epilogue of this CTA's share of the token rows, one warp per row; all loads of a row are in flight
// together. Ends with this thread's arrival at the cluster barrier behind which the partial tiles may go away.
template <int kSplits>
__device__ __forceinline__ void skinny_finish(const FewRowParams& p, uint32_t part, int split, int n0, const float* s_rstd) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint32_t at[kSplits];
#pragma unroll
  for (int c = 0; c < kSplits; ++c) at[c] = kSplits > 1 ? map_to_cta(part, c) : part;
  const int n = n0 + lane * (p.swiglu ? 2 : 4);
  for (int m = split + kSplits * warp; m < p.M; m += kSplits * (kThreads / 32)) {
    float f[4] = {0.f, 0.f, 0.f, 0.f};
    const float alpha = p.ss_in ? p.alpha * s_rstd[m] : p.alpha;
    if (p.swiglu) {
      float2 g[kSplits], u[kSplits];
#pragma unroll
      for (int c = 0; c < kSplits; ++c) {
        g[c] = ld_cluster_f2(at[c] + (m * 128 + lane * 2) * 4);
        u[c] = ld_cluster_f2(at[c] + (m * 128 + 64 + lane * 2) * 4);
      }
#pragma unroll
      for (int c = 0; c < kSplits; ++c) { f[0] += g[c].x; f[1] += g[c].y; f[2] += u[c].x; f[3] += u[c].y; }
      if (n < p.N) {                  // N is even
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const float gv = f[e] * alpha, uv = f[2 + e] * alpha;
          f[e] = gv / (1.f + __expf(-gv)) * uv;
        }
        if (p.res) {
          const __nv_bfloat162 rv = *reinterpret_cast<const __nv_bfloat162*>(p.res + m * p.ldr + n);
          f[0] += __bfloat162float(rv.x);
          f[1] += __bfloat162float(rv.y);
        }
        *reinterpret_cast<uint32_t*>(p.y + m * p.ldy + n) = pack_bf16x2(f[0], f[1]);
      }
    } else {
      float4 v[kSplits];
#pragma unroll
      for (int c = 0; c < kSplits; ++c) v[c] = ld_cluster_f4(at[c] + (m * 128 + lane * 4) * 4);
      uint2 rv = make_uint2(0u, 0u);
      if (p.res && n < p.N) rv = *reinterpret_cast<const uint2*>(p.res + m * p.ldr + n);
#pragma unroll
      for (int c = 0; c < kSplits; ++c) { f[0] += v[c].x; f[1] += v[c].y; f[2] += v[c].z; f[3] += v[c].w; }
      float ss = 0.f;
      if (n < p.N) {                  // N is a multiple of 8
        f[0] = fmaf(f[0], alpha, bf16_bits_to_float(rv.x & 0xFFFFu)); f[1] = fmaf(f[1], alpha, bf16_bits_to_float(rv.x >> 16));
        f[2] = fmaf(f[2], alpha, bf16_bits_to_float(rv.y & 0xFFFFu)); f[3] = fmaf(f[3], alpha, bf16_bits_to_float(rv.y >> 16));
        const uint2 yv = make_uint2(pack_bf16x2(f[0], f[1]), pack_bf16x2(f[2], f[3]));
        *reinterpret_cast<uint2*>(p.y + m * p.ldy + n) = yv;
        if (p.y2) {
          const uint2 nv = *reinterpret_cast<const uint2*>(p.nw_out + n);
          const float y[4] = {bf16_bits_to_float(yv.x & 0xFFFFu), bf16_bits_to_float(yv.x >> 16), bf16_bits_to_float(yv.y & 0xFFFFu),
                              bf16_bits_to_float(yv.y >> 16)};
          ss = y[0] * y[0] + y[1] * y[1] + y[2] * y[2] + y[3] * y[3];
          *reinterpret_cast<uint2*>(p.y2 + m * p.ldy + n) =
              make_uint2(pack_bf16x2(y[0] * bf16_bits_to_float(nv.x & 0xFFFFu), y[1] * bf16_bits_to_float(nv.x >> 16)),
                         pack_bf16x2(y[2] * bf16_bits_to_float(nv.y & 0xFFFFu), y[3] * bf16_bits_to_float(nv.y >> 16)));
        }
      }
      if (p.y2) {
#pragma unroll
        for (int e = 16; e > 0; e >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, e);
        if (lane == 0) p.ss_out[(n0 >> 7) * 128 + m] = ss;
      }
    }
  }
  __syncwarp();
  if (kSplits > 1) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}

// kMT token columns. Shared memory: stages x [weights 128 x 64 | tokens kMT x 64], read again as the fp32 partial tile
// [kMT][128] once the MMAs are done.
template <int kMT>
__global__ void __launch_bounds__(kThreads)
skinny_linear_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const FewRowParams p) {
  constexpr int kStage = kSkW + kMT * 128;
  constexpr int kCols = kMT < 32 ? 32 : kMT;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ uint64_t full_bar[kMaxStages], empty_bar[kMaxStages], done_bar;
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_word;
  __shared__ float s_rstd[128];
  volatile int* abort_flag = &abort_word;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int split = p.splits > 1 ? static_cast<int>(cluster_ctarank()) : 0;
  const int tile = blockIdx.x / p.splits;
  const int n0 = tile * (p.swiglu ? 64 : 128);
  const int kb0 = split * p.per, nkb = max(min(p.nkb, kb0 + p.per) - kb0, 0);

  pdl_launch_dependents();
  if (threadIdx.x == 0) {
    tma_prefetch_desc(&map_w);
    tma_prefetch_desc(&map_x);
    for (int i = 0; i < p.stages; ++i) {
      mbar_init(&full_bar[i], 1);
      mbar_init(&empty_bar[i], 1);
    }
    mbar_init(&done_bar, 1);
    abort_word = 0;
    mbar_init_fence();
  }
  if (warp == 1) {
    tmem_alloc(&tmem_slot, kCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA: weights of the first stages, wait, tokens
    const bool elected = elect_one();
    auto load_w = [&](int kb, int s) {
      uint8_t* dst = smem + s * kStage;
      const int k = (kb0 + kb) * kBK;
      mbar_expect_tx(&full_bar[s], kStage);
      if (p.swiglu) {
        tma_load_2d(dst, &map_w, &full_bar[s], k, n0);
        tma_load_2d(dst + kSkW / 2, &map_w, &full_bar[s], k, p.N + n0);
      } else {
        tma_load_2d(dst, &map_w, &full_bar[s], k, n0);
      }
    };
    const int early = min(nkb, p.stages);
    if (elected)
      for (int kb = 0; kb < early; ++kb) load_w(kb, kb);
    pdl_wait();
    if (elected)
      for (int kb = 0; kb < early; ++kb) tma_load_2d(smem + kb * kStage + kSkW, &map_x, &full_bar[kb], (kb0 + kb) * kBK, 0);
    int s = 0;
    uint32_t ph = 0;
    for (int kb = early; kb < nkb; ++kb) {
      if (!mbar_wait(&empty_bar[s], ph, abort_flag, p.status, kTimeoutProducer)) break;
      if (elected) {
        load_w(kb, s);
        tma_load_2d(smem + s * kStage + kSkW, &map_x, &full_bar[s], (kb0 + kb) * kBK, 0);
      }
      if (++s == p.stages) { s = 0; ph ^= 1; }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA
    const bool elected = elect_one();
    const uint32_t sbase = smem_u32(smem);
    const uint32_t idesc = make_idesc_bf16(kMT, 0, 0);
    const uint64_t da0 = make_smem_desc(sbase, 16u, 1024u), db0 = make_smem_desc(sbase + kSkW, 16u, 1024u);
    int s = 0;
    uint32_t ph = 0;
    bool ok = true;
    for (int kb = 0; kb < nkb; ++kb) {
      if (!mbar_wait(&full_bar[s], ph, abort_flag, p.status, kTimeoutMma)) { ok = false; break; }
      tc_fence_after();
      if (elected) {
        const uint64_t da = da0 + static_cast<uint32_t>(s * (kStage >> 4)), db = db0 + static_cast<uint32_t>(s * (kStage >> 4));
#pragma unroll
        for (int j = 0; j < 4; ++j) umma_f16(tmem, da + 2 * j, db + 2 * j, idesc, kb > 0 || j > 0);
        umma_commit(&empty_bar[s]);
      }
      if (++s == p.stages) { s = 0; ph ^= 1; }
    }
    if (ok && elected && nkb > 0) umma_commit(&done_bar);
  } else {
    // ------------------------------------------------------------------ accumulator -> shared memory, [token][weight row]
    float* part = reinterpret_cast<float*>(smem);
    const int r = (warp & 3) * 32 + lane;
    if (p.ss_in) {                    // while the products are on their way
      pdl_wait();
      float ss = 0.f;
      if (r < p.M)
        for (int i = 0; i < p.parts_in; ++i) ss += __ldcg(p.ss_in + i * 128 + r);
      s_rstd[r] = rsqrtf(ss / static_cast<float>(p.K) + p.eps);
    }
    const bool have = nkb > 0 && mbar_wait(&done_bar, 0, abort_flag, p.status, kTimeoutEpilogue);
    tc_fence_after();
    const uint32_t t0 = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16);
#pragma unroll
    for (int c = 0; c < kCols / 32; ++c) {
      uint32_t v[32];
      tmem_ld_32x32b_x32(t0 + c * 32, v);
      tmem_ld_wait();
#pragma unroll
      for (int e = 0; e < (kMT < 32 ? kMT : 32); ++e) part[(c * 32 + e) * 128 + r] = have ? __uint_as_float(v[e]) : 0.f;
    }
    tc_fence_before();
  }
  __syncwarp();
  if (*abort_flag) {                  // an abandoned wait: let the copies in flight land first
    const unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) { }
  }
  __syncthreads();
  if (p.splits > 1) cluster_sync_all();
  if (warp != 0) pdl_wait();          // the residual and the output belong to earlier kernels until here (warp 0 has waited)
  switch (p.splits) {
    case 1: skinny_finish<1>(p, smem_u32(smem), split, n0, s_rstd); break;
    case 2: skinny_finish<2>(p, smem_u32(smem), split, n0, s_rstd); break;
    case 4: skinny_finish<4>(p, smem_u32(smem), split, n0, s_rstd); break;
    default: skinny_finish<8>(p, smem_u32(smem), split, n0, s_rstd); break;
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, kCols);
  }
  if (p.splits > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");   // the peers have read this CTA's partial tile
}

// What a chain that starts from plain rows needs: x * nw and the rows' sums of squares. One CTA per row.
__global__ void __launch_bounds__(256) skinny_prep_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ nw,
                                                          __nv_bfloat16* __restrict__ y2, float* __restrict__ ss_out, int H) {
  pdl_launch_dependents();
  pdl_wait();
  __shared__ float red[8];
  const long long base = static_cast<long long>(blockIdx.x) * H;
  float ss = 0.f;
  for (int c = threadIdx.x * 4; c < H; c += 1024) {
    const uint2 xv = *reinterpret_cast<const uint2*>(x + base + c), nv = *reinterpret_cast<const uint2*>(nw + c);
    const uint32_t xw[2] = {xv.x, xv.y}, nq[2] = {nv.x, nv.y};
    uint32_t o[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const float a = bf16_bits_to_float(xw[e] & 0xFFFFu), b = bf16_bits_to_float(xw[e] >> 16);
      ss += a * a + b * b;
      o[e] = pack_bf16x2(a * bf16_bits_to_float(nq[e] & 0xFFFFu), b * bf16_bits_to_float(nq[e] >> 16));
    }
    *reinterpret_cast<uint2*>(y2 + base + c) = make_uint2(o[0], o[1]);
  }
#pragma unroll
  for (int e = 16; e > 0; e >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, e);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) t += red[i];
    ss_out[blockIdx.x] = t;
  }
}

template <int kMT>
static int launch_skinny(const CUtensorMap& mw, const CUtensorMap& mx, FewRowParams p, int tiles, int chain, cudaStream_t st) {
  constexpr int kStage = kSkW + kMT * 128;
  // two CTAs to an SM, so that the next kernel of a chain can move in: about 100 KB each
  p.stages = std::min(std::min(kMaxStages, 100 * 1024 / kStage), std::max(p.per, 1));
  const int smem = std::max(p.stages * kStage, kMT * 512) + 1024;
  static DeviceOnce once;
  if (once.pending()) {
    cudaError_t e = cudaFuncSetAttribute(skinny_linear_kernel<kMT>, cudaFuncAttributeMaxDynamicSharedMemorySize, 104 * 1024);
    if (e != cudaSuccess) return static_cast<int>(e);
    once.mark();
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(static_cast<unsigned>(tiles) * p.splits);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  int n = 0;
  if (p.splits > 1) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = p.splits;
    attr[n].val.clusterDim.y = attr[n].val.clusterDim.z = 1;
    ++n;
  }
  if (chain) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n].val.programmaticStreamSerializationAllowed = 1;
    ++n;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  return static_cast<int>(cudaLaunchKernelEx(&cfg, skinny_linear_kernel<kMT>, mw, mx, p));
}

}  // namespace pm

using namespace pm;

// pm_linear_skinny inside a chain of RMSNorms. ss_in non-null: x is rows * norm weight and ss_in [parts_in][128] their partial sums of squares
// (row m of part i at i * 128 + m), the product is that of the normalised rows. y2 non-null (not with swiglu): y2 = y * nw_out with y's
// strides and ss_out [(N + 127) / 128][128] for the next link.
extern "C" int pm_linear_skinny_norm(const void* x, long long ldx, const void* w, long long ldw, void* y, long long ldy, const void* res,
                                     long long ldr, int M, int N, int K, int swiglu, float alpha, int splits, int chain,
                                     const float* ss_in, int parts_in, float eps, const void* nw_out, void* y2, float* ss_out,
                                     int* status, cudaStream_t st) {
  if (M <= 0 || M > 128 || N <= 0 || K <= 0) return -1;
  if ((N | K) % 8 || (ldx | ldw | ldy) % 8 || (res && ldr % 8)) return -2;
  if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(y) |
       reinterpret_cast<uintptr_t>(res) | reinterpret_cast<uintptr_t>(y2) | reinterpret_cast<uintptr_t>(nw_out)) & 15)
    return -3;
  if (y2 && (swiglu || !nw_out || !ss_out)) return -5;
  FewRowParams p{};
  p.y = static_cast<__nv_bfloat16*>(y); p.ldy = ldy;
  p.res = static_cast<const __nv_bfloat16*>(res); p.ldr = ldr;
  p.M = M; p.N = N; p.K = K; p.swiglu = swiglu; p.alpha = alpha; p.status = status;
  p.ss_in = ss_in; p.parts_in = parts_in; p.eps = eps;
  p.nw_out = static_cast<const __nv_bfloat16*>(nw_out); p.y2 = static_cast<__nv_bfloat16*>(y2); p.ss_out = ss_out;
  p.nkb = (K + kBK - 1) / kBK;
  const int rows = swiglu ? 64 : 128, tiles = (N + rows - 1) / rows;
  if (splits <= 0) {
    // up to 4/3 CTAs per SM with at least two k blocks each: 64 rows of 4096 x 1024 take 9.1, 7.7, 6.1, 7.6 us on 32, 64, 128, 256 CTAs
    splits = 1;
    while (splits < 8 && tiles * splits * 6 <= 4 * num_sms() && p.nkb >= splits * 4) splits *= 2;
  }
  if (splits != 1 && splits != 2 && splits != 4 && splits != 8) return -4;
  p.splits = splits;
  p.per = (p.nkb + splits - 1) / splits;
  const int mt = M <= 16 ? 16 : M <= 32 ? 32 : M <= 64 ? 64 : 128;
  CUtensorMap mw, mx;
  int rc;
  if ((rc = make_map(&mw, w, K, static_cast<uint64_t>(swiglu ? 2 * static_cast<long long>(N) : N), ldw, kBK, rows))) return rc;
  if ((rc = make_map(&mx, x, K, M, ldx, kBK, mt))) return rc;
  switch (mt) {
    case 16: return launch_skinny<16>(mw, mx, p, tiles, chain, st);
    case 32: return launch_skinny<32>(mw, mx, p, tiles, chain, st);
    case 64: return launch_skinny<64>(mw, mx, p, tiles, chain, st);
    default: return launch_skinny<128>(mw, mx, p, tiles, chain, st);
  }
}

// x: [M, K] rows ldx apart, w: [N, K] (swiglu: [2 N, K], gate rows first) rows ldw apart, y / res: [M, N] rows ldy / ldr apart (res
// nullable, may be y). M <= 128; K, N and the row strides multiples of 8, pointers 16-byte aligned. splits 0: chosen here. chain: see
// the head of this file. Returns a negative value for arguments outside of that.
extern "C" int pm_linear_skinny(const void* x, long long ldx, const void* w, long long ldw, void* y, long long ldy, const void* res,
                                long long ldr, int M, int N, int K, int swiglu, float alpha, int splits, int chain, int* status,
                                cudaStream_t st) {
  return pm_linear_skinny_norm(x, ldx, w, ldw, y, ldy, res, ldr, M, N, K, swiglu, alpha, splits, chain, nullptr, 0, 0.f, nullptr, nullptr,
                               nullptr, status, st);
}

// First link of such a chain: y2 = x * nw [M, H] and ss [128] = the rows' sums of squares. M <= 128, H a multiple of 8.
extern "C" int pm_skinny_prep(const void* x, const void* nw, void* y2, float* ss, int M, int H, cudaStream_t st) {
  if (M <= 0 || M > 128 || H <= 0 || H % 8) return -1;
  return static_cast<int>(launch_pdl(skinny_prep_kernel, dim3(static_cast<unsigned>(M)), dim3(256), 0, st,
                                     static_cast<const __nv_bfloat16*>(x), static_cast<const __nv_bfloat16*>(nw),
                                     static_cast<__nv_bfloat16*>(y2), ss, H));
}

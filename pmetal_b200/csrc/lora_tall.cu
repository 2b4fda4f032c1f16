// The narrow products of a LoRA layer: D[M, 64] = alpha * X[M, K] B with B a factor of at most 64 columns, M tokens: t = x A^T
// (A [nr, K] as it lies) and dt = dY B (B [N, r], read in place as an MN-major operand; the part of the reduction that belongs to
// segment s lands in columns [s r, (s + 1) r) because its tile is fetched s r columns left of the origin, zero fill elsewhere).
//
// Each is one pass over X, which a few thousand tokens give to only a handful of 128-row tiles: K is cut over the CTAs of a
// cluster, which add their partial tiles through distributed shared memory in a fixed order and share the output rows. Measured (tile GEMM
// on 128-row tiles that walk all of K, here, bytes at 6.5 TB/s), r = 16, captured: 2048 rows x 1024, t 7.7, 6.1, 0.6 us; x 3072 t 17.1, 9.0,
// 1.9 us; dt over 4096 22.4, 9.8, 2.6 us, over 6144 31.4, 11.3, 3.9 us; 8192 rows, dt over 19456 93.9, 61.5, 49.0 us. What is left at 2048
// rows is launch, first bytes, sum and store.
#include <algorithm>

#include "gemm_pair.cuh"
#include "pmetal_b200.h"

namespace pm {

struct TallParams {
  __nv_bfloat16* d;
  long long ldd;
  int M, K, nkb, per, splits, stages, b_mn, seg_r;
  int seg_end[4];
  float alpha;
  int* status;
};

constexpr int kTlStage = 128 * 128 + 64 * 128;      // X [128][64], B [64][64]
constexpr int kTlLd = 68;                           // floats per row of the partial tile: 16-byte rows on different banks

template <int kSplits>
__device__ __forceinline__ void tall_finish(const TallParams& p, uint32_t part, int split, int m0) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, c = (lane & 15) * 4;
  uint32_t at[kSplits];
#pragma unroll
  for (int i = 0; i < kSplits; ++i) at[i] = kSplits > 1 ? map_to_cta(part, i) : part;
  constexpr int kShare = 128 / kSplits;
  for (int r = warp * 2 + (lane >> 4); r < kShare; r += kThreads / 16) {
    const int row = split * kShare + r;
    float4 v[kSplits];
#pragma unroll
    for (int i = 0; i < kSplits; ++i) v[i] = ld_cluster_f4(at[i] + (row * kTlLd + c) * 4);
    float f[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int i = 0; i < kSplits; ++i) { f[0] += v[i].x; f[1] += v[i].y; f[2] += v[i].z; f[3] += v[i].w; }
    if (m0 + row < p.M)
      *reinterpret_cast<uint2*>(p.d + (m0 + row) * p.ldd + c) =
          make_uint2(pack_bf16x2(f[0] * p.alpha, f[1] * p.alpha), pack_bf16x2(f[2] * p.alpha, f[3] * p.alpha));
  }
  __syncwarp();
  if (kSplits > 1) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}

__global__ void __launch_bounds__(kThreads)
lora_tall_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_b, const TallParams p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ uint64_t full_bar[kMaxStages], empty_bar[kMaxStages], done_bar;
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_word;
  volatile int* abort_flag = &abort_word;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int split = p.splits > 1 ? static_cast<int>(cluster_ctarank()) : 0;
  const int m0 = blockIdx.x / p.splits * 128;
  const int kb0 = split * p.per, nkb = max(min(p.nkb, kb0 + p.per) - kb0, 0);

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&map_x);
    tma_prefetch_desc(&map_b);
    for (int i = 0; i < p.stages; ++i) {
      mbar_init(&full_bar[i], 1);
      mbar_init(&empty_bar[i], 1);
    }
    mbar_init(&done_bar, 1);
    abort_word = 0;
    mbar_init_fence();
  }
  if (warp == 1) {
    tmem_alloc(&tmem_slot, 64);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;

  if (warp == 0) {
    const bool elected = elect_one();
    int s = 0;
    uint32_t ph = 1;
    for (int kb = 0; kb < nkb; ++kb) {
      if (!mbar_wait(&empty_bar[s], ph, abort_flag, p.status, kTimeoutProducer)) break;
      if (elected) {
        const int k = (kb0 + kb) * kBK;
        uint8_t* dst = smem + s * kTlStage;
        mbar_expect_tx(&full_bar[s], kTlStage);
        tma_load_2d(dst, &map_x, &full_bar[s], k, m0);
        if (p.b_mn) {
          int seg = 0;
#pragma unroll
          for (int i = 0; i < 3; ++i) seg += k >= p.seg_end[i] ? 1 : 0;
          tma_load_2d(dst + 128 * 128, &map_b, &full_bar[s], -seg * p.seg_r, k);
        } else {
          tma_load_2d(dst + 128 * 128, &map_b, &full_bar[s], k, 0);
        }
      }
      if (++s == p.stages) { s = 0; ph ^= 1; }
    }
  } else if (warp == 1) {
    const bool elected = elect_one();
    const uint32_t sbase = smem_u32(smem);
    const uint32_t idesc = make_idesc_bf16(64, 0, p.b_mn);
    const uint64_t da0 = make_smem_desc(sbase, 16u, 1024u), db0 = make_smem_desc(sbase + 128 * 128, p.b_mn ? 8192u : 16u, 1024u);
    const uint32_t bstep = p.b_mn ? 128u : 2u;
    int s = 0;
    uint32_t ph = 0;
    bool ok = true;
    for (int kb = 0; kb < nkb; ++kb) {
      if (!mbar_wait(&full_bar[s], ph, abort_flag, p.status, kTimeoutMma)) { ok = false; break; }
      tc_fence_after();
      if (elected) {
        const uint64_t da = da0 + static_cast<uint32_t>(s * (kTlStage >> 4)), db = db0 + static_cast<uint32_t>(s * (kTlStage >> 4));
#pragma unroll
        for (int j = 0; j < 4; ++j) umma_f16(tmem, da + 2 * j, db + bstep * j, idesc, kb > 0 || j > 0);
        umma_commit(&empty_bar[s]);
      }
      if (++s == p.stages) { s = 0; ph ^= 1; }
    }
    if (ok && elected && nkb > 0) umma_commit(&done_bar);
  } else {
    const int r = (warp & 3) * 32 + lane;
    const bool have = nkb > 0 && mbar_wait(&done_bar, 0, abort_flag, p.status, kTimeoutEpilogue);
    tc_fence_after();
    uint32_t v[2][32];
    tmem_ld_32x32b_x32(tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16), v[0]);
    tmem_ld_32x32b_x32(tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16) + 32, v[1]);
    tmem_ld_wait();
    float4* row = reinterpret_cast<float4*>(reinterpret_cast<float*>(smem) + r * kTlLd);
#pragma unroll
    for (int e = 0; e < 16; ++e) {
      const uint32_t* q = &v[e >> 3][(e & 7) * 4];
      row[e] = have ? make_float4(__uint_as_float(q[0]), __uint_as_float(q[1]), __uint_as_float(q[2]), __uint_as_float(q[3]))
                    : make_float4(0.f, 0.f, 0.f, 0.f);
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
  switch (p.splits) {
    case 1: tall_finish<1>(p, smem_u32(smem), split, m0); break;
    case 2: tall_finish<2>(p, smem_u32(smem), split, m0); break;
    case 4: tall_finish<4>(p, smem_u32(smem), split, m0); break;
    default: tall_finish<8>(p, smem_u32(smem), split, m0); break;
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 64);
  }
  if (p.splits > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");   // the peers have read this CTA's partial tile
}

}  // namespace pm

using namespace pm;

// x: [M, K] rows ldx apart. b_mn 0: b is [nr, K] rows ldb apart and d = alpha x b^T; b_mn 1: b is [K, nr], d[:, seg nr ..] = alpha x[:, seg] b[seg]
// with the cumulative ends of the segments in seg_end[4] (multiples of 64; 0x7fffffff beyond the last but one). d: [M, 64] rows ldd apart, all 64 columns
// are written (zeros beyond the factors). nr and segments * nr up to 64, multiples of 8; K, the row strides multiples of 8, pointers
// 16-byte aligned. splits 0: chosen here.
extern "C" int pm_lora_tall(const void* x, long long ldx, const void* b, long long ldb, int b_mn, int nr, void* d, long long ldd, int M, int K,
                            const int* seg_end, float alpha, int splits, int* status, cudaStream_t st) {
  if (M <= 0 || K <= 0 || nr <= 0 || nr > 64 || nr % 8 || K % 8) return -1;
  if ((ldx | ldb) % 8 || ldd % 4) return -2;
  if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(d)) & 15) return -3;
  TallParams p{};
  p.d = static_cast<__nv_bfloat16*>(d);
  p.ldd = ldd; p.M = M; p.K = K; p.b_mn = b_mn; p.seg_r = nr; p.alpha = alpha; p.status = status;
  for (int i = 0; i < 4; ++i) {
    p.seg_end[i] = b_mn && seg_end ? seg_end[i] : 0x7fffffff;
    if (p.seg_end[i] != 0x7fffffff && (p.seg_end[i] % 64 || (i + 2) * nr > 64)) return -5;
  }
  p.nkb = (K + kBK - 1) / kBK;
  const int tiles = (M + 127) / 128;
  if (splits <= 0) {
    // up to two CTAs per SM with at least four k blocks each; past one per SM only long reductions gain (16384 rows: K = 1024 9.3 us on
    // 128 CTAs, 10.4 on 256, K = 3072 24.7, 22.8)
    splits = 1;
    while (splits < 8 && tiles * splits <= num_sms() && p.nkb >= splits * 8 && (tiles * splits * 2 <= num_sms() || p.nkb >= 32)) splits *= 2;
  }
  if (splits != 1 && splits != 2 && splits != 4 && splits != 8) return -4;
  p.splits = splits;
  p.per = (p.nkb + splits - 1) / splits;
  p.stages = std::min(4, std::max(p.per, 2));
  CUtensorMap mx, mb;
  int rc;
  if ((rc = make_map(&mx, x, K, M, ldx, kBK, 128))) return rc;
  if ((rc = b_mn ? make_map(&mb, b, nr, K, ldb, 64, kBK) : make_map(&mb, b, K, nr, ldb, kBK, 64))) return rc;
  const int smem = p.stages * kTlStage + 1024;
  static DeviceOnce once;
  if (once.pending()) {
    cudaError_t e = cudaFuncSetAttribute(lora_tall_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 4 * kTlStage + 1024);
    if (e != cudaSuccess) return static_cast<int>(e);
    once.mark();
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(static_cast<unsigned>(tiles) * splits);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = splits;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = splits > 1 ? 1 : 0;
  return static_cast<int>(cudaLaunchKernelEx(&cfg, lora_tall_kernel, mx, mb, p));
}

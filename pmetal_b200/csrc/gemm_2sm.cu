// bf16 GEMM on CTA pairs: tcgen05.mma.cta_group::2 computes a 256 x 256 output tile across two SMs.
//
// Same math and operand options as gemm_tcgen05.cu:
//   D[M,N] = alpha * ( A[M,K] * B[N,K]^T + A2[M,K2] * B2[N,K2]^T ) (+ R[M,N])
// but launched as clusters of two CTAs. CTA r of a pair stages A rows [m0+128r, +128) and B rows
// [n0+128r, +128) of each 64-wide K block in its own shared memory; one thread of the leader CTA
// (cluster rank 0) issues the MMAs, which read both CTAs' shared memory and write 128 x 256 fp32
// accumulators into each CTA's TMEM. Per SM this moves 32 KB of operands per K block instead of the
// 48 KB a single CTA needs for 128 x 256, which is what lifts the kernel off the L2->SM bandwidth limit.
// No operand is multicast: every CTA fetches its own half with plain tiled TMA loads whose completion
// is counted on the leader's "full" barrier.
//
// Cross-CTA signalling:
//   full[s]   (leader)      <- TMA bytes of both CTAs + the leader producer's expect_tx arrive
//   empty[s]  (each CTA)    <- tcgen05.commit from the leader, once to its own and once to the peer's barrier
//   tfull[b]  (each CTA)    <- tcgen05.commit from the leader after the last K block (own + peer)
//   tempty[b] (leader)      <- 4 epilogue warps of each CTA (remote mbarrier.arrive from the peer)
// All waits are bounded (see common.cuh); the pair leaves through a cluster barrier so neither CTA
// exits while its partner can still touch its shared memory.
#include <algorithm>

#include "gemm_pair.cuh"
#include "pmetal_b200.h"

namespace pm {

// Shared memory of a CTA: [stages][A 16 KB | B kBN/2 rows] | epilogue staging, two 4 KB buffers per warp | barriers
constexpr int kEpiBytes = 4 * 2 * 4096;
template <int kBN>
struct PairTile {
  static constexpr int kHalf = kBN / 2;
  static constexpr int kABytes = kBM * kBK * 2;
  static constexpr int kStage = kABytes + kHalf * kBK * 2;
  static constexpr int kStages = (227 * 1024 - 1024 - 512 - kEpiBytes) / kStage;
  static constexpr int kSmem = kStages * kStage + kEpiBytes + 1024 + 512;
};

// What bounds it: the tensor cores, as long as one k block (64 wide) costs the two issuing threads less than the
// 512 cycles that its MMAs take. The loops below therefore carry nothing but the wait, the copies or MMAs and the commit:
// the ring position is a counter (no division), descriptors and barrier addresses are sums of precomputed bases, and the
// operand layout is looked at once per tile. Measured at 16384 x 4096 x 1024: 84.9 us (1620 TFLOP/s); 145.0 us with the ring
// position divided out, two k blocks to a stage, per-block branches (about 1100 cycles per k block) and results stored
// from registers. 2048 x 1024 x 3072, where 256-wide tiles leave half of the SMs idle: 14.9 us (33.4 us).
//
// Tile order: groups of `group_m` row blocks, inside a group row blocks vary fastest. The 74 pairs at work then share a
// few row blocks and a few column blocks, and B is read from DRAM once per group instead of once per row block.
template <int kBN>
__global__ void __launch_bounds__(kThreads, 1)
gemm_bf16_2sm_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                     const __grid_constant__ CUtensorMap map_a2, const __grid_constant__ CUtensorMap map_b2,
                     const __grid_constant__ CUtensorMap map_d, const __grid_constant__ CUtensorMap map_r,
                     const GemmParams p) {
  using T = PairTile<kBN>;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* epi = smem + T::kStages * T::kStage;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(epi + kEpiBytes);
  uint64_t* empty_bar = full_bar + kMaxStages;
  uint64_t* tfull_bar = empty_bar + kMaxStages;   // [2]
  uint64_t* tempty_bar = tfull_bar + 2;           // [2]
  uint64_t* r_bar = tempty_bar + 2;               // [4 warps][2]: a piece of the residual has landed
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(r_bar + 8);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();        // 0 = leader
  const bool leader = rank == 0;

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&map_a);
    tma_prefetch_desc(&map_b);
    for (int i = 0; i < T::kStages; ++i) {
      mbar_init(&full_bar[i], 1);     // leader producer's expect_tx arrive; bytes from both CTAs
      mbar_init(&empty_bar[i], 1);    // one tcgen05.commit
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&tfull_bar[i], 1);    // one tcgen05.commit
      mbar_init(&tempty_bar[i], 8);   // 4 epilogue warps of each CTA (used on the leader only)
    }
    for (int i = 0; i < 8; ++i) mbar_init(&r_bar[i], 1);
    *abort_flag = 0;
    mbar_init_fence();
    if (p.nk2) {
      tma_prefetch_desc(&map_a2);
      tma_prefetch_desc(&map_b2);
    }
  }
  if (warp == 1) {
    tmem_alloc_pair(tmem_slot, 2 * kBN);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();   // both CTAs' barriers are initialised before any remote signal
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  const int m_tiles = (p.M + 2 * kBM - 1) / (2 * kBM);
  const int n_tiles = (p.N + kBN - 1) / kBN;
  const int total = m_tiles * n_tiles * p.splits;
  const int nk = p.nk1 + p.nk2;
  const int per_split = (nk + p.splits - 1) / p.splits;
  const int first = static_cast<int>(cluster_id_x());
  const int stride = static_cast<int>(num_clusters_x());

  // work item -> (row block, column block, k range)
  auto item = [&](int w, int& mb, int& nb, int& kb0, int& kb1) {
    int tile = w, split = 0;
    if (p.splits > 1) {
      split = w % p.splits;
      tile = w / p.splits;
    }
    const int per_group = p.group_m * n_tiles;
    const int g = tile / per_group, in = tile - g * per_group;
    const int rows = min(p.group_m, m_tiles - g * p.group_m);
    nb = in / rows;
    mb = g * p.group_m + in - nb * rows;
    kb0 = split * per_split;
    kb1 = min(nk, kb0 + per_split);
  };

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer (one per CTA)
    const bool elected = elect_one();
    const uint32_t sbase = smem_u32(smem);
    const uint32_t full0 = map_to_cta(smem_u32(full_bar), 0);       // both CTAs' bytes are counted on the leader's barrier
    int s = 0;
    uint32_t ph = 1;
    bool ok = true;
    for (int w = first; w < total && ok; w += stride) {
      int mb, nb, kb0, kb1;
      item(w, mb, nb, kb0, kb1);
      const int m0 = mb * 2 * kBM + static_cast<int>(rank) * kBM;
      const int n_tile0 = nb * kBN;
      const int n0 = n_tile0 + static_cast<int>(rank) * T::kHalf;
      for (int part = 0; part < 2 && ok; ++part) {
        // the two products of the sum one after the other: [kb0, kb1) cut at nk1
        const int lo = part ? max(kb0, p.nk1) : kb0, hi = part ? kb1 : min(kb1, p.nk1);
        if (lo >= hi) continue;
        const CUtensorMap* ma = part ? &map_a2 : &map_a;
        const CUtensorMap* mbp = part ? &map_b2 : &map_b;
        const int amn = part ? p.a2_mn : p.a_mn, bmn = part ? p.b2_mn : p.b_mn;
        int ka = (lo - (part ? p.nk1 : 0)) * kBK, kb_ = ka;
        int brow = n0;
        if (part && p.seg_mode == 1) ka += seg_of(p, n_tile0) * p.seg_r;
        if (!part && p.seg_mode == 2) brow += seg_of(p, mb * 2 * kBM) * p.seg_r;
        for (int kb = lo; kb < hi; ++kb) {
          if (!mbar_wait(&empty_bar[s], ph, abort_flag, p.status, kTimeoutProducer)) { ok = false; break; }
          if (elected) {
            const uint32_t sa = sbase + s * T::kStage, sb = sa + T::kABytes, fb = full0 + s * 8;
            if (leader) mbar_expect_tx(&full_bar[s], 2 * T::kStage);
            if (!amn) {
              tma_load_2d_pair(sa, ma, fb, ka, m0);
            } else {
              tma_load_2d_pair(sa, ma, fb, m0, ka);
              tma_load_2d_pair(sa + 8192, ma, fb, m0 + 64, ka);
            }
            if (!bmn) {
              tma_load_2d_pair(sb, mbp, fb, kb_, brow);
            } else {
#pragma unroll
              for (int j = 0; j < T::kHalf / 64; ++j) tma_load_2d_pair(sb + j * 8192, mbp, fb, brow + 64 * j, kb_);
            }
          }
          ka += kBK;
          kb_ += kBK;
          if (++s == T::kStages) { s = 0; ph ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (leader CTA only)
    if (leader) {
      const bool elected = elect_one();
      const uint32_t sbase = smem_u32(smem);
      int s = 0;
      uint32_t ph = 0, acc_it = 0;
      bool ok = true;
      for (int w = first; w < total && ok; w += stride) {
        int mb, nb, kb0, kb1;
        item(w, mb, nb, kb0, kb1);
        if (kb0 >= kb1) continue;
        const int buf = acc_it & 1;
        const uint32_t aph = (acc_it >> 1) & 1;
        if (!mbar_wait_cluster(&tempty_bar[buf], aph ^ 1, abort_flag, p.status, kTimeoutMma)) { ok = false; break; }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + buf * kBN;
        uint32_t accumulate = 0;
        for (int part = 0; part < 2 && ok; ++part) {
          const int lo = part ? max(kb0, p.nk1) : kb0, hi = part ? kb1 : min(kb1, p.nk1);
          if (lo >= hi) continue;
          const int amn = part ? p.a2_mn : p.a_mn, bmn = part ? p.b2_mn : p.b_mn;
          const uint32_t idesc = make_idesc_bf16_m256(kBN, amn, bmn);
          const uint64_t da0 = make_smem_desc(sbase, amn ? 8192u : 16u, 1024u);
          const uint64_t db0 = make_smem_desc(sbase + T::kABytes, bmn ? 8192u : 16u, 1024u);
          const uint32_t astep = amn ? 128u : 2u, bstep = bmn ? 128u : 2u;   // 16 K elements, in units of 16 bytes
          for (int kb = lo; kb < hi; ++kb) {
            if (!mbar_wait(&full_bar[s], ph, abort_flag, p.status, kTimeoutMma)) { ok = false; break; }
            tc_fence_after();
            if (elected) {
              const uint64_t da = da0 + static_cast<uint32_t>(s * (T::kStage >> 4));
              const uint64_t db = db0 + static_cast<uint32_t>(s * (T::kStage >> 4));
              const int nmma = part ? min(4, (p.K2 - (kb - p.nk1) * kBK + 15) / 16) : 4;
              umma_f16_pair(d_tmem, da, db, idesc, accumulate);
#pragma unroll
              for (int j = 1; j < 4; ++j)
                if (j < nmma) umma_f16_pair(d_tmem, da + astep * j, db + bstep * j, idesc, 1);
              umma_commit_both(&empty_bar[s]);   // the stage is free in both CTAs once these MMAs have read it
            }
            accumulate = 1;
            if (++s == T::kStages) { s = 0; ph ^= 1; }
          }
        }
        if (ok && elected) umma_commit_both(&tfull_bar[buf]);
        ++acc_it;
      }
    }
  } else {
    // ------------------------------------------------------------------ epilogue (warps 2..5 of each CTA)
    // bf16 results go through shared memory, 32 rows x 64 columns at a time in the 128-byte swizzle, and leave as TMA
    // stores (whole 128-byte lines; a store from registers writes 16 bytes to each of 32 rows per instruction, which at
    // K = 1024 took longer than the tile's MMAs). A residual piece is brought into the same buffer by TMA beforehand.
    const int q = warp & 3;
    const bool staged = p.staged;
    uint8_t* ebuf = epi + (warp - 2) * 8192;
    uint64_t* rb = r_bar + (warp - 2) * 2;
    const uint32_t row_off = static_cast<uint32_t>(lane) * 128u;
    const uint32_t tempty0 = map_to_cta(smem_u32(tempty_bar), 0);
    uint32_t acc_it = 0, piece = 0, rph = 0;
    bool ok = true;
    for (int w = first; w < total && ok; w += stride) {
      int mb, nb, kb0, kb1;
      item(w, mb, nb, kb0, kb1);
      if (kb0 >= kb1) continue;
      const int buf = acc_it & 1;
      const uint32_t aph = (acc_it >> 1) & 1;
      const int row0 = mb * 2 * kBM + static_cast<int>(rank) * kBM + q * 32;
      const int col_base = nb * kBN;
      const uint32_t tm = tmem_base + buf * kBN + (static_cast<uint32_t>(q * 32) << 16);
      if (staged) {
        const int pieces = row0 < p.M ? max(0, min(kBN / 64, (p.n_store - col_base + 63) / 64)) : 0;   // none past n_store
        if (p.R && lane == 0) {
          tma_store_wait_read<0>();
          for (int c = 0; c < min(2, pieces); ++c) {
            const int b = (piece + c) & 1;
            mbar_expect_tx(&rb[b], 4096);
            tma_load_2d(ebuf + b * 4096, &map_r, &rb[b], col_base + c * 64, row0);
          }
        }
        if (!mbar_wait(&tfull_bar[buf], aph, abort_flag, p.status, kTimeoutEpilogue)) { ok = false; break; }
        tc_fence_after();
        for (int c = 0; c < pieces; ++c, ++piece) {
          const int b = piece & 1;
          uint8_t* dst = ebuf + b * 4096;
          uint32_t r[2][32];
          tmem_ld_32x32b_x32(tm + c * 64, r[0]);
          tmem_ld_32x32b_x32(tm + c * 64 + 32, r[1]);
          if (p.R) {
            if (!mbar_wait(&rb[b], (rph >> b) & 1, abort_flag, p.status, kTimeoutEpilogue)) { ok = false; break; }
            rph ^= 1u << b;
          } else {
            if (lane == 0) tma_store_wait_read<1>();
            __syncwarp();
          }
          tmem_ld_wait();
          if (c == pieces - 1) {      // the accumulator is in registers: the next tile may use its columns
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(tempty0 + buf * 8);
          }
#pragma unroll
          for (int v = 0; v < 8; ++v) {
            uint4* at = reinterpret_cast<uint4*>(dst + row_off + ((v ^ (lane & 7)) << 4));
            float f[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) f[e] = __uint_as_float(r[v >> 2][(v & 3) * 8 + e]) * p.alpha;
            if (p.R) {
              const uint4 rv = *at;
              const uint32_t rw[4] = {rv.x, rv.y, rv.z, rv.w};
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                f[2 * e] += bf16_bits_to_float(rw[e] & 0xFFFFu);
                f[2 * e + 1] += bf16_bits_to_float(rw[e] >> 16);
              }
            }
            *at = make_uint4(pack_bf16x2(f[0], f[1]), pack_bf16x2(f[2], f[3]), pack_bf16x2(f[4], f[5]),
                             pack_bf16x2(f[6], f[7]));
          }
          fence_async_smem();
          __syncwarp();
          if (lane == 0) {
            tma_store_2d(&map_d, dst, col_base + c * 64, row0);
            tma_store_commit();
            if (p.R && c + 2 < pieces) {
              tma_store_wait_read<0>();
              mbar_expect_tx(&rb[b], 4096);
              tma_load_2d(dst, &map_r, &rb[b], col_base + (c + 2) * 64, row0);
            }
          }
        }
        if (pieces == 0) {
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster(tempty0 + buf * 8);
        }
        ++acc_it;
        continue;
      }
      if (!mbar_wait(&tfull_bar[buf], aph, abort_flag, p.status, kTimeoutEpilogue)) { ok = false; break; }
      tc_fence_after();
      const int row = row0 + lane;
      const bool row_ok = row < p.M;
      for (int c = 0; c < kBN / 32; ++c) {
        uint32_t r[32];
        tmem_ld_32x32b_x32(tm + c * 32, r);
        tmem_ld_wait();
        const int col0 = col_base + c * 32;
        if (!row_ok || col0 >= p.n_store) continue;
        epilogue_store_chunk(p, r, row, col0);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(tempty0 + buf * 8);
      ++acc_it;
    }
    if (staged && lane == 0) tma_store_wait_all();
  }

  // ------------------------------------------------------------------ tail
  __syncwarp();
  if (*abort_flag) {
    const unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) { }
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();   // the partner is done with this CTA's shared memory, barriers and TMEM
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, 2 * kBN);
  }
}

template <int kBN>
static int launch_pair(GemmParams p, const void* A, int lda, int a_rows, const void* B, int ldb, int b_rows, const void* A2,
                       int lda2, int a2_k, const void* B2, int ldb2, int b2_rows, int pairs_cap, cudaStream_t stream) {
  using T = PairTile<kBN>;
  p.bn = kBN;
  p.stages = T::kStages;
  CUtensorMap ma, mb, ma2, mb2, md, mr;
  int rc;
  if ((rc = operand_map(&ma, A, p.a_mn, a_rows, p.K, lda, kBM))) return rc * 10 - 1;
  if ((rc = operand_map(&mb, B, p.b_mn, b_rows, p.K, ldb, T::kHalf))) return rc * 10 - 2;
  ma2 = ma;
  mb2 = mb;
  if (p.K2 > 0) {
    if ((rc = operand_map(&ma2, A2, p.a2_mn, a_rows, a2_k, lda2, kBM))) return rc * 10 - 3;
    if ((rc = operand_map(&mb2, B2, p.b2_mn, b2_rows, p.K2, ldb2, T::kHalf))) return rc * 10 - 4;
  }
  md = mr = ma;
  // columns past n_store and rows past M lie outside the map and the store leaves them alone, but it cuts a row off at 16 bytes: where
  // n_store ends inside 8 columns the results are stored from registers
  p.staged = p.out_mode == 0 && !p.tail && p.n_store % 8 == 0;
  if (p.staged) {
    if ((rc = make_map(&md, p.D, p.n_store, p.M, p.ldd, 64, 32))) return rc * 10 - 5;
    if (p.R && (rc = make_map(&mr, p.R, p.n_store, p.M, p.ldr, 64, 32))) return rc * 10 - 6;
  }
  static DeviceOnce configured;
  if (configured.pending()) {
    cudaError_t e = cudaFuncSetAttribute(gemm_bf16_2sm_kernel<kBN>, cudaFuncAttributeMaxDynamicSharedMemorySize, T::kSmem);
    if (e != cudaSuccess) return static_cast<int>(e);
    configured.mark();
  }
  const int m_tiles = (p.M + 2 * kBM - 1) / (2 * kBM), n_tiles = (p.N + kBN - 1) / kBN;
  // rows of A that one group of tiles keeps in L2: up to 24 MB and 16 row blocks
  const long long block = 2ll * kBM * p.K * 2;
  p.group_m = static_cast<int>(std::min<long long>(std::min(m_tiles, 16), std::max<long long>(1, (24ll << 20) / block)));
  const long long items = static_cast<long long>(m_tiles) * n_tiles * p.splits;
  const int pairs = static_cast<int>(std::min<long long>(items, pairs_cap));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * pairs, 1, 1);
  cfg.blockDim = dim3(kThreads, 1, 1);
  cfg.dynamicSmemBytes = T::kSmem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return static_cast<int>(cudaLaunchKernelEx(&cfg, gemm_bf16_2sm_kernel<kBN>, ma, mb, ma2, mb2, md, mr, p));
}

// Width of the tile: the one whose last wave of pairs costs less. A pair walks its tiles one after the other; a k block of
// 128 columns takes about 0.65 of one of 256 (it moves three quarters of the bytes), and a tile about 4 blocks' time more
// than its blocks. LoRA segments must end on tile boundaries.
static int pair_width(const GemmParams& p, int pairs) {
  if (p.seg_mode == 1)
    for (int i = 0; i < 3; ++i)
      if (p.seg_end[i] != 0x7fffffff && p.seg_end[i] % 256) return 128;
  const long long m_tiles = (p.M + 2 * kBM - 1) / (2 * kBM), per = (p.nk1 + p.nk2 + p.splits - 1) / p.splits;
  auto cost = [&](int bn, int per_block) {
    const long long items = m_tiles * ((p.N + bn - 1) / bn) * p.splits;
    return (items + pairs - 1) / pairs * (per * per_block + 400);
  };
  return cost(128, 65) < cost(256, 100) ? 128 : 256;
}

}  // namespace pm

using namespace pm;

// Same contract as pm_gemm_bf16 with the tile 256 rows high per CTA pair; its width (256 or 128 columns) is chosen here.
extern "C" int pm_gemm_bf16_2sm(const void* A, int a_mn, int lda, int a_rows, const void* B, int b_mn, int ldb,
                                int b_rows, const void* A2, int a2_mn, int lda2, int a2_k, const void* B2, int b2_mn,
                                int ldb2, int b2_rows, void* D, int out_mode, int ldd, const void* R, int ldr, int M,
                                int N, int K, int K2, int n_store, float alpha, int splits, int seg_mode,
                                const int* seg_end, int seg_r, int max_ctas, float* tail, int tail_from, int ld_tail,
                                int* status, cudaStream_t stream) {
  if (tail && (out_mode != 0 || R || tail_from % 8 || (reinterpret_cast<uintptr_t>(tail) & 15))) return -20;
  if (splits < 1 || (splits > 1 && (out_mode < 2 || out_mode > 3))) return -12;   // split-K needs the atomic modes
  if (M <= 0 || N <= 0 || K <= 0) return -13;
  if (seg_mode < 0 || seg_mode > 2) return -16;
  if (out_mode == 0 && ((ldd % 8) || (reinterpret_cast<uintptr_t>(D) & 15))) return -14;
  if (R && ((ldr % 8) || (reinterpret_cast<uintptr_t>(R) & 15))) return -15;
  GemmParams p{};
  p.M = M; p.N = N; p.K = K; p.K2 = K2;
  p.a_mn = a_mn; p.b_mn = b_mn; p.a2_mn = a2_mn; p.b2_mn = b2_mn;
  p.nk1 = (K + kBK - 1) / kBK;
  p.nk2 = K2 > 0 ? (K2 + kBK - 1) / kBK : 0;
  p.splits = splits;
  p.out_mode = out_mode; p.ldd = ldd; p.ldr = ldr; p.n_store = n_store > 0 ? n_store : N;
  p.alpha = alpha; p.D = D; p.R = R;
  p.seg_mode = seg_mode; p.seg_r = seg_r;
  for (int i = 0; i < 4; ++i) p.seg_end[i] = (seg_mode && seg_end) ? seg_end[i] : 0x7fffffff;
  p.status = status;
  p.tail = tail; p.tail_from = tail_from; p.ld_tail = ld_tail;
  const int cap = std::max(1, (max_ctas > 0 ? max_ctas : num_sms()) / 2);
  return pair_width(p, cap) == 256
             ? launch_pair<256>(p, A, lda, a_rows, B, ldb, b_rows, A2, lda2, a2_k, B2, ldb2, b2_rows, cap, stream)
             : launch_pair<128>(p, A, lda, a_rows, B, ldb, b_rows, A2, lda2, a2_k, B2, ldb2, b2_rows, cap, stream);
}

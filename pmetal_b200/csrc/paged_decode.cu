// Attention of a decode step over the paged cache: one or a few new tokens per sequence, head_dim 128, up to 8 query heads per
// kv head, bf16 or int8 cache (layouts as in attention.cu).
//
// The work is one pass over the cached keys and values, so what counts is bytes in flight: one warp brings whole blocks (64 keys)
// by TMA into a ring of 2 to 6 stages, four warps take a quarter of each block (16 keys) into the fragments of mma.m16n8k16 and
// share nothing until the end. S = Q K^T has the heads as rows; its accumulators are, as they stand, the B operand of
// O^T = V^T P^T, whose A operand pairs the values of two keys with one byte permute per pair. The MMAs only need their operands
// to agree on which channel sits in which slot, so the slots follow 16-byte shared-memory loads.
//
// The keys of a row are cut over the CTAs of a cluster, which merge their partial results through distributed shared memory.
//
// int8: codes become bf16 exactly (|code| <= 127 has 7 bits); the scale of a (key, 64 channels) multiplies the partial score in
// fp32, and the probability before its rounding to bf16, so a cached value is never rounded itself.
//
// The last block may hold anything past the keys, what a sequence that gave the block back left there included (NaN, infinities): scores
// there are replaced, values are taken as zero, since a probability of zero would not silence them.
//
// Probabilities meet bf16 values as two bf16 (the rounded one and what it leaves, two products), about 2^-17 of each: one bf16 alone
// costs 2 to 12 % of a sum whose terms nearly cancel. The second product takes up to 3 % of the kernel's time.
//
// Measured, captured over cold caches (here; 64-row tiles, split keys and a merge kernel; bytes at 6.5 TB/s):
//   64 x 450 keys, 16 heads on 8: 28.9, 30.4, 18.1 us      16 x 700: 12.5, 15.7, 7.1 us      1 x 6000: 11.5, 18.0, 3.8 us
//   8 x 6000 keys: 34.5, 42.0, 30.2 us; int8: 35.5, 69.3, 15.1 us (expanding the codes)
#include <algorithm>

#include "gemm_pair.cuh"
#include "pdl.cuh"
#include "pmetal_b200.h"

namespace pm {

struct PagedDecodeParams {
  const __nv_bfloat16* q;        // [total_q, hq, 128]
  const void* k_cache;           // [num_blocks, 64, hkv, 128]
  const void* v_cache;
  const float* k_scale;          // int8: [num_blocks, 64, hkv, 2]
  const float* v_scale;
  __nv_bfloat16* out;            // [total_q, hq, 128]
  const int *block_table, *seq_lens, *q_start, *q_lens;
  int max_blocks, max_q, hq, hkv, rep, splits, stages;
  float scale;
  int* status;
};

// Groups of four warps on keys, block b goes to group b % groups; one more warp fetches. Expanding int8 codes is most of an int8
// step's work, so it has two groups.
template <bool kQ8>
struct PdShape {
  static constexpr int kGroups = kQ8 ? 2 : 1, kWarps = 4 * kGroups, kThreads = 32 * kWarps + 32, kPerSm = kQ8 ? 2 : 3;
};
constexpr int kPdHeads = 8;

__device__ __forceinline__ void pd_mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ float pd_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// what the two bf16 of `packed` leave of (a, b), as bf16
__device__ __forceinline__ uint32_t pd_rest(float a, float b, uint32_t packed) {
  return pack_bf16x2(a - __uint_as_float(packed << 16), b - __uint_as_float(packed & 0xffff0000u));
}
// byte i of a word of biased codes (code + 128) as the fp32 bits of the code: 2^23 + u has u in its low bits
__device__ __forceinline__ uint32_t pd_code(uint32_t biased, int i) {
  return __float_as_uint(__uint_as_float(__byte_perm(biased, 0x4B000000u, 0x7540u | i)) - 8388736.f);
}
// 16 bytes of row `row` (128 bytes, 128B-swizzled box) of a stage
__device__ __forceinline__ uint4 pd_lds16(uint32_t box, int row, int chunk) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "r"(box + row * 128 + ((chunk ^ (row & 7)) << 4)));
  return v;
}
__device__ __forceinline__ uint2 pd_lds8(uint32_t box, int row, int half) {      // half: 8-byte piece
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];"
               : "=r"(v.x), "=r"(v.y)
               : "r"(box + row * 128 + (((half >> 1) ^ (row & 7)) << 4) + (half & 1) * 8));
  return v;
}

constexpr int kPdBox = 64 * 128;                 // 64 keys x 128 bytes
// bytes of a ring stage: keys, values, int8: their scales (64 x 8 bytes each)
__host__ __device__ constexpr int pd_stage(bool q8) { return q8 ? 2 * kPdBox + 1024 : 4 * kPdBox; }
__device__ __forceinline__ void pd_cp_async8(uint32_t dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}
// one arrival on `bar` once this thread's cp.async copies so far have landed
__device__ __forceinline__ void pd_cp_async_arrive(uint64_t* bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

template <bool kQ8>
__global__ void __launch_bounds__(PdShape<kQ8>::kThreads, PdShape<kQ8>::kPerSm)
paged_decode_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v, const PagedDecodeParams p) {
  constexpr int kBoxes = kQ8 ? 1 : 2, kStage = pd_stage(kQ8), kGroups = PdShape<kQ8>::kGroups, kWarps = PdShape<kQ8>::kWarps;
  pdl_launch_dependents();
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  float (*s_o)[kPdHeads][128] = reinterpret_cast<float (*)[kPdHeads][128]>(smem);   // after the loop: per warp; then [0] the CTA's result
  __shared__ float s_ml[kWarps][kPdHeads][2];
  __shared__ float s_part_ml[kPdHeads][2];
  __shared__ uint64_t full_bar[kMaxStages], empty_bar[kMaxStages];
  __shared__ int abort_word;
  volatile int* abort_flag = &abort_word;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
  const int row = blockIdx.x / p.splits, rank = blockIdx.x - row * p.splits, hk = blockIdx.y;
  const int seq = row / p.max_q, qi = row - seq * p.max_q;
  // lengths, table and the keys of earlier steps were there before the chain of launches began; the tokens of this step and the
  // queries are the previous kernel's
  const int q_len = p.q_lens[seq], seq_len = p.seq_lens[seq], q_first = p.q_start[seq];
  const int kv = seq_len - q_len + qi + 1;
  if (qi >= q_len || kv <= 0) {                 // the whole cluster
    pdl_wait();
    return;
  }
  if (threadIdx.x == 0) {
    for (int i = 0; i < p.stages; ++i) {
      mbar_init(&full_bar[i], kQ8 ? 33 : 1);    // the bytes of the boxes; int8: and every lane's scales
      mbar_init(&empty_bar[i], 4);
    }
    abort_word = 0;
    mbar_init_fence();
  }
  const long long out_row = static_cast<long long>(q_first + qi) * p.hq + hk * p.rep;
  const int n_blocks = (kv + 63) >> 6, per = (n_blocks + p.splits - 1) / p.splits;
  const int b0 = rank * per, b1 = min(n_blocks, b0 + per);
  const int* bt = p.block_table + static_cast<long long>(seq) * p.max_blocks;
  __syncthreads();

  float m_run = -INFINITY, l_run = 0.f;         // of head g; l: this lane's keys only
  if (warp == kWarps) {
    // ------------------------------------------------------------------ TMA: blocks b0 .. b1 - 1
    const bool elected = elect_one();
    if (elected) {
      tma_prefetch_desc(&map_k);
      tma_prefetch_desc(&map_v);
    }
    const int old_blocks = (seq_len - q_len) >> 6;       // blocks without a token of this step
    bool waited = false, ok = true;
    int s = 0;
    uint32_t ph = 1;
    int entry = 0;
    for (int b = b0; b < b1 && ok; ++b) {
      if (((b - b0) & 31) == 0) entry = bt[min(b + lane, n_blocks - 1)];
      const int blk = __shfl_sync(0xffffffffu, entry, (b - b0) & 31);
      if (!waited && b >= old_blocks) {
        pdl_wait();
        waited = true;
      }
      ok = mbar_wait(&empty_bar[s], ph, abort_flag, p.status, kTimeoutProducer);
      if (ok && elected) {
        uint8_t* dst = smem + s * kStage;
        mbar_expect_tx(&full_bar[s], 2 * kBoxes * kPdBox);
#pragma unroll
        for (int c = 0; c < kBoxes; ++c) tma_load_2d(dst + c * kPdBox, &map_k, &full_bar[s], hk * (kQ8 ? 64 : 128) + c * 64, blk * 64);
#pragma unroll
        for (int c = 0; c < kBoxes; ++c) tma_load_2d(dst + (kBoxes + c) * kPdBox, &map_v, &full_bar[s], hk * (kQ8 ? 64 : 128) + c * 64, blk * 64);
      }
      if (kQ8 && ok) {
        const uint32_t dst = smem_u32(smem + s * kStage + 2 * kPdBox) + lane * 8;
        const long long at = ((static_cast<long long>(blk) * 64 + lane) * p.hkv + hk) * 2, half = 64ll * p.hkv;
        pd_cp_async8(dst, p.k_scale + at);
        pd_cp_async8(dst + 256, p.k_scale + at + half);
        pd_cp_async8(dst + 512, p.v_scale + at);
        pd_cp_async8(dst + 768, p.v_scale + at + half);
        pd_cp_async_arrive(&full_bar[s]);
      }
      if (++s == p.stages) { s = 0; ph ^= 1; }
    }
    if (!waited) pdl_wait();
  }
  // ---------------------------------------------------------------------- keys: a warp takes a quarter of every block
  const int quarter = (warp & 3) * 16, group = warp >> 2;
  float o[8][4];                                // O^T: tile (h, w): channels h * 64 + 8 g + 2 w + {0, 1}, heads 2 t4 + {0, 1}
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int e = 0; e < 4; ++e) o[i][e] = 0.f;
  const float sl2 = p.scale * 1.4426950408889634f;

  if (warp < kWarps) {
  pdl_wait();
  // Q fragments. Channel slots: bf16 chunk c holds channels 32 c + 8 t4 .. + 7 of a lane, int8 chunk c 64 c + 16 t4 .. + 15
  uint32_t qf[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) qf[i] = 0u;
  if (g < p.rep) {
    const __nv_bfloat16* qr = p.q + (out_row + g) * 128;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int ch = kQ8 ? (c >> 1) * 64 + t4 * 16 + (c & 1) * 8 : c * 32 + t4 * 8;
      const uint4 v = *reinterpret_cast<const uint4*>(qr + ch);
      qf[4 * c] = v.x; qf[4 * c + 1] = v.y; qf[4 * c + 2] = v.z; qf[4 * c + 3] = v.w;
    }
  }
  int st = group;                               // stages are a multiple of the groups
  uint32_t ph = 0;
  bool ok = true;
  for (int b = b0 + group; b < b1; b += kGroups) {
    const int j0 = b * 64 + quarter;
    ok = mbar_wait(&full_bar[st], ph, abort_flag, p.status, kTimeoutEpilogue);
    if (!ok) break;
    if (j0 < kv) {                              // the quarter of the last block may lie past the keys
    const uint32_t kbox = smem_u32(smem + st * kStage), vbox = kbox + kBoxes * kPdBox;
    float2 ks[2][2], vs[4];
    if (kQ8) {
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int key = 2 * t4 + (u & 1) + (u >> 1) * 8;
        const float2* sc = reinterpret_cast<const float2*>(smem + st * kStage + 2 * kPdBox) + quarter + key;
        ks[u >> 1][u & 1] = sc[0];
        vs[u] = j0 + key < kv ? sc[64] : make_float2(0.f, 0.f);
      }
    }
    float s[2][2];
#pragma unroll
    for (int nt = 0; nt < 2; ++nt) {
      float acc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
      if (kQ8) {
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const uint4 kr = pd_lds16(kbox, quarter + nt * 8 + g, c * 4 + t4);
          const uint32_t w[4] = {kr.x, kr.y, kr.z, kr.w};
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const uint32_t u = w[j] ^ 0x80808080u;
            pd_mma(acc[c & 1], qf[8 * c + 2 * j], 0u, qf[8 * c + 2 * j + 1], 0u, __byte_perm(pd_code(u, 0), pd_code(u, 1), 0x7632),
                   __byte_perm(pd_code(u, 2), pd_code(u, 3), 0x7632));
          }
        }
#pragma unroll
        for (int e = 0; e < 2; ++e) s[nt][e] = fmaf(acc[0][e], ks[nt][e].x, acc[1][e] * ks[nt][e].y) * sl2;
      } else {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const uint4 kr = pd_lds16(kbox + (c >> 1) * kPdBox, quarter + nt * 8 + g, (c & 1) * 4 + t4);
          pd_mma(acc[0], qf[4 * c], 0u, qf[4 * c + 1], 0u, kr.x, kr.y);
          pd_mma(acc[1], qf[4 * c + 2], 0u, qf[4 * c + 3], 0u, kr.z, kr.w);
        }
#pragma unroll
        for (int e = 0; e < 2; ++e) s[nt][e] = (acc[0][e] + acc[1][e]) * sl2;
      }
    }
    float mx = -INFINITY;
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        if (j0 + nt * 8 + 2 * t4 + e >= kv) s[nt][e] = -INFINITY;
        mx = fmaxf(mx, s[nt][e]);
      }
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
    const float m_new = fmaxf(m_run, mx), m_use = m_new == -INFINITY ? 0.f : m_new;
    const float corr = m_run == -INFINITY ? 0.f : pd_exp2(m_run - m_use);
    m_run = m_new;
    float pr[2][2];
    l_run *= corr;
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        pr[nt][e] = pd_exp2(s[nt][e] - m_use);
        l_run += pr[nt][e];
      }
    if (__any_sync(0xffffffffu, corr != 1.f)) {
      const float ca = __shfl_sync(0xffffffffu, corr, t4 * 8), cb = __shfl_sync(0xffffffffu, corr, t4 * 8 + 4);
#pragma unroll
      for (int i = 0; i < 8; ++i) { o[i][0] *= ca; o[i][1] *= cb; o[i][2] *= ca; o[i][3] *= cb; }
    }
    if (kQ8) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float f[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) f[u] = pr[u >> 1][u & 1] * (h ? vs[u].y : vs[u].x);
        const uint32_t pb0 = pack_bf16x2(f[0], f[1]), pb1 = pack_bf16x2(f[2], f[3]);
        uint2 vr[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) vr[u] = pd_lds8(vbox, quarter + 2 * t4 + (u & 1) + (u >> 1) * 8, h * 8 + g);
#pragma unroll
        for (int w = 0; w < 4; ++w) {
          uint32_t x[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) x[u] = (w < 2 ? vr[u].x : vr[u].y) ^ 0x80808080u;
          const int i0 = (w & 1) * 2, i1 = i0 + 1;
          pd_mma(o[h * 4 + w], __byte_perm(pd_code(x[0], i0), pd_code(x[1], i0), 0x7632), __byte_perm(pd_code(x[0], i1), pd_code(x[1], i1), 0x7632),
                 __byte_perm(pd_code(x[2], i0), pd_code(x[3], i0), 0x7632), __byte_perm(pd_code(x[2], i1), pd_code(x[3], i1), 0x7632), pb0, pb1);
        }
      }
    } else {
      // probabilities keep 16 bits of their mantissa: the bf16 value and, in a second product, what it leaves
      const uint32_t pb0 = pack_bf16x2(pr[0][0], pr[0][1]), pb1 = pack_bf16x2(pr[1][0], pr[1][1]);
      const uint32_t pl0 = pd_rest(pr[0][0], pr[0][1], pb0), pl1 = pd_rest(pr[1][0], pr[1][1], pb1);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint4 vr[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int key = 2 * t4 + (u & 1) + (u >> 1) * 8;
          vr[u] = pd_lds16(vbox + h * kPdBox, quarter + key, g);
          if (j0 + key >= kv) vr[u] = make_uint4(0u, 0u, 0u, 0u);
        }
#pragma unroll
        for (int w = 0; w < 4; ++w) {
          uint32_t x[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) x[u] = w == 0 ? vr[u].x : w == 1 ? vr[u].y : w == 2 ? vr[u].z : vr[u].w;
          const uint32_t a0 = __byte_perm(x[0], x[1], 0x5410), a1 = __byte_perm(x[0], x[1], 0x7632), a2 = __byte_perm(x[2], x[3], 0x5410),
                         a3 = __byte_perm(x[2], x[3], 0x7632);
          pd_mma(o[h * 4 + w], a0, a1, a2, a3, pb0, pb1);
          pd_mma(o[h * 4 + w], a0, a1, a2, a3, pl0, pl1);
        }
      }
    }
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&empty_bar[st]);
    if ((st += kGroups) >= p.stages) { st = group; ph ^= 1; }
  }
  }

  // ---- merge the warps; the ring has been read and is the exchange area from here on
  __syncwarp();
  if (*abort_flag) {                            // an abandoned wait: let the copies in flight land first
    const unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) { }
  }
  __syncthreads();
  if (warp < kWarps) {
    l_run += __shfl_xor_sync(0xffffffffu, l_run, 1);
    l_run += __shfl_xor_sync(0xffffffffu, l_run, 2);
    if (t4 == 0) {
      s_ml[warp][g][0] = m_run;
      s_ml[warp][g][1] = l_run;
    }
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int head = 2 * t4 + e;
      if (head < p.rep) {
#pragma unroll
        for (int i = 0; i < 8; ++i)
          *reinterpret_cast<float2*>(&s_o[warp][head][(i >> 2) * 64 + g * 8 + (i & 3) * 2]) = make_float2(o[i][e], o[i][2 + e]);
      }
    }
  }
  __syncthreads();
  const int d = threadIdx.x;                    // channel
  for (int h = 0; h < p.rep && d < 128; ++h) {
    float m = -INFINITY;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) m = fmaxf(m, s_ml[w][h][0]);
    float acc = 0.f, l = 0.f;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      const float f = s_ml[w][h][0] == -INFINITY ? 0.f : pd_exp2(s_ml[w][h][0] - m);
      acc += f * s_o[w][h][d];
      l += f * s_ml[w][h][1];
    }
    if (p.splits == 1) {
      p.out[(out_row + h) * 128 + d] = __float2bfloat16(l > 0.f ? acc / l : 0.f);
    } else {
      s_o[0][h][d] = acc;                       // only this thread reads or writes channel d of the partial results
      if (d == 0) { s_part_ml[h][0] = m; s_part_ml[h][1] = l; }
    }
  }
  if (p.splits == 1) return;

  // ---- merge the cluster: every CTA finishes its share of the (head, channel) pairs
  cluster_sync_all();
  const int share = p.rep * 128 / p.splits;
  const uint32_t o_addr = smem_u32(&s_o[0][0][0]), ml_addr = smem_u32(&s_part_ml[0][0]);
  for (int e = rank * share + threadIdx.x; e < (rank + 1) * share; e += PdShape<kQ8>::kThreads) {
    const int h = e >> 7;
    float mv[8], lv[8], ov[8], m = -INFINITY;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      mv[c] = -INFINITY;
      lv[c] = ov[c] = 0.f;
      if (c < p.splits) {
        const uint32_t ml = map_to_cta(ml_addr, c) + h * 8;
        mv[c] = ld_cluster_f32(ml);
        lv[c] = ld_cluster_f32(ml + 4);
        ov[c] = ld_cluster_f32(map_to_cta(o_addr, c) + e * 4);
      }
    }
#pragma unroll
    for (int c = 0; c < 8; ++c) m = fmaxf(m, mv[c]);
    float acc = 0.f, l = 0.f;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const float f = mv[c] == -INFINITY ? 0.f : pd_exp2(mv[c] - m);
      acc += f * ov[c];
      l += f * lv[c];
    }
    p.out[out_row * 128 + e] = __float2bfloat16(l > 0.f ? acc / l : 0.f);
  }
  cluster_sync_all();                           // the peers have read this CTA's partial result
}

}  // namespace pm

using namespace pm;

// q, out: [total_q, hq, 128]; caches, table and lengths as for pm_paged_attn_ex, no window. k_scale / v_scale null: bf16 cache. Token i of
// sequence s sees the keys j <= seq_lens[s] - q_lens[s] + i. hq / hkv up to 8. splits 0: chosen here (1, 2, 4 or 8 slices of the keys).
extern "C" int pm_paged_decode(const void* q, const void* k_cache, const void* v_cache, const float* k_scale, const float* v_scale,
                               void* out, const int* block_table, const int* seq_lens, const int* q_start, const int* q_lens,
                               int num_seqs, int max_blocks, int num_blocks, int max_q, int hq, int hkv, float scale, int splits, int* status,
                               cudaStream_t st) {
  if (num_seqs <= 0 || num_blocks <= 0 || max_q <= 0 || hkv <= 0 || hkv > 65535 || hq % hkv || hq / hkv > kPdHeads) return -1;
  if ((k_scale == nullptr) != (v_scale == nullptr)) return -4;
  if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k_cache) | reinterpret_cast<uintptr_t>(v_cache)) & 15) return -5;
  PagedDecodeParams p{};
  p.q = static_cast<const __nv_bfloat16*>(q);
  p.k_cache = k_cache; p.v_cache = v_cache; p.k_scale = k_scale; p.v_scale = v_scale;
  p.out = static_cast<__nv_bfloat16*>(out);
  p.block_table = block_table; p.seq_lens = seq_lens; p.q_start = q_start; p.q_lens = q_lens;
  p.max_blocks = max_blocks; p.max_q = max_q; p.hq = hq; p.hkv = hkv; p.rep = hq / hkv; p.scale = scale;
  const long long rows = static_cast<long long>(num_seqs) * max_q;
  const long long ctas = rows * hkv;
  if (splits <= 0) {
    // up to two CTAs per SM where the table has that many blocks; captured steps have tables of at least 8
    const int blocks = std::max(max_blocks, 8);
    splits = 1;
    while (splits < 8 && ctas * splits * 2 <= 2ll * num_sms() && splits * 2 <= blocks) splits *= 2;
  }
  if (splits != 1 && splits != 2 && splits != 4 && splits != 8) return -2;
  if (rows * splits > 0x7fffffffll) return -3;
  p.splits = splits;
  p.status = status;
  // the ring: as deep as the CTAs that share an SM allow, at most six stages, an even number
  const int stage = pd_stage(k_scale != nullptr), most = k_scale ? PdShape<true>::kPerSm : PdShape<false>::kPerSm;
  const int warps = k_scale ? PdShape<true>::kWarps : PdShape<false>::kWarps;
  const int per_sm = static_cast<int>(std::min<long long>(most, (ctas * splits + num_sms() - 1) / num_sms()));
  p.stages = std::max(2, std::min(6, (220 * 1024 / per_sm - 4096) / stage)) & ~1;
  const int smem = std::max(p.stages * stage, warps * kPdHeads * 128 * 4) + 1024;
  static DeviceOnce once;
  if (once.pending()) {
    cudaError_t e = cudaFuncSetAttribute(paged_decode_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(paged_decode_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024);
    if (e != cudaSuccess) return static_cast<int>(e);
    once.mark();
  }
  CUtensorMap mk, mv;
  int rc;
  for (int i = 0; i < 2; ++i) {
    CUtensorMap* m = i ? &mv : &mk;
    const void* base = i ? v_cache : k_cache;
    // an int8 row of 128 channels is mapped as 64 pairs of bytes
    const uint64_t width = static_cast<uint64_t>(hkv) * (k_scale ? 64 : 128);
    if ((rc = make_map(m, base, width, 64ull * num_blocks, width, 64, 64))) return rc;
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(static_cast<unsigned>(rows * splits), static_cast<unsigned>(hkv));
  cfg.blockDim = dim3(32 * warps + 32);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  int n = 0;
  if (splits > 1) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = splits;
    attr[n].val.clusterDim.y = attr[n].val.clusterDim.z = 1;
    ++n;
  }
  if (pdl_scope_depth > 0 || pdl_enabled()) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n].val.programmaticStreamSerializationAllowed = 1;
    ++n;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  return static_cast<int>(k_scale ? cudaLaunchKernelEx(&cfg, paged_decode_kernel<true>, mk, mv, p)
                                  : cudaLaunchKernelEx(&cfg, paged_decode_kernel<false>, mk, mv, p));
}

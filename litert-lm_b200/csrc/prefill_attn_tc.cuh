// Prefill attention on the 5th-generation tensor cores (tcgen05 + TMEM + TMA).
//
// One CTA owns a 128-row query tile of one kv head: 128 / G consecutive tokens
// times the G query heads of the group (GQA packing: every K/V tile is loaded
// once for all heads that share it).  Keys are walked in tiles of 64:
//
//   S  = Q K^T        tcgen05.mma  M128 N64  K=hd   (Q, K tiles by TMA, K-major)
//   P  = exp(S - B)   softmax warps: tcgen05.ld, mask, exp2, bf16, tcgen05.st back
//                     into the columns S came from
//   O += P V          tcgen05.mma  M128 N=hd K64    (P is the A operand in tensor
//                                                    memory; V comes from a TRANSPOSED
//                                                    bf16 copy of the cache, so it is
//                                                    K-major in shared memory)
//
// Q and K are RMS-normalised per head before the product, so every score obeys
// |s| <= B = sqrt(hd) max|g_q| max|g_k|.  The softmax is therefore shifted by the
// constant B instead of a running maximum: exact by shift invariance, no
// overflow, and the O accumulator in tensor memory never has to be rescaled.
// (Layers whose bound is too large for fp32 exponents use the CUDA-core kernel.)
//
// At head size 256 the queries are copied to tensor memory and enter S = Q K^T from there: an M128 N64 K16 product takes 32
// cycles, but reading its 4 KB of Q from shared memory about 60.
//
// S is double buffered in tensor memory and the MMA warp issues S(j+1) before
// P(j) V(j), so the tensor pipe works on the next scores while the softmax
// warps turn the current ones into probabilities.  K and V tiles have their
// own two-stage rings: a K stage is released by the S product that read it, a
// V stage by the P V product.
//
// Warp roles: warp 0 TMA producer, warp 1 MMA issuer (owns TMEM), warps 2-9
// softmax + epilogue (two threads per query row = TMEM lane, 32 keys each).
// All waits are bounded.
#pragma once
#include <cuda.h>

#include "common.cuh"
#include "prefill_ops.cuh"
#include "prefill_gemm_ts.cuh"

namespace b200lm {

constexpr int kFaThreads = 320;
constexpr int kFaBN = 64;            // keys per tile
constexpr float kFaMaxBound = 40.0f; // exp(-2 * 40) is still a normal fp32 number

template <int HD>
struct FaSmem {
  static constexpr int kQ = 128 * HD * 2;            // 128 rows, HD/64 sub-tiles of 128 B rows
  static constexpr int kK = kFaBN * HD * 2;          // per stage
  static constexpr int kV = HD * kFaBN * 2;          // per stage: HD rows of 64 keys
  static constexpr int kTotal = kQ + 2 * kK + 2 * kV + 1024 + 1024;
};

struct FaArgs {
  int T, start, hq, hkv, window, is_global;
  const int* page_table;
  __nv_bfloat16* out;      // [T][hq][hd]
  float bound;             // B
  int* err;
};

__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

template <int HD>
__global__ void __launch_bounds__(kFaThreads, 1)
flash_prefill_tc_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                        const __grid_constant__ CUtensorMap tmVt, FaArgs g) {
  extern __shared__ unsigned char fa_raw[];
  unsigned char* sm = reinterpret_cast<unsigned char*>(((uintptr_t)fa_raw + 1023) & ~(uintptr_t)1023);
  using L = FaSmem<HD>;
  unsigned char* sQ = sm;
  unsigned char* sK = sQ + L::kQ;
  unsigned char* sV = sK + 2 * L::kK;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sV + 2 * L::kV);
  uint64_t* q_full = bars;            // Q tile landed
  uint64_t* k_full = bars + 1;        // [2]
  uint64_t* k_empty = bars + 3;       // [2] S = Q K^T of the tile is done with the stage
  uint64_t* v_full = bars + 5;        // [2]
  uint64_t* v_empty = bars + 7;       // [2] P V of the tile is done with the stage
  uint64_t* s_full = bars + 9;        // [2] scores complete in S buffer
  uint64_t* p_full = bars + 11;       // [2] probabilities written over the scores
  uint64_t* o_full = bars + 13;       // all MMAs complete
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 14);
  float* l_part = reinterpret_cast<float*>(bars + 16);     // [128] row sums of the upper 32 keys
  uint64_t* q_tmem = bars + 80;       // Q copied to tensor memory

  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int G = g.hq / g.hkv;
  const int TT = 128 / G;                       // tokens per tile
  // later query tiles see more keys: they are scheduled first so the longest CTAs do not start last
  const int t0 = ((int)gridDim.x - 1 - (int)blockIdx.x) * TT, kvh = blockIdx.y;
  constexpr int KB = HD / 64;                   // 64-column blocks of the head dimension
  constexpr uint32_t kTmemCols = HD + 2 * kFaBN <= 256 ? 256 : 512;
  constexpr uint32_t kOCol = 0, kSCol = HD;     // O, then two S buffers of 64 columns, then Q where it fits
  constexpr bool kQTmem = HD == 256;            // with head size 128, two CTAs share an SM's tensor memory
  constexpr uint32_t kQCol = HD + 2 * kFaBN;

  // key range of this query tile
  const int qpos_min = g.start + t0;
  const int qpos_max = g.start + min(t0 + TT, g.T) - 1;
  const int k_lo = g.is_global ? 0 : max(0, qpos_min - g.window + 1);
  const int tile_lo = k_lo / kFaBN, tile_hi = qpos_max / kFaBN;
  const int ntiles = tile_hi - tile_lo + 1;

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(&k_full[s], 1);
      mbar_init(&k_empty[s], 1);
      mbar_init(&v_full[s], 1);
      mbar_init(&v_empty[s], 1);
      mbar_init(&s_full[s], 1);
      mbar_init(&p_full[s], 8);
    }
    mbar_init(o_full, 1);
    mbar_init(q_tmem, 8);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) tmem_alloc(tmem_slot, kTmemCols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  pdl_wait();                 // set-up done; Q, K, V below come from the preceding kernel
  pdl_launch_dependents();

  bool ok = true;             // none of this thread's waits has given up
  if (warp == 0) {
    // ---- producer
    const bool leader = elect_one();
    if (leader) {
      // Q tile: KB boxes of 64 columns x (G heads x TT tokens) rows
      mbar_arrive_expect_tx(q_full, L::kQ);
      for (int kb = 0; kb < KB; ++kb) {
        asm volatile(
            "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
            ::"r"(smem_u32(sQ + kb * 128 * 128)), "l"(&tmQ), "r"(kb * 64), "r"(kvh * G), "r"(t0), "r"(smem_u32(q_full))
            : "memory");
      }
    }
    for (int j = 0; j < ntiles && ok; ++j) {
      const int s = j & 1, n = j >> 1;
      const int key0 = (tile_lo + j) * kFaBN;
      const int page = g.page_table[key0 / kPage], slot0 = key0 % kPage;
      if (n > 0) ok = __all_sync(0xffffffffu, mbar_wait(&k_empty[s], (n - 1) & 1, g.err));
      if (ok && leader) {
        mbar_arrive_expect_tx(&k_full[s], L::kK);
        const int krow = (page * g.hkv + kvh) * kPage + slot0;
        for (int kb = 0; kb < KB; ++kb)
          tma_load_2d(sK + s * L::kK + kb * kFaBN * 128, &tmK, kb * 64, krow, &k_full[s]);
      }
      if (ok && n > 0) ok = __all_sync(0xffffffffu, mbar_wait(&v_empty[s], (n - 1) & 1, g.err));
      if (ok && leader) {
        mbar_arrive_expect_tx(&v_full[s], L::kV);
        tma_load_2d(sV + s * L::kV, &tmVt, slot0, (page * g.hkv + kvh) * HD, &v_full[s]);
      }
      __syncwarp();
    }
  } else if (warp == 1) {
    // ---- MMA issue: S(0), then per tile S(j+1) before P(j) V(j)
    const uint32_t idesc_s = umma_idesc_bf16(128, kFaBN);
    const uint32_t idesc_o = umma_idesc_bf16(128, HD);
    auto issue_s = [&](int j) {
      const int s = j & 1;
#pragma unroll
      for (int kb = 0; kb < KB; ++kb) {
        const uint64_t qd = umma_desc_sw128(smem_u32(sQ + kb * 128 * 128));
        const uint64_t kd = umma_desc_sw128(smem_u32(sK + s * L::kK + kb * kFaBN * 128));
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if constexpr (kQTmem) umma_bf16_ts(tmem + kSCol + s * kFaBN, tmem + kQCol + (kb * 4 + k) * 8, kd + (uint64_t)(k * 2), idesc_s, (kb | k) ? 1u : 0u);
          else umma_bf16(tmem + kSCol + s * kFaBN, qd + (uint64_t)(k * 2), kd + (uint64_t)(k * 2), idesc_s, (kb | k) ? 1u : 0u);
      }
      umma_commit(&s_full[s]);
      umma_commit(&k_empty[s]);
    };
    const bool leader = elect_one();
    ok = __all_sync(0xffffffffu, mbar_wait2(kQTmem ? q_tmem : q_full, 0, &k_full[0], 0, g.err));
    if (ok) {
      tc_fence_after();
      if (leader) issue_s(0);
      __syncwarp();
    }
    for (int j = 0; j < ntiles && ok; ++j) {
      const int s = j & 1, n = j >> 1;
      if (j + 1 < ntiles) {
        ok = __all_sync(0xffffffffu, mbar_wait(&k_full[(j + 1) & 1], ((j + 1) >> 1) & 1, g.err));
        if (!ok) break;
        tc_fence_after();
        if (leader) issue_s(j + 1);
        __syncwarp();
      }
      ok = __all_sync(0xffffffffu, mbar_wait(&v_full[s], n & 1, g.err) && mbar_wait(&p_full[s], n & 1, g.err));
      if (!ok) break;
      tc_fence_after();
      if (leader) {
        const uint64_t vd = umma_desc_sw128(smem_u32(sV + s * L::kV));
#pragma unroll
        for (int k = 0; k < kFaBN / 16; ++k)      // P: 8 TMEM columns per 16 keys
          umma_bf16_ts(tmem + kOCol, tmem + kSCol + s * kFaBN + k * 8, vd + (uint64_t)(k * 2), idesc_o, (j | k) ? 1u : 0u);
        umma_commit(&v_empty[s]);
      }
      __syncwarp();
    }
    if (ok && leader) umma_commit(o_full);
    __syncwarp();
  } else {
    // ---- softmax warps: two threads per query row (TMEM lane), 32 keys each
    const int quarter = warp & 3;
    const int khalf = (warp - 2) >> 2;                 // which 32 keys of the tile
    const int r = quarter * 32 + lane;                 // row of the tile: token r / G, head r % G
    const int tok = t0 + r / G;
    const int qpos = g.start + tok;
    const uint32_t lane_addr = tmem + ((uint32_t)(quarter * 32) << 16);
    const float log2e = 1.4426950408889634f;
    const float shift = g.bound * log2e;
    float lsum = 0.f;
    if constexpr (kQTmem) {                            // half of the row's queries into tensor memory
      if (__all_sync(0xffffffffu, mbar_wait(q_full, 0, g.err))) {
#pragma unroll
        for (int c = 0; c < HD / 2; c += 32) {
          uint32_t q[16];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int col = khalf * (HD / 2) + c + 8 * i;
            const uint4 w = *reinterpret_cast<const uint4*>(sQ + col / 64 * 128 * 128 + r * 128 + (((col % 64 / 8) ^ (r & 7)) << 4));
            q[4 * i] = w.x; q[4 * i + 1] = w.y; q[4 * i + 2] = w.z; q[4 * i + 3] = w.w;
          }
          tmem_st16(lane_addr + kQCol + (khalf * (HD / 2) + c) / 2, q);
        }
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(q_tmem);
      }
    }
    // The eight warps leave this loop together: the named barrier tells all of them
    // whether a wait of one gave up.
    for (int j = 0; j < ntiles; ++j) {
      const int s = j & 1, n = j >> 1;
      uint32_t packed[16];
      const bool got = __all_sync(0xffffffffu, mbar_wait(&s_full[s], n & 1, g.err));
      if (got) {
        tc_fence_after();
        uint32_t v[32];
        tmem_ld32(lane_addr + kSCol + s * kFaBN + khalf * 32, v);
        const int key0 = (tile_lo + j) * kFaBN + khalf * 32;
        // every row of the tile sees every key of an interior tile: no mask needed there
        const bool interior = key0 + 31 <= qpos_min && (g.is_global || qpos_max - key0 < g.window);
        if (interior) {
#pragma unroll
          for (int c = 0; c < 32; c += 2) {
            const float p0 = ex2_approx(fmaf(__uint_as_float(v[c]), log2e, -shift));
            const float p1 = ex2_approx(fmaf(__uint_as_float(v[c + 1]), log2e, -shift));
            lsum += p0 + p1;
            __nv_bfloat162 h = __floats2bfloat162_rn(p0, p1);
            packed[c >> 1] = *reinterpret_cast<uint32_t*>(&h);
          }
        } else {
#pragma unroll
          for (int c = 0; c < 32; c += 2) {
            float p[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const int kpos = key0 + c + e;
              const bool open = kpos <= qpos && (g.is_global || qpos - kpos < g.window);
              p[e] = open ? ex2_approx(fmaf(__uint_as_float(v[c + e]), log2e, -shift)) : 0.f;
            }
            lsum += p[0] + p[1];
            __nv_bfloat162 h = __floats2bfloat162_rn(p[0], p[1]);
            packed[c >> 1] = *reinterpret_cast<uint32_t*>(&h);
          }
        }
      }
      // The 16 columns a thread writes lie inside the 32 that it or the other thread
      // of its row has just read, so all eight warps meet before anyone overwrites.
      ok = !block_gave_up([&] { return !got; }, bar_or<1, 256>);
      if (!ok) break;
      tmem_st16(lane_addr + kSCol + s * kFaBN + khalf * 16, packed);
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_full[s]);
    }
    // ---- epilogue: O / l -> bf16; this thread writes half of the head dimension
    if (khalf == 1) l_part[r] = lsum;
    asm volatile("bar.sync 1, 256;" ::: "memory");
    if (khalf == 0) lsum += l_part[r];
    asm volatile("bar.sync 1, 256;" ::: "memory");
    if (khalf == 0) l_part[r] = lsum;
    asm volatile("bar.sync 1, 256;" ::: "memory");
    lsum = l_part[r];
    ok = ok && __all_sync(0xffffffffu, mbar_wait(o_full, 0, g.err));
    if (ok) {
      tc_fence_after();
      const float inv = lsum > 0.f ? 1.0f / lsum : 0.f;
      const int head = kvh * G + (r % G);
      __nv_bfloat16* dst = g.out + ((size_t)tok * g.hq + head) * HD + khalf * (HD / 2);
#pragma unroll 1
      for (int cb = 0; cb < HD / 64; ++cb) {
        uint32_t o[32];
        tmem_ld32(lane_addr + kOCol + khalf * (HD / 2) + cb * 32, o);
        if (tok < g.T) {
#pragma unroll
          for (int c = 0; c < 32; c += 8) {
            uint4 w;
            __nv_bfloat162 h0 = __floats2bfloat162_rn(__uint_as_float(o[c]) * inv, __uint_as_float(o[c + 1]) * inv);
            __nv_bfloat162 h1 = __floats2bfloat162_rn(__uint_as_float(o[c + 2]) * inv, __uint_as_float(o[c + 3]) * inv);
            __nv_bfloat162 h2 = __floats2bfloat162_rn(__uint_as_float(o[c + 4]) * inv, __uint_as_float(o[c + 5]) * inv);
            __nv_bfloat162 h3 = __floats2bfloat162_rn(__uint_as_float(o[c + 6]) * inv, __uint_as_float(o[c + 7]) * inv);
            w.x = *reinterpret_cast<uint32_t*>(&h0); w.y = *reinterpret_cast<uint32_t*>(&h1);
            w.z = *reinterpret_cast<uint32_t*>(&h2); w.w = *reinterpret_cast<uint32_t*>(&h3);
            *reinterpret_cast<uint4*>(dst + cb * 32 + c) = w;
          }
        }
      }
    }
  }
  tc_fence_before();
  sync_after_waits(ok);
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, kTmemCols);
  }
}

}  // namespace b200lm

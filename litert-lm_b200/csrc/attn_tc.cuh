// Attention of many single-token queries over one bf16 cache on the 5th-generation tensor cores: the shape of
// attn_mma.cuh where a kv head has more rows than mma.sync handles well.
//
// A CTA owns 128 query rows of a kv head and a range of keys, walked in tiles of 32.  The contract is fp32: queries and
// probabilities enter the bf16 products as three bf16 terms each (x = hi + mid + lo, 24 bits).
//
//   S  = Q K^T    three products a 16-wide step.  hi and mid sit in shared memory, lo is the A operand in tensor memory
//                 (three 64 KB planes do not fit beside the ring).  The tensor core cuts its sums off rather than rounding
//                 them, so the leading products are spread out: a quarter of the head's hi products each, in two accumulators
//                 that are read twice a tile.  Part A is two quarters; part B the third, and in one chain of 36 (head size 256)
//                 lo, mid and the last quarter.
//   P          running maximum, exp2, three terms back into tensor memory
//   O_t = P V     V rows as they lie in the cache: the B operand with hd contiguous.  Every tile's product, a chain of six
//                 over 32 keys, leaves tensor memory and is added to fp32 registers, which is also where the running
//                 maximum rescales the sum.
// attn_mma.cuh has shorter chains in places (P V three over 16 keys, lo and mid apart from hi); atc_splits has both errors.
//
// Four CTAs with neighbouring key ranges are a cluster: they exchange their sums through distributed shared memory, a
// quarter of the head each, so that only a fourth of the splits goes through the scratch.
//
// The issue order is A(j + 1), B(j + 1), PV(j): the softmax of tile j runs beside PV(j - 1) and A(j + 1), the reading of A(j + 1)
// and the sum of O(j - 1) ahead of and beside B(j + 1).
//
// What bounds it: the products.  An M128 N32 K16 step reads 4 KB of Q from shared memory and takes about 60 cycles where
// the product takes 16; 32 of them, 16 with Q in tensor memory and six of PV (768 cycles) are 3300 cycles a tile of 32 keys
// at head size 256.
//
// Warps: 0 copies (TMA, no multicast), 1 issues the products and owns tensor memory, 4 - 11 softmax and sums (two threads
// per row: half of the tile's keys, then half of the head).  The latter take the registers that the first four give up
// (launched with 168: 4 warps x 56 + 8 warps x 224 = 12 x 168).  All waits on mbarriers are bounded; the cluster's barriers
// wait for CTAs whose every path comes to them.
#pragma once
#include <cuda.h>

#include "attn_mma.cuh"
#include "common.cuh"
#include "prefill_gemm_ts.cuh"
#include "prefill_ops.cuh"

namespace b200lm {

constexpr int kAtcThreads = 384, kAtcKeys = 32, kAtcStages = 3, kAtcCluster = 4;

template <int HD>
struct AtcShape {
  static constexpr int KB = HD / 64;                                 // 64-wide blocks of the head
  static constexpr int kPlane = 128 * HD * 2;                        // a term of the queries
  static constexpr int kTile = kAtcKeys * HD * 2;                    // 32 K or V rows
  static constexpr int kMRow = HD / 4 + 4;                           // floats: padded row of the exchange
  static constexpr int kExchange = kAtcCluster * 128 * kMRow * 4;    // [quarter of the head][128][kMRow], over the planes and the ring
  static constexpr int kMl = kExchange;                              // [128][2]: maximum and sum of the CTA's keys
  static constexpr int kWt = kMl + 128 * 8;                          // [128][8]: weights of the cluster's ranges, 1 / sum or 1
  static constexpr int kRing = 2 * kPlane;
  static constexpr int kLo = kRing + 2 * kTile;                      // the lo plane on its way: over the ring but for its first two K tiles
  static constexpr int kMax = kRing + 2 * kAtcStages * kTile;        // [2][2][128] row maxima
  static constexpr int kBars = kMax + 2 * 2 * 128 * 4;
  static constexpr int kSmem = kBars + 256;
  static_assert(kLo + kPlane == kMax && kAtcStages == 3 && kWt + 128 * 32 <= kMax && kSmem <= 227 * 1024, "shared memory budget");
  // tensor memory columns
  static constexpr uint32_t kO = 0, kQlo = HD, kS = HD + HD / 2, kP = kS + 2 * kAtcKeys;
  static_assert(kP + 3 * kAtcKeys / 2 <= 512, "tensor memory budget");
};

// Two fp32 values as three bf16 pairs, cut off instead of rounded: 8 of the 24 bits each, so that they add up to the values
// exactly, and byte moves and logic where conversions would queue.
__device__ __forceinline__ void atc_split3(float x, float y, uint32_t& t0, uint32_t& t1, uint32_t& t2) {
  uint32_t t[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    t[i] = __byte_perm(__float_as_uint(x), __float_as_uint(y), 0x7632);
    if (i < 2) {
      x -= __uint_as_float(__float_as_uint(x) & 0xFFFF0000u);
      y -= __uint_as_float(__float_as_uint(y) & 0xFFFF0000u);
    }
  }
  t0 = t[0]; t1 = t[1]; t2 = t[2];
}
// Address of this CTA's shared-memory location in the cluster's CTA `rank`.
__device__ __forceinline__ uint32_t atc_map(uint32_t addr, int rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ float4 atc_get4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ float2 atc_get2(uint32_t addr) {
  float2 v;
  asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void atc_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void atc_tma_3d(void* dst, const CUtensorMap* map, int x, int y, int z, uint64_t* bar) {
  asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
               ::"r"(smem_u32(dst)), "l"(map), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar)) : "memory");
}
// Operand with the non-contracted dimension contiguous (V: rows of 64 head elements, one row a key), 128-byte swizzle:
// groups of eight keys are 1024 bytes apart, blocks of 64 elements `block` bytes.
__device__ __forceinline__ uint64_t atc_desc_mn(uint32_t saddr, uint32_t block) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3FFFF) >> 4);
  d |= (uint64_t)(block >> 4) << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}
__device__ __forceinline__ void atc_tmem_st8(uint32_t taddr, const uint32_t* r) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
               ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}

template <int HD>
__global__ void __launch_bounds__(kAtcThreads, 1)
attn_tc_kernel(const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v, const AmArgs a) {
  using S = AtcShape<HD>;
  extern __shared__ __align__(1024) unsigned char atc_sm[];
  unsigned char* ring = atc_sm + S::kRing;                            // [stage] K tile, then [stage] V tile
  float* row_max = reinterpret_cast<float*>(atc_sm + S::kMax);
  uint64_t* bars = reinterpret_cast<uint64_t*>(atc_sm + S::kBars);
  uint64_t* k_full = bars;                                            // [stages]
  uint64_t* k_empty = k_full + kAtcStages;
  uint64_t* v_full = k_empty + kAtcStages;
  uint64_t* v_empty = v_full + kAtcStages;
  uint64_t* q_ready = v_empty + kAtcStages;                           // query terms in place
  uint64_t* a_full = q_ready + 1;                                     // part A of a tile's scores complete
  uint64_t* a_empty = a_full + 1;                                     // and read
  uint64_t* b_full = a_empty + 1;                                     // part B
  uint64_t* b_empty = b_full + 1;
  uint64_t* p_full = b_empty + 1;                                     // probabilities written, O of the tile before read
  uint64_t* o_full = p_full + 1;                                      // P V of a tile complete
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(o_full + 1);
  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int rank = blockIdx.x % kAtcCluster, group = blockIdx.x / kAtcCluster;      // of the cluster; key range, then unit
  const int split = group % a.nsplit, unit = group / a.nsplit;
  const int row_tiles = (a.rows + 127) / 128, kvh = unit / row_tiles, r0 = (unit % row_tiles) * 128;
  if (threadIdx.x == 0) {
#pragma unroll 1
    for (int s = 0; s < kAtcStages; ++s) {
      mbar_init(&k_full[s], 1);
      mbar_init(&k_empty[s], 1);
      mbar_init(&v_full[s], 1);
      mbar_init(&v_empty[s], 1);
    }
    mbar_init(q_ready, 8);
    mbar_init(a_full, 1);
    mbar_init(a_empty, 8);
    mbar_init(b_full, 1);
    mbar_init(b_empty, 8);
    mbar_init(p_full, 8);
    mbar_init(o_full, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) tmem_alloc(tmem_slot, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  pdl_wait();
  pdl_launch_dependents();
  // key tiles of this CTA: the launcher gives every one at least one
  const int tfirst = a.lo / kAtcKeys, ntiles = (a.k1 + kAtcKeys - 1) / kAtcKeys - tfirst;
  const int nsub = a.nsplit * kAtcCluster, sub = split * kAtcCluster + rank;
  const int c0 = tfirst + (int)((long long)ntiles * sub / nsub), n = tfirst + (int)((long long)ntiles * (sub + 1) / nsub) - c0;

  // The two kinds of warps do not meet in common code again (it would have the fewer registers): each has its own tail, of
  // sync_after_waits and the two cluster barriers.  Nobody leaves it early: a CTA whose wait gave up comes to the
  // cluster's barriers like the rest.
  bool ok = true;                                                     // none of this thread's waits has given up
  if (warp < 4) {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
  if (warp == 0) {
    const bool leader = elect_one();
#pragma unroll 1
    for (int j = 0; j < n && ok; ++j) {
      const int s = j % kAtcStages, use = j / kAtcStages, key0 = (c0 + j) * kAtcKeys;
      const int page = __ldg(a.page_table + key0 / kPage), y = kvh * kPage + key0 % kPage;
      if (use > 0) ok = __all_sync(0xffffffffu, mbar_wait(&k_empty[s], (use - 1) & 1, a.err));
      if (ok && leader) {
        mbar_arrive_expect_tx(&k_full[s], S::kTile);
#pragma unroll
        for (int b = 0; b < S::KB; ++b) atc_tma_3d(ring + s * S::kTile + b * kAtcKeys * 128, &tm_k, b * 64, y, page, &k_full[s]);
      }
      if (j == 0) ok = __all_sync(0xffffffffu, mbar_wait(q_ready, 0, a.err));      // the lo plane has left the ring
      if (ok && use > 0) ok = __all_sync(0xffffffffu, mbar_wait(&v_empty[s], (use - 1) & 1, a.err));
      if (ok && leader) {
        mbar_arrive_expect_tx(&v_full[s], S::kTile);
#pragma unroll
        for (int b = 0; b < S::KB; ++b) atc_tma_3d(ring + (kAtcStages + s) * S::kTile + b * kAtcKeys * 128, &tm_v, b * 64, y, page, &v_full[s]);
      }
      __syncwarp();
    }
  } else if (warp == 1) {
    constexpr uint32_t idesc_s = umma_idesc_bf16(128, kAtcKeys), idesc_o = umma_idesc_bf16(128, HD) | 1u << 16;   // V: hd contiguous
    const bool leader = elect_one();
    constexpr int Q4 = HD / 64;                                       // 16-wide steps of a quarter of the head
    const uint32_t first = tmem + S::kS, second = first + kAtcKeys, hi_plane = smem_u32(atc_sm), mid_plane = hi_plane + S::kPlane;
    auto kd = [&](int s, int i) { return umma_desc_sw128(smem_u32(ring) + s * S::kTile + i / 4 * kAtcKeys * 128) + (uint64_t)(i % 4 * 2); };
    auto qd = [&](uint32_t plane, int i) { return umma_desc_sw128(plane + i / 4 * 128 * 128) + (uint64_t)(i % 4 * 2); };
    auto part_a = [&](int s) {
#pragma unroll
      for (int i = 0; i < Q4; ++i) umma_bf16(first, qd(hi_plane, i), kd(s, i), idesc_s, i > 0);
#pragma unroll
      for (int i = Q4; i < 2 * Q4; ++i) umma_bf16(second, qd(hi_plane, i), kd(s, i), idesc_s, i > Q4);
      umma_commit(a_full);
    };
    auto part_b = [&](int s) {
#pragma unroll
      for (int i = 0; i < HD / 16; ++i) umma_bf16_ts(second, tmem + S::kQlo + i * 8, kd(s, i), idesc_s, i > 0);
#pragma unroll
      for (int i = 0; i < HD / 16; ++i) umma_bf16(second, qd(mid_plane, i), kd(s, i), idesc_s, 1);
#pragma unroll
      for (int i = 2 * Q4; i < 3 * Q4; ++i) umma_bf16(first, qd(hi_plane, i), kd(s, i), idesc_s, i > 2 * Q4);
#pragma unroll
      for (int i = 3 * Q4; i < 4 * Q4; ++i) umma_bf16(second, qd(hi_plane, i), kd(s, i), idesc_s, 1);
      umma_commit(b_full);
      umma_commit(&k_empty[s]);
    };
    ok = __all_sync(0xffffffffu, mbar_wait2(q_ready, 0, &k_full[0], 0, a.err));
    if (ok) {
      tc_fence_after();
      if (leader) part_a(0);
      __syncwarp();
      ok = __all_sync(0xffffffffu, mbar_wait(a_empty, 0, a.err));
    }
    if (ok) {
      tc_fence_after();
      if (leader) part_b(0);
      __syncwarp();
    }
#pragma unroll 1
    for (int j = 0; j < n && ok; ++j) {
      const int s = j % kAtcStages, s1 = (j + 1) % kAtcStages;
      if (j + 1 < n) {
        ok = __all_sync(0xffffffffu, mbar_wait2(&k_full[s1], ((j + 1) / kAtcStages) & 1, b_empty, j & 1, a.err));
        if (!ok) break;
        tc_fence_after();
        if (leader) part_a(s1);
        __syncwarp();
        ok = __all_sync(0xffffffffu, mbar_wait(a_empty, (j + 1) & 1, a.err));
        if (!ok) break;
        tc_fence_after();
        if (leader) part_b(s1);
        __syncwarp();
      }
      ok = __all_sync(0xffffffffu, mbar_wait(&v_full[s], (j / kAtcStages) & 1, a.err));
      if (!ok) break;
      const int key0 = (c0 + j) * kAtcKeys, lo = max(a.lo - key0, 0), hi = min(a.k1 - key0, kAtcKeys);
      if (lo > 0 || hi < kAtcKeys) {                                  // rows outside the visible keys may hold anything: a NaN would pass a zero
        for (int i = lane; i < kAtcKeys * S::KB * 8; i += 32) {
          const int key = i / 8 % kAtcKeys;
          if (key < lo || key >= hi) *reinterpret_cast<uint4*>(ring + (kAtcStages + s) * S::kTile + i * 16) = make_uint4(0u, 0u, 0u, 0u);
        }
        fence_async_smem();
        __syncwarp();
      }
      ok = __all_sync(0xffffffffu, mbar_wait(p_full, j & 1, a.err));
      if (!ok) break;
      tc_fence_after();
      if (leader) {
        const uint32_t vt = smem_u32(ring + (kAtcStages + s) * S::kTile);
#pragma unroll
        for (int p = 2; p >= 0; --p)                                  // the smallest terms first
#pragma unroll
          for (int k = 0; k < kAtcKeys / 16; ++k)
            umma_bf16_ts(tmem + S::kO, tmem + S::kP + p * (kAtcKeys / 2) + k * 8, atc_desc_mn(vt + k * 2048, kAtcKeys * 128), idesc_o, p < 2 || k > 0);
        umma_commit(o_full);
        umma_commit(&v_empty[s]);
      }
      __syncwarp();
    }
  }
  tc_fence_before();
  sync_after_waits(ok);
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
  atc_cluster_sync();
  atc_cluster_sync();
  } else {
  asm volatile("setmaxnreg.inc.sync.aligned.u32 224;");
  const int quarter = warp & 3, half = (warp - 4) >> 2, row = quarter * 32 + lane;    // warps 4 - 11
  // the state of a row: this thread's half of the head, the maximum, the sum over its keys
  constexpr int HH = HD / 2;
  float o[HH], m = -INFINITY, l = 0.f;
#pragma unroll
  for (int i = 0; i < HH; ++i) o[i] = 0.f;
  {
    const uint32_t lane_addr = tmem + ((uint32_t)(quarter * 32) << 16);
    {   // ---- the queries, scaled, as three terms in swizzled planes; lo goes on into tensor memory
      constexpr int C4 = HD / 4, N = 128 * C4 / 256, B = 16;          // float4 of a row, of a thread, in flight
      const int t = threadIdx.x - 128, glog = 31 - __clz(a.G);        // groups are of 1, 2 or 4
#pragma unroll 1
      for (int i0 = 0; i0 < N; i0 += B) {                             // whole rows by warps
        float4 x[B];
#pragma unroll
        for (int i = 0; i < B; ++i) {
          const int r = (t + 256 * (i0 + i)) / C4, c = (t + 256 * (i0 + i)) % C4, g = r0 + r;
          x[i] = g < a.rows ? *reinterpret_cast<const float4*>(a.q + (size_t)(g >> glog) * a.q_stride + ((kvh << glog) + (g & (a.G - 1))) * HD + 4 * c)
                            : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int i = 0; i < B; ++i) {
          const int r = (t + 256 * (i0 + i)) / C4, c = (t + 256 * (i0 + i)) % C4;
          uint2 hi, mid, lo;
          atc_split3(x[i].x * a.qscale, x[i].y * a.qscale, hi.x, mid.x, lo.x);
          atc_split3(x[i].z * a.qscale, x[i].w * a.qscale, hi.y, mid.y, lo.y);
          unsigned char* at = atc_sm + c / 16 * 128 * 128 + r * 128 + (((c % 16 / 2) ^ (r & 7)) << 4) + c % 2 * 8;
          *reinterpret_cast<uint2*>(at) = hi;
          *reinterpret_cast<uint2*>(at + S::kPlane) = mid;
          *reinterpret_cast<uint2*>(at + S::kLo) = lo;
        }
      }
      asm volatile("bar.sync 1, 256;" ::: "memory");
#pragma unroll 4
      for (int e = half * HH; e < half * HH + HH; e += 16) {
        const unsigned char* line = atc_sm + S::kLo + e / 64 * 128 * 128 + row * 128;
        const uint4 u = *reinterpret_cast<const uint4*>(line + (((e % 64 / 8) ^ (row & 7)) << 4));
        const uint4 v = *reinterpret_cast<const uint4*>(line + (((e % 64 / 8 + 1) ^ (row & 7)) << 4));
        const uint32_t w[8] = {u.x, u.y, u.z, u.w, v.x, v.y, v.z, v.w};
        atc_tmem_st8(lane_addr + S::kQlo + e / 2, w);
      }
      tmem_st_wait();
      tc_fence_before();
      fence_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(q_ready);
    }
    float corr = 0.f;                                                 // of the tile whose O comes next
    auto add_tile = [&]() {
#pragma unroll
      for (int c = 0; c < HH; c += 32) {
        uint32_t v[32];
        tmem_ld32(lane_addr + S::kO + half * HH + c, v);
#pragma unroll
        for (int i = 0; i < 32; ++i) o[c + i] = fmaf(o[c + i], corr, __uint_as_float(v[i]));
      }
    };
    float s[16];
    auto read_scores = [&](uint64_t* full, uint64_t* empty, int j, bool add) {
      if (!__all_sync(0xffffffffu, mbar_wait(full, j & 1, a.err))) return false;
      tc_fence_after();
      uint32_t x[16], y[16];
      tmem_ld16(lane_addr + S::kS + half * 16, x);
      tmem_ld16(lane_addr + S::kS + kAtcKeys + half * 16, y);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(empty);
#pragma unroll
      for (int i = 0; i < 16; ++i) s[i] = (add ? s[i] : 0.f) + (__uint_as_float(x[i]) + __uint_as_float(y[i]));
      return true;
    };
    bool late = false;
#pragma unroll 1
    for (int j = 0; j < n; ++j) {
      // 16 keys of the row.  The eight warps leave the loop together: the barrier tells them whether a wait of one gave up.
      const int key0 = (c0 + j) * kAtcKeys + half * 16;
      bool got = true;
      if (j == 0) got = read_scores(a_full, a_empty, 0, false);       // the later ones are read ahead, below
      got = got && !late && read_scores(b_full, b_empty, j, true);
      if (got) {
        const bool inside = key0 >= a.lo && key0 + 16 <= a.k1;
        float mx = -INFINITY;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          if (!inside && (key0 + i < a.lo || key0 + i >= a.k1)) s[i] = -INFINITY;
          mx = fmaxf(mx, s[i]);
        }
        row_max[((j & 1) * 2 + half) * 128 + row] = mx;
      }
      ok = !block_gave_up([&] { return !got; }, bar_or<1, 256>);
      if (!ok) break;
      const float mn = fmaxf(m, fmaxf(row_max[(j & 1) * 256 + row], row_max[(j & 1) * 256 + 128 + row]));
      const float f = am_ex2(m - mn);
      m = mn;
      float p[16], sum = 0.f;
#pragma unroll
      for (int i = 0; i < 16; i += 2) {
        p[i] = am_ex2(s[i] - mn);
        p[i + 1] = am_ex2(s[i + 1] - mn);
        sum += p[i] + p[i + 1];
      }
      l = fmaf(l, f, sum);
      if (j + 1 < n) late = !read_scores(a_full, a_empty, j + 1, false);      // ahead of the rest, so that part B can follow
      uint32_t t3[3][8];
#pragma unroll
      for (int i = 0; i < 16; i += 2) atc_split3(p[i], p[i + 1], t3[0][i / 2], t3[1][i / 2], t3[2][i / 2]);
      // the products of the tile before: probabilities free, sums out
      if (j > 0) {
        late = !__all_sync(0xffffffffu, mbar_wait(o_full, (j - 1) & 1, a.err)) || late;      // said ahead of the next barrier
        tc_fence_after();
      }
#pragma unroll
      for (int i = 0; i < 3; ++i) atc_tmem_st8(lane_addr + S::kP + i * (kAtcKeys / 2) + half * 8, t3[i]);
      if (j > 0) add_tile();
      corr = f;
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_full);
    }
    ok = ok && !late && __all_sync(0xffffffffu, mbar_wait(o_full, (n - 1) & 1, a.err));
    if (ok) {
      tc_fence_after();
      add_tile();
    }
  }
  tc_fence_before();
  sync_after_waits(ok);
  // ---- the cluster's four ranges meet: CTA q adds quarter q of the head, out of all four CTAs' shared memory
  {                                                                   // the CTA's products and copies are done: over the planes and the ring
    float* at = reinterpret_cast<float*>(atc_sm) + row * S::kMRow;
#pragma unroll
    for (int q2 = 0; q2 < 2; ++q2)
#pragma unroll
      for (int i = 0; i < HD / 4; i += 4)
        *reinterpret_cast<float4*>(at + (half * 2 + q2) * 128 * S::kMRow + i) =
            make_float4(o[q2 * (HD / 4) + i], o[q2 * (HD / 4) + i + 1], o[q2 * (HD / 4) + i + 2], o[q2 * (HD / 4) + i + 3]);
    row_max[half * 128 + row] = l;
    asm volatile("bar.sync 1, 256;" ::: "memory");
    if (half == 0) *reinterpret_cast<float2*>(atc_sm + S::kMl + row * 8) = make_float2(m, l + row_max[128 + row]);
  }
  atc_cluster_sync();
  {
    const int t = threadIdx.x - 128;
    const uint32_t own = smem_u32(atc_sm);
    float* wt = reinterpret_cast<float*>(atc_sm + S::kWt);
    if (t < 128) {
      float2 x[kAtcCluster];
      float M = -INFINITY, L = 0.f;
#pragma unroll
      for (int k = 0; k < kAtcCluster; ++k) x[k] = atc_get2(atc_map(own + S::kMl + t * 8, k));
#pragma unroll
      for (int k = 0; k < kAtcCluster; ++k) M = fmaxf(M, x[k].x);
#pragma unroll
      for (int k = 0; k < kAtcCluster; ++k) {
        const float w = M > -INFINITY ? am_ex2(x[k].x - M) : 0.f;
        wt[t * 8 + k] = w;
        L += w * x[k].y;
      }
      wt[t * 8 + 4] = a.nsplit > 1 ? 1.0f : L > 0.f ? 1.0f / L : 0.f;
      if (a.nsplit > 1 && rank == 0 && r0 + t < a.rows)
        *reinterpret_cast<float2*>(a.part_ml + (((size_t)kvh * a.rows + r0 + t) * a.nsplit + split) * 2) = make_float2(M, L);
    }
    asm volatile("bar.sync 1, 256;" ::: "memory");
    constexpr int C4 = HD / 16;                                       // float4 of a quarter's row
    constexpr int N = 128 * C4 / 256, B = N < 4 ? N : 4;              // of a thread; in flight
#pragma unroll 1
    for (int i0 = 0; i0 < N; i0 += B) {
      float4 x[B][kAtcCluster];
#pragma unroll
      for (int b = 0; b < B; ++b) {
        const int i = t + (i0 + b) * 256;
#pragma unroll
        for (int k = 0; k < kAtcCluster; ++k) x[b][k] = atc_get4(atc_map(own + (uint32_t)((rank * 128 + i / C4) * S::kMRow + i % C4 * 4) * 4, k));
      }
#pragma unroll
      for (int b = 0; b < B; ++b) {
        const int i = t + (i0 + b) * 256, r = i / C4, e = i % C4 * 4;
        if (r0 + r >= a.rows) continue;
        const float4 w = *reinterpret_cast<const float4*>(wt + r * 8);
        const float f = wt[r * 8 + 4];
        const size_t pi = ((size_t)kvh * a.rows + r0 + r) * a.nsplit + split;
        float* dst = (a.nsplit > 1 ? a.part_o + pi * HD : a.out + am_out_row(a, kvh, r0 + r) * HD) + rank * (HD / 4) + e;
        const float4* y = x[b];
        *reinterpret_cast<float4*>(dst) = make_float4(f * (w.x * y[0].x + w.y * y[1].x + w.z * y[2].x + w.w * y[3].x),
                                                      f * (w.x * y[0].y + w.y * y[1].y + w.z * y[2].y + w.w * y[3].y),
                                                      f * (w.x * y[0].z + w.y * y[1].z + w.z * y[2].z + w.w * y[3].z),
                                                      f * (w.x * y[0].w + w.y * y[1].w + w.z * y[2].w + w.w * y[3].w));
      }
    }
  }
  atc_cluster_sync();                                                 // the others have read this CTA's part
  }
}

// Clusters of the kernel that the device holds at once; sets the kernel's attributes.
template <int HD>
inline int atc_prepare() {
  raise_dyn_smem(attn_tc_kernel<HD>, (size_t)AtcShape<HD>::kSmem);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(kAtcCluster);
  cfg.blockDim = dim3(kAtcThreads);
  cfg.dynamicSmemBytes = AtcShape<HD>::kSmem;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = kAtcCluster;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  int n = 0;
  B2_CUDA(cudaOccupancyMaxActiveClusters(&n, attn_tc_kernel<HD>, &cfg));
  return n;
}

// Splits of a call (clusters of a unit), or 0 where the kernel is not the one to take it.  Setting up the three planes and
// the exchange cost about 10 us, so mma.sync keeps the short and the narrow calls.  At 64 rows and more the line is at 1000
// keys (80 rows of head size 256: 18.2 us against 19.0; at 300 keys 20.1 against 18.8; at 32768 34.8 against 63.0), for 33 -
// 48 rows at 8000 of all kv heads together (48 rows, one kv head: 19.5 against 19.4 at 2500, 25.8 against 27.6 at 14000).
// 256 rows over 32768 keys take 50 us, mma.sync 121; 16 kv heads of 128 with 128 rows each 159 us and 532.  The error
// against 64 bits is that of mma.sync within 1 % at head size 256 and 8 % below it at 128 (geometric means of these shapes).
inline int atc_splits(const AmArgs& a, int hd, int clusters, int cap) {
  if ((hd != 128 && hd != 256) || clusters <= 0) return 0;
  const int units = a.hkv * ((a.rows + 127) / 128), nkeys = a.k1 - a.lo;
  if (a.rows <= 32 || (a.rows > 48 ? nkeys < 1000 : nkeys < 2500 || (long long)nkeys * a.hkv < 8000)) return 0;
  const int ntiles = (a.k1 + kAtcKeys - 1) / kAtcKeys - a.lo / kAtcKeys;
  return std::max(1, std::min(std::min(clusters / units, cap), std::min(256, ntiles / kAtcCluster)));
}

template <int HD>
inline void launch_attn_tc(cudaStream_t st, const CUtensorMap& tm_k, const CUtensorMap& tm_v, AmArgs a, int nsplit) {
  a.nsplit = nsplit;
  const int units = a.hkv * ((a.rows + 127) / 128);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(units * nsplit * kAtcCluster);
  cfg.blockDim = dim3(kAtcThreads);
  cfg.dynamicSmemBytes = AtcShape<HD>::kSmem;
  cfg.stream = st;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = kAtcCluster;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 2;
  B2_CUDA(cudaLaunchKernelEx(&cfg, attn_tc_kernel<HD>, tm_k, tm_v, AmArgs(a)));
  if (nsplit > 1)
    launch_pdl(attn_shared_sum_kernel, dim3(a.hkv * a.rows * (HD / 64)), dim3(kAmSumThreads), (size_t)0, st, a, (int)HD);
}

}  // namespace b200lm

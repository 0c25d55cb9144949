// Int4 weight-only GEMM for at most 16 token rows (wide decode steps, very short prompts) on mma.sync.
//
//   out[token][n] = scale[n] * sum_k W[n][k] X[token][k],  X bf16, W the 16 x 64 tiles of decode_ops.cuh
//
// With few token rows the work is streaming the weights.  The tcgen05 kernel passes every weight block through four
// roles (copy, expand, tensor memory, MMA), whose hand-overs cost a block as much at 16 tokens as at 64 (2560 x 10240 and the
// norm behind it, 5 rows: 11.1 us there, 9.4 here; 2560 x 2048: 6.3 and 5.7).  Here a warp expands a tile from its own 16 bytes per lane straight into the A operand: a
// shift and a mask turn two of the tile's nibbles into bf16(136 + q), one packed subtract takes the bias off.  The k
// order inside a 16-wide step is the tile's own (lane t holds k = 4t .. 4t + 3, even ones first), and X follows it.
//
// X of the CTA's K slice stays in shared memory (one CTA per SM: read once per SM, where a CTA per few row tiles read
// as many bytes of X as of W).  The CTA's row tiles x k tiles are dealt to the 16 warps as contiguous runs.  A row tile
// that one run covers is written from its registers; those that several runs met are added in warp order through
// shared memory.  Weights stream through a private ring per warp by cp.async: a lane reads back what it copied itself,
// so there is no barrier on the way, and the ring's first fill is requested ahead of griddepcontrol.wait.
// The issue slots bound it (a tile of 512 bytes takes about 60 for the operand and the products, the logic half at
// half rate), so the loop over a run keeps to a pointer, a slot and two counters.
#pragma once
#include <algorithm>

#include "attn_mma.cuh"
#include "common.cuh"
#include "decode_ops.cuh"
#include "prefill_ops.cuh"

namespace b200lm {

constexpr int kGsThreads = 512, kGsWarps = kGsThreads / 32, kGsMaxT = 16;
constexpr int kGsDepth = 8;                       // tiles in the ring of a warp (64 KB in all)
constexpr int kGsRing = kGsWarps * kGsDepth * 512;
constexpr int kGsPairTiles = 64;                  // most row tiles of a CTA with EPI 1
constexpr int kGsTable = kGsPairTiles * 16 * 4 + kGsPairTiles * 4 + 128;     // scales; which warps met a row tile; how many
inline int gs_nt(int T) { return T <= 8 ? 1 : 2; }
__host__ __device__ constexpr int gs_part_bytes(int nt) { return 16 * (nt * 8 + 1) * 4; }                 // a partial sum of a row tile
__host__ __device__ inline int gs_per(int ntile, int KTs) { return (ntile * KTs + kGsWarps - 1) / kGsWarps; }
__host__ __device__ inline int gs_slots(int epi, int per, int KTs) { return epi == 1 ? (per + KTs - 1) / KTs + 1 : 2; }   // of a warp
__host__ __device__ inline int gs_xrow(int KTs) { return KTs * 128 + 32; }         // bytes: 32 past a multiple of 128, conflict-free 8-byte reads
inline int gs_smem(int epi, int nt, int ntile, int KTs) {
  return kGsRing + kGsTable + kGsWarps * gs_slots(epi, gs_per(ntile, KTs), KTs) * gs_part_bytes(nt) + nt * 8 * gs_xrow(KTs);
}
constexpr int kGsMaxSmem = 227 * 1024;

struct GsArgs {
  const uint4* w;             // [row_tile][k_tile]
  const float* wscale;        // [row_tile][16]
  const __nv_bfloat16* x;     // [T][K]
  int T, N, KT;
  int ksplit, KTs;            // K splits, k tiles of one
  int cps, tile_base, tile_rem;      // CTAs per split; row tiles (EPI 1: pairs) per CTA: base, one more for the first rem
  float* outF;                // EPI 0: [ksplit][T][N]
  __nv_bfloat16* outB;        // EPI 1: [T][N / 2], tiles alternate gate, up
};

__device__ __forceinline__ void gs_mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// (v & 0x000F000F) ^ 0x43084308: bf16(136 + q) of the two's complement nibbles at bits 0 and 16, in one instruction.
__device__ __forceinline__ uint32_t gs_136(uint32_t v) {
  uint32_t r;
  asm("lop3.b32 %0, %1, %2, %3, 0x6a;" : "=r"(r) : "r"(v), "r"(0x000F000Fu), "r"(0x43084308u));
  return r;
}

template <int EPI, int NT>
__global__ void __launch_bounds__(kGsThreads, 1)
gemm_w4_small_kernel(const GsArgs g) {
  extern __shared__ __align__(128) unsigned char gs_sm[];
  constexpr int PS = NT * 8 + 1;                                         // floats of a partial sum's row
  constexpr int unit = EPI == 1 ? 2 : 1;
  const int warp = __shfl_sync(~0u, threadIdx.x >> 5, 0), lane = threadIdx.x & 31, gr = lane >> 2, tq = lane & 3;
  const int KTs = g.KTs, xrow = gs_xrow(KTs);
  const int split = g.ksplit == 1 ? 0 : (int)blockIdx.x / g.cps, local = blockIdx.x - split * g.cps;
  const int t0 = (local * g.tile_base + min(local, g.tile_rem)) * unit, ntile = (g.tile_base + (local < g.tile_rem ? 1 : 0)) * unit;
  const int per = gs_per(ntile, KTs), slots = gs_slots(EPI, gs_per((g.tile_base + (g.tile_rem ? 1 : 0)) * unit, KTs), KTs);
  unsigned char* ring = gs_sm + warp * (kGsDepth * 512) + lane * 16;
  float* scales = reinterpret_cast<float*>(gs_sm + kGsRing);             // [entry][16]
  uint32_t* met = reinterpret_cast<uint32_t*>(scales + kGsPairTiles * 16);     // [entry]: row tile << 16 | last warp << 8 | first warp
  volatile uint32_t& nmet = *(met + kGsPairTiles);
  float* part = reinterpret_cast<float*>(gs_sm + kGsRing + kGsTable);    // [warp][slot][16 rows][PS]
  unsigned char* xs = reinterpret_cast<unsigned char*>(part) + kGsWarps * slots * gs_part_bytes(NT);
  // ---- this warp's run: tile by tile, first row tile and k tile, tiles left to request and to use
  const int beg = min(ntile * KTs, warp * per), total = min(ntile * KTs - beg, per), rt0 = beg / KTs, kt0 = beg - rt0 * KTs;
  const uint4* src = g.w + ((size_t)(t0 + rt0) * g.KT + split * KTs + kt0) * 32 + lane;
  int pleft = total, pseg = KTs - kt0, ps = 0;
  auto request = [&]() {
    if (pleft > 0) {
      am_cp16(smem_u32(ring) + ps, src, 16);
      src += 32;
      --pleft;
      if (--pseg == 0) { pseg = KTs; src += (size_t)(g.KT - KTs) * 32; } // the split's part of the next row tile
    }
    asm volatile("cp.async.commit_group;" ::: "memory");                 // always one, so that the wait counts tiles
    ps = (ps + 512) & (kGsDepth * 512 - 1);
  };
#pragma unroll 1
  for (int s = 0; s < kGsDepth - 1; ++s) request();
  // ---- row tiles whose sums meet in shared memory (EPI 1: all), and their scales
  if constexpr (EPI == 1) {
    if (threadIdx.x < ntile) met[threadIdx.x] = threadIdx.x << 16 | ((threadIdx.x * KTs + KTs - 1) / per) << 8 | threadIdx.x * KTs / per;
    if (threadIdx.x == 0) nmet = ntile;
  } else if (warp == 0) {
    const int b = lane * per, tile = b / KTs;                            // the run of warp `lane` begins inside this row tile,
    const bool first = lane > 0 && lane < kGsWarps && b < ntile * KTs && b != tile * KTs && b - per <= tile * KTs;     // and no run before it does
    const uint32_t mask = __ballot_sync(~0u, first);
    if (first) met[__popc(mask & ((1u << lane) - 1))] = tile << 16 | (min(ntile * KTs - 1, tile * KTs + KTs - 1) / per) << 8 | (lane - 1);
    if (lane == 0) nmet = __popc(mask);
  }
  __syncthreads();
  const int nshared = nmet;
  for (int i = threadIdx.x; i < nshared * 16; i += kGsThreads) scales[i] = __ldg(g.wscale + (t0 + (met[i >> 4] >> 16)) * 16 + (i & 15));
  pdl_launch_dependents();                         // ahead of the wait, as in the tcgen05 kernel
  pdl_wait();
  // ---- X of the slice
  for (int row = warp; row < g.T; row += kGsWarps) {
    const uint4* from = reinterpret_cast<const uint4*>(g.x + (size_t)row * (g.KT * 64) + split * KTs * 64);
#pragma unroll 8
    for (int u = lane; u < KTs * 8; u += 32) {
      const uint4 v = __ldcg(from + u);                                  // of four k: 0, 2 and 1, 3 to a word, as the weights' nibbles come
      *reinterpret_cast<uint4*>(xs + row * xrow + u * 16) = make_uint4(__byte_perm(v.x, v.y, 0x5410), __byte_perm(v.x, v.y, 0x7632),
                                                                       __byte_perm(v.z, v.w, 0x5410), __byte_perm(v.z, v.w, 0x7632));
    }
  }
  __syncthreads();
  const __nv_bfloat162 bias = __float2bfloat162_rn(136.0f);
  const unsigned char* xb = xs + gr * xrow + tq * 8;
  int left = total, cs = 0, kt = kt0;
#pragma unroll 1
  for (int rt = rt0, seg = 0; left > 0; ++rt, ++seg) {                   // a row tile of the run
    int n = min(KTs - kt, left);
    const bool whole = EPI == 0 && n == KTs;
    left -= n;
    float s0 = 0.f, s1 = 0.f;
    if (whole) { s0 = __ldg(g.wscale + (t0 + rt) * 16 + gr); s1 = __ldg(g.wscale + (t0 + rt) * 16 + gr + 8); }
    float acc[NT][4];
#pragma unroll
    for (int m = 0; m < NT; ++m) acc[m][0] = acc[m][1] = acc[m][2] = acc[m][3] = 0.f;
    const unsigned char* xt = xb + kt * 128;
#pragma unroll 1
    for (; n > 0; --n, xt += 128) {
      request();
      asm volatile("cp.async.wait_group %0;" ::"n"(kGsDepth - 1) : "memory");
      const uint4 w = *reinterpret_cast<const uint4*>(ring + cs);
      cs = (cs + 512) & (kGsDepth * 512 - 1);
      const uint32_t wj[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        uint2 b[NT];
#pragma unroll
        for (int m = 0; m < NT; ++m) b[m] = *reinterpret_cast<const uint2*>(xt + m * 8 * xrow + j * 32);
        // nibble 2 i = row g, 2 i + 1 = row g + 8, two's complement, i = k - 4t: nibbles four apart are one operand word
        uint32_t a[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) a[i] = gs_136(wj[j] >> (4 * i));
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const __nv_bfloat162 h = __hsub2(*reinterpret_cast<__nv_bfloat162*>(&a[i]), bias);
          a[i] = *reinterpret_cast<const uint32_t*>(&h);
        }
#pragma unroll
        for (int m = 0; m < NT; ++m) gs_mma(acc[m], a, b[m].x, b[m].y);
      }
    }
    kt = 0;
    if (whole) {
      float* out = g.outF + (size_t)split * g.T * g.N + (t0 + rt) * 16 + gr;
#pragma unroll
      for (int m = 0; m < NT; ++m) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int t = m * 8 + 2 * tq + i;
          if (t < g.T) {
            out[(size_t)t * g.N] = acc[m][i] * s0;
            out[(size_t)t * g.N + 8] = acc[m][2 + i] * s1;
          }
        }
      }
    } else {
      const int slot = EPI == 1 ? seg : (seg > 0 ? 1 : 0);
      float* p = part + ((size_t)(warp * slots + slot) * 16 + gr) * PS + 2 * tq;
#pragma unroll
      for (int m = 0; m < NT; ++m) {
        p[m * 8] = acc[m][0]; p[m * 8 + 1] = acc[m][1];
        p[8 * PS + m * 8] = acc[m][2]; p[8 * PS + m * 8 + 1] = acc[m][3];
      }
    }
  }
  __syncthreads();
  // ---- the row tiles that several runs met: a group of 16 threads takes a token's 16 outputs
  const int row = threadIdx.x & 15, t = (threadIdx.x >> 4) & 15;
  if (t >= g.T) return;
  auto sum = [&](int e) {
    const uint32_t m = met[e];
    const int tile = m >> 16, w1 = (m >> 8) & 255;
    float s = 0.f;
#pragma unroll 1
    for (int w = m & 255; w <= w1; ++w) {
      const int before = tile * KTs - w * per;                           // tiles of w's run ahead of this row tile, where positive
      const int slot = before <= 0 ? 0 : EPI == 1 ? (before + KTs - 1) / KTs : 1;
      s += part[((size_t)(w * slots + slot) * 16 + row) * PS + t];
    }
    return s * scales[e * 16 + row];
  };
#pragma unroll 1
  for (int e = (threadIdx.x >> 8) * unit; e < nshared; e += 2 * unit) {
    const int tile = t0 + (met[e] >> 16);
    if constexpr (EPI == 0) g.outF[((size_t)split * g.T + t) * g.N + tile * 16 + row] = sum(e);
    else g.outB[(size_t)t * (g.N / 2) + tile * 8 + row] = __float2bfloat16(gelu_tanh(sum(e)) * sum(e + 1));
  }
}

// A CTA's part of the row tiles (EPI 1: pairs), at most.
inline int gs_tiles(int epi, int N, int ksplit, int sms) {
  const int unit = epi == 1 ? 2 : 1, units = N / (16 * unit), cps = std::max(1, std::min(units, sms / ksplit));
  return (units + cps - 1) / cps * unit;
}
// Whether a GEMM fits the kernel: token rows, and X of a split beside the ring and the partial sums.
inline bool gs_fits(int T, int N, int KT, int ksplit, bool geglu, int sms) {
  if (T > kGsMaxT || N % (geglu ? 32 : 16) || KT % ksplit) return false;
  const int ntile = gs_tiles(geglu, N, ksplit, sms);
  return (!geglu || ntile <= kGsPairTiles) && ntile < 65536 && gs_smem(geglu, gs_nt(T), ntile, KT / ksplit) <= kGsMaxSmem;
}

// K splits: tiles of the busiest CTA, plus what each part costs its consumer.
inline int gs_ksplit(int T, int N, int KT, int sms, int most) {
  int best = 0;
  double best_cost = 1e30;
  for (int s = 1; s <= 8 && s <= most; ++s) {
    if (KT % s || (s > 1 && KT / s < 4) || !gs_fits(T, N, KT, s, false, sms)) continue;
    const double cost = (double)gs_tiles(0, N, s, sms) * (KT / s) + 6.0 * s;
    if (cost < best_cost - 1e-9) { best_cost = cost; best = s; }
  }
  return best;
}

inline void launch_gemm_small(cudaStream_t st, int sms, int device, const uint4* w, const float* wscale, const __nv_bfloat16* x, int T, int N, int K,
                              int ksplit, bool geglu, float* outF, __nv_bfloat16* outB) {
  const int nt = gs_nt(T);
  GsArgs g{};
  g.w = w; g.wscale = wscale; g.x = x; g.T = T; g.N = N; g.KT = K / 64; g.ksplit = ksplit; g.KTs = g.KT / ksplit; g.outF = outF; g.outB = outB;
  const int units = geglu ? N / 32 : N / 16;
  g.cps = std::max(1, std::min(units, sms / ksplit));
  g.tile_base = units / g.cps;
  g.tile_rem = units % g.cps;
  static unsigned char ready[64] = {};                                   // per device; a race only repeats the calls
  if (!ready[device]) {
    raise_dyn_smem(gemm_w4_small_kernel<0, 1>, (size_t)kGsMaxSmem);
    raise_dyn_smem(gemm_w4_small_kernel<1, 1>, (size_t)kGsMaxSmem);
    raise_dyn_smem(gemm_w4_small_kernel<0, 2>, (size_t)kGsMaxSmem);
    raise_dyn_smem(gemm_w4_small_kernel<1, 2>, (size_t)kGsMaxSmem);
    share_memory(gemm_w4_small_kernel<0, 1>);
    share_memory(gemm_w4_small_kernel<1, 1>);
    share_memory(gemm_w4_small_kernel<0, 2>);
    share_memory(gemm_w4_small_kernel<1, 2>);
    ready[device] = 1;
  }
  const dim3 grid(g.cps * ksplit), block(kGsThreads);
  const size_t smem = (size_t)gs_smem(geglu, nt, gs_tiles(geglu, N, ksplit, sms), g.KTs);
  if (nt == 1) {
    if (geglu) launch_pdl(gemm_w4_small_kernel<1, 1>, grid, block, smem, st, g);
    else launch_pdl(gemm_w4_small_kernel<0, 1>, grid, block, smem, st, g);
  } else {
    if (geglu) launch_pdl(gemm_w4_small_kernel<1, 2>, grid, block, smem, st, g);
    else launch_pdl(gemm_w4_small_kernel<0, 2>, grid, block, smem, st, g);
  }
}

}  // namespace b200lm

// Attention of many single-token queries over ONE cache (all at the same position) on mma.sync.
//
// batch * G query rows of a kv head see the same keys, so the cache is read once per 64 rows instead of once
// per query.  The operator's contract is fp32: queries, probabilities and (fp32) cache rows enter the bf16
// tensor-core products as up to three bf16 terms each (x = hi + mid + lo, 24 bits) and the products whose
// weight is above 2^-24 are accumulated in fp32.  The tensor core cuts its sums off rather than rounding them, so no
// long sum stays in its accumulators: scores leave them every 64 elements, P V every 16 keys (left in them over 32768
// keys, the result was off by 2e-6 where fp32 adds are off by 3e-7).  Many rows over a long
// bf16 cache run on tcgen05 instead (attn_tc.cuh), with an O accumulator per tile of keys for the same reason.
//
// A warp owns (row tile of 16 query rows) x (every KG-th chunk of 16 keys): scores, online softmax and P V of a
// chunk stay in its registers, so warps meet only at the end.  The warps of a key group stream the chunks' K
// and V rows into the group's ring with 16-byte asynchronous copies, into rows padded so that the fragment loads hit
// all banks (one bulk copy per row took its warp 1450 cycles per 16 rows, half of the loop; no producer warp: a ninth warp would cap the kernel at 168 registers, and the O accumulator alone takes 128).
//   MT = 1, 2, 4 row tiles per CTA (16 / 32 / 64 rows), the key groups fill the rest of the eight warps.
//   PACK: at most four rows: the three query terms share ONE 16-row tile (row 4 * term + r), which takes a third
//   of the products; that is the shape bound by the cache bytes.
//
// What bounds it: the mma.sync pipe for many rows (54 % busy), the cache's bytes for few rows over a long cache, and for
// short caches one chain of latencies.
#pragma once
#include <algorithm>

#include "common.cuh"
#include "decode_ops.cuh"
#include "prefill_ops.cuh"
#include "split_ticket.h"

namespace b200lm {

__device__ __forceinline__ void am_ldsm4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void am_ldsm4t(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
// volatile: the order of products and fragment loads is the written one (left to the compiler, the loads of a whole
// chunk move up front and the accumulators spill)
__device__ __forceinline__ void am_mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ float am_ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// 16 bytes global -> shared (the rest of them zero), and this thread's arrival on `bar` once all its copies so far have landed
__device__ __forceinline__ void am_cp16(uint32_t dst, const void* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void am_cp_arrive(uint64_t* bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// Two fp32 values as three bf16 pairs: x = t0 + t1 + t2 up to 2^-24 |x|.
__device__ __forceinline__ void am_split3(float x, float y, uint32_t (&t)[3]) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
    t[i] = *reinterpret_cast<const uint32_t*>(&h);
    if (i < 2) {
      x -= __low2float(h);
      y -= __high2float(h);
    }
  }
}

template <typename T, int HD, int MT, bool PACK>
struct AmShape {
  static constexpr int QT = PACK ? 1 : 3;                            // bf16 planes of the query tile
  static constexpr int KT = sizeof(T) == 4 ? 3 : 1;                  // bf16 terms of a cache value
  static constexpr int kQRow = HD * 2 + 16;
  static constexpr int kQ = QT * MT * 16 * kQRow;
  // row strides: 16 (bf16, V) or 32 (fp32 K, read as pairs of floats) bytes past a multiple of 128
  static constexpr int kKRow = sizeof(T) == 4 ? HD * 4 + 32 : HD * 2 + 16;
  static constexpr int kVRow = HD * (int)sizeof(T) + 16;
  static constexpr int kHalf = 16 * kKRow;                           // one ring entry: 16 K rows or 16 V rows
  static constexpr int kRoom = 226 * 1024 - kQ - 1024;
  static constexpr int KG = MT == 4 ? 2 : MT == 2 ? 4 : kRoom / kHalf >= 24 ? 8 : 4;    // key groups
  static constexpr int NSraw = kRoom / kHalf / KG;
  static constexpr int NS = NSraw < 8 ? NSraw : 8;                   // ring entries per key group
  static constexpr int kWarps = MT * KG;
  static constexpr int kThreads = 32 * kWarps;
  static constexpr int kRows = PACK ? 4 : MT * 16;                   // query rows per CTA
  static constexpr int kWRows = PACK ? 4 : 16;                       // of a warp
  static constexpr int kMRow = HD + 8;                               // floats: padded row of the merge area
  static constexpr int kMerge = kWarps * kWRows * (kMRow + 2) * 4 + kRows * (KG + 2) * 4;
  static constexpr int kMain = kQ + KG * NS * kHalf > kMerge ? kQ + KG * NS * kHalf : kMerge;
  static constexpr int kBars = (kMain + 127) & ~127;
  static constexpr int kSmem = kBars + 2 * KG * NS * 8 + 16;
  static_assert(NS >= 2 && kSmem <= 227 * 1024, "shared memory budget");
};

struct AmArgs {
  const float* q;           // [batch] rows of q_stride floats, the q heads first
  int q_stride;
  const void *k, *v;        // [page][hkv][kPage][hd]
  const int* page_table;
  int rows, G, hkv;         // rows = batch * G per kv head
  int lo, k1;               // visible keys [lo, k1)
  int nsplit;
  float qscale;             // log2(e) / sqrt(hd)
  float* out;               // [batch][hkv * G][hd]
  float* part_o;            // [hkv][rows][nsplit][hd]   (nsplit > 1)
  float* part_ml;           // [hkv][rows][nsplit][2]
  unsigned* tickets;        // one per (kv head, row tile): the last split to arrive sums up; null: a second kernel does
  int* err;
};

// Output row of (kv head, row).
__device__ __forceinline__ size_t am_out_row(const AmArgs& a, int kvh, int r) {
  return (size_t)(r / a.G) * (a.hkv * a.G) + kvh * a.G + r % a.G;
}

template <typename T, int HD, int MT, bool PACK>
__global__ void __launch_bounds__((AmShape<T, HD, MT, PACK>::kThreads), 1)
attn_shared_kernel(const AmArgs a) {
  using S = AmShape<T, HD, MT, PACK>;
  constexpr int KG = S::KG, NS = S::NS, QT = S::QT, KT = S::KT, NT = HD / 8;
  constexpr int NA = PACK ? KT : 2, RW = sizeof(T) == 2 ? 4 : 8;
  extern __shared__ __align__(128) unsigned char am_sm[];
  unsigned char* ring = am_sm + S::kQ;
  uint64_t* full = reinterpret_cast<uint64_t*>(am_sm + S::kBars);     // [KG][NS]
  uint64_t* empty = full + KG * NS;
  int* last_s = reinterpret_cast<int*>(empty + KG * NS);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int split = blockIdx.x % a.nsplit, unit = blockIdx.x / a.nsplit;
  const int row_tiles = (a.rows + S::kRows - 1) / S::kRows;
  const int kvh = unit / row_tiles, r0 = (unit % row_tiles) * S::kRows;
  if (threadIdx.x < KG * NS) {
    mbar_init(&full[threadIdx.x], 32 * MT);   // every lane of the group, once its copies have landed
    mbar_init(&empty[threadIdx.x], MT);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  pdl_wait();
  pdl_launch_dependents();
  const int cfirst = a.lo >> 4, nchunks = ((a.k1 + 15) >> 4) - cfirst;
  const int c0 = cfirst + (int)((long long)nchunks * split / a.nsplit), c1 = cfirst + (int)((long long)nchunks * (split + 1) / a.nsplit);

  float o[NT][4];
#pragma unroll
  for (int j = 0; j < NT; ++j) o[j][0] = o[j][1] = o[j][2] = o[j][3] = 0.f;
  float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};             // rows g and g + 8; PACK: row g & 3 in [0]
  const int g = lane >> 2, t = lane & 3;

  // ---- ring entries of a key group: K rows, then V rows of its chunks; entry n is chunk c0 + kg + (n / 2) KG.  The
  // group's warps issue them, each its share of the copies, NS - 1 ahead.  Chunks start at multiples of 16, so one never
  // spans two pages and is contiguous in the cache: every copy of the loop has a constant offset.
  const int mt = warp % MT, kg = warp / MT;
  // None of this lane's waits has given up.  A lane that gave up waits no more and asks for nothing, but goes on with what is
  // there: the products are the whole warp's, and lanes that left would be waited for (a vote a wait cost 0.4 %).
  bool ok = true;
  int page = 0;                                // of the next chunk to issue
  auto next_page = [&](int c) {                // volatile: a load that may sink to its use is a round trip to L2 in the loop
    if (c < c1) asm volatile("ld.global.nc.s32 %0, [%1];" : "=r"(page) : "l"(a.page_table + c * 16 / kPage));
  };
  next_page(c0 + kg);
  // a short query tile is asked for ahead of the cache rows, whose copies wait for the page number
  constexpr int NQ = S::kRows * (HD / 2) / S::kThreads;
  constexpr bool kQAhead = NQ <= 8 && NQ * S::kThreads == S::kRows * (HD / 2);
  auto q_pair = [&](int i) {
    const int r = i / (HD / 2), e = 2 * (i % (HD / 2));
    return r0 + r < a.rows ? *reinterpret_cast<const float2*>(a.q + (size_t)((r0 + r) / a.G) * a.q_stride + (kvh * a.G + (r0 + r) % a.G) * HD + e)
                           : make_float2(0.f, 0.f);
  };
  float2 qa[kQAhead ? NQ : 1];
  if constexpr (kQAhead) {
#pragma unroll
    for (int u = 0; u < NQ; ++u) qa[u] = q_pair(threadIdx.x + u * S::kThreads);
  }
  int is_slot = 0, is_round = 0;               // slot and use of the slot of the next entry to issue
  auto issue = [&](int n) {
    const int isv = n & 1, c = c0 + kg + (n >> 1) * KG, slot = is_slot, round = is_round;
    if (c >= c1) return;
    if (++is_slot == NS) { is_slot = 0; ++is_round; }
    uint64_t* fb = &full[kg * NS + slot];
    if (round > 0) ok = ok && mbar_wait(&empty[kg * NS + slot], (round - 1) & 1, a.err);
    if (!ok) return;
    constexpr int UPR = HD * (int)sizeof(T) / 16;               // 16-byte units per row; 32 / UPR or fewer rows per round
    const unsigned char* src = reinterpret_cast<const unsigned char*>(isv ? a.v : a.k) +
                               (((size_t)page * a.hkv + kvh) * kPage + c * 16 % kPage) * (UPR * 16) + lane * 16;
    const uint32_t drow = isv ? S::kVRow : S::kKRow;
    const uint32_t dst = smem_u32(ring + (size_t)(kg * NS + slot) * S::kHalf) + lane / UPR * drow + lane % UPR * 16;
    if (c * 16 >= a.lo && c * 16 + 16 <= a.k1) {
#pragma unroll
      for (int i = 0; i < UPR / 2; ++i)
        if (i % MT == mt) am_cp16(dst + (i * 32 / UPR) * drow + i * 32 % UPR * 16, src + i * 512, 16);
    } else {                                                     // rows outside the visible keys become zeros
#pragma unroll
      for (int i = 0; i < UPR / 2; ++i) {
        if (i % MT != mt) continue;
        const int key = c * 16 + (i * 32 + lane) / UPR;
        am_cp16(dst + (i * 32 / UPR) * drow + i * 32 % UPR * 16, src + i * 512, key >= a.lo && key < a.k1 ? 16 : 0);
      }
    }
    am_cp_arrive(fb);
    if (isv) next_page(c + KG);
  };
  for (int n = 0; n < NS - 1; ++n) issue(n);
  {
    // ---- query rows, scaled, as bf16 planes
    auto place = [&](int i, float2 x) {
      const int r = i / (HD / 2), e = 2 * (i % (HD / 2));
      uint32_t s3[3];
      am_split3(x.x * a.qscale, x.y * a.qscale, s3);
#pragma unroll
      for (int p = 0; p < 3; ++p) {
        const int row = PACK ? 4 * p + r : p * MT * 16 + r;
        *reinterpret_cast<uint32_t*>(am_sm + row * S::kQRow + e * 2) = s3[p];
      }
      if (PACK) *reinterpret_cast<uint32_t*>(am_sm + (12 + r) * S::kQRow + e * 2) = 0u;
    };
    if constexpr (kQAhead) {
#pragma unroll
      for (int u = 0; u < NQ; ++u) place(threadIdx.x + u * S::kThreads, qa[u]);
    } else {
#pragma unroll 8
      for (int i = threadIdx.x; i < S::kRows * (HD / 2); i += S::kThreads) place(i, q_pair(i));
    }
    __syncthreads();
    const uint32_t q_addr = smem_u32(am_sm) + (uint32_t)((mt * 16 + (lane & 15)) * S::kQRow + (lane >> 4) * 16);
    int slot = 0, phase = 0;
    auto advance = [&]() { if (++slot == NS) { slot = 0; phase ^= 1; } };
    for (int c = c0 + kg, n = 0; c < c1; c += KG, n += 2) {
      issue(n + NS - 1);
      // ---- scores of 16 keys: two n-tiles of 8, the leading and the other terms in accumulators of their own
      float acc[2][NA][4], sum[2][4];
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        sum[x][0] = sum[x][1] = sum[x][2] = sum[x][3] = 0.f;
#pragma unroll
        for (int p = 0; p < NA; ++p) acc[x][p][0] = acc[x][p][1] = acc[x][p][2] = acc[x][p][3] = 0.f;
      }
      ok = ok && mbar_wait(&full[kg * NS + slot], phase, a.err);
      const unsigned char* ks = ring + (size_t)(kg * NS + slot) * S::kHalf;
      const uint32_t k_addr = smem_u32(ks) + (uint32_t)(((lane & 7) + ((lane >> 4) << 3)) * S::kKRow + ((lane >> 3) & 1) * 16);
      uint32_t af[2][QT][4], raw[2][RW];                              // fragments of this k step and the next
      auto fetch = [&](int k) {
#pragma unroll
        for (int p = 0; p < QT; ++p) am_ldsm4(af[k & 1][p], q_addr + (uint32_t)(p * MT * 16 * S::kQRow + k * 32));
        if constexpr (sizeof(T) == 2) {
          am_ldsm4(raw[k & 1], k_addr + (uint32_t)(k * 32));          // {b0, b1} of n-tile 0, then of n-tile 1
        } else {
#pragma unroll
          for (int x = 0; x < 4; ++x) {
            const uint2 kv = *reinterpret_cast<const uint2*>(ks + ((x >> 1) * 8 + g) * S::kKRow + (k * 16 + (x & 1) * 8 + 2 * t) * 4);
            raw[k & 1][2 * x] = kv.x;
            raw[k & 1][2 * x + 1] = kv.y;
          }
        }
      };
      fetch(0);
#pragma unroll
      for (int k = 0; k < HD / 16; ++k) {
        if (k + 1 < HD / 16) fetch(k + 1);
        uint32_t bf[KT][4];
        if constexpr (sizeof(T) == 2) {
#pragma unroll
          for (int x = 0; x < 4; ++x) bf[0][x] = raw[k & 1][x];
        } else {
#pragma unroll
          for (int x = 0; x < 4; ++x) {
            uint32_t s3[3];
            am_split3(__uint_as_float(raw[k & 1][2 * x]), __uint_as_float(raw[k & 1][2 * x + 1]), s3);
#pragma unroll
            for (int p = 0; p < 3; ++p) bf[p][x] = s3[p];
          }
        }
#pragma unroll
        for (int w = 0; w < KT; ++w)
#pragma unroll
          for (int p = 0; p < QT; ++p)
            if (PACK || p + w <= 2) {
              am_mma(acc[0][PACK ? w : p + w > 0], af[k & 1][p], bf[w][0], bf[w][1]);
              am_mma(acc[1][PACK ? w : p + w > 0], af[k & 1][p], bf[w][2], bf[w][3]);
            }
        if (k % 4 == 3 && k + 1 < HD / 16) {                          // the leading term leaves the tensor core's accumulator
#pragma unroll
          for (int x = 0; x < 2; ++x)
#pragma unroll
            for (int y = 0; y < 4; ++y) { sum[x][y] += acc[x][0][y]; acc[x][0][y] = 0.f; }
        }
      }
      // the smallest terms first
#pragma unroll
      for (int x = 0; x < 2; ++x)
#pragma unroll
        for (int p = NA - 2; p >= 0; --p)
#pragma unroll
          for (int y = 0; y < 4; ++y) acc[x][p][y] += acc[x][p + 1][y];
#pragma unroll
      for (int x = 0; x < 2; ++x)
#pragma unroll
        for (int y = 0; y < 4; ++y) acc[x][0][y] += sum[x][y];
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty[kg * NS + slot]);
      advance();
      // ---- online softmax (base 2: the scale carries log2 e); P as the A operand of the second product
      const int key0 = c * 16 + 2 * t;                          // columns of this thread: key0, +1, +8, +9
      uint32_t pa[QT][4];
      if constexpr (PACK) {
        float s[4];
#pragma unroll
        for (int x = 0; x < 2; ++x)
#pragma unroll
          for (int y = 0; y < 2; ++y) {
            float v = acc[x][0][y] + acc[x][0][2 + y];                 // rows g and g + 8
            v += __shfl_xor_sync(0xffffffffu, v, 16);                  // rows g ^ 4
            s[2 * x + y] = key0 + 8 * x + y >= a.lo && key0 + 8 * x + y < a.k1 ? v : -INFINITY;
          }
        float mx = fmaxf(fmaxf(s[0], s[1]), fmaxf(s[2], s[3]));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
        const float mn = fmaxf(m[0], mx);
        const float corr = am_ex2(m[0] - mn);
        if (__any_sync(0xffffffffu, mn > m[0])) {
#pragma unroll
          for (int j = 0; j < NT; ++j) { o[j][0] *= corr; o[j][1] *= corr; o[j][2] *= corr; o[j][3] *= corr; }
        }
        m[0] = mn;
        float p[4];
#pragma unroll
        for (int x = 0; x < 4; ++x) p[x] = am_ex2(s[x] - mn);
        l[0] = l[0] * corr + ((p[0] + p[1]) + (p[2] + p[3]));
        uint32_t u[3], v[3];
        am_split3(p[0], p[1], u);
        am_split3(p[2], p[3], v);
        const bool upper = g >= 4;                                     // row g: term 0 of rows 0..3, term 1 of rows 4..7; row g + 8: term 2
        pa[0][0] = upper ? u[1] : u[0];
        pa[0][1] = upper ? 0u : u[2];
        pa[0][2] = upper ? v[1] : v[0];
        pa[0][3] = upper ? 0u : v[2];
      } else {
#pragma unroll
        for (int h = 0; h < 2; ++h) {                                  // rows g + 8 h
          float s[4];
#pragma unroll
          for (int x = 0; x < 2; ++x)
#pragma unroll
            for (int y = 0; y < 2; ++y) {
              s[2 * x + y] = key0 + 8 * x + y >= a.lo && key0 + 8 * x + y < a.k1 ? acc[x][0][2 * h + y] : -INFINITY;
            }
          float mx = fmaxf(fmaxf(s[0], s[1]), fmaxf(s[2], s[3]));
          mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
          mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
          const float mn = fmaxf(m[h], mx);
          const float corr = am_ex2(m[h] - mn);
          if (__any_sync(0xffffffffu, mn > m[h])) {
#pragma unroll
            for (int j = 0; j < NT; ++j) { o[j][2 * h] *= corr; o[j][2 * h + 1] *= corr; }
          }
          m[h] = mn;
          float p[4];
#pragma unroll
          for (int x = 0; x < 4; ++x) p[x] = am_ex2(s[x] - mn);
          l[h] = l[h] * corr + ((p[0] + p[1]) + (p[2] + p[3]));
          uint32_t u[3], v[3];
          am_split3(p[0], p[1], u);
          am_split3(p[2], p[3], v);
#pragma unroll
          for (int x = 0; x < QT; ++x) {
            pa[x][h] = u[x];
            pa[x][2 + h] = v[x];
          }
        }
      }
      // ---- O += P V
      issue(n + NS);
      ok = ok && mbar_wait(&full[kg * NS + slot], phase, a.err);
      const unsigned char* vs = ring + (size_t)(kg * NS + slot) * S::kHalf;
      const uint32_t v_addr = smem_u32(vs) + (uint32_t)(((lane & 7) + ((lane >> 3) & 1) * 8) * S::kVRow + (lane >> 4) * 16);
      uint32_t vraw[2][2][RW];                                        // two pairs of n-tiles at a time, fetched one step ahead
      auto vfetch = [&](int j4) {
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int j = 4 * j4 + 2 * u;
          if constexpr (sizeof(T) == 2) {
            am_ldsm4t(vraw[j4 & 1][u], v_addr + (uint32_t)(j * 16));
          } else {
#pragma unroll
            for (int x = 0; x < 4; ++x) {
              const unsigned char* p = vs + ((x & 1) * 8 + 2 * t) * S::kVRow + ((j + (x >> 1)) * 8 + g) * 4;
              vraw[j4 & 1][u][2 * x] = *reinterpret_cast<const uint32_t*>(p);
              vraw[j4 & 1][u][2 * x + 1] = *reinterpret_cast<const uint32_t*>(p + S::kVRow);
            }
          }
        }
      };
      vfetch(0);
#pragma unroll
      for (int j4 = 0; j4 < NT / 4; ++j4) {
        if (j4 + 1 < NT / 4) vfetch(j4 + 1);
        uint32_t bf[KT][2][4];
#pragma unroll
        for (int u = 0; u < 2; ++u)
#pragma unroll
          for (int x = 0; x < 4; ++x) {
            if constexpr (sizeof(T) == 2) {
              bf[0][u][x] = vraw[j4 & 1][u][x];
            } else {
              uint32_t s3[3];
              am_split3(__uint_as_float(vraw[j4 & 1][u][2 * x]), __uint_as_float(vraw[j4 & 1][u][2 * x + 1]), s3);
#pragma unroll
              for (int w = 0; w < 3; ++w) bf[w][u][x] = s3[w];
            }
          }
        // smallest terms first, four accumulators between two products of one chain
        float pv[4][4];
#pragma unroll
        for (int u = 0; u < 4; ++u) pv[u][0] = pv[u][1] = pv[u][2] = pv[u][3] = 0.f;
#pragma unroll
        for (int w = KT - 1; w >= 0; --w)
#pragma unroll
          for (int p = QT - 1; p >= 0; --p)
            if (PACK || p + w <= 2) {
#pragma unroll
              for (int u = 0; u < 4; ++u) am_mma(pv[u], pa[p], bf[w][u >> 1][2 * (u & 1)], bf[w][u >> 1][2 * (u & 1) + 1]);
            }
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
          for (int y = 0; y < 4; ++y) o[4 * j4 + u][y] += pv[u][y];
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty[kg * NS + slot]);
      advance();
    }
    // sums over the key columns of a row: the four lanes of a quad
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      l[h] += __shfl_xor_sync(0xffffffffu, l[h], 1);
      l[h] += __shfl_xor_sync(0xffffffffu, l[h], 2);
    }
  }
  // ---- the key groups of a row meet in shared memory (the query tile and the ring are done with)
  __syncthreads();
  float* mo = reinterpret_cast<float*>(am_sm);                          // [warps][kWRows][kMRow]
  float* mm = mo + S::kWarps * S::kWRows * S::kMRow;                    // [warps][kWRows][2]
  float* wt = mm + S::kWarps * S::kWRows * 2;                           // [rows][KG + 2]: weights, then M and L
  {
    float* wo = mo + (size_t)warp * S::kWRows * S::kMRow;
    if constexpr (PACK) {
#pragma unroll
      for (int j = 0; j < NT; ++j) {
#pragma unroll
        for (int y = 0; y < 2; ++y) {
          float v = o[j][y] + o[j][2 + y];
          v += __shfl_xor_sync(0xffffffffu, v, 16);
          if (g < 4) wo[g * S::kMRow + j * 8 + 2 * t + y] = v;
        }
      }
      if (t == 0 && g < 4) { mm[(warp * 4 + g) * 2] = m[0]; mm[(warp * 4 + g) * 2 + 1] = l[0]; }
    } else {
#pragma unroll
      for (int j = 0; j < NT; ++j) {
        *reinterpret_cast<float2*>(wo + g * S::kMRow + j * 8 + 2 * t) = make_float2(o[j][0], o[j][1]);
        *reinterpret_cast<float2*>(wo + (g + 8) * S::kMRow + j * 8 + 2 * t) = make_float2(o[j][2], o[j][3]);
      }
      if (t == 0) {
#pragma unroll
        for (int h = 0; h < 2; ++h) { mm[(warp * 16 + g + 8 * h) * 2] = m[h]; mm[(warp * 16 + g + 8 * h) * 2 + 1] = l[h]; }
      }
    }
  }
  __syncthreads();
  for (int r = threadIdx.x; r < S::kRows; r += S::kThreads) {
    const int mt = r / S::kWRows, rr = r % S::kWRows;
    float M = -INFINITY, L = 0.f;
#pragma unroll
    for (int k = 0; k < KG; ++k) M = fmaxf(M, mm[((k * MT + mt) * S::kWRows + rr) * 2]);
#pragma unroll
    for (int k = 0; k < KG; ++k) {
      const float w = M > -INFINITY ? am_ex2(mm[((k * MT + mt) * S::kWRows + rr) * 2] - M) : 0.f;
      L += w * mm[((k * MT + mt) * S::kWRows + rr) * 2 + 1];
      wt[r * (KG + 2) + k] = w;
    }
    wt[r * (KG + 2) + KG] = M;
    wt[r * (KG + 2) + KG + 1] = L;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < S::kRows * (HD / 4); i += S::kThreads) {
    const int r = i / (HD / 4), e = 4 * (i % (HD / 4));
    if (r0 + r >= a.rows) continue;
    const int mt = r / S::kWRows, rr = r % S::kWRows;
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int k = 0; k < KG; ++k) {
      const float w = wt[r * (KG + 2) + k];
      const float4 x = *reinterpret_cast<const float4*>(mo + ((size_t)(k * MT + mt) * S::kWRows + rr) * S::kMRow + e);
      s.x += w * x.x; s.y += w * x.y; s.z += w * x.z; s.w += w * x.w;
    }
    const float M = wt[r * (KG + 2) + KG], L = wt[r * (KG + 2) + KG + 1];
    if (a.nsplit == 1) {
      const float inv = L > 0.f ? 1.0f / L : 0.f;
      *reinterpret_cast<float4*>(a.out + am_out_row(a, kvh, r0 + r) * HD + e) = make_float4(s.x * inv, s.y * inv, s.z * inv, s.w * inv);
    } else {
      const size_t pi = ((size_t)kvh * a.rows + r0 + r) * a.nsplit + split;
      *reinterpret_cast<float4*>(a.part_o + pi * HD + e) = s;
      if (e == 0) *reinterpret_cast<float2*>(a.part_ml + pi * 2) = make_float2(M, L);
    }
  }
  if (a.nsplit > 1 && a.tickets) {
    // ---- the split that arrives last sums up this unit's rows
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) *last_s = ticket_last(a.tickets + unit, a.nsplit, [](unsigned* t, unsigned top) { return atomicInc(t, top); });
    __syncthreads();
    if (*last_s) {
      __threadfence();
      const int nr = min(S::kRows, a.rows - r0);
      float* w_s = reinterpret_cast<float*>(am_sm);                    // [row][nsplit]: exp2(m - M) / L
      const float2* ml = reinterpret_cast<const float2*>(a.part_ml) + ((size_t)kvh * a.rows + r0) * a.nsplit;
      // A chain of round trips to L2 if written so: sixteen partials are in flight at once, the first of them ahead of the
      // weights, and the (m, l) pairs of up to 32 splits are read once.
      constexpr int P = 16;
      const int items = nr * (HD / 4);
      float4 x[P];
      auto request = [&](int i, int p0) {
        const float* po = a.part_o + ((size_t)kvh * a.rows + r0 + i / (HD / 4)) * a.nsplit * HD + 4 * (i % (HD / 4));
#pragma unroll
        for (int u = 0; u < P; ++u)
          if (i < items && p0 + u < a.nsplit) x[u] = __ldcg(reinterpret_cast<const float4*>(po + (size_t)(p0 + u) * HD));
      };
      request(threadIdx.x, 0);
      for (int r = warp; r < nr; r += S::kThreads / 32) {
        const float2 own = lane < a.nsplit ? __ldcg(ml + (size_t)r * a.nsplit + lane) : make_float2(-INFINITY, 0.f);
        float M = own.x, L = 0.f;
        for (int s = lane + 32; s < a.nsplit; s += 32) M = fmaxf(M, __ldcg(ml + (size_t)r * a.nsplit + s).x);
        M = warp_max(M);
        for (int s = lane; s < a.nsplit; s += 32) {
          const float2 y = s < 32 ? own : __ldcg(ml + (size_t)r * a.nsplit + s);
          const float w = M > -INFINITY ? am_ex2(y.x - M) : 0.f;
          w_s[r * a.nsplit + s] = w;
          L += w * y.y;
        }
        L = warp_sum(L);
        const float inv = L > 0.f ? 1.0f / L : 0.f;
        for (int s = lane; s < a.nsplit; s += 32) w_s[r * a.nsplit + s] *= inv;
      }
      __syncthreads();
      for (int i = threadIdx.x; i < items; i += S::kThreads) {
        const int r = i / (HD / 4), e = 4 * (i % (HD / 4));
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int p0 = 0; p0 < a.nsplit; p0 += P) {
          if (i != (int)threadIdx.x || p0 > 0) request(i, p0);
#pragma unroll
          for (int u = 0; u < P; ++u)
            if (p0 + u < a.nsplit) {
              const float w = w_s[r * a.nsplit + p0 + u];
              s.x += w * x[u].x; s.y += w * x[u].y; s.z += w * x[u].z; s.w += w * x[u].w;
            }
        }
        *reinterpret_cast<float4*>(a.out + am_out_row(a, kvh, r0 + r) * HD + e) = s;
      }
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");       // only a wait that gave up leaves copies behind
}

// Sum of the splits where one CTA would take too long over them: one CTA per (row, up to 64 elements), 16 lanes of
// splits by up to 16 float4 columns.
constexpr int kAmSumThreads = 256;
static __global__ void __launch_bounds__(kAmSumThreads)
attn_shared_sum_kernel(const AmArgs a, int hd) {
  __shared__ float w_s[256];
  __shared__ float4 red[16][16];
  pdl_wait();
  pdl_launch_dependents();
  const int cols = hd < 64 ? hd / 4 : 16, blocks = hd / (4 * cols);
  const int row = blockIdx.x / blocks, eb = (blockIdx.x % blocks) * 4 * cols;
  const int kvh = row / a.rows, r = row % a.rows;
  const float2* ml = reinterpret_cast<const float2*>(a.part_ml) + (size_t)row * a.nsplit;
  if (threadIdx.x < 32) {
    float M = -INFINITY, L = 0.f;
    for (int s = threadIdx.x; s < a.nsplit; s += 32) M = fmaxf(M, __ldcg(ml + s).x);
    M = warp_max(M);
    for (int s = threadIdx.x; s < a.nsplit; s += 32) {
      const float2 x = __ldcg(ml + s);
      const float w = M > -INFINITY ? am_ex2(x.x - M) : 0.f;
      w_s[s] = w;
      L += w * x.y;
    }
    L = warp_sum(L);
    const float inv = L > 0.f ? 1.0f / L : 0.f;
    for (int s = threadIdx.x; s < a.nsplit; s += 32) w_s[s] *= inv;
  }
  __syncthreads();
  const int col = threadIdx.x % 16, sl = threadIdx.x / 16;
  float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
  if (col < cols) {
    const float* po = a.part_o + (size_t)row * a.nsplit * hd + eb + 4 * col;
    for (int p = sl; p < a.nsplit; p += 16) {
      const float4 x = __ldcg(reinterpret_cast<const float4*>(po + (size_t)p * hd));
      const float w = w_s[p];
      s.x += w * x.x; s.y += w * x.y; s.z += w * x.z; s.w += w * x.w;
    }
  }
  red[sl][col] = s;
  __syncthreads();
  if (threadIdx.x < cols) {
    float4 v = red[0][threadIdx.x];
#pragma unroll
    for (int p = 1; p < 16; ++p) {
      const float4 x = red[p][threadIdx.x];
      v.x += x.x; v.y += x.y; v.z += x.z; v.w += x.w;
    }
    *reinterpret_cast<float4*>(a.out + am_out_row(a, kvh, r) * hd + eb + 4 * threadIdx.x) = v;
  }
}

// ---- host side

// The shape and split count of one call: as many splits as fill the SMs, no fewer than one chunk of 16 keys per key
// group of a split, no more partials than `cap` splits' worth of scratch.
template <typename T, int HD, int MT, bool PACK>
inline void launch_attn_shared_t(cudaStream_t st, AmArgs a, int device, int sms, int cap, unsigned* tickets) {
  using S = AmShape<T, HD, MT, PACK>;
  const int units = a.hkv * ((a.rows + S::kRows - 1) / S::kRows);
  const int nchunks = (a.k1 + 15) / 16 - a.lo / 16;
  a.nsplit = std::max(1, std::min(std::min(sms / units, cap), std::min(kTicketSplits, (nchunks + S::KG - 1) / S::KG)));
  // One CTA sums up to 128 KB of partials in about the time that a second launch costs; more is spread over a grid.
  const size_t part = (size_t)a.nsplit * std::min(a.rows, S::kRows) * HD * 4;
  a.tickets = part <= 128 * 1024 && units <= kTicketUnits ? ticket_row(tickets, a.nsplit) : nullptr;
  static unsigned char ready[64] = {};                                // per device; a race only repeats the call
  if (!ready[device]) {
    raise_dyn_smem(attn_shared_kernel<T, HD, MT, PACK>, (size_t)S::kSmem);
    ready[device] = 1;
  }
  launch_pdl(attn_shared_kernel<T, HD, MT, PACK>, dim3(units * a.nsplit), dim3(S::kThreads), (size_t)S::kSmem, st, a);
  if (a.nsplit > 1 && !a.tickets)
    launch_pdl(attn_shared_sum_kernel, dim3(a.hkv * a.rows * (HD < 64 ? 1 : HD / 64)), dim3(kAmSumThreads), (size_t)0, st, a, (int)HD);
}
template <typename T, int HD>
inline void launch_attn_shared_r(cudaStream_t st, const AmArgs& a, int device, int sms, int cap, unsigned* tickets) {
  if (a.rows <= 4) launch_attn_shared_t<T, HD, 1, true>(st, a, device, sms, cap, tickets);
  else if (a.rows <= 16) launch_attn_shared_t<T, HD, 1, false>(st, a, device, sms, cap, tickets);
  else if (a.rows <= 32) launch_attn_shared_t<T, HD, 2, false>(st, a, device, sms, cap, tickets);
  else launch_attn_shared_t<T, HD, 4, false>(st, a, device, sms, cap, tickets);
}
template <typename T>
inline void launch_attn_shared(cudaStream_t st, const AmArgs& a, int hd, int device, int sms, int cap, unsigned* tickets) {
  switch (hd) {
    case 32: launch_attn_shared_r<T, 32>(st, a, device, sms, cap, tickets); break;
    case 64: launch_attn_shared_r<T, 64>(st, a, device, sms, cap, tickets); break;
    case 128: launch_attn_shared_r<T, 128>(st, a, device, sms, cap, tickets); break;
    default: launch_attn_shared_r<T, 256>(st, a, device, sms, cap, tickets); break;
  }
}
// The kernels of one cache type are a translation unit.
void launch_attn_shared_f32(cudaStream_t st, const AmArgs& a, int hd, int device, int sms, int cap, unsigned* tickets);
void launch_attn_shared_bf16(cudaStream_t st, const AmArgs& a, int hd, int device, int sms, int cap, unsigned* tickets);

}  // namespace b200lm

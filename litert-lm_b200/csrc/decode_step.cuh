// Decode step as a chain of small kernels, one per phase, replayed from a CUDA graph with programmatic edges.
//
//   qkv      residual update + pre-attention norm -> QKV projection
//   attn     QK-norm, RoPE, cache append, one CTA per (session, kv head, key split)
//   o        combine of the splits -> O projection (K split over whole heads)
//   gate/up  residual update + pre-FFN norm -> gate / up + GeGLU
//   down     down projection (K split)
//   head     residual update + final norm -> LM head, arg-max, next token and position
//
// What bounds a step of one to four sessions is the chain, not the bytes: 5 kernels a layer, each of which needs all
// of its predecessor.  A kernel boundary with programmatic dependent launch costs 1.7 us on this chip including the
// first read of the predecessor's output (a chain of 130 kernels of 148 CTAs, measured), less than the same hand-over
// inside one persistent kernel with its prologue (2.5 - 3 us with flag-carrying words), and everything that does not
// depend on the predecessor happens before griddepcontrol.wait: barriers, the first weight tiles of every warp, the
// scales, the cached K / V rows and the gains.  So the weights stream while the previous kernel still works, and two
// generations of CTAs share an SM (shared memory is sized for that).
//
// The projections are the int4 x int8 tiles of decode_ops.cuh: activations as up to three int8 terms against the
// vector's own maximum, exact integer sums.  A CTA's row tiles x k tiles are dealt to its 16 warps as contiguous
// runs; every warp streams its run through a private ring of bulk copies (no barrier between warps) and adds its
// fragments into the tile's integer sums in shared memory.
#pragma once
#include <algorithm>

#include "common.cuh"
#include "decode_ops.cuh"
#include "prefill_ops.cuh"

namespace b200lm {

constexpr int kStThreads = 512, kStWarps = kStThreads / 32;
constexpr int kStMaxSlots = 2;            // ring slots of a warp
constexpr int kStKeys = 32;               // keys of one attention round (one per lane of the softmax warps)
constexpr int kStMaxSplits = 64;
constexpr int kAtThreads = 256;
constexpr int kStShortSlice = 256;        // widest slice of K that kStCombineShort takes
static_assert(kStShortSlice <= kStThreads, "less than a float4 a thread with four sessions");

enum StepPrologue { kStResid = 0, kStAct = 1, kStCombine = 2, kStCombineShort = 3 };
enum StepEpilogue { kStPlain = 0, kStGeglu = 1, kStHead = 2 };

// Byte offsets of a projection's shared-memory areas (made on the host).
struct StepSmem {
  int ring, bars, xq, red, vals, scratch, total;
};

struct StepGemv {
  const uint4* w;             // [row_tile][k_tile] tiles of 512 bytes
  const float* wscale;        // [row_tile][16]
  int tiles, KT;              // row tiles, k tiles
  int slices, cps;            // K slices, CTAs per slice (grid = slices * cps)
  int KTs;                    // k tiles of a slice
  int tile_base, tile_rem;    // row tiles (gate / up: pairs) per CTA of a slice: base, one more for the first rem
  int slot_tiles, nslots;     // ring of a warp: slots of up to slot_tiles k tiles of its run
  int round_tiles;            // row tiles whose sums are held at once
  StepSmem sm;
  int xstride;                // bytes between rows of the quantised activations (== 64 mod 128)
  float* y;                   // plain [slices][ncols][16 tiles]; geglu [ncols][8 tiles]; head: logits [ncols][16 tiles]
  int kmax;                   // values per session the prologue quantises (K of a slice)
  float inv_k;                // resid: 1 / d
  // resid
  const float* parts;         // [nparts][ncols][d], or null: x is the embedding of the session's token
  int nparts;                 // at most four
  const float* xin;           // [ncols][d]
  float* xout;
  const float *g_post, *g_pre;
  // act
  const float* act;           // [ncols][slices * kmax]
  // combine
  const float *part_o, *part_ml;    // [ncols][hkv][nsplit][G][hd], [..][2]
  int nsplit, is_global, heads, hd_log2;   // heads of a slice
  int* ticket;                // head: CTAs that have published their candidate
  int bar;                    // index of this kernel in the step (timeline)
};

// Session groups of a CTA: three sessions take the instantiation of four, a quarter of whose warps then have no vector in the
// prologue.  A step of the 1B model at 300 keys is 485 / 621 / 688 / 732 us with 1 / 2 / 3 / 4 sessions; two took 658 with the
// instantiation of four.
__host__ __device__ inline int st_cols(int ncols) { return ncols <= 2 ? (ncols <= 1 ? 1 : 2) : 4; }
__host__ __device__ inline int st_xstride(int kmax) { return (kmax + 127) / 128 * 128 + 64; }

inline StepSmem st_smem(const StepGemv& g, int ncols, int nterms) {
  StepSmem s;
  int o = 0;
  s.ring = o; o += kStWarps * g.nslots * g.slot_tiles * 512;
  s.bars = o; o += kStWarps * kStMaxSlots * 8;
  s.xq = o; o += ncols * nterms * g.xstride;
  s.red = o; o += g.round_tiles * 16 * kQCols * 4;
  s.vals = o;
  if (g.heads) {              // combine: split sums, then split weights
    const int v = ncols * g.kmax * 4;
    o += (v > kStThreads * 16 ? v : kStThreads * 16) + ncols * g.heads * kStMaxSplits * 4;
  }
  s.scratch = o; o += 64 * 4 + 2 * kMaxCols * 4 + 2 * kStWarps * kMaxCols * 4;
  s.total = (o + 127) & ~127;
  return s;
}

// Keys of an attention split: at least a round, more when the context is longer than nsplit rounds.
__host__ __device__ inline int st_chunk(int nkeys, int nsplit) {
  const int c = (nkeys + nsplit - 1) / nsplit;
  return c > kStKeys ? c : kStKeys;
}
__device__ __forceinline__ int st_visible(const ModelDims& dm, int pos, int is_global) {
  return is_global ? pos + 1 : min(pos + 1, dm.window);
}

// Four consecutive values scaled into [-127, 127] as int8 terms (x = t0 + t1 / 128 + t2 / 16384), permuted inside each
// 64-wide k tile so that lane t of an MMA quad finds its words for k = 4t, 16 + 4t, 32 + 4t, 48 + 4t in one 16-byte load.
// Adding 1.5 * 2^23 rounds to the nearest integer and leaves it in the low byte: adds on the FMA pipe, where rounding
// and conversion instructions would queue on the quarter-rate pipe (430 cycles per projection).
__device__ __forceinline__ void st_quantize4(float4 r, int nterms, int8_t* row0, int k, int stride) {
  const float M = 12582912.0f;
  const float v[4] = {r.x, r.y, r.z, r.w};
  uint32_t b[3][4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float u0 = v[i] + M, r1 = (v[i] - (u0 - M)) * 128.0f;
    const float u1 = r1 + M, r2 = (r1 - (u1 - M)) * 128.0f;
    b[0][i] = __float_as_uint(u0);
    b[1][i] = __float_as_uint(u1);
    b[2][i] = __float_as_uint(r2 + M);
  }
  const int kk = k & 63;
  int8_t* q = row0 + (k & ~63) + ((kk >> 2) & 3) * 16 + (kk >> 4) * 4;
#pragma unroll
  for (int t = 0; t < 3; ++t)
    if (t < nterms)
      *reinterpret_cast<uint32_t*>(q + t * stride) = __byte_perm(__byte_perm(b[t][0], b[t][1], 0x0040), __byte_perm(b[t][2], b[t][3], 0x0040), 0x5410);
}

// Timeline of one step (B200Lm_TraceDecodeStep): stamps of kernel `bar`, in nanoseconds of the device-wide timer.
// 0 start, 1 predecessor complete, 2 activations ready, 3 tiles done, 4 end; the end is also "arrive" of this kernel
// and stamp 1 "release" of the one before.
__device__ __forceinline__ void st_stamp(const DecodeArgs& a, int bar, int k) {
  if (a.trace == nullptr || threadIdx.x != 0) return;
  long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  const size_t i = (size_t)bar * a.trace_ctas + blockIdx.x;
  if ((int)blockIdx.x >= a.trace_ctas) return;
  a.trace_pts[i * 8 + k] = t;
  if (k == 4) a.trace[i * 2] = t;
  if (k == 1 && bar > 0) a.trace[(i - a.trace_ctas) * 2 + 1] = t;
}

// Asks for a line ahead of its use, without waiting for it or keeping the value.
__device__ __forceinline__ void st_touch(const float* p) {
  float x;
  asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(x) : "l"(p));
}
__device__ __forceinline__ float4 st_ld4(const float* p) { return __ldcg(reinterpret_cast<const float4*>(p)); }

// Maximum over the warp in one instruction: of floats that are not negative (their bits order as they do), and of any.
__device__ __forceinline__ float st_warp_absmax(float v) { return __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(v))); }
__device__ __forceinline__ float st_warp_max(float v) {
  const int b = __float_as_int(v), k = __reduce_max_sync(0xffffffffu, b ^ ((b >> 31) & 0x7fffffff));
  return __int_as_float(k ^ ((k >> 31) & 0x7fffffff));
}
__device__ __forceinline__ float st_absmax(float4 v) { return fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))); }
__device__ __forceinline__ float st_sq(float4 v) { return (v.x * v.x + v.y * v.y) + (v.z * v.z + v.w * v.w); }

// Sum or maximum of N floats in shared memory (N = 4, 8 or 16, 16-byte aligned): wide loads, a tree.
template <int N>
__device__ __forceinline__ float st_sum_row(const float* p) {
  float4 v[N / 4];
#pragma unroll
  for (int i = 0; i < N / 4; ++i) v[i] = reinterpret_cast<const float4*>(p)[i];
  float s[N / 4];
#pragma unroll
  for (int i = 0; i < N / 4; ++i) s[i] = (v[i].x + v[i].y) + (v[i].z + v[i].w);
#pragma unroll
  for (int n = N / 8; n >= 1; n /= 2)
#pragma unroll
    for (int i = 0; i < n; ++i) s[i] += s[i + n];
  return s[0];
}
template <int N>
__device__ __forceinline__ float st_max_row(const float* p) {
  float4 v[N / 4];
#pragma unroll
  for (int i = 0; i < N / 4; ++i) v[i] = reinterpret_cast<const float4*>(p)[i];
  float m = fmaxf(fmaxf(v[0].x, v[0].y), fmaxf(v[0].z, v[0].w));
#pragma unroll
  for (int i = 1; i < N / 4; ++i) m = fmaxf(m, fmaxf(fmaxf(v[i].x, v[i].y), fmaxf(v[i].z, v[i].w)));
  return m;
}

// One projection.  NV: float4 of a session's vector per thread; CP: session groups (one session: three terms and all
// 16 warps on its vector; two: eight warps each; up to four: four).
// STREAM: the warps' runs are longer than the ring (else a run is one slot, requested ahead of the wait and awaited
// once).  A kernel runs its code once, so the code is kept short: nothing with a run-time count is unrolled (with the
// compiler's unrolling these kernels were 60 - 120 KB each, and five of them in turn waited for instructions).
template <int PRO, int EPI, int NV, int CP, bool STREAM>
__global__ void __launch_bounds__(kStThreads, NV <= 4 && !STREAM ? 2 : 1)
step_gemv_kernel(const __grid_constant__ DecodeArgs a, const __grid_constant__ StepGemv g) {
  constexpr int W = kStWarps / CP, T = W * 32;                          // warps, threads of a session group
  extern __shared__ __align__(128) unsigned char st_sm[];
  const int ncols = CP == 1 ? 1 : a.ncols, nterms = CP == 1 ? 3 : a.nterms;
  const int warp = warp_index(), lane = threadIdx.x & 31;
  st_stamp(a, g.bar, 0);
  uint64_t* bars = reinterpret_cast<uint64_t*>(st_sm + g.sm.bars) + warp * kStMaxSlots;
  int8_t* xq = reinterpret_cast<int8_t*>(st_sm + g.sm.xq);
  int* red = reinterpret_cast<int*>(st_sm + g.sm.red);
  float* scratch = reinterpret_cast<float*>(st_sm + g.sm.scratch);      // 3 x 16 reduction words
  float* colscale = scratch + 64;
  const int xstride = g.xstride, KTs = g.KTs;
  int* err = &a.st->err;

  // ---- this CTA's row tiles [t0, t0 + ntile) and k tiles [kt0, kt0 + KTs)
  const int slice = g.slices == 1 ? 0 : (int)blockIdx.x / g.cps, local = blockIdx.x - slice * g.cps;
  const int kt0 = slice * KTs;
  constexpr int unit = EPI == kStGeglu ? 2 : 1;                          // gate / up pairs stay together
  const int t0 = (local * g.tile_base + min(local, g.tile_rem)) * unit, ntile = (g.tile_base + (local < g.tile_rem ? 1 : 0)) * unit;

  // ---- weight stream: a round's row tiles x k tiles, dealt to the warps as contiguous runs
  struct Cursor {
    int round, left, tile, kt;                                           // k tiles left in the run; tile counted from t0
  };
  auto start_round = [&](Cursor& c) {
    const int nt = min(g.round_tiles, ntile - c.round * g.round_tiles);
    if (nt <= 0) { c.left = -1; return; }
    const int total = nt * KTs, per = (total + kStWarps - 1) / kStWarps, beg = min(total, warp * per), tile = beg / KTs;
    c.left = min(per, total - beg);
    c.tile = c.round * g.round_tiles + tile;
    c.kt = beg - tile * KTs;
  };
  Cursor cc{0, 0, 0, 0};
  start_round(cc);
  Cursor pc = cc;
  const int nslots = STREAM ? g.nslots : 1, slot_tiles = g.slot_tiles;
  unsigned char* wring = st_sm + g.sm.ring + (size_t)warp * nslots * slot_tiles * 512;
  int ps = 0;                                                            // slot of the next fill
  const bool leader = elect_one();
  auto issue = [&]() {
    if (STREAM) {
#pragma unroll 1
      while (pc.left == 0) { ++pc.round; start_round(pc); }
    }
    if (pc.left <= 0) return;
    int n = STREAM ? min(slot_tiles, pc.left) : pc.left;
    uint64_t* bar = &bars[ps];
    if (leader) mbar_arrive_expect_tx(bar, (uint32_t)n * 512u);
    unsigned char* dst = wring + (size_t)ps * slot_tiles * 512;
    const uint4* src = g.w + ((size_t)(t0 + pc.tile) * g.KT + kt0 + pc.kt) * 32;
    pc.left -= n;
#pragma unroll 1
    while (n > 0) {                                                      // one copy per row tile (one in all when K is not split)
      const int len = g.slices == 1 ? n : min(n, KTs - pc.kt);
      if (leader) bulk_load_1d(dst, src, (uint32_t)len * 512u, bar);
      dst += len * 512;
      n -= len;
      pc.kt += len;
      src += len * 32;
      if (g.slices > 1 && pc.kt == KTs) { pc.kt = 0; ++pc.tile; src += (g.KT - KTs) * 32; }
    }
    if (STREAM) {
      if (g.slices == 1) {
#pragma unroll 1
        while (pc.kt >= KTs) { pc.kt -= KTs; ++pc.tile; }
      }
      if (++ps == nslots) ps = 0;
    }
  };
  if (leader) {
#pragma unroll 1
    for (int s = 0; s < nslots; ++s) mbar_init(&bars[s], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncwarp();
  if (STREAM) {
#pragma unroll 1
    for (int s = 0; s < nslots; ++s) issue();
  } else {
    issue();
  }
  {
    const int n4 = min(g.round_tiles, ntile) * 16 * kQCols / 4;
#pragma unroll 1
    for (int i = threadIdx.x; i < n4; i += kStThreads) reinterpret_cast<int4*>(red)[i] = make_int4(0, 0, 0, 0);
  }
  // the row scales this thread will need first
  float wsc[2] = {0.f, 0.f};
  {
    const int rows = min(g.round_tiles, ntile) * 16;
    const float* src = g.wscale + t0 * 16;
    if (EPI == kStGeglu) {
      const int f = threadIdx.x, row = (f >> 4) * 32 + (f & 15);
      if (f < rows / 2) { wsc[0] = __ldg(src + row); wsc[1] = __ldg(src + row + 16); }
    } else if ((int)threadIdx.x < rows) {
      wsc[0] = __ldg(src + threadIdx.x);
    }
  }
  const int col = CP == 1 ? 0 : warp / W, gw = CP == 1 ? warp : warp % W, tl = gw * 32 + lane;
  const bool colok = CP == 1 || col < ncols;
  int8_t* q0 = xq + (size_t)(col * nterms) * xstride;

  // ---- prologue: the session's vector, quantised against its own maximum
  float4 v[NV];
  int vi[NV];                                                            // float4 index, or -1
  float m = 0.f, post = 1.0f;                                            // column scale = maximum * post / 127
  if constexpr (PRO == kStResid) {
    const int d = g.kmax, d4 = d / 4, nch = (d4 + 31) / 32;
    // Every CTA reads the same few lines at the same time: each starts at another one.  The warps' sums are filed by
    // chunk, so that all CTAs add them in the same order (equal rows of the head give bit-equal logits).
    const int rot = NV == 1 ? (int)blockIdx.x % nch : 0;
    int slot_r = warp;                                                   // where this warp's sums go
    constexpr bool kGainsAhead = NV <= (STREAM ? 4 : 2);                 // as far as the registers go
    float4 gp[NV], gq[NV];
#pragma unroll
    for (int u = 0; u < NV; ++u) {
      int ch = gw + u * W;
      const bool in = ch < nch;
      if (NV == 1 && in) {
        ch += rot;
        if (ch >= nch) ch -= nch;
        slot_r = col * W + ch;
      }
      vi[u] = in && colok && ch * 32 + lane < d4 ? ch * 32 + lane : -1;
      gp[u] = gq[u] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (kGainsAhead && vi[u] >= 0) {
        if (g.parts) gp[u] = __ldg(reinterpret_cast<const float4*>(g.g_post) + vi[u]);
        gq[u] = __ldg(reinterpret_cast<const float4*>(g.g_pre) + vi[u]);
      } else if (vi[u] >= 0) {                                           // else into L1: they come from HBM in every step
        if (g.parts) st_touch(g.g_post + 4 * vi[u]);
        st_touch(g.g_pre + 4 * vi[u]);
      }
    }
    pdl_wait();
    pdl_launch_dependents();
    st_stamp(a, g.bar, 1);
    if (g.parts) {
      float4 f[NV];
      float ss = 0.f;
#pragma unroll
      for (int u = 0; u < NV; ++u) {
        v[u] = f[u] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (vi[u] >= 0) {
          const float* p = g.parts + (size_t)col * d + 4 * vi[u];
          const size_t ps_ = (size_t)ncols * d;
          float4 t[4];
          t[0] = st_ld4(p);
#pragma unroll
          for (int q = 1; q < 4; ++q) t[q] = q < g.nparts ? st_ld4(p + q * ps_) : make_float4(0.f, 0.f, 0.f, 0.f);
          v[u] = st_ld4(g.xin + (size_t)col * d + 4 * vi[u]);
          f[u] = make_float4((t[0].x + t[1].x) + (t[2].x + t[3].x), (t[0].y + t[1].y) + (t[2].y + t[3].y), (t[0].z + t[1].z) + (t[2].z + t[3].z),
                             (t[0].w + t[1].w) + (t[2].w + t[3].w));
        }
        ss += st_sq(f[u]);
      }
      ss = warp_sum(ss);
      if (lane == 0) scratch[slot_r] = ss;
      __syncthreads();
      const float r = rsqrtf(st_sum_row<W>(scratch + col * W) * g.inv_k + a.dims.eps);
#pragma unroll
      for (int u = 0; u < NV; ++u) {
        if (!kGainsAhead && vi[u] >= 0) gp[u] = __ldg(reinterpret_cast<const float4*>(g.g_post) + vi[u]);
        v[u].x += f[u].x * r * gp[u].x; v[u].y += f[u].y * r * gp[u].y; v[u].z += f[u].z * r * gp[u].z; v[u].w += f[u].w * r * gp[u].w;
      }
    } else {
      int tok = colok ? __ldcg(&a.st->token[col]) : 0;
      if (tok < 0 || tok >= a.dims.vocab) {
        if (tl == 0) atomicExch(err, (int)kDevBadToken);
        tok = 0;
      }
      const unsigned short* row = reinterpret_cast<const unsigned short*>(a.embed_rows + (size_t)tok * (d / 2));
      const float sc = __ldg(a.embed_scale + tok) * sqrtf((float)d);
#pragma unroll
      for (int u = 0; u < NV; ++u) {
        v[u] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (vi[u] >= 0) {
          const int b = __ldg(row + vi[u]);         // four nibbles, low first, two's complement
          v[u] = make_float4((float)((b << 28) >> 28) * sc, (float)((b << 24) >> 28) * sc, (float)((b << 20) >> 28) * sc,
                             (float)((b << 16) >> 28) * sc);
        }
      }
    }
    float ss2 = 0.f;
#pragma unroll
    for (int u = 0; u < NV; ++u) {
      if (vi[u] >= 0 && blockIdx.x == 0) *reinterpret_cast<float4*>(g.xout + (size_t)col * d + 4 * vi[u]) = v[u];
      if (!kGainsAhead && vi[u] >= 0) gq[u] = __ldg(reinterpret_cast<const float4*>(g.g_pre) + vi[u]);
      ss2 += st_sq(v[u]);
      v[u].x *= gq[u].x; v[u].y *= gq[u].y; v[u].z *= gq[u].z; v[u].w *= gq[u].w;
      m = fmaxf(m, st_absmax(v[u]));
    }
    // sum and maximum share one pass through shared memory
    ss2 = warp_sum(ss2);
    m = st_warp_absmax(m);
    if (lane == 0) { scratch[16 + slot_r] = ss2; scratch[32 + slot_r] = m; }
    __syncthreads();
    m = st_max_row<W>(scratch + 32 + col * W);
    post = rsqrtf(st_sum_row<W>(scratch + 16 + col * W) * g.inv_k + a.dims.eps);   // the row factor leaves with the column scale
  } else if constexpr (PRO == kStCombineShort) {
    // The combine below for a slice of at most 256 values and heads of 128 and more: a warp's 128 values belong to one
    // head, so it makes the weights of that head's splits itself and takes them out of its lanes; one warp of the session
    // then adds the split groups, and the vector's maximum is a maximum over its lanes.  Two barriers of the CTA instead of
    // four: the prologue of the 1B model's O projection takes 2.2 us, 2.6 with the general form.
    const int k4 = g.kmax / 4, wide = k4 > 32, sg = W >> wide, sgi = gw >> wide, c4 = (wide ? (gw & 1) * 32 : 0) + lane;
    const int hd = 1 << g.hd_log2, G = a.dims.hq / a.dims.hkv, h = slice * g.heads + ((4 * c4) >> g.hd_log2), kvh = h / G;
    const int pos = colok ? __ldcg(&a.st->pos[col]) : 0;                 // has not changed since the step began
    const int nkeys = st_visible(a.dims, min(max(pos, 0), a.dims.max_ctx - 1), g.is_global);
    const int chunk = st_chunk(nkeys, g.nsplit), na = colok ? (nkeys + chunk - 1) / chunk : 0;      // splits that hold keys
    const size_t base = (((size_t)col * a.dims.hkv + kvh) * g.nsplit) * G + (h - kvh * G), sstride = (size_t)G << g.hd_log2;
    const float* p = g.part_o + (base << g.hd_log2) + ((4 * c4) & (hd - 1));
    const float* ml = g.part_ml + base * 2;
    float4* part = reinterpret_cast<float4*>(st_sm + g.sm.vals);         // [split groups][ncols][k4]
    pdl_wait();
    pdl_launch_dependents();
    st_stamp(a, g.bar, 1);
    float2 x[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int s = lane + 32 * q;
      x[q] = s < na ? __ldcg(reinterpret_cast<const float2*>(ml + (size_t)s * G * 2)) : make_float2(-INFINITY, 0.f);
    }
    constexpr int kAhead = 4;
    float4 pre[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; ++u) pre[u] = sgi + u * sg < na ? st_ld4(p + (sgi + u * sg) * sstride) : make_float4(0.f, 0.f, 0.f, 0.f);
    const float M = st_warp_max(fmaxf(x[0].x, x[1].x));
    float w0 = __expf(x[0].x - M), w1 = __expf(x[1].x - M);
    const float Lsum = warp_sum(x[0].y * w0 + x[1].y * w1), inv = Lsum > 0.f ? __fdividef(1.0f, Lsum) : 0.f;
    w0 *= inv;
    w1 *= inv;
    auto weight = [&](int s) { return __shfl_sync(0xffffffffu, s < 32 ? w0 : w1, s & 31); };
    float4 s4 = make_float4(0.f, 0.f, 0.f, 0.f);
    auto add = [&](const float4& o, float w) { s4.x += w * o.x; s4.y += w * o.y; s4.z += w * o.z; s4.w += w * o.w; };
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      const float w = weight(sgi + u * sg);                              // zero past the last split, or read as zero
      add(pre[u], sgi + u * sg < na ? w : 0.f);
    }
#pragma unroll 2
    for (int s = sgi + kAhead * sg; s < na; s += sg) add(st_ld4(p + s * sstride), weight(s));
    if (colok) part[(sgi * ncols + col) * k4 + c4] = s4;
    __syncthreads();
    if (gw == 0 && colok) {
      float4 y[2];
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        y[c] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (c <= wide) {
#pragma unroll
          for (int q = 0; q < W; ++q)
            if (q < sg && c * 32 + lane < k4) {
              const float4 o = part[(q * ncols + col) * k4 + c * 32 + lane];
              y[c].x += o.x; y[c].y += o.y; y[c].z += o.z; y[c].w += o.w;
            }
        }
        m = fmaxf(m, st_absmax(y[c]));
      }
      m = st_warp_absmax(m);
      const float k = m > 0.f ? __fdividef(127.0f, m) * 0.9999999f : 0.f;
      if (lane == 0) colscale[col] = k > 0.f ? __fdividef(post, k) : 0.f;
#pragma unroll
      for (int c = 0; c < 2; ++c)
        if (c * 32 + lane < k4) st_quantize4(make_float4(y[c].x * k, y[c].y * k, y[c].z * k, y[c].w * k), nterms, q0, 4 * (c * 32 + lane), xstride);
    }
  } else {
    const int K = g.kmax, k4 = K / 4;
#pragma unroll
    for (int u = 0; u < NV; ++u) vi[u] = colok && tl + u * T < k4 ? tl + u * T : -1;
    if constexpr (PRO == kStAct) {
      pdl_wait();
      pdl_launch_dependents();
      st_stamp(a, g.bar, 1);
      const float* src = g.act + (size_t)col * (g.slices * K) + (size_t)slice * K;
#pragma unroll
      for (int u = 0; u < NV; ++u) v[u] = vi[u] >= 0 ? st_ld4(src + 4 * vi[u]) : make_float4(0.f, 0.f, 0.f, 0.f);
    } else {
      // combine of the key splits of this slice's heads: sum_s o_s exp(m_s - M) / sum_s l_s exp(m_s - M).  The position
      // has not changed since the step began, so it is read ahead of the wait.
      const int heads = g.heads, G = a.dims.hq / a.dims.hkv, hd = 1 << g.hd_log2;
      float* part = reinterpret_cast<float*>(st_sm + g.sm.vals);         // [split groups][ncols][K]
      float* wsp = part + (ncols * K > kStThreads * 4 ? ncols * K : kStThreads * 4);   // [ncols][heads][kStMaxSplits]
      const int pos = colok ? __ldcg(&a.st->pos[col]) : 0;
      const int nkeys = st_visible(a.dims, min(max(pos, 0), a.dims.max_ctx - 1), g.is_global);
      const int chunk = st_chunk(nkeys, g.nsplit), na = (nkeys + chunk - 1) / chunk;   // splits that hold keys
      const int sg = max(1, T / k4), sgi = tl / k4, c4 = tl - sgi * k4;  // split groups, this thread's group and first float4
      const bool lead = colok && sgi < sg;
      auto head_base = [&](int hh) {                                     // first partial of head hh of the slice
        const int h = slice * heads + hh, kvh = h / G;
        return (((size_t)col * a.dims.hkv + kvh) * g.nsplit) * G + (h - kvh * G);
      };
      const float* p0 = g.part_o + (head_base((4 * c4) >> g.hd_log2) << g.hd_log2) + ((4 * c4) & (hd - 1));
      const size_t sstride = (size_t)G << g.hd_log2;
      const float* ml0 = g.part_ml + head_base(gw) * 2;
      pdl_wait();
      pdl_launch_dependents();
      st_stamp(a, g.bar, 1);
      // every head's first partials are requested before its weights are known
      constexpr int kAhead = 4;
      float4 pre[kAhead];
#pragma unroll
      for (int u = 0; u < kAhead; ++u) {
        const int s = sgi + u * sg;
        pre[u] = lead && s < na ? st_ld4(p0 + s * sstride) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
#pragma unroll 1
      for (int hh = gw; hh < heads && colok; hh += W) {
        const float* ml = hh == gw ? ml0 : g.part_ml + head_base(hh) * 2;
        float2 x[2];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const int s = lane + 32 * q;
          x[q] = s < na ? __ldcg(reinterpret_cast<const float2*>(ml + (size_t)s * G * 2)) : make_float2(-INFINITY, 0.f);
        }
        const float M = warp_max(fmaxf(x[0].x, x[1].x));
        const float w0 = __expf(x[0].x - M), w1 = __expf(x[1].x - M);
        const float Lsum = warp_sum(x[0].y * w0 + x[1].y * w1);
        const float inv = Lsum > 0.f ? __fdividef(1.0f, Lsum) : 0.f;
        float* wd = wsp + ((size_t)col * heads + hh) * kStMaxSplits;
        wd[lane] = w0 * inv;
        wd[lane + 32] = w1 * inv;
      }
      __syncthreads();
      if (lead) {
#pragma unroll 1
        for (int i = c4; i < k4; i += T) {
          const int hh = (4 * i) >> g.hd_log2;
          const float* wd = wsp + ((size_t)col * heads + hh) * kStMaxSplits;
          const float* p = i == c4 ? p0 : g.part_o + (head_base(hh) << g.hd_log2) + ((4 * i) & (hd - 1));
          float4 s4 = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
          for (int u = 0; u < kAhead; ++u) {
            const int s = sgi + u * sg;
            if (s < na) {
              const float4 o = i == c4 ? pre[u] : st_ld4(p + s * sstride);
              const float w = wd[s];
              s4.x += w * o.x; s4.y += w * o.y; s4.z += w * o.z; s4.w += w * o.w;
            }
          }
#pragma unroll 2
          for (int s = sgi + kAhead * sg; s < na; s += sg) {
            const float4 o = st_ld4(p + s * sstride);
            const float w = wd[s];
            s4.x += w * o.x; s4.y += w * o.y; s4.z += w * o.z; s4.w += w * o.w;
          }
          *reinterpret_cast<float4*>(part + ((size_t)sgi * ncols + col) * K + 4 * i) = s4;
        }
      }
      __syncthreads();
#pragma unroll
      for (int u = 0; u < NV; ++u) {
        v[u] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (vi[u] >= 0)
#pragma unroll 2
          for (int q = 0; q < sg; ++q) {
            const float4 o = *reinterpret_cast<const float4*>(part + ((size_t)q * ncols + col) * K + 4 * vi[u]);
            v[u].x += o.x; v[u].y += o.y; v[u].z += o.z; v[u].w += o.w;
          }
      }
    }
#pragma unroll
    for (int u = 0; u < NV; ++u) m = fmaxf(m, st_absmax(v[u]));
    m = st_warp_absmax(m);
    if (lane == 0) scratch[warp] = m;
    __syncthreads();
    m = st_max_row<W>(scratch + col * W);
  }
  if constexpr (PRO != kStCombineShort) {
    const float k = m > 0.f ? __fdividef(127.0f, m) * 0.9999999f : 0.f;    // never above 127, whatever the quotient's last bit
    if (tl == 0 && colok) colscale[col] = k > 0.f ? __fdividef(post, k) : 0.f;
#pragma unroll
    for (int u = 0; u < NV; ++u)
      if (vi[u] >= 0) st_quantize4(make_float4(v[u].x * k, v[u].y * k, v[u].z * k, v[u].w * k), nterms, q0, 4 * vi[u], xstride);
  }
  __syncthreads();
  st_stamp(a, g.bar, 2);

  // ---- tiles
  const int gr = lane >> 2, tq = lane & 3, nq = ncols * nterms;
  const bool xok = gr < nq;
  const uint4* bp = reinterpret_cast<const uint4*>(xq + (size_t)(xok ? gr : 0) * xstride + tq * 16);
  float bv[CP];
  int bi[CP];
#pragma unroll
  for (int c = 0; c < CP; ++c) { bv[c] = -INFINITY; bi[c] = 0x7fffffff; }
  int cs = 0, par = 0;
  bool ok = true;
#pragma unroll 1
  for (int round = 0; round * g.round_tiles < ntile; ++round) {
    const int tb = round * g.round_tiles, nt = min(g.round_tiles, ntile - tb);
    if (STREAM && round > 0) { cc.round = round; start_round(cc); }
    int acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0;
    const uint32_t msk = 0xF0F0F0F0u;         // high nibble of every byte = 16 * q as int8
    auto tile_mma = [&](int (&c0)[4], int (&c1)[4], const uint4& w, const uint4& b) {
      mma_s8s8(c0, (w.x << 4) & msk, w.x & msk, (w.y << 4) & msk, w.y & msk, b.x, b.y);
      mma_s8s8(c1, (w.z << 4) & msk, w.z & msk, (w.w << 4) & msk, w.w & msk, b.z, b.w);
    };
#pragma unroll 1
    while (cc.left > 0) {
      int n = STREAM ? min(slot_tiles, cc.left) : cc.left;
      // A lane whose wait gave up goes on with what is there: the products are the whole warp's, and lanes that left would be
      // waited for.  It asks for nothing more.  (256 steps of the 1B model: 130.9 ms when they left, 131.5 so, 132.1 with a vote.)
      ok = mbar_wait(&bars[cs], par, err) && ok;
      const uint4* wt = reinterpret_cast<const uint4*>(wring + (size_t)cs * slot_tiles * 512) + lane;
      cc.left -= n;
#pragma unroll 1
      while (n > 0) {
        const int len = min(n, KTs - cc.kt);
        const uint4* xb = bp + cc.kt * 4;
        const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
        int j = 0;
#pragma unroll 1
        for (; j + 1 < len; j += 2) {
          const uint4 w0 = wt[j * 32], w1 = wt[j * 32 + 32];
          const uint4 b0 = xok ? xb[j * 4] : zero, b1 = xok ? xb[j * 4 + 4] : zero;
          tile_mma(acc[0], acc[1], w0, b0);
          tile_mma(acc[2], acc[3], w1, b1);
        }
        if (j < len) tile_mma(acc[0], acc[1], wt[j * 32], xok ? xb[j * 4] : zero);
        wt += len * 32;
        n -= len;
        cc.kt += len;
        if (cc.kt == KTs || (n == 0 && cc.left == 0)) {    // the run leaves this row tile: its sums join the tile's
          int* rd = red + (size_t)(cc.tile - tb) * 16 * kQCols + gr * kQCols + 2 * tq;
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            if (2 * tq < nq) atomicAdd(rd + 8 * h * kQCols, (acc[0][2 * h] + acc[1][2 * h]) + (acc[2][2 * h] + acc[3][2 * h]));
            if (2 * tq + 1 < nq) atomicAdd(rd + 8 * h * kQCols + 1, (acc[0][2 * h + 1] + acc[1][2 * h + 1]) + (acc[2][2 * h + 1] + acc[3][2 * h + 1]));
          }
#pragma unroll
          for (int i = 0; i < 4; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0;
          if (cc.kt == KTs) { cc.kt = 0; ++cc.tile; }
        }
      }
      if (STREAM) {
        __syncwarp();
        if (ok) issue();                       // the slot just read is the next to fill
        if (++cs == nslots) { cs = 0; par ^= 1; }
      }
    }
    __syncthreads();
    st_stamp(a, g.bar, 3);
    // ---- values: terms, column scale; weights entered the MMA as 16 * q
    auto value = [&](int row, int c) {         // row counted from the round's first tile
      const int* r = red + (size_t)row * kQCols + c * nterms;
      float x = (float)r[0] + (float)r[1] * (1.0f / 128.0f);
      if (nterms > 2) x += (float)r[2] * (1.0f / 16384.0f);
      return x * (colscale[c] * (1.0f / 16.0f));
    };
    const int rows = nt * 16, base = (t0 + tb) * 16;
    if constexpr (EPI == kStGeglu) {
      const int n = rows / 2;
#pragma unroll
      for (int c = 0; c < CP; ++c)
        if (c < ncols)
#pragma unroll 1
          for (int f = threadIdx.x; f < n; f += kStThreads) {
            const int row = (f >> 4) * 32 + (f & 15);
            const bool first = round == 0 && f < kStThreads;
            const float s0 = first ? wsc[0] : __ldg(g.wscale + base + row), s1 = first ? wsc[1] : __ldg(g.wscale + base + row + 16);
            g.y[(size_t)c * (g.tiles * 8) + base / 2 + f] = gelu_tanh(value(row, c) * s0) * (value(row + 16, c) * s1);
          }
    } else {
#pragma unroll
      for (int c = 0; c < CP; ++c)
        if (c < ncols)
#pragma unroll 1
          for (int row = threadIdx.x; row < rows; row += kStThreads) {
            const float x = value(row, c) * (round == 0 && row < kStThreads ? wsc[0] : __ldg(g.wscale + base + row));
            g.y[((size_t)slice * ncols + c) * (g.tiles * 16) + base + row] = x;
            if (EPI == kStHead && (x > bv[c] || (x == bv[c] && base + row < bi[c]))) { bv[c] = x; bi[c] = base + row; }
          }
    }
    if ((round + 1) * g.round_tiles < ntile) {
      __syncthreads();
#pragma unroll 1
      for (int i = threadIdx.x; i < g.round_tiles * 16 * kQCols; i += kStThreads) red[i] = 0;
      __syncthreads();
    }
  }
  if constexpr (EPI == kStHead) {
    // ---- arg-max (lowest index wins ties): CTA candidate, then the last CTA to arrive picks the token
    float* sv = scratch + 64 + 2 * kMaxCols;                              // [ncols][warps]
    int* si = reinterpret_cast<int*>(sv + kStWarps * kMaxCols);
    auto better = [](float& v, int& i, float ov, int oi) {
      if (ov > v || (ov == v && oi < i)) { v = ov; i = oi; }
    };
#pragma unroll
    for (int c = 0; c < CP; ++c) {
      if (c < ncols) {
        float v = bv[c];
        int ix = bi[c];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          const float ov = __shfl_xor_sync(0xffffffffu, v, o);
          const int oi = __shfl_xor_sync(0xffffffffu, ix, o);
          better(v, ix, ov, oi);
        }
        if (lane == 0) { sv[c * kStWarps + warp] = v; si[c * kStWarps + warp] = ix; }
      }
    }
    __syncthreads();
    if (warp == 0) {
#pragma unroll 1
      for (int c = 0; c < ncols; ++c) {
        float v = lane < kStWarps ? sv[c * kStWarps + lane] : -INFINITY;
        int ix = lane < kStWarps ? si[c * kStWarps + lane] : 0x7fffffff;
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) {
          const float ov = __shfl_xor_sync(0xffffffffu, v, o);
          const int oi = __shfl_xor_sync(0xffffffffu, ix, o);
          better(v, ix, ov, oi);
        }
        if (lane == 0) {
          a.amax_val[(size_t)blockIdx.x * ncols + c] = v;
          a.amax_idx[(size_t)blockIdx.x * ncols + c] = ix;
        }
      }
      int last = 0;
      if (lane == 0) {
        __threadfence();
        last = atomicAdd(g.ticket, 1) == (int)gridDim.x - 1;
        if (last) { *g.ticket = 0; __threadfence(); }
      }
      if (__shfl_sync(0xffffffffu, last, 0)) {
        const int sd = __ldcg(&a.st->steps_done);
#pragma unroll 1
        for (int c = 0; c < ncols; ++c) {
          float v = -INFINITY;
          int ix = 0x7fffffff;
#pragma unroll 1
          for (int b = lane; b < (int)gridDim.x; b += 32)
            better(v, ix, __ldcg(a.amax_val + (size_t)b * ncols + c), __ldcg(a.amax_idx + (size_t)b * ncols + c));
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, v, o);
            const int oi = __shfl_xor_sync(0xffffffffu, ix, o);
            better(v, ix, ov, oi);
          }
          if (lane == 0) {
            if (ix == 0x7fffffff) ix = 0;
            a.st->out_token[c] = ix;
            if (a.step_tokens && sd < a.step_capacity) a.step_tokens[(size_t)sd * ncols + c] = ix;
            a.st->token[c] = ix;
            a.st->pos[c] = __ldcg(&a.st->pos[c]) + 1;
          }
        }
        if (lane == 0) a.st->steps_done = sd + 1;
      }
    }
  }
  st_stamp(a, g.bar, 4);
  if (!ok) {                                   // a wait gave up: let the bulk copies in flight land before the CTA retires
#pragma unroll 1
    for (int i = 0; i < 2000; ++i) __nanosleep(100);
  }
}

// Attention of one (session, kv head, key split): the split's cached rows arrive by bulk copies issued before the wait
// on the QKV projection, in rounds of kStKeys keys over `nbuf` buffers; the step's own key joins the last split in
// shared memory and is appended to the cache by it.  A round is: scores (a warp takes four keys, the G * 4 sums of a
// warp fold together), softmax (one warp per head, one lane per key), P V (two elements and a share of the keys per
// thread).
struct StepAttn {
  const float* qkv;           // [ncols][nqkv]
  const float *g_q, *g_k;
  const float *cosT, *sinT;
  LayerKv kv;
  int is_global, nsplit, nbuf;
  float *part_o, *part_ml;    // [ncols][hkv][nsplit][G][hd], [..][2]
  int bar;
};

template <typename T, int HD>
__host__ __device__ constexpr int st_kv_bytes() { return 2 * kStKeys * HD * (int)sizeof(T); }    // one buffer: K rows, V rows
template <typename T, int HD, int G>
__host__ __device__ constexpr int st_attn_smem(int nbuf) {
  return nbuf * st_kv_bytes<T, HD>() + ((G + 2) * HD + kStKeys * G + 4 * G + 2 * kAtThreads * G) * 4 + 64 + 128;
}

template <typename T, int HD, int G>
__global__ void __launch_bounds__(kAtThreads, 2)
step_attn_kernel(const __grid_constant__ DecodeArgs a, const __grid_constant__ StepAttn g) {
  constexpr int half = HD / 2, VEC = HD / 32, PARTS = kAtThreads / half;      // key shares of the P V stage
  extern __shared__ __align__(128) unsigned char st_sm[];
  const ModelDims& dm = a.dims;
  const int warp = warp_index(), lane = threadIdx.x & 31;
  unsigned char* kvbuf = st_sm;
  float* q_s = reinterpret_cast<float*>(st_sm + (size_t)g.nbuf * st_kv_bytes<T, HD>());   // [G][HD], scaled by 1/sqrt(HD)
  float* k_s = q_s + G * HD;
  float* v_s = k_s + HD;
  float* sc = v_s + HD;                        // [kStKeys][G] scores, then probabilities
  float* cr = sc + kStKeys * G;                // [G] factor of the sums of earlier rounds, [G] running max, [G] running sum
  float* ored = cr + 4 * G;                    // [PARTS][G][HD]
  uint64_t* bars = reinterpret_cast<uint64_t*>(ored + 2 * kAtThreads * G);          // [nbuf]
  int* err = &a.st->err;
  st_stamp(a, g.bar, 0);
  const int split = blockIdx.x % g.nsplit, kvh = (blockIdx.x / g.nsplit) % dm.hkv, col = blockIdx.x / (g.nsplit * dm.hkv);
  int pos = __ldcg(&a.st->pos[col]);
  if (pos < 0 || pos >= dm.max_ctx) {
    if (threadIdx.x == 0) atomicExch(err, (int)kDevBadPosition);
    pos = 0;
  }
  const int* ptab = a.page_table + (size_t)col * a.pages_per_seq;
  const int nkeys = st_visible(dm, pos, g.is_global), lo = pos + 1 - nkeys, chunk = st_chunk(nkeys, g.nsplit);
  const int k0 = lo + split * chunk, k1 = min(k0 + chunk, pos + 1);
  if (k0 >= k1) {                              // no keys for this split: the combine does not read it
    pdl_wait();
    pdl_launch_dependents();
    return;
  }
  const bool has_new = k1 == pos + 1;
  const int k1c = has_new ? pos : k1;          // cached keys [k0, k1c)
  const int nrounds = (k1 - k0 + kStKeys - 1) / kStKeys;
  auto issue = [&](int r) {                    // one thread
    const int b = r % g.nbuf, ka = k0 + r * kStKeys, n = min(kStKeys, k1c - ka);
    if (n <= 0) { mbar_arrive(&bars[b]); return; }
    constexpr uint32_t rowb = HD * sizeof(T);
    unsigned char* dst = kvbuf + (size_t)b * st_kv_bytes<T, HD>();
    mbar_arrive_expect_tx(&bars[b], 2u * (uint32_t)n * rowb);
#pragma unroll 1
    for (int done = 0; done < n;) {            // rows of one page are contiguous
      const int key = ka + done, len = min(n - done, kPage - key % kPage);
      const size_t off = (((size_t)__ldg(ptab + key / kPage) * dm.hkv + kvh) * kPage + key % kPage) * rowb;
      bulk_load_1d(dst + (size_t)done * rowb, reinterpret_cast<const unsigned char*>(g.kv.k) + off, (uint32_t)len * rowb, &bars[b]);
      bulk_load_1d(dst + (size_t)(kStKeys + done) * rowb, reinterpret_cast<const unsigned char*>(g.kv.v) + off, (uint32_t)len * rowb, &bars[b]);
      done += len;
    }
  };
  if (warp == 0 && elect_one()) {
#pragma unroll 1
    for (int b = 0; b < g.nbuf; ++b) mbar_init(&bars[b], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
#pragma unroll 1
    for (int r = 0; r < min(g.nbuf, nrounds); ++r) issue(r);
  }
  // ---- q heads and k head: a warp per head, gains and RoPE rows requested before the wait
  float v[VEC], ga[VEC], cs[(VEC + 1) / 2], sn[(VEC + 1) / 2];
  if (warp <= G) {
    const float* gain = warp < G ? g.g_q : g.g_k;
#pragma unroll
    for (int i = 0; i < VEC; ++i) ga[i] = __ldg(gain + lane + 32 * i);
#pragma unroll
    for (int i = 0; i < (VEC + 1) / 2; ++i) {  // HD 32: the pair of element e sits 16 lanes away
      const int e = HD == 32 ? lane & 15 : lane + 32 * i;
      cs[i] = __ldg(g.cosT + (size_t)pos * half + e);
      sn[i] = __ldg(g.sinT + (size_t)pos * half + e);
    }
  }
  pdl_wait();
  pdl_launch_dependents();
  st_stamp(a, g.bar, 1);
  const float* row = g.qkv + (size_t)col * dm.nqkv();
  if (warp < G + 2) {
    if (warp <= G ? warp < G || has_new : has_new) {
      const float* src = row + (warp < G ? (kvh * G + warp) * HD : dm.nq() + (warp == G ? 0 : dm.nkv()) + kvh * HD);
      float ss = 0.f;
#pragma unroll
      for (int i = 0; i < VEC; ++i) v[i] = __ldcg(src + lane + 32 * i);
      if (warp <= G) {
#pragma unroll
        for (int i = 0; i < VEC; ++i) ss += v[i] * v[i];
        ss = warp_sum(ss);
        const float r = rsqrtf(ss / (float)HD + dm.eps), post = warp < G ? rsqrtf((float)HD) : 1.0f;
        float* dst = q_s + warp * HD;          // k_s follows the q heads
        if constexpr (HD == 32) {
          const float x = v[0] * r * ga[0], y = __shfl_xor_sync(0xffffffffu, x, 16);
          dst[lane] = (lane < 16 ? x * cs[0] - y * sn[0] : x * cs[0] + y * sn[0]) * post;
        } else {
#pragma unroll
          for (int i = 0; i < VEC / 2; ++i) {
            const float a0 = v[i] * r * ga[i], b0 = v[i + VEC / 2] * r * ga[i + VEC / 2];
            dst[lane + 32 * i] = (a0 * cs[i] - b0 * sn[i]) * post;
            dst[lane + 32 * i + half] = (b0 * cs[i] + a0 * sn[i]) * post;
          }
        }
      } else {
#pragma unroll
        for (int i = 0; i < VEC; ++i) v_s[lane + 32 * i] = v[i];
      }
    }
  }
  if (threadIdx.x < G) { cr[G + threadIdx.x] = -INFINITY; cr[2 * G + threadIdx.x] = 0.f; }
  __syncthreads();
  st_stamp(a, g.bar, 2);
  float q[G][VEC];
#pragma unroll
  for (int h = 0; h < G; ++h)
#pragma unroll
    for (int c = 0; c < VEC; ++c) q[h][c] = q_s[h * HD + head_elem<HD>(lane, c)];
  const int e2 = 2 * (threadIdx.x % half), part = threadIdx.x / half;
  float o[G][2];
#pragma unroll
  for (int h = 0; h < G; ++h) o[h][0] = o[h][1] = 0.f;
  auto append = [&](int first, int step) {
    T* kbase = reinterpret_cast<T*>(g.kv.k);
    T* vbase = reinterpret_cast<T*>(g.kv.v);
    const int page = ptab[pos / kPage], slot = pos % kPage;
    const size_t off = (((size_t)page * dm.hkv + kvh) * kPage + slot) * HD;
#pragma unroll 1
    for (int e = first; e < HD; e += step) {
      if constexpr (sizeof(T) == 4) {
        kbase[off + e] = k_s[e];
        vbase[off + e] = v_s[e];
        if (g.kv.k16) g.kv.k16[off + e] = __float2bfloat16(k_s[e]);
      } else {
        kbase[off + e] = __float2bfloat16(k_s[e]);
        vbase[off + e] = __float2bfloat16(v_s[e]);
      }
      if (g.kv.v16) g.kv.v16[(((size_t)page * dm.hkv + kvh) * HD + e) * kPage + slot] = __float2bfloat16(v_s[e]);
    }
    asm volatile("fence.proxy.async.global;" ::: "memory");     // later steps fetch these rows with bulk copies
  };
  bool ok = true;
#pragma unroll 1
  for (int r = 0; r < nrounds; ++r) {
    const int b = r % g.nbuf, ka = k0 + r * kStKeys, n = min(kStKeys, k1 - ka);
    T* ks = reinterpret_cast<T*>(kvbuf + (size_t)b * st_kv_bytes<T, HD>());
    T* vs = ks + kStKeys * HD;
    ok = mbar_wait(&bars[b], (r / g.nbuf) & 1, err) && ok;
    if (has_new && r == nrounds - 1) {         // the step's own rows, as the cache will hand them back
#pragma unroll 1
      for (int e = threadIdx.x; e < HD; e += kAtThreads) {
        if constexpr (sizeof(T) == 4) { ks[(n - 1) * HD + e] = k_s[e]; vs[(n - 1) * HD + e] = v_s[e]; }
        else { ks[(n - 1) * HD + e] = __float2bfloat16(k_s[e]); vs[(n - 1) * HD + e] = __float2bfloat16(v_s[e]); }
      }
      __syncthreads();
    }
    // ---- scores of keys 4 * warp .. + 3: the 4 G sums of the warp fold together, each exchange halving what a lane carries
    if (4 * warp < n) {
      constexpr int NK = 4, NSUM = NK * G;
      float s[NSUM];
#pragma unroll
      for (int j = 0; j < NK; ++j) {
        float x[VEC];
        load_head_row_smem<T, HD>(ks + (size_t)min(NK * warp + j, n - 1) * HD, lane, x);
#pragma unroll
        for (int h = 0; h < G; ++h) {
          float d = 0.f;
#pragma unroll
          for (int c = 0; c < VEC; ++c) d += q[h][c] * x[c];
          s[j * G + h] = d;
        }
      }
#pragma unroll
      for (int w = NSUM / 2, bit = 16; w >= 1; w /= 2, bit /= 2) {
        const bool up = lane & bit;
#pragma unroll
        for (int i = 0; i < w; ++i) {
          const float give = up ? s[i] : s[i + w], keep = up ? s[i + w] : s[i];
          s[i] = keep + __shfl_xor_sync(0xffffffffu, give, bit);
        }
      }
#pragma unroll
      for (int bit = 16 / NSUM; bit >= 1; bit /= 2) s[0] += __shfl_xor_sync(0xffffffffu, s[0], bit);
      if (lane % (32 / NSUM) == 0) {
        const int i = lane / (32 / NSUM), key = NK * warp + i / G;     // value i: key i / G, head i % G
        if (key < n) sc[key * G + i % G] = s[0];
      }
    }
    __syncthreads();
    // ---- softmax: warp = head, lane = key
    if (warp < G) {
      const float s = lane < n ? sc[lane * G + warp] : -INFINITY;
      const float m0 = cr[G + warp], m1 = fmaxf(m0, warp_max(s)), f = __expf(m0 - m1);
      const float p = __expf(s - m1), ps = warp_sum(p);
      if (lane < n) sc[lane * G + warp] = p;
      __syncwarp();
      if (lane == 0) { cr[warp] = f; cr[G + warp] = m1; cr[2 * G + warp] = cr[2 * G + warp] * f + ps; }
    } else if (has_new && r == 0) {            // the other warps append meanwhile: at the end, the stores held up the kernel's completion
      append(threadIdx.x - 32 * G, kAtThreads - 32 * G);
    }
    __syncthreads();
    // ---- P V: elements e2, e2 + 1, keys part, part + PARTS, ...
#pragma unroll
    for (int h = 0; h < G; ++h) { o[h][0] *= cr[h]; o[h][1] *= cr[h]; }
#pragma unroll 4
    for (int kk = part; kk < n; kk += PARTS) {
      float x0, x1;
      if constexpr (sizeof(T) == 4) {
        const float2 x = *reinterpret_cast<const float2*>(vs + (size_t)kk * HD + e2);
        x0 = x.x; x1 = x.y;
      } else {
        const __nv_bfloat162 x = *reinterpret_cast<const __nv_bfloat162*>(vs + (size_t)kk * HD + e2);
        x0 = __low2float(x); x1 = __high2float(x);
      }
      float p[G];
      ld_vec<G>(sc + kk * G, p);
#pragma unroll
      for (int h = 0; h < G; ++h) {
        o[h][0] += p[h] * x0;
        o[h][1] += p[h] * x1;
      }
    }
    if (r + 1 < nrounds) {
      __syncthreads();                         // everyone is done with the buffer, the probabilities and cr
      if (warp == 0 && r + g.nbuf < nrounds && elect_one()) issue(r + g.nbuf);
    }
  }
  // ---- the key shares meet, the split's state goes out
  st_stamp(a, g.bar, 3);
#pragma unroll
  for (int h = 0; h < G; ++h) *reinterpret_cast<float2*>(ored + ((size_t)part * G + h) * HD + e2) = make_float2(o[h][0], o[h][1]);
  __syncthreads();
  const size_t pi = (((size_t)col * dm.hkv + kvh) * g.nsplit + split) * G;
#pragma unroll 1
  for (int i = threadIdx.x; i < G * HD; i += kAtThreads) {
    float s = 0.f;
#pragma unroll
    for (int p = 0; p < PARTS; ++p) s += ored[(size_t)p * G * HD + i];
    g.part_o[pi * HD + i] = s;
  }
  if (threadIdx.x < G) {
    g.part_ml[(pi + threadIdx.x) * 2] = cr[G + threadIdx.x];
    g.part_ml[(pi + threadIdx.x) * 2 + 1] = cr[2 * G + threadIdx.x];
  }
  st_stamp(a, g.bar, 4);
  if (!ok)
#pragma unroll 1
    for (int i = 0; i < 2000; ++i) __nanosleep(100);
}

// ------------------------------------------------------------------ host side

// Everything a step's launches need for one executor: K splits, key splits and scratch.
struct StepPlan {
  int sms = 0, max_splits = 0;
  size_t smem_optin = 0;
  int o_slices = 1, down_slices = 1;
  int nsplit[2] = {1, 1};                      // key splits of local and global layers
  int keys[2] = {1, 1};                        // keys they can hold at most
  float *part_o = nullptr, *part_ml = nullptr;      // attention partials
  float *opart = nullptr, *fpart = nullptr;         // [slices][ncols][d]
  int* ticket = nullptr;
};

// Called around each collective of tensor parallelism; null otherwise.
typedef void (*StepReduceFn)(void* ctx, float* buf, size_t count);

// Fills in the splits; false when the model's geometry does not fit the kernels.
bool step_plan(const ModelDims& d, int sms, size_t smem_optin, int max_tokens, StepPlan* pl);
// Raises the kernels' shared-memory limits (outside any capture); false when a projection of a.ncols sessions does not
// fit: a vector longer than twelve float4 per thread, or too long for shared memory.
bool step_prepare(const DecodeArgs& a, const StepPlan& pl, const LayerWeights* layers, const LayerKv* kv);
// Queues one step of a.ncols sessions; returns the number of launches.
int step_launch(cudaStream_t st, const DecodeArgs& a, const StepPlan& pl, const LayerWeights* layers, const LayerKv* kv, StepReduceFn reduce,
                void* reduce_ctx);

}  // namespace b200lm

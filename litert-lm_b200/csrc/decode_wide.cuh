// Wide lockstep decode: one greedy step for MANY sessions at once, with the projections on the
// tensor-core int4 GEMM of the prefill path (the sessions' current tokens are the GEMM's token rows)
// and attention CTAs per (session, kv head, key split) over that session's own pages.  The weights stream
// once per step for the whole group, which is what a group of more sessions than the GEMV kernels
// carry (kMaxCols) needs.  Activations are bf16 as in prefill.
//
// This file holds the two kernels the step adds to the prefill kernels, its attention and its arg-max; the
// step itself is Executor::wide_step.
#pragma once
#include <algorithm>
#include "decode_ops.cuh"
#include "prefill_ops.cuh"

namespace b200lm {

constexpr int kWideMax = 128;          // sessions of one wide step (half a token tile of the GEMM)
constexpr int kWideArgThreads = 1024;
constexpr int kWideMaxSplits = 16;    // key splits of one (session, kv head) in the wide attention

// Per-session state of a wide run, device resident: [0, n) token of the next step, [kWideMax, +n)
// its position, [2 kWideMax, +n) the position of the run's first step.
struct WideState {
  int* tok;
  int* pos;
  int* pos0;
  float* part_val;            // arg-max of the parts of a row
  int* part_idx;
  int* ticket;                // parts of a row that are done; zero between launches
};

// Arg-max of the sessions' logits rows (lowest index among equal maxima, the rule of
// runtime/components/sampling_cpu_util.cc:32-41), recorded as the step's id and as the next input.  `parts` CTAs share
// a row, so that a few rows (9 rows of 1 MB took one CTA each 17.4 us) draw on the whole chip; the last one to finish
// joins them, and equal maxima go by index whatever the order.
constexpr int kWideArgParts = 16;
static __global__ void __launch_bounds__(kWideArgThreads)
wide_argmax_kernel(const float* __restrict__ logits, int vocab, int n, int parts, WideState st, int* __restrict__ step_tokens) {
  __shared__ float sv[kWideArgThreads / 32];
  __shared__ int si[kWideArgThreads / 32];
  pdl_wait();
  pdl_launch_dependents();
  const int row = blockIdx.x / parts, part = blockIdx.x % parts, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const float4* src = reinterpret_cast<const float4*>(logits + (size_t)row * vocab);
  float bv = -INFINITY;
  int bi = 0x7fffffff;
  const int v4 = vocab / 4, per = (v4 + parts - 1) / parts, beg = min(v4, part * per), end = min(v4, beg + per);
#pragma unroll 4
  for (int i = beg + threadIdx.x; i < end; i += kWideArgThreads) {     // ascending per thread: > keeps the first
    const float4 v = __ldcs(src + i);
    if (v.x > bv) { bv = v.x; bi = 4 * i; }
    if (v.y > bv) { bv = v.y; bi = 4 * i + 1; }
    if (v.z > bv) { bv = v.z; bi = 4 * i + 2; }
    if (v.w > bv) { bv = v.w; bi = 4 * i + 3; }
  }
  if (part == parts - 1)
    for (int i = v4 * 4 + threadIdx.x; i < vocab; i += kWideArgThreads) {
      const float v = logits[(size_t)row * vocab + i];
      if (v > bv) { bv = v; bi = i; }
    }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
    const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
    if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
  }
  if (lane == 0) { sv[warp] = bv; si[warp] = bi; }
  __syncthreads();
  if (warp == 0) {
    bv = lane < kWideArgThreads / 32 ? sv[lane] : -INFINITY;
    bi = lane < kWideArgThreads / 32 ? si[lane] : 0x7fffffff;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
    }
    if (parts > 1) {
      float* pv = st.part_val + (size_t)row * kWideArgParts;
      int* pi = st.part_idx + (size_t)row * kWideArgParts;
      int last = 0;
      if (lane == 0) {
        pv[part] = bv;
        pi[part] = bi;
        __threadfence();
        last = atomicAdd(st.ticket + row, 1) == parts - 1;
        if (last) st.ticket[row] = 0;
        __threadfence();
      }
      if (!__shfl_sync(0xffffffffu, last, 0)) return;
      bv = lane < parts ? __ldcg(pv + lane) : -INFINITY;
      bi = lane < parts ? __ldcg(pi + lane) : 0x7fffffff;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
      }
    }
    if (lane == 0) {
      if (bi == 0x7fffffff) bi = 0;                 // a row of NaNs: id 0, as the host path casts
      const int p = st.pos[row];
      step_tokens[(size_t)(p - st.pos0[row]) * n + row] = bi;
      st.tok[row] = bi;
      st.pos[row] = p + 1;
    }
  }
}

// ------------------------------------------------------------------ attention of a wide step
// One CTA per (session, kv head, key split).  The session's K / V rows of this head are contiguous inside a page
// ([page][kv head][slot][hd]), so a round's 16 or 32 keys are one or two bulk copies each for K and V, into a ring of
// rounds that is requested ahead of griddepcontrol.wait.  Scores: a warp takes 2 or 4 keys of the round for all G query
// heads, and the sums fold together, each exchange halving what a lane carries.  Softmax: a warp per head, a lane per
// key.  P V: a thread per pair of elements.  So a round has one chain of exchanges and exponentials, where a warp that
// owned its keys had one per key (9 sessions x 530 keys of 256 fp32: 17.5 us a layer and 6.1 for a kernel of its own
// that joined the splits).  The last CTA of a (session, kv head) to finish joins the splits, in split order.  The CTA
// whose keys end at the current position norms, rotates and appends the step's own K / V row.
constexpr int kWaThreads = 256, kWaWarps = 8, kWaMaxStages = 6;
// Keys of a round: 32 KB a stage for the largest rows, so that two CTAs of an SM hold three stages each.
template <typename T, int HD>
__host__ __device__ constexpr int wa_keys() { return HD * (int)sizeof(T) >= 1024 ? 16 : 32; }

struct WideAttnArgs {
  const float* qkv;          // [sessions][nqkv] raw projections of this step
  const int* pos;            // [sessions] position of this step's token
  const int* page_table;     // first session's row; rows of pages_per_seq entries
  int pages_per_seq;
  int is_global;
  int nsplit;
  int stages;                // ring depth (2 .. kWaMaxStages), sized by the host to the shared memory
  const float *g_q, *g_k, *cosT, *sinT;
  LayerKv kv;
  float* part;               // nsplit > 1: [session][kv head] partial states, nsplit * G * (hd + 4) floats each (16-byte rows)
  int* ticket;               // nsplit > 1: [session][kv head], zero before and after
  __nv_bfloat16* out;        // [session][hq * hd], optional
  int* err;
  int seq_stride;            // 1: session i has row i of the page table; 0: every query reads sequence 0
  int appended;              // 1: q rows are final (no norm, no rotation) and every K / V row is already in the cache
  float* out_f32;            // the same output in fp32 (operator-level callers), optional
  int ctas_per_sm;           // host-side hint: size the ring so that this many CTAs fit one SM (0 = 1)
  int qkv_parts;             // > 1: qkv is that many split-K partials, qkv_part_stride floats apart, summed on load
  size_t qkv_part_stride;
};

template <typename T, int HD>
__host__ __device__ constexpr int wa_stage_bytes() { return 2 * wa_keys<T, HD>() * HD * (int)sizeof(T); }
__host__ __device__ inline size_t wa_fixed_bytes(int hd, int G) {
  return sizeof(float) * ((size_t)(G + 2) * hd + 32 * G + 4 * G + 2 * kWaThreads * G) + 8 * kWaMaxStages + 128;
}

template <typename T, int HD, int G>
__global__ void __launch_bounds__(kWaThreads, 2)
wide_attn_kernel(ModelDims dm, WideAttnArgs a) {
  constexpr int VEC = HD / 32, half = HD / 2, KEYS = wa_keys<T, HD>(), PARTS = kWaThreads / half;   // PARTS: key shares of P V
  constexpr int kStage = wa_stage_bytes<T, HD>();
  extern __shared__ __align__(128) unsigned char wa_sm[];
  const int S = a.stages;
  float* q_s = reinterpret_cast<float*>(wa_sm + (size_t)S * kStage);   // [G][HD], scaled by 1/sqrt(HD)
  float* k_s = q_s + G * HD;
  float* v_s = k_s + HD;
  float* sc = v_s + HD;                        // [KEYS][G] scores, then probabilities
  float* cr = sc + 32 * G;                     // [G] factor of the sums of earlier rounds, [G] running max, [G] running sum
  float* ored = cr + 4 * G;                    // [PARTS][G][HD]
  uint64_t* full = reinterpret_cast<uint64_t*>(ored + 2 * kWaThreads * G);
  int* last = reinterpret_cast<int*>(full + kWaMaxStages);

  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int split = blockIdx.x % a.nsplit, pair = blockIdx.x / a.nsplit, kvh = pair % dm.hkv, qi = pair / dm.hkv;
  int pos = __ldcg(a.pos + qi);                // written two kernels back or earlier, as the cached rows are
  if (pos < 0 || pos >= dm.max_ctx) {
    if (threadIdx.x == 0) atomicExch(a.err, (int)kDevBadPosition);
    pos = 0;
  }
  const int* ptab = a.page_table + (size_t)(a.seq_stride ? qi : 0) * a.pages_per_seq;
  const T* kbase = reinterpret_cast<const T*>(a.kv.k);
  const T* vbase = reinterpret_cast<const T*>(a.kv.v);
  int k0, k1;
  attn_split_range(dm, pos, a.is_global, a.nsplit, split, &k0, &k1);
  const bool has_new = !a.appended && k1 == pos + 1 && k1 > k0;
  const int k1c = has_new ? pos : k1;          // cached keys [k0, k1c)
  const int nrounds = k1 > k0 ? (k1 - k0 + KEYS - 1) / KEYS : 0;
  auto issue = [&](int r) {                    // one thread
    const int b = r % S, ka = k0 + r * KEYS, n = min(KEYS, k1c - ka);
    if (n <= 0) { mbar_arrive(&full[b]); return; }
    unsigned char* dst = wa_sm + (size_t)b * kStage;
    constexpr uint32_t rowb = HD * sizeof(T);
    mbar_arrive_expect_tx(&full[b], 2u * (uint32_t)n * rowb);
#pragma unroll 1
    for (int done = 0; done < n;) {            // rows of one page are contiguous
      const int key = ka + done, len = min(n - done, kPage - key % kPage);
      const size_t off = (((size_t)__ldg(ptab + key / kPage) * dm.hkv + kvh) * kPage + key % kPage) * HD;
      bulk_load_1d(dst + (size_t)done * rowb, kbase + off, (uint32_t)len * rowb, &full[b]);
      bulk_load_1d(dst + (size_t)(KEYS + done) * rowb, vbase + off, (uint32_t)len * rowb, &full[b]);
      done += len;
    }
  };
  if (warp == 0 && elect_one()) {
#pragma unroll 1
    for (int s = 0; s < S; ++s) mbar_init(&full[s], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
#pragma unroll 1
    for (int r = 0; r < min(S, nrounds); ++r) issue(r);
  }
  // ---- q heads, k head and v head: a warp per head (or two), gains and RoPE rows requested before the wait
  float ga[VEC], cs[(VEC + 1) / 2], sn[(VEC + 1) / 2];
  if (warp <= G && !a.appended) {
    const float* gain = warp < G ? a.g_q : a.g_k;
#pragma unroll
    for (int i = 0; i < VEC; ++i) ga[i] = __ldg(gain + lane + 32 * i);
#pragma unroll
    for (int i = 0; i < (VEC + 1) / 2; ++i) {  // HD 32: the pair of element e sits 16 lanes away
      const int e = HD == 32 ? lane & 15 : lane + 32 * i;
      cs[i] = __ldg(a.cosT + (size_t)pos * half + e);
      sn[i] = __ldg(a.sinT + (size_t)pos * half + e);
    }
  }
  pdl_wait();
  pdl_launch_dependents();
  if (warp < G || (warp < G + 2 && has_new)) {
    const float* src = a.qkv + (size_t)qi * dm.nqkv() + (warp < G ? (kvh * G + warp) * HD : dm.nq() + (warp == G ? 0 : dm.nkv()) + kvh * HD);
    float v[VEC];
#pragma unroll
    for (int i = 0; i < VEC; ++i) v[i] = __ldcg(src + lane + 32 * i);
#pragma unroll 3
    for (int p = 1; p < a.qkv_parts; ++p)      // a projection is the sum of its split-K partials, in order
#pragma unroll
      for (int i = 0; i < VEC; ++i) v[i] += __ldcg(src + p * a.qkv_part_stride + lane + 32 * i);
    float* dst = q_s + warp * HD;              // k_s and v_s follow the q heads
    const float post = warp < G ? rsqrtf((float)HD) : 1.0f;
    if (a.appended || warp > G) {
#pragma unroll
      for (int i = 0; i < VEC; ++i) dst[lane + 32 * i] = v[i] * post;
    } else {
      float ss = 0.f;
#pragma unroll
      for (int i = 0; i < VEC; ++i) ss += v[i] * v[i];
      ss = warp_sum(ss);
      const float r = rsqrtf(ss / (float)HD + dm.eps);
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
    }
  }
  if (threadIdx.x < G) { cr[G + threadIdx.x] = -INFINITY; cr[2 * G + threadIdx.x] = 0.f; }
  __syncthreads();
  if (has_new) {                               // append: exactly one CTA per (session, kv head)
    const int page = ptab[pos / kPage], slot = pos % kPage;
    const size_t off = (((size_t)page * dm.hkv + kvh) * kPage + slot) * HD;
    T* kw = reinterpret_cast<T*>(a.kv.k);
    T* vw = reinterpret_cast<T*>(a.kv.v);
#pragma unroll 1
    for (int e = threadIdx.x; e < HD; e += kWaThreads) {
      if constexpr (sizeof(T) == 4) {
        kw[off + e] = k_s[e];
        vw[off + e] = v_s[e];
        if (a.kv.k16) a.kv.k16[off + e] = __float2bfloat16(k_s[e]);
      } else {
        kw[off + e] = __float2bfloat16(k_s[e]);
        vw[off + e] = __float2bfloat16(v_s[e]);
      }
      if (a.kv.v16) a.kv.v16[(((size_t)page * dm.hkv + kvh) * HD + e) * kPage + slot] = __float2bfloat16(v_s[e]);
    }
    asm volatile("fence.proxy.async.global;" ::: "memory");     // later steps fetch these rows with bulk copies
  }
  float q[G][VEC];
#pragma unroll
  for (int h = 0; h < G; ++h)
#pragma unroll
    for (int c = 0; c < VEC; ++c) q[h][c] = q_s[h * HD + head_elem<HD>(lane, c)];
  const int e2 = 2 * (threadIdx.x % half), share = threadIdx.x / half;
  float o[G][2];
#pragma unroll
  for (int h = 0; h < G; ++h) o[h][0] = o[h][1] = 0.f;
  bool ok = true;
#pragma unroll 1
  for (int r = 0; r < nrounds; ++r) {
    const int b = r % S, n = min(KEYS, k1 - k0 - r * KEYS);
    T* ks = reinterpret_cast<T*>(wa_sm + (size_t)b * kStage);
    T* vs = ks + KEYS * HD;
    ok = mbar_wait(&full[b], (uint32_t)((r / S) & 1), a.err) && ok;
    if (has_new && r == nrounds - 1) {         // the step's own rows, as the cache will hand them back
#pragma unroll 1
      for (int e = threadIdx.x; e < HD; e += kWaThreads) {
        if constexpr (sizeof(T) == 4) { ks[(n - 1) * HD + e] = k_s[e]; vs[(n - 1) * HD + e] = v_s[e]; }
        else { ks[(n - 1) * HD + e] = __float2bfloat16(k_s[e]); vs[(n - 1) * HD + e] = __float2bfloat16(v_s[e]); }
      }
      __syncthreads();
    }
    constexpr int NK = KEYS / kWaWarps, NSUM = NK * G;
    if (NK * warp < n) {
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
    if (warp < G) {                            // softmax: warp = head, lane = key
      const float s = lane < n ? sc[lane * G + warp] : -INFINITY;
      const float m0 = cr[G + warp], m1 = fmaxf(m0, warp_max(s)), f = __expf(m0 - m1);
      const float p = __expf(s - m1), ps = warp_sum(p);
      if (lane < n) sc[lane * G + warp] = p;
      __syncwarp();
      if (lane == 0) { cr[warp] = f; cr[G + warp] = m1; cr[2 * G + warp] = cr[2 * G + warp] * f + ps; }
    }
    __syncthreads();
#pragma unroll
    for (int h = 0; h < G; ++h) { o[h][0] *= cr[h]; o[h][1] *= cr[h]; }
#pragma unroll 4
    for (int kk = share; kk < n; kk += PARTS) {
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
      __syncthreads();                         // everyone is done with the stage, the probabilities and cr
      if (warp == 0 && r + S < nrounds && elect_one()) issue(r + S);
    }
  }
  // ---- the key shares meet
#pragma unroll
  for (int h = 0; h < G; ++h) *reinterpret_cast<float2*>(ored + ((size_t)share * G + h) * HD + e2) = make_float2(o[h][0], o[h][1]);
  __syncthreads();
  // part: [split][G][HD] sums, then [split][G] maxima and [split][G] sums of the probabilities
  constexpr int UNITS = G * HD / 4;
  float* part = a.part + (size_t)pair * a.nsplit * G * (HD + 4);
  float* part_m = part + (size_t)a.nsplit * G * HD;
  float* part_l = part_m + a.nsplit * G;
  auto put = [&](int i, float4 v, float f) {
    v.x *= f; v.y *= f; v.z *= f; v.w *= f;
    const size_t oi = ((size_t)qi * dm.hq + kvh * G) * HD + 4 * i;
    if (a.out) {
      const __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y), hi = __floats2bfloat162_rn(v.z, v.w);
      *reinterpret_cast<uint2*>(a.out + oi) = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
    }
    if (a.out_f32) *reinterpret_cast<float4*>(a.out_f32 + oi) = v;
  };
  for (int i = threadIdx.x; i < UNITS; i += kWaThreads) {
    float4 v = reinterpret_cast<const float4*>(ored)[i];
#pragma unroll
    for (int p = 1; p < PARTS; ++p) {
      const float4 x = reinterpret_cast<const float4*>(ored)[p * UNITS + i];
      v.x += x.x; v.y += x.y; v.z += x.z; v.w += x.w;
    }
    if (a.nsplit > 1) {
      reinterpret_cast<float4*>(part)[split * UNITS + i] = v;
    } else {
      const float L = cr[2 * G + i / (HD / 4)];
      put(i, v, L > 0.f ? 1.0f / L : 0.f);
    }
  }
  if (a.nsplit > 1) {
    if (threadIdx.x < G) { part_m[split * G + threadIdx.x] = cr[G + threadIdx.x]; part_l[split * G + threadIdx.x] = cr[2 * G + threadIdx.x]; }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
      *last = atomicAdd(a.ticket + pair, 1) == a.nsplit - 1;
      if (*last) a.ticket[pair] = 0;
    }
    __syncthreads();
    if (*last) {
      __threadfence();
      if (warp < G) {                          // weights of the splits, two to a lane: kMaxSplits in all
        float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.f, l1 = 0.f;
        if (lane < a.nsplit) { m0 = __ldcg(part_m + lane * G + warp); l0 = __ldcg(part_l + lane * G + warp); }
        if (lane + 32 < a.nsplit) { m1 = __ldcg(part_m + (lane + 32) * G + warp); l1 = __ldcg(part_l + (lane + 32) * G + warp); }
        const float M = warp_max(fmaxf(m0, m1));
        m0 = M > -INFINITY ? __expf(m0 - M) : 0.f;
        m1 = M > -INFINITY ? __expf(m1 - M) : 0.f;
        const float L = warp_sum(l0 * m0 + l1 * m1), inv = L > 0.f ? 1.0f / L : 0.f;
        float* w = ored + warp * kMaxSplits;
        w[lane] = m0 * inv;
        w[lane + 32] = m1 * inv;
      }
      __syncthreads();
      for (int i = threadIdx.x; i < UNITS; i += kWaThreads) {
        const float* w = ored + i / (HD / 4) * kMaxSplits;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
        for (int s = 0; s < a.nsplit; ++s) {
          const float4 x = __ldcg(reinterpret_cast<const float4*>(part) + s * UNITS + i);
          v.x += x.x * w[s]; v.y += x.y * w[s]; v.z += x.z * w[s]; v.w += x.w * w[s];
        }
        put(i, v, 1.0f);
      }
    }
  }
  if (!ok)                                     // a wait gave up: let the bulk copies still in flight land before the CTA retires
#pragma unroll 1
    for (int i = 0; i < 2000; ++i) __nanosleep(100);
}

// Host side: the kernel instantiated for the cache type, head size and group size.  nb <= 0 only sets the
// kernel's shared-memory attributes (executor creation, outside any stream capture).
template <typename T, int HD, int G>
inline void launch_wide_attn_t(cudaStream_t st, const ModelDims& d, int nb, size_t smem_optin, WideAttnArgs a) {
  const size_t fixed = wa_fixed_bytes(HD, G);
  const int stage = wa_stage_bytes<T, HD>();
  // A round is a chain of exchanges, exponentials and barriers: with two CTAs per SM the ring is shallower, but one
  // CTA's chain runs beside the other's.
  int per_sm = std::max(1, a.ctas_per_sm);
  int stages = 0;
  for (; per_sm >= 1; --per_sm) {
    const size_t budget = smem_optin / per_sm - 1024;
    stages = budget > fixed ? (int)std::min<size_t>(kWaMaxStages, (budget - fixed) / stage) : 0;
    if (stages >= 2) break;
  }
  B2_CHECK(stages >= 2, kUnimplemented, "the streaming decode attention does not fit the device's shared memory");
  a.stages = stages;
  const size_t smem = fixed + (size_t)stages * stage;
  raise_dyn_smem(wide_attn_kernel<T, HD, G>, smem);
  if (nb <= 0) { share_memory(wide_attn_kernel<T, HD, G>); return; }
  launch_pdl(wide_attn_kernel<T, HD, G>, dim3(nb * d.hkv * a.nsplit), dim3(kWaThreads), smem, st, d, a);
}
template <typename T, int HD>
inline void launch_wide_attn_g(cudaStream_t st, const ModelDims& d, int nb, size_t smem_optin, const WideAttnArgs& a) {
  switch (d.group()) {
    case 1: launch_wide_attn_t<T, HD, 1>(st, d, nb, smem_optin, a); break;
    case 2: launch_wide_attn_t<T, HD, 2>(st, d, nb, smem_optin, a); break;
    case 4: launch_wide_attn_t<T, HD, 4>(st, d, nb, smem_optin, a); break;
    default: throw Error{kUnimplemented, "query heads per kv head must be 1, 2 or 4"};
  }
}
template <typename T>
inline void launch_wide_attn_h(cudaStream_t st, const ModelDims& d, int nb, size_t smem_optin, const WideAttnArgs& a) {
  switch (d.hd) {
    case 32: launch_wide_attn_g<T, 32>(st, d, nb, smem_optin, a); break;
    case 64: launch_wide_attn_g<T, 64>(st, d, nb, smem_optin, a); break;
    case 128: launch_wide_attn_g<T, 128>(st, d, nb, smem_optin, a); break;
    case 256: launch_wide_attn_g<T, 256>(st, d, nb, smem_optin, a); break;
    default: throw Error{kUnimplemented, "head size must be 32, 64, 128 or 256"};
  }
}
// The kernels of one cache type are a translation unit.
void launch_wide_attn_f32(cudaStream_t st, const ModelDims& d, int nb, size_t smem_optin, const WideAttnArgs& a);
void launch_wide_attn_bf16(cudaStream_t st, const ModelDims& d, int nb, size_t smem_optin, const WideAttnArgs& a);
inline void launch_wide_attn(cudaStream_t st, const ModelDims& d, int nb, size_t smem_optin, const WideAttnArgs& a) {
  if (d.kv_dtype == 0) launch_wide_attn_f32(st, d, nb, smem_optin, a);
  else launch_wide_attn_bf16(st, d, nb, smem_optin, a);
}

}  // namespace b200lm

// Host side of the decode step (decode_step.cuh) and its kernel instantiations.
#include "decode_step.cuh"

namespace b200lm {

bool step_plan(const ModelDims& d, int sms, size_t smem_optin, int max_tokens, StepPlan* pl) {
  const int G = d.group();
  if (d.d % 64 || d.ffn % 64 || d.nq() % 64 || d.nqkv() % 16 || d.vocab % 16 || d.d / 4 > 12 * kStThreads) return false;
  if (G != 1 && G != 2 && G != 4) return false;
  if (d.hd != 32 && d.hd != 64 && d.hd != 128 && d.hd != 256) return false;
  pl->sms = sms;
  pl->smem_optin = smem_optin;
  // K splits (up to four): they cut the vector a CTA has to fetch and quantise, and the next kernel adds the parts.
  // The O projection splits over whole heads.
  for (int s = 4; s >= 1; --s)
    if (d.hq % s == 0 && (d.nq() / s) % 64 == 0) { pl->o_slices = s; break; }
  for (int s = 4; s >= 1; --s)
    if ((d.ffn / 64) % s == 0) { pl->down_slices = s; break; }
  const int keys[2] = {std::min(d.window, max_tokens), max_tokens};
  for (int g = 0; g < 2; ++g) {
    pl->keys[g] = keys[g];
    pl->nsplit[g] = std::max(1, std::min(kStMaxSplits, (keys[g] + kStKeys - 1) / kStKeys));
  }
  pl->max_splits = std::max(pl->nsplit[0], pl->nsplit[1]);
  return true;
}

namespace {

// Shared memory of a projection: two generations of CTAs fit an SM, so that a kernel's first tiles arrive while its
// predecessor still runs; the ring takes what the other areas leave.
constexpr int kStSmemTarget = 112 * 1024;

struct Launch {
  cudaStream_t st;
  bool* fits = nullptr;                        // dry run: raise the shared-memory limits, note what does not fit
  bool pdl = true;
};

template <typename... KArgs, typename... Args>
void go(const Launch& l, void (*kernel)(KArgs...), int grid, int block, size_t smem, Args&&... args) {
  if (l.fits) { raise_dyn_smem(kernel, smem); share_memory(kernel); return; }
  if (l.pdl) launch_pdl(kernel, dim3(grid), dim3(block), smem, l.st, std::forward<Args>(args)...);
  else kernel<<<grid, block, smem, l.st>>>(std::forward<Args>(args)...);
}

template <int PRO, int EPI, int NV, int CP>
void launch_gemv_s(const Launch& l, const DecodeArgs& a, const StepGemv& g) {
  const size_t smem = (size_t)g.sm.total;
  if (g.nslots > 1) go(l, step_gemv_kernel<PRO, EPI, NV, CP, true>, g.slices * g.cps, kStThreads, smem, a, g);
  else go(l, step_gemv_kernel<PRO, EPI, NV, CP, false>, g.slices * g.cps, kStThreads, smem, a, g);
}
template <int PRO, int EPI, int NV>
void launch_gemv_cp(const Launch& l, const DecodeArgs& a, const StepGemv& g) {
  if (st_cols(a.ncols) == 1) launch_gemv_s<PRO, EPI, NV, 1>(l, a, g);
  else if (st_cols(a.ncols) == 2) launch_gemv_s<PRO, EPI, NV, 2>(l, a, g);
  else launch_gemv_s<PRO, EPI, NV, 4>(l, a, g);
}

template <int PRO, int EPI>
void launch_gemv(const Launch& l, const DecodeArgs& a, const StepPlan& pl, StepGemv g) {
  constexpr int unit = EPI == kStGeglu ? 2 : 1;
  const int units = g.tiles / unit;
  g.cps = std::max(1, std::min(pl.sms / g.slices, units));
  g.tile_base = units / g.cps;
  g.tile_rem = units % g.cps;
  const int most = (g.tile_base + (g.tile_rem ? 1 : 0)) * unit;          // row tiles of the busiest CTA
  g.KTs = g.KT / g.slices;
  g.kmax = g.KTs * 64;
  g.xstride = st_xstride(g.kmax);
  g.inv_k = 1.0f / (float)g.kmax;
  g.heads = PRO == kStCombine || PRO == kStCombineShort ? g.kmax / a.dims.hd : 0;
  for (g.hd_log2 = 0; (1 << g.hd_log2) < a.dims.hd;) ++g.hd_log2;
  // sums of a head CTA's tiles are held in two goes, so that the ring keeps most of the shared memory
  g.round_tiles = std::min(most, 64);
  const int per = (g.round_tiles * g.KTs + kStWarps - 1) / kStWarps;     // k tiles of a warp's run in a round
  // A run that fits is one slot: everything is requested before the wait and awaited once.  Longer ones stream through
  // slots of 4 KB: a bulk copy costs an SM about 70 ns whatever its size, so 1 KB copies held the 27B gate / up stream at
  // 2.1 TB/s and 4 KB ones run it at 6.7.
  g.nslots = 0;
  g.slot_tiles = 0;
  const int fixed = st_smem(g, a.ncols, a.nterms).total;
  const int room = (kStSmemTarget - fixed) / (kStWarps * 512);
  if (per <= room && most <= g.round_tiles) {
    g.slot_tiles = per;
    g.nslots = 1;
  } else {
    g.slot_tiles = 8;
    g.nslots = kStMaxSlots;
  }
  g.sm = st_smem(g, a.ncols, a.nterms);
  const int T = kStThreads / st_cols(a.ncols);
  const int nv = (g.kmax / 4 + T - 1) / T;                               // float4 of a vector per thread
  // one limit for every group: what the instantiation of four holds (two sessions alone would hold twice as much)
  const int widest = 12 * (a.ncols <= 1 ? kStThreads : kStThreads / 4);
  if ((size_t)g.sm.total > pl.smem_optin || g.kmax / 4 > widest) {
    B2_CHECK(l.fits != nullptr, kInternal, "the decode step does not fit, but was planned");
    *l.fits = false;
    return;
  }
  // the short combine's slices are at most 256 wide, which is less than a float4 a thread in every group
  if constexpr (PRO == kStCombineShort) {
    launch_gemv_cp<PRO, EPI, 1>(l, a, g);
  } else {
    if (nv <= 1) launch_gemv_cp<PRO, EPI, 1>(l, a, g);
    else if (nv <= 3) launch_gemv_cp<PRO, EPI, 3>(l, a, g);
    else if (nv <= 4) launch_gemv_cp<PRO, EPI, 4>(l, a, g);
    else launch_gemv_cp<PRO, EPI, 12>(l, a, g);
  }
}

template <typename T, int HD, int G>
void launch_attn_t(const Launch& l, const DecodeArgs& a, const StepPlan& pl, StepAttn g) {
  // a second buffer only where a split can hold more than one round
  g.nbuf = g.nsplit * kStKeys >= pl.keys[g.is_global] ? 1 : 2;
  go(l, step_attn_kernel<T, HD, G>, a.ncols * a.dims.hkv * g.nsplit, kAtThreads, (size_t)st_attn_smem<T, HD, G>(g.nbuf), a, g);
}
template <typename T, int HD>
void launch_attn_g(const Launch& l, const DecodeArgs& a, const StepPlan& pl, const StepAttn& g) {
  switch (a.dims.group()) {
    case 1: launch_attn_t<T, HD, 1>(l, a, pl, g); break;
    case 2: launch_attn_t<T, HD, 2>(l, a, pl, g); break;
    default: launch_attn_t<T, HD, 4>(l, a, pl, g); break;
  }
}
template <typename T>
void launch_attn(const Launch& l, const DecodeArgs& a, const StepPlan& pl, const StepAttn& g) {
  switch (a.dims.hd) {
    case 32: launch_attn_g<T, 32>(l, a, pl, g); break;
    case 64: launch_attn_g<T, 64>(l, a, pl, g); break;
    case 128: launch_attn_g<T, 128>(l, a, pl, g); break;
    default: launch_attn_g<T, 256>(l, a, pl, g); break;
  }
}

int run(Launch l, const DecodeArgs& a, const StepPlan& pl, const LayerWeights* layers, const LayerKv* kv, StepReduceFn reduce, void* ctx) {
  const ModelDims& d = a.dims;
  const int KTd = d.d / 64, KTo = d.nq() / 64, KTf = d.ffn / 64;
  int n = 0;
  const int nl = l.fits ? 1 : d.n_layers;
  auto resid = [&](StepGemv& g, const float* parts, int nparts, int from, const float* g_post, const float* g_pre) {
    g.parts = parts;
    g.nparts = nparts;
    g.xin = a.xres[from];
    g.xout = a.xres[from ^ 1];
    g.g_post = g_post;
    g.g_pre = g_pre;
  };
  int x = 0;                                   // which copy of the residual the next kernel reads
  for (int i = 0; i < nl; ++i) {
    const LayerWeights& L = layers[i];
    StepGemv q{};
    q.w = L.wqkv; q.wscale = L.sqkv; q.tiles = d.nqkv() / 16; q.KT = KTd; q.slices = 1; q.y = a.qkv;
    resid(q, i > 0 ? pl.fpart : nullptr, pl.down_slices, x, i > 0 ? layers[i - 1].g_post_ffn : nullptr, L.g_pre_attn);
    x ^= 1;
    l.pdl = !(reduce && i > 0);                // an ordinary edge behind a collective
    q.bar = 5 * i;
    launch_gemv<kStResid, kStPlain>(l, a, pl, q);
    l.pdl = true;
    for (int glob = l.fits ? 0 : L.is_global; glob <= (l.fits ? 1 : L.is_global); ++glob) {
      StepAttn t{};
      t.qkv = a.qkv; t.g_q = L.g_q; t.g_k = L.g_k; t.cosT = a.rope_cos[glob]; t.sinT = a.rope_sin[glob]; t.kv = kv[i];
      t.is_global = glob; t.nsplit = pl.nsplit[glob]; t.part_o = pl.part_o; t.part_ml = pl.part_ml;
      t.bar = 5 * i + 1;
      if (d.kv_dtype == 0) launch_attn<float>(l, a, pl, t);
      else launch_attn<__nv_bfloat16>(l, a, pl, t);
    }
    StepGemv o{};
    o.w = L.wo; o.wscale = L.so; o.tiles = d.d / 16; o.KT = KTo; o.slices = pl.o_slices; o.y = pl.opart;
    o.part_o = pl.part_o; o.part_ml = pl.part_ml; o.nsplit = pl.nsplit[L.is_global ? 1 : 0]; o.is_global = L.is_global;
    o.bar = 5 * i + 2;
    // one head of 256, or one or two of 128 in a slice of K: a warp's 128 values belong to one head
    if (d.hd >= 128 && d.nq() / pl.o_slices <= kStShortSlice) launch_gemv<kStCombineShort, kStPlain>(l, a, pl, o);
    else launch_gemv<kStCombine, kStPlain>(l, a, pl, o);
    if (reduce) reduce(ctx, pl.opart, (size_t)pl.o_slices * a.ncols * d.d);
    StepGemv gu{};
    gu.w = L.wgu; gu.wscale = L.sgu; gu.tiles = 2 * d.ffn / 16; gu.KT = KTd; gu.slices = 1; gu.y = a.act;
    resid(gu, pl.opart, pl.o_slices, x, L.g_post_attn, L.g_pre_ffn);
    x ^= 1;
    l.pdl = !reduce;
    gu.bar = 5 * i + 3;
    launch_gemv<kStResid, kStGeglu>(l, a, pl, gu);
    l.pdl = true;
    StepGemv dn{};
    dn.w = L.wdown; dn.wscale = L.sdown; dn.tiles = d.d / 16; dn.KT = KTf; dn.slices = pl.down_slices; dn.y = pl.fpart; dn.act = a.act;
    dn.bar = 5 * i + 4;
    launch_gemv<kStAct, kStPlain>(l, a, pl, dn);
    if (reduce) reduce(ctx, pl.fpart, (size_t)pl.down_slices * a.ncols * d.d);
    n += 5;
  }
  StepGemv h{};
  h.w = a.head_w; h.wscale = a.embed_scale; h.tiles = d.vocab / 16; h.KT = KTd; h.slices = 1; h.y = a.logits; h.ticket = pl.ticket;
  resid(h, pl.fpart, pl.down_slices, x, layers[d.n_layers - 1].g_post_ffn, a.g_final);
  l.pdl = !reduce;
  h.bar = 5 * d.n_layers;
  launch_gemv<kStResid, kStHead>(l, a, pl, h);
  if (!l.fits) B2_CUDA(cudaGetLastError());
  return n + 1;
}

}  // namespace

bool step_prepare(const DecodeArgs& a, const StepPlan& pl, const LayerWeights* layers, const LayerKv* kv) {
  bool fits = true;
  Launch l{nullptr};
  l.fits = &fits;
  run(l, a, pl, layers, kv, nullptr, nullptr);
  return fits;
}

int step_launch(cudaStream_t st, const DecodeArgs& a, const StepPlan& pl, const LayerWeights* layers, const LayerKv* kv, StepReduceFn reduce,
                void* reduce_ctx) {
  return run(Launch{st}, a, pl, layers, kv, reduce, reduce_ctx);
}

}  // namespace b200lm

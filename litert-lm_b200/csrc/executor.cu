// The B200 executor: model upload, paged KV cache, the reference's executor
// state machine (token hold-back, step counter, bucketed work groups) and the
// kernel orchestration for prefill and decode, behind the C ABI of b200lm.h.
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdio.h>
#include <stdlib.h>

#include <algorithm>
#include <cmath>
#include <fstream>
#include <memory>
#include <string>
#include <vector>

#include "../../include/b200lm.h"
#include "common.cuh"
#include "decode_ops.cuh"
#include "decode_stream.cuh"
#include "decode_step.cuh"
#include "model_host.h"
#include "prefill_ops.cuh"
#include "prefill_gemm_ts.cuh"
#include "gemm_small.cuh"
#include "prefill_attn_tc.cuh"
#include "runtime.h"

namespace b200lm {

// ------------------------------------------------------------------ the model

Model::~Model() {
  cudaSetDevice(device);
  for (void* p : allocations) cudaFree(p);
}

void* Model::alloc(size_t bytes) {
  void* p = nullptr;
  B2_CUDA(cudaMalloc(&p, std::max<size_t>(bytes, 256)));
  allocations.push_back(p);
  return p;
}

template <typename T>
static T* upload(Model& m, const T* host, size_t count) {
  T* d = reinterpret_cast<T*>(m.alloc(count * sizeof(T)));
  B2_CUDA(cudaMemcpy(d, host, count * sizeof(T), cudaMemcpyHostToDevice));
  return d;
}

static const uint4* upload_w4t(Model& m, const uint8_t* packed, int64_t rows, int64_t K) {
  std::vector<uint32_t> buf((size_t)rows * K / 8);
  repack_w4t(packed, rows, K, [](int64_t r) { return r; }, buf.data());
  return reinterpret_cast<const uint4*>(upload(m, buf.data(), buf.size()));
}

// Host-side W4T tiles of a matrix.
template <typename RowMap>
static std::vector<uint32_t> w4t_host(const uint8_t* packed, int64_t rows, int64_t K, RowMap map) {
  std::vector<uint32_t> buf((size_t)rows * K / 8);
  repack_w4t(packed, rows, K, map, buf.data());
  return buf;
}
// W4G with rows padded to 128; scales padded with 1.0.
static void upload_w4g(Model& m, const uint8_t* packed, const float* scale, int64_t rows, int64_t K,
                       const uint8_t** w_out, const float** s_out) {
  int64_t tiles = (rows + 127) / 128;
  std::vector<uint32_t> buf((size_t)tiles * 128 * K / 8);
  repack_w4g(packed, tiles, K, [rows](int64_t r) { return r < rows ? r : (int64_t)-1; }, buf.data());
  std::vector<float> sc((size_t)tiles * 128, 1.0f);
  std::copy(scale, scale + rows, sc.begin());
  *w_out = reinterpret_cast<const uint8_t*>(upload(m, buf.data(), buf.size()));
  *s_out = upload(m, sc.data(), sc.size());
}

std::shared_ptr<Model> Model::load(const uint8_t* image, size_t n, int device, bool want_tc) {
  WeightsRecord rec = locate_weights(image, n);
  auto m = std::make_shared<Model>();
  m->device = device;
  m->dims = rec.dims;
  const ModelDims& d = m->dims;
  B2_CUDA(cudaSetDevice(device));
  auto bytes = [&](const TensorEntry& e) { return rec.base + e.offset; };
  auto fvec = [&](const std::string& nm, size_t count) {
    const TensorEntry& e = rec.need(nm, 1);
    B2_CHECK(e.nbytes == count * 4, kInvalidArgument, "tensor has the wrong size: " + nm);
    return upload(*m, reinterpret_cast<const float*>(bytes(e)), count);
  };
  auto qmat = [&](const std::string& nm, int64_t rows, int64_t K) -> const TensorEntry& {
    const TensorEntry& e = rec.need(nm + ".q", 0);
    B2_CHECK((int64_t)e.rows == rows && (int64_t)e.cols == K && (int64_t)e.nbytes == rows * K / 2,
             kInvalidArgument, "matrix has the wrong shape: " + nm);
    return e;
  };
  // tied embedding: canonical rows for the gather, mma tiles for the head
  {
    const TensorEntry& e = qmat("embed", d.vocab, d.d);
    m->embed_rows = upload(*m, bytes(e), (size_t)e.nbytes);
    m->embed_scale = fvec("embed.scale", d.vocab);
    if (want_tc) {
      const TensorEntry& es = rec.need("embed.scale", 1);
      upload_w4g(*m, bytes(e), reinterpret_cast<const float*>(bytes(es)), d.vocab, d.d, &m->head_g, &m->head_gs);
    }
    auto ht = w4t_host(bytes(e), d.vocab, d.d, [](int64_t r) { return r; });
    m->head_w = reinterpret_cast<const uint4*>(upload(*m, ht.data(), ht.size()));
  }
  m->g_final = fvec("final_norm", d.d);
  {
    const float* g = reinterpret_cast<const float*>(bytes(rec.need("final_norm", 1)));
    m->gmax_final = 0.f;
    for (int k = 0; k < d.d; ++k) m->gmax_final = std::max(m->gmax_final, std::fabs(g[k]));
  }
  m->layers_host.resize(d.n_layers);
  m->gemm_host.resize(d.n_layers);
  auto fptr = [&](const std::string& nm) { return reinterpret_cast<const float*>(bytes(rec.need(nm, 1))); };
  for (int i = 0; i < d.n_layers; ++i) {
    std::string p = "L" + std::to_string(i) + ".";
    LayerWeights& L = m->layers_host[i];
    LayerGemmWeights& Gm = m->gemm_host[i];
    memset(&L, 0, sizeof L);
    memset(&Gm, 0, sizeof Gm);
    const TensorEntry& eqkv = qmat(p + "wqkv", d.nqkv(), d.d);
    const TensorEntry& eo = qmat(p + "wo", d.d, d.nq());
    const TensorEntry& eg = qmat(p + "wgate", d.ffn, d.d);
    const TensorEntry& eu = qmat(p + "wup", d.ffn, d.d);
    const TensorEntry& ed = qmat(p + "wdown", d.d, d.ffn);
    const float* sqkv = reinterpret_cast<const float*>(bytes(rec.need(p + "wqkv.scale", 1)));
    const float* so = reinterpret_cast<const float*>(bytes(rec.need(p + "wo.scale", 1)));
    const float* sg = reinterpret_cast<const float*>(bytes(rec.need(p + "wgate.scale", 1)));
    const float* su = reinterpret_cast<const float*>(bytes(rec.need(p + "wup.scale", 1)));
    const float* sd = reinterpret_cast<const float*>(bytes(rec.need(p + "wdown.scale", 1)));
    auto ident = [](int64_t r) { return r; };
    {
      auto t = w4t_host(bytes(eqkv), d.nqkv(), d.d, ident);
      L.wqkv = reinterpret_cast<const uint4*>(upload(*m, t.data(), t.size()));
    }
    L.sqkv = upload(*m, sqkv, d.nqkv());
    {
      auto t = w4t_host(bytes(eo), d.d, d.nq(), ident);
      L.wo = reinterpret_cast<const uint4*>(upload(*m, t.data(), t.size()));
    }
    L.so = upload(*m, so, d.d);
    {
      auto t = w4t_host(bytes(ed), d.d, d.ffn, ident);
      L.wdown = reinterpret_cast<const uint4*>(upload(*m, t.data(), t.size()));
    }
    L.sdown = upload(*m, sd, d.d);
    // gate and up share one matrix: canonical rows [gate ; up]
    std::vector<uint8_t> gu((size_t)2 * d.ffn * d.d / 2);
    memcpy(gu.data(), bytes(eg), (size_t)eg.nbytes);
    memcpy(gu.data() + eg.nbytes, bytes(eu), (size_t)eu.nbytes);
    const int64_t ffn = d.ffn;
    {   // decode layout: 16-row tiles alternate gate, up
      std::vector<uint32_t> buf((size_t)2 * ffn * d.d / 8);
      auto map = [ffn](int64_t r) {
        int64_t tile = r / 16, pair = tile / 2;
        return (tile & 1 ? ffn : (int64_t)0) + pair * 16 + (r % 16);
      };
      repack_w4t(gu.data(), 2 * ffn, d.d, map, buf.data());
      L.wgu = reinterpret_cast<const uint4*>(upload(*m, buf.data(), buf.size()));
      std::vector<float> sc((size_t)2 * ffn);
      for (int64_t r = 0; r < 2 * ffn; ++r) {
        int64_t src = map(r);
        sc[r] = src < ffn ? sg[src] : su[src - ffn];
      }
      L.sgu = upload(*m, sc.data(), sc.size());
    }
    auto gmax = [&](const std::string& nm) {
      const float* g = reinterpret_cast<const float*>(bytes(rec.need(nm, 1)));
      float m = 0.f;
      for (int k = 0; k < d.d; ++k) m = std::max(m, std::fabs(g[k]));
      return m;
    };
    L.gmax_pre_attn = gmax(p + "pre_attn");
    L.gmax_pre_ffn = gmax(p + "pre_ffn");
    L.g_pre_attn = fvec(p + "pre_attn", d.d);
    L.g_post_attn = fvec(p + "post_attn", d.d);
    L.g_pre_ffn = fvec(p + "pre_ffn", d.d);
    L.g_post_ffn = fvec(p + "post_ffn", d.d);
    {
      const float* gq = reinterpret_cast<const float*>(bytes(rec.need(p + "q_norm", 1)));
      const float* gk = reinterpret_cast<const float*>(bytes(rec.need(p + "k_norm", 1)));
      float mq = 0.f, mk = 0.f;
      for (int k = 0; k < d.hd; ++k) { mq = std::max(mq, std::fabs(gq[k])); mk = std::max(mk, std::fabs(gk[k])); }
      m->attn_bound.push_back(std::sqrt((float)d.hd) * mq * mk * 1.01f);
      L.attn_bound = m->attn_bound.back();
    }
    L.g_q = fvec(p + "q_norm", d.hd);
    L.g_k = fvec(p + "k_norm", d.hd);
    L.is_global = d.is_global(i) ? 1 : 0;
    if (want_tc) {
      upload_w4g(*m, bytes(eqkv), sqkv, d.nqkv(), d.d, &Gm.wqkv, &Gm.sqkv);
      upload_w4g(*m, bytes(eo), so, d.d, d.nq(), &Gm.wo, &Gm.so);
      upload_w4g(*m, bytes(ed), sd, d.d, d.ffn, &Gm.wdown, &Gm.sdown);
      // 128-row tiles of 64 ffn features: gate row of a feature, then its up row
      int64_t tiles = ffn / 64;
      std::vector<uint32_t> buf((size_t)tiles * 128 * d.d / 8);
      auto map = [ffn](int64_t r) {
        int64_t j = r / 128, c = r % 128;
        return (c & 1 ? ffn : (int64_t)0) + j * 64 + (c >> 1);
      };
      repack_w4g(gu.data(), tiles, d.d, map, buf.data());
      Gm.wgu = reinterpret_cast<const uint8_t*>(upload(*m, buf.data(), buf.size()));
      std::vector<float> sc((size_t)tiles * 128);
      for (int64_t r = 0; r < tiles * 128; ++r) {
        int64_t src = map(r);
        sc[r] = src < ffn ? sg[src] : su[src - ffn];
      }
      Gm.sgu = upload(*m, sc.data(), sc.size());
    }
  }
  m->has_tc = want_tc;
  m->layers_dev = upload(*m, m->layers_host.data(), m->layers_host.size());
  for (int t = 0; t < 2; ++t) {
    std::vector<float> c, s;
    build_rope_table(t ? d.rope_global : d.rope_local, d.hd, d.max_ctx, c, s);
    m->rope_cos[t] = upload(*m, c.data(), c.size());
    m->rope_sin[t] = upload(*m, s.data(), s.size());
  }
  return m;
}

// --------------------------------------------------------------- tensor maps

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_tiled_fn() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    B2_CUDA(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q));
    B2_CHECK(p != nullptr && q == cudaDriverEntryPointSuccess, kInternal, "cuTensorMapEncodeTiled unavailable");
    fn = reinterpret_cast<EncodeTiledFn>(p);
  }
  return fn;
}

// bf16 row-major [rows][cols]; box = 64 columns x 128 rows, 128-byte swizzle.
ActMap make_activation_map(const __nv_bfloat16* base, int rows, int cols) {
  ActMap m;
  for (int i = 0; i < 4; ++i) m.box[i] = make_activation_map_box(base, rows, cols, 16 << i);
  return m;
}

CUtensorMap make_activation_map_box(const __nv_bfloat16* base, int rows, int cols, int box_rows) {
  CUtensorMap tm;
  cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)cols * 2};
  cuuint32_t box[2] = {(cuuint32_t)kGemmBK, (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = encode_tiled_fn()(&tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<__nv_bfloat16*>(base), dims,
                                 strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                                 CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  B2_CHECK(r == CUDA_SUCCESS, kInternal, "cuTensorMapEncodeTiled failed: " + std::to_string((int)r));
  return tm;
}

// bf16 tensor of rank 2 or 3 (innermost dimension first), 128-byte swizzle.
static CUtensorMap make_bf16_map(const void* base, int rank, const cuuint64_t* dims, const cuuint64_t* strides_bytes,
                                 const cuuint32_t* box) {
  CUtensorMap tm;
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = encode_tiled_fn()(&tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, (cuuint32_t)rank, const_cast<void*>(base), dims,
                                 strides_bytes, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                                 CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  B2_CHECK(r == CUDA_SUCCESS, kInternal, "cuTensorMapEncodeTiled failed: " + std::to_string((int)r));
  return tm;
}

// What a GEMM of the tcgen05 kernel and its consumer's pass over the partial sums take, in us, for one choice of token
// tile and K split.  The terms are what the kernel spends its time on: rounds of tiles over the CTA slots, each a row of k
// blocks whose price depends on the tile's width (tensor-bound at 256 tokens, the expansion's chain of waits below; dearer
// where two CTAs share an SM), then the accumulators' stores, then the partials once more out of L2.  The constants are a
// least-squares fit to timed pairs of GEMM and residual norm (14 projections of four models, 20 - 1023 tokens), made while
// a split's K went into one accumulator.  With the present kernel the choice takes 1.5 % more than the best split on average and up
// to 22 % at 36 tokens (15 projections, 2048 tokens and shards of layers among them: profiles/gemm_split_choice.md), where filling
// 90 % of the last round with the widest tile had eight splits for 2560 x 2048 at 1023 tokens: 45.6 us with the norm, 22.5 with one.
static double ts_cost(int T, int N, int K, bool geglu, int ntok, int ks, int sms) {
  struct Width { int ntok; double kb, kb_shared, round; };
  static const Width widths[] = {{16, 0.172, 0.325, 0.0}, {32, 0.188, 0.312, 0.0}, {64, 0.209, 0.317, 0.0}, {128, 0.281, 0.281, 0.0}, {256, 0.331, 0.331, 0.6}};
  const Width* w = widths;
  while (w->ntok != ntok) ++w;
  const int tiles = ((N + kTsRows - 1) / kTsRows) * ((T + ntok - 1) / ntok) * ks, slots = ts_ctas_per_sm(ntok) * sms;
  const double mb = 1e-6 * 4, rounds = (tiles + slots - 1) / slots;
  double us = rounds * ((double)(K / kGemmBK / ks) * (tiles > sms ? w->kb_shared : w->kb) + w->round);
  us += 0.126 * mb * std::min(tiles, slots) * ntok * kTsRows * (geglu ? 0.5 : 1.0);
  if (!geglu) us += 0.25 * mb * ks * T * N + 0.15 * ks;
  return us;
}
// Token tile of the tcgen05 kernel for a given K split.
static int ts_tile_tokens(int T, int N, int K, bool geglu, int ks, int sms) {
  int best = 16;
  double best_us = ts_cost(T, N, K, geglu, best, ks, sms);
  for (int ntok : {32, 64, 128, 256}) {
    const double us = ts_cost(T, N, K, geglu, ntok, ks, sms);
    if (us < best_us) { best_us = us; best = ntok; }
  }
  return best;
}

// K that one accumulator of the tcgen05 GEMM takes, by what its rows are.  Short chains lose less in the accumulators,
// which cut off, long ones less in rounding the sums of their parts.  Which of the two counts depends on the rows: products of
// two values (GeGLU) spread over more binades than normed rows, and attention's rows, whose heads differ in size, lie between.
// 2-norm errors against 64 bits: GeGLU rows, K = 6912 in 1 / 2 / 4 / 6 chains 1.2e-6 / 5.0e-7 / 2.3e-7 / 1.6e-7; normed rows,
// K = 5376 in 1 / 2 / 4 / 6 / 9 chains 1.5e-7 / 8.6e-8 / 6.5e-8 / 6.4e-8 / 7.0e-8; attention's, K = 2048 in 1 / 2 / 4 / 8 chains
// 1.1e-7 / 6.7e-8 / 5.6e-8 / 6.2e-8.
int gemm_chain(GemmRows rows, int K) {
  if (rows == GemmRows::kNormed) return 1024;
  if (rows == GemmRows::kAttention) return std::min(512, K / 2);
  return std::max(256, K / 8);
}

// Split-K factor of a GEMM: a divisor of the 64-wide k blocks, at most `most` (what the partials buffer holds) and eight,
// four blocks a split and more.
int pick_ksplit(int T, int N, int K, int sms, int most) {
  const int KB = K / kGemmBK;
  if (const int s = gs_ksplit(T, N, KB, sms, most)) return s;
  int best = 1;
  double best_us = 1e30;
  for (int s = 1; s <= std::min(8, most); ++s) {
    if (KB % s || (s > 1 && KB / s < 4)) continue;
    const double us = ts_cost(T, N, K, false, ts_tile_tokens(T, N, K, false, s, sms), s, sms);
    if (us < best_us) { best_us = us; best = s; }
  }
  return best;
}

// Launches one int4 GEMM.  a_map must describe `A` ([rows >= T][K] bf16).
void launch_gemm(cudaStream_t st, int mode, const ActMap& a_map, const __nv_bfloat16* A,
                 const uint4* w4t, const float* s4t, const uint8_t* w4g, const float* s4g, int T, int N, int K,
                 int ksplit, int chain, bool geglu, float* outF, __nv_bfloat16* outB, int* err, int64_t* launches) {
  if (mode == B200LM_GEMM_TCGEN05) {
    const int stages = (K / kGemmBK / ksplit + kTsKb - 1) / kTsKb, most = std::max(1, (chain + kTsKb * kGemmBK - 1) / (kTsKb * kGemmBK));
    const int chains = (stages + most - 1) / most;
    GemmArgs g{w4g, s4g, T, N, K, ksplit, (stages + chains - 1) / chains, outF, outB, err};
    static int sms_of[64] = {0};              // per device: SM count, set once together with the kernel attributes
    int dev = 0;
    B2_CUDA(cudaGetDevice(&dev));
    B2_CHECK(dev >= 0 && dev < 64, kInternal, "device ordinal out of range");
    if (!sms_of[dev]) {
#define B2_TS_PREP(NTOK_)                                              \
  raise_dyn_smem(gemm_w4_ts_kernel<0, NTOK_>, (size_t)ts_smem(NTOK_)); \
  raise_dyn_smem(gemm_w4_ts_kernel<1, NTOK_>, (size_t)ts_smem(NTOK_)); \
  share_memory(gemm_w4_ts_kernel<0, NTOK_>);                           \
  share_memory(gemm_w4_ts_kernel<1, NTOK_>)
      B2_TS_PREP(16);
      B2_TS_PREP(32);
      B2_TS_PREP(64);
      B2_TS_PREP(128);
      B2_TS_PREP(256);
#undef B2_TS_PREP
#define B2_TS_REGS(NTOK_)                                                    \
  B2_CUDA(cudaFuncGetAttributes(&fa, gemm_w4_ts_kernel<0, NTOK_>));          \
  B2_CHECK(fa.numRegs == ts_regs(NTOK_).launch, kInternal, "GEMM kernel: not the registers that its warps share out")
      cudaFuncAttributes fa;                  // a warp would wait for ever for registers that the block does not have
      B2_TS_REGS(64);
      B2_TS_REGS(128);
      B2_TS_REGS(256);
#undef B2_TS_REGS
      B2_CUDA(cudaDeviceGetAttribute(&sms_of[dev], cudaDevAttrMultiProcessorCount, dev));
    }
    const int sms = sms_of[dev];
    // At most 16 rows whose slice of X fits beside the weight ring: mma.sync (20480 x 2560 with GeGLU, 16 rows: 11.9 us against
    // 13.2 on tcgen05; 4096 x 2560 and what follows it 7.0 against 7.3; of the 1B model's only gate/up loses, 6.8 against 6.1).
    // From 17 rows on it loses (13824 x 1152: 10.2 against 6.9 us at 20 rows, 12.8 against 8.2 at 36).
    if (gs_fits(T, N, K / 64, ksplit, geglu, sms)) {
      launch_gemm_small(st, sms, dev, w4t, s4t, A, T, N, K, ksplit, geglu, outF, outB);
      B2_CUDA(cudaGetLastError());
      if (launches) ++*launches;
      return;
    }
    const int ntok = ts_tile_tokens(T, N, K, geglu, ksplit, sms);
    const int total = ((N + kTsRows - 1) / kTsRows) * ((T + ntok - 1) / ntok) * ksplit;
    const int slots = ts_ctas_per_sm(ntok) * sms, grid = total < slots ? total : slots;
#define B2_TS(EPI_, NTOK_, MAP_) launch_pdl(gemm_w4_ts_kernel<EPI_, NTOK_>, dim3(grid), dim3(ts_threads(NTOK_)), ts_smem(NTOK_), st, MAP_, g)
#define B2_TS2(NTOK_, MAP_) do { if (geglu) B2_TS(1, NTOK_, MAP_); else B2_TS(0, NTOK_, MAP_); } while (0)
    switch (ntok) {
      case 16: B2_TS2(16, a_map.box[0]); break;
      case 32: B2_TS2(32, a_map.box[1]); break;
      case 64: B2_TS2(64, a_map.box[2]); break;
      case 128: B2_TS2(128, a_map.box[3]); break;
      default: B2_TS2(256, a_map.box[3]); break;
    }
#undef B2_TS2
#undef B2_TS
  } else {
    B2_CHECK(ksplit == 1, kInternal, "the check GEMM does not split K");
    dim3 grid(geglu ? N / 32 : N / 16, (T + 7) / 8);
    gemm_w4_simple_kernel<<<grid, 128, 0, st>>>(A, w4t, s4t, T, N, K, geglu ? 1 : 0, outF, outB);
  }
  B2_CUDA(cudaGetLastError());
  if (launches) ++*launches;
}

// --------------------------------------------------------------- the executor

template <typename T>
static auto kv_append_kernel(const ModelDims& d) {
  switch (d.hd) {
    case 32: return pf_kv_append_kernel<T, 32>;
    case 64: return pf_kv_append_kernel<T, 64>;
    case 128: return pf_kv_append_kernel<T, 128>;
    default: return pf_kv_append_kernel<T, 256>;
  }
}

static int round_up(int v, int a) { return (v + a - 1) / a * a; }

Executor::~Executor() {
  cudaSetDevice(device);
  if (stream) cudaStreamSynchronize(stream);
  for (auto& g : step_graphs) {
    if (g.second.graph) cudaGraphDestroy(g.second.graph);
    if (g.second.exec) cudaGraphExecDestroy(g.second.exec);
  }
  for (auto& g : wide_graphs) cudaGraphExecDestroy(g.second);
  for (cudaEvent_t ev : logit_part)
    if (ev) cudaEventDestroy(ev);
  if (tp_comm) {
    try { NcclApi::get().CommDestroy(tp_comm); } catch (...) {}
  }
  for (void* p : allocations) cudaFree(p);
  for (int i = 0; i < kTokRing; ++i)
    if (tok_ring_done[i]) cudaEventDestroy(tok_ring_done[i]);
  if (pinned) cudaFreeHost(pinned);
  if (own_stream && stream) cudaStreamDestroy(stream);
}

void* Executor::alloc(size_t bytes, bool zero) {
  void* p = nullptr;
  B2_CUDA(cudaMalloc(&p, std::max<size_t>(bytes, 256)));
  allocations.push_back(p);
  if (zero) B2_CUDA(cudaMemset(p, 0, std::max<size_t>(bytes, 256)));
  return p;
}

std::unique_ptr<Executor> Executor::create(std::shared_ptr<Model> model, const B200LmConfig& cfg) {
  auto e = std::unique_ptr<Executor>(new Executor());
  e->model = model;
  e->device = model->device;
  const ModelDims& d = model->dims;
  B2_CUDA(cudaSetDevice(e->device));
  cudaDeviceProp prop;
  B2_CUDA(cudaGetDeviceProperties(&prop, e->device));
  B2_CHECK(prop.major == 10, kFailedPrecondition,
           "this library is built for sm_100a (B200); device reports sm_" + std::to_string(prop.major) +
               std::to_string(prop.minor));
  e->n_sms = prop.multiProcessorCount;
  e->smem_optin = (size_t)prop.sharedMemPerBlockOptin;
  if (cfg.stream) {
    e->stream = reinterpret_cast<cudaStream_t>(cfg.stream);
  } else {
    B2_CUDA(cudaStreamCreateWithFlags(&e->stream, cudaStreamNonBlocking));
    e->own_stream = true;
  }
  if (cfg.tp_world > 1) {
    B2_CHECK(cfg.tp_rank >= 0 && cfg.tp_rank < cfg.tp_world && cfg.tp_unique_id != nullptr, kInvalidArgument,
             "tensor parallelism needs 0 <= tp_rank < tp_world and the group's unique id");
    const NcclApi& nccl = NcclApi::get();
    NcclApi::UniqueId id;
    memcpy(&id, cfg.tp_unique_id, sizeof id);
    nccl.check(nccl.CommInitRank(&e->tp_comm, cfg.tp_world, id, cfg.tp_rank), "ncclCommInitRank");
    e->tp_rank = cfg.tp_rank;
    e->tp_world = cfg.tp_world;
  }
  e->max_num_tokens = cfg.max_num_tokens > 0 ? std::min(cfg.max_num_tokens, d.max_ctx) : d.max_ctx;
  B2_CHECK(cfg.prefill_gemm >= B200LM_GEMM_AUTO && cfg.prefill_gemm <= B200LM_GEMM_TCGEN05, kInvalidArgument,
           "prefill_gemm must be B200LM_GEMM_AUTO, _CHECK or _TCGEN05");
  e->prefill_gemm = cfg.prefill_gemm == B200LM_GEMM_AUTO ? (model->has_tc ? B200LM_GEMM_TCGEN05 : B200LM_GEMM_CHECK)
                                                          : cfg.prefill_gemm;
  B2_CHECK(e->prefill_gemm != B200LM_GEMM_TCGEN05 || model->has_tc, kFailedPrecondition,
           "tensor-core GEMM weights were not loaded for this model");
  B2_CHECK(cfg.page_order == 0 || cfg.page_order == 1, kInvalidArgument, "page_order must be 0 or 1");
  B2_CHECK(cfg.decode_mode >= B200LM_DECODE_AUTO && cfg.decode_mode <= B200LM_DECODE_WIDE, kInvalidArgument,
           "decode_mode must be one of B200LM_DECODE_*");
  e->decode_mode = cfg.decode_mode == B200LM_DECODE_AUTO ? B200LM_DECODE_CHAINED : cfg.decode_mode;
  // more sessions than the GEMV kernels carry per step: the projections run on the tensor-core GEMM
  if (cfg.n_sessions > kMaxCols && cfg.decode_mode == B200LM_DECODE_AUTO) e->decode_mode = B200LM_DECODE_WIDE;
  if (e->decode_mode == B200LM_DECODE_WIDE)
    B2_CHECK(e->prefill_gemm == B200LM_GEMM_TCGEN05 && cfg.tp_world <= 1, kFailedPrecondition,
             "the wide decode mode needs the tensor-core GEMM weights and no tensor parallelism");
  // a collective cannot run inside a persistent kernel: tensor-parallel decode launches its kernels one by one
  if (cfg.tp_world > 1) e->decode_mode = B200LM_DECODE_PHASE_KERNELS;
  const int esz = d.kv_dtype == 0 ? 4 : 2;
  // ---- paged KV cache
  e->pages_per_seq = (e->max_num_tokens + kPage - 1) / kPage;     // the cache holds max_num_tokens positions per session
  e->n_sessions = cfg.n_sessions > 0 ? cfg.n_sessions : 1;
  {
    const int cap = e->decode_mode == B200LM_DECODE_WIDE ? kWideMax : kMaxCols;
    B2_CHECK(e->n_sessions <= cap, kInvalidArgument,
             "n_sessions exceeds the " + std::to_string(cap) + " sessions one decode step of this mode can carry");
  }
  const int max_cols = std::max(kMaxCols, e->n_sessions);
  e->parked.resize(e->n_sessions);
  const int total_pages = e->pages_per_seq * e->n_sessions;
  size_t pool = (size_t)total_pages * d.hkv * kPage * d.hd;
  e->kv_host.resize(d.n_layers);
  // tensor-core prefill attention: head_dim 128 / 256, and every layer's score bound small enough
  e->attn_tc = e->prefill_gemm == B200LM_GEMM_TCGEN05 && (d.hd == 128 || d.hd == 256);
  for (float b : model->attn_bound) e->attn_tc = e->attn_tc && b <= kFaMaxBound;
  for (int i = 0; i < d.n_layers; ++i) {
    e->kv_host[i].k = e->alloc(pool * esz, true);
    e->kv_host[i].v = e->alloc(pool * esz, true);
    e->kv_host[i].k16 = nullptr;
    e->kv_host[i].v16 = nullptr;
    if (e->attn_tc) {
      if (d.kv_dtype == 0) e->kv_host[i].k16 = reinterpret_cast<__nv_bfloat16*>(e->alloc(pool * 2, true));
      e->kv_host[i].v16 = reinterpret_cast<__nv_bfloat16*>(e->alloc(pool * 2, true));
    }
  }
  LayerKv* kvd = reinterpret_cast<LayerKv*>(e->alloc(sizeof(LayerKv) * d.n_layers, false));
  B2_CUDA(cudaMemcpy(kvd, e->kv_host.data(), sizeof(LayerKv) * d.n_layers, cudaMemcpyHostToDevice));
  e->kv_dev = kvd;
  // one page-table row per session, each over its own block of physical pages
  e->page_table_host.resize(total_pages);
  for (int sn = 0; sn < e->n_sessions; ++sn)
    for (int i = 0; i < e->pages_per_seq; ++i)
      e->page_table_host[(size_t)sn * e->pages_per_seq + i] =
          sn * e->pages_per_seq + (cfg.page_order == 1 ? e->pages_per_seq - 1 - i : i);
  int* ptd = reinterpret_cast<int*>(e->alloc(sizeof(int) * total_pages, false));
  B2_CUDA(cudaMemcpy(ptd, e->page_table_host.data(), sizeof(int) * total_pages, cudaMemcpyHostToDevice));
  e->page_table_dev = ptd;
  // ---- decode buffers
  DecodeArgs& a = e->dargs;
  memset(&a, 0, sizeof a);
  a.dims = d;
  a.ncols = 1;
  a.nterms = 3;
  // a split of 32 (local) / 64 (global, at full context) keys fits one staged chunk
  a.n_attn_splits_local = std::max(1, std::min(kMaxSplits, d.window / 32));
  a.n_attn_splits_global = std::max(1, std::min(kMaxSplits, d.max_ctx / 64));
  int hps = 1;
  while ((hps * d.hd) % 64 != 0) ++hps;
  B2_CHECK(d.hq % hps == 0, kUnimplemented, "q heads cannot be grouped into 64-wide slices");
  a.o_slices = d.hq / hps;
  while (a.o_slices > e->n_sms) a.o_slices /= 2;
  {   // the combine of split partials stages (m, l) of one head slice in 512 floats
    int heads_per_slice = d.hq / a.o_slices;
    int cap = std::max(1, 256 / heads_per_slice);
    a.n_attn_splits_local = std::min(a.n_attn_splits_local, cap);
    a.n_attn_splits_global = std::min(a.n_attn_splits_global, cap);
  }
  int KTd = d.ffn / 64;
  a.down_slices = 1;
  for (int s = 4; s >= 2; --s)
    if (KTd % s == 0 && (d.d / 16) * s <= e->n_sms) { a.down_slices = s; break; }
  a.layers = model->layers_dev;
  a.kv = e->kv_dev;
  a.page_table = e->page_table_dev;
  a.pages_per_seq = e->pages_per_seq;
  a.embed_rows = model->embed_rows;
  a.embed_scale = model->embed_scale;
  a.head_w = model->head_w;
  a.g_final = model->g_final;
  a.gmax_final = model->gmax_final;
  for (int t = 0; t < 2; ++t) { a.rope_cos[t] = model->rope_cos[t]; a.rope_sin[t] = model->rope_sin[t]; }
  a.st = reinterpret_cast<DecodeState*>(e->alloc(sizeof(DecodeState), true));
  const int G = d.group();
  a.xres[0] = reinterpret_cast<float*>(e->alloc(sizeof(float) * kMaxCols * d.d, true));
  a.xres[1] = reinterpret_cast<float*>(e->alloc(sizeof(float) * kMaxCols * d.d, true));
  a.qkv = reinterpret_cast<float*>(e->alloc(sizeof(float) * kMaxCols * d.nqkv(), true));
  a.act = reinterpret_cast<float*>(e->alloc(sizeof(float) * kMaxCols * d.ffn, true));
  a.logits = reinterpret_cast<float*>(e->alloc(sizeof(float) * max_cols * d.vocab, true));
  a.amax_val = reinterpret_cast<float*>(e->alloc(sizeof(float) * e->n_sms * kMaxCols, true));
  a.amax_idx = reinterpret_cast<int*>(e->alloc(sizeof(int) * e->n_sms * kMaxCols, true));
  a.step_capacity = d.max_ctx;
  a.step_tokens = reinterpret_cast<int*>(e->alloc(sizeof(int) * a.step_capacity * max_cols, true));
  if (e->decode_mode == B200LM_DECODE_WIDE) {
    int* ws = reinterpret_cast<int*>(e->alloc(sizeof(int) * (4 + 2 * kWideArgParts) * kWideMax, true));
    e->wide = WideState{ws, ws + kWideMax, ws + 2 * kWideMax, reinterpret_cast<float*>(ws + 4 * kWideMax), ws + (4 + kWideArgParts) * kWideMax,
                        ws + 3 * kWideMax};
    {
      WideAttnArgs prep{};
      prep.ctas_per_sm = 2;
      launch_wide_attn(e->stream, d, 0, e->smem_optin, prep);
    }
    e->wide_part = reinterpret_cast<float*>(
        e->alloc(sizeof(float) * (size_t)e->n_sessions * d.hkv * kWideMaxSplits * d.group() * (d.hd + 4), true));
    e->wide_ticket = reinterpret_cast<int*>(e->alloc(sizeof(int) * (size_t)e->n_sessions * d.hkv, true));
  }
  // Which kernels carry a step, and how many sessions at once.  The chain gives way to the persistent kernel, that to the
  // chain with the sessions of a group one after another, that to one kernel per phase; the persistent kernels give way
  // to the chain.  No persistent kernel under tensor parallelism, whose collectives run between the phases.
  e->step_cols = e->n_sessions;
  if (e->decode_mode != B200LM_DECODE_WIDE) {
    const bool coop = prop.cooperativeLaunch && cfg.tp_world <= 1;
    bool placed = false;
    if (e->decode_mode == B200LM_DECODE_PERSISTENT) placed = e->plan_persistent(coop);
    if (e->decode_mode == B200LM_DECODE_PERSISTENT_BASIC) {
      e->dec_smem = dec_smem_bytes(d, e->n_sessions);
      B2_CHECK(e->dec_smem <= e->smem_optin, kUnimplemented, "the persistent decode kernel needs more shared memory than the device offers");
      raise_dyn_smem(decode_persistent_kernel, e->dec_smem);
      int occ = 0;
      B2_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, decode_persistent_kernel, kDecThreads, e->dec_smem));
      placed = occ >= 1 && coop;
    }
    if (!placed) placed = e->chain = e->plan_chain();
    if (!placed && e->decode_mode == B200LM_DECODE_CHAINED && e->plan_persistent(coop)) {
      placed = true;
      e->decode_mode = B200LM_DECODE_PERSISTENT;
    }
    if (!placed && e->n_sessions > 1) {
      e->step_cols = 1;
      placed = e->chain = e->plan_chain();
    }
    if (e->chain && e->decode_mode != B200LM_DECODE_PHASE_KERNELS) e->decode_mode = B200LM_DECODE_CHAINED;
    if (!placed) {
      e->dec_smem = dec_smem_bytes(d, 1);
      B2_CHECK(e->dec_smem <= e->smem_optin, kUnimplemented, "decode kernels need more shared memory than the device offers");
      raise_dyn_smem(decode_phase_kernel, e->dec_smem);
      e->decode_mode = B200LM_DECODE_PHASE_KERNELS;
    }
  }
  // split partials of the kernels that run (the wide step has its own)
  if (e->decode_mode != B200LM_DECODE_WIDE) {
    auto floats = [&](size_t n) { return reinterpret_cast<float*>(e->alloc(sizeof(float) * kMaxCols * n, true)); };
    StepPlan& sp = e->step;
    const size_t splits = e->chain ? sp.max_splits : std::max(a.n_attn_splits_local, a.n_attn_splits_global);
    (e->chain ? sp.part_o : a.part_o) = floats(d.hkv * splits * G * d.hd);
    (e->chain ? sp.part_ml : a.part_ml) = floats(d.hkv * splits * G * 2);
    (e->chain ? sp.opart : a.opart) = floats((size_t)(e->chain ? sp.o_slices : a.o_slices) * d.d);
    (e->chain ? sp.fpart : a.fpart) = floats((size_t)(e->chain ? sp.down_slices : a.down_slices) * d.d);
    if (e->chain) sp.ticket = reinterpret_cast<int*>(e->alloc(sizeof(int), true));
  }
  // ---- prefill buffers (rows padded to whole 128-token tiles, zero-filled)
  e->t_max = d.buckets[0];
  e->t_pad = round_up(e->t_max, kGemmBM);
  const size_t tp = e->t_pad;
  e->pf_tokens = reinterpret_cast<int*>(e->alloc(sizeof(int) * tp, true));
  e->pf_xres = reinterpret_cast<float*>(e->alloc(sizeof(float) * tp * d.d, true));
  e->pf_h = reinterpret_cast<__nv_bfloat16*>(e->alloc(2 * tp * d.d, true));
  e->pf_qkv = reinterpret_cast<float*>(e->alloc(sizeof(float) * tp * d.nqkv(), true));
  e->pf_attn = reinterpret_cast<__nv_bfloat16*>(e->alloc(2 * tp * d.nq(), true));
  e->pf_act = reinterpret_cast<__nv_bfloat16*>(e->alloc(2 * tp * d.ffn, true));
  e->pf_parts = reinterpret_cast<float*>(e->alloc(sizeof(float) * 8 * tp * d.d, true));
  if (e->attn_tc) {
    const int G = d.group();
    e->pf_q = reinterpret_cast<__nv_bfloat16*>(e->alloc(2 * tp * d.nq(), true));
    {
      cuuint64_t dims[3] = {(cuuint64_t)d.hd, (cuuint64_t)d.hq, (cuuint64_t)tp};
      cuuint64_t str[2] = {(cuuint64_t)d.hd * 2, (cuuint64_t)d.nq() * 2};
      cuuint32_t box[3] = {64, (cuuint32_t)G, (cuuint32_t)(128 / G)};
      e->tm_q = make_bf16_map(e->pf_q, 3, dims, str, box);
    }
    const cuuint64_t rows = (cuuint64_t)total_pages * d.hkv * kPage;
    for (int i = 0; i < d.n_layers; ++i) {
      const void* kbase = d.kv_dtype == 0 ? (const void*)e->kv_host[i].k16 : (const void*)e->kv_host[i].k;
      cuuint64_t kd[2] = {(cuuint64_t)d.hd, rows};
      cuuint64_t ks[1] = {(cuuint64_t)d.hd * 2};
      cuuint32_t kb[2] = {64, (cuuint32_t)kFaBN};
      e->tm_k.push_back(make_bf16_map(kbase, 2, kd, ks, kb));
      cuuint64_t vd[2] = {(cuuint64_t)kPage, (cuuint64_t)total_pages * d.hkv * d.hd};
      cuuint64_t vs[1] = {(cuuint64_t)kPage * 2};
      cuuint32_t vb[2] = {(cuuint32_t)kFaBN, (cuuint32_t)d.hd};
      e->tm_vt.push_back(make_bf16_map(e->kv_host[i].v16, 2, vd, vs, vb));
    }
    if (d.hd == 256) {
      raise_dyn_smem(flash_prefill_tc_kernel<256>, (size_t)(FaSmem<256>::kTotal));
      share_memory(flash_prefill_tc_kernel<256>);
    } else {
      raise_dyn_smem(flash_prefill_tc_kernel<128>, (size_t)(FaSmem<128>::kTotal));
      share_memory(flash_prefill_tc_kernel<128>);
    }
  }
  share_memory(pf_embed_norm_kernel);
  share_memory(pf_resid_norm_reg_kernel<128, 3, 4>);
  share_memory(pf_resid_norm_reg_kernel<256, 3, 4>);
  share_memory(pf_resid_norm_reg_kernel<512, 3, 4>);
  if (d.kv_dtype == 0) share_memory(kv_append_kernel<float>(d));
  else share_memory(kv_append_kernel<__nv_bfloat16>(d));
  share_memory(wide_argmax_kernel);
  raise_dyn_smem(pf_attn_kernel, sizeof(float) * ((size_t)(d.group() + 2) * d.hd + (size_t)8 * d.group() * (d.hd + 2)));
  if (e->prefill_gemm == B200LM_GEMM_TCGEN05) {
    e->tm_h = make_activation_map(e->pf_h, (int)tp, d.d);
    e->tm_attn = make_activation_map(e->pf_attn, (int)tp, d.nq());
    e->tm_act = make_activation_map(e->pf_act, (int)tp, d.ffn);
  }
  // page-locked staging: logits | kTokRing slices of prompt ids | sampled ids of a decode call | state words
  size_t pin = sizeof(float) * (size_t)d.vocab + sizeof(int) * (kTokRing * tp + (size_t)d.max_ctx * max_cols + 3 * kWideMax) + 4096;
  B2_CUDA(cudaMallocHost(&e->pinned, pin));
  e->pin_logits = reinterpret_cast<float*>(e->pinned);
  e->pin_ints = reinterpret_cast<int*>(e->pin_logits + d.vocab);
  e->pin_steps = e->pin_ints + (size_t)kTokRing * tp;
  e->pin_wide = e->pin_steps + (size_t)d.max_ctx * max_cols;
  e->pin_state = reinterpret_cast<DecodeState*>(e->pin_wide + 3 * kWideMax);
  for (int i = 0; i < kTokRing; ++i) B2_CUDA(cudaEventCreateWithFlags(&e->tok_ring_done[i], cudaEventDisableTiming));
  B2_CUDA(cudaDeviceSynchronize());
  return e;
}

bool Executor::plan_chain() {
  if (!step_plan(model->dims, n_sms, smem_optin, max_num_tokens, &step)) return false;
  for (int nc : {1, step_cols}) {
    DecodeArgs p = dargs;
    p.ncols = nc;
    p.nterms = nc * 3 <= kQCols ? 3 : kQCols / nc;
    if (!step_prepare(p, step, model->layers_host.data(), kv_host.data())) return false;
  }
  return true;
}

bool Executor::plan_persistent(bool cooperative) {
  const ModelDims& d = model->dims;
  if (!cooperative) return false;
  for (float b : model->attn_bound)
    if (b > kFaMaxBound) return false;              // its attention shifts the softmax by the bound
  // staging halves take what shared memory the activation staging leaves, up to 96 KiB each
  const size_t fixed = stream_fixed_bytes(d, n_sessions);
  const long room = ((long)smem_optin - (long)fixed - 2048) / 2;   // margin: static shared memory
  const int half = (int)std::min<long>(room, 96 * 1024) / 1024 * 1024;
  if (half <= 0 || !stream_model_fits(d, dargs.o_slices, dargs.down_slices, half)) return false;
  const void* kfn = decode_stream_kernel_for(d);
  stream_half = half;
  stream_smem = fixed + 2 * (size_t)half;
  raise_dyn_smem(kfn, stream_smem);
  cudaFuncAttributes fa;
  B2_CUDA(cudaFuncGetAttributes(&fa, kfn));
  return fa.maxThreadsPerBlock >= kStreamThreads;
}

void Executor::tp_allreduce(float* buf, size_t count) {
  const NcclApi& nccl = NcclApi::get();
  nccl.check(nccl.AllReduce(buf, buf, count, kNcclFloat32, kNcclSum, tp_comm, stream), "ncclAllReduce");
}

// err, barrier and steps_done are adjacent
constexpr size_t kErrTail = sizeof(DecodeState) - offsetof(DecodeState, err);

void Executor::queue_device_error() {
  B2_CUDA(cudaMemcpyAsync(&pin_state->err, &dargs.st->err, kErrTail, cudaMemcpyDeviceToHost, stream));
}

void Executor::check_device_error(const char* where) {
  queue_device_error();
  B2_CUDA(cudaStreamSynchronize(stream));
  raise_device_error(where);
}

// The words queued by queue_device_error have arrived.
void Executor::raise_device_error(const char* where) {
  const int err = pin_state->err;
  if (err == kDevOk) return;
  B2_CUDA(cudaStreamSynchronize(stream));
  // clear the words and the barrier count so the handle stays usable
  B2_CUDA(cudaMemsetAsync(&dargs.st->err, 0, kErrTail, stream));
  B2_CUDA(cudaStreamSynchronize(stream));
  barrier_epoch = 0;
  std::string w(where);
  if (err == kDevBarrierTimeout) {
    throw Error{kDeadlineExceeded, w + ": a bounded device-side wait gave up"};
  }
  if (err == kDevBadToken) throw Error{kInvalidArgument, w + ": token id outside the vocabulary"};
  if (err == kDevBadPosition) throw Error{kInvalidArgument, w + ": position outside the KV capacity"};
  throw Error{kInternal, w + ": device error word " + std::to_string(err)};
}

// ------------------------------------------------------------------- prefill

// x += rmsnorm(sum of split-K partials) * g_post ; h = bf16(rmsnorm(x) * g_pre)
static void launch_resid_norm(cudaStream_t st, const float* parts, int nparts, int T, const ModelDims& d,
                              const float* g_post, const float* g_pre, float* xres, __nv_bfloat16* h) {
  const int d4 = d.d / 4;
  const size_t stride = (size_t)T * d.d;
  if (d4 <= 128 * 3)
    launch_pdl(pf_resid_norm_reg_kernel<128, 3, 4>, dim3(T), dim3(128), 0, st, parts, nparts, stride, d.d, d.eps, g_post, g_pre, xres, h);
  else if (d4 <= 256 * 3)
    launch_pdl(pf_resid_norm_reg_kernel<256, 3, 4>, dim3(T), dim3(256), 0, st, parts, nparts, stride, d.d, d.eps, g_post, g_pre, xres, h);
  else if (d4 <= 512 * 3)
    launch_pdl(pf_resid_norm_reg_kernel<512, 3, 4>, dim3(T), dim3(512), 0, st, parts, nparts, stride, d.d, d.eps, g_post, g_pre, xres, h);
  else
    pf_resid_norm_kernel<<<T, kPfThreads, sizeof(float) * d.d, st>>>(parts, nparts, stride, d.d, d.eps, g_post, g_pre,
                                                                    xres, h);
}

template <typename T>
static void launch_kv_append(cudaStream_t st, const ModelDims& d, int T_, const float* qkv, int nparts, int pos0, const int* pt,
                             const LayerWeights& L, const float* c, const float* s, const LayerKv& kv,
                             __nv_bfloat16* qout) {
  const int groups = (T_ + pos0 % kKvaTok + kKvaTok - 1) / kKvaTok;
  const int grid = groups * d.hkv + (qout ? (T_ * d.hq + kKvaTok - 1) / kKvaTok : 0);
  const size_t stride = (size_t)T_ * d.nqkv();
  launch_pdl(kv_append_kernel<T>(d), dim3(grid), dim3(kKvaThreads), 0, st, d, qkv, nparts, stride, T_, pos0, pt, L.g_k, c, s, kv, L.g_q, qout);
}

void Executor::run_prefill_chunk(const int* tokens, int T, int start) {
  const ModelDims& d = model->dims;
  B2_CHECK(T <= t_max, kInternal, "prefill chunk larger than the largest bucket");
  B2_CHECK(start + T <= max_num_tokens, kInvalidArgument,
           "Input token ids are too long. Exceeding the maximum number of tokens allowed: " +
               std::to_string(start + T) + " > " + std::to_string(max_num_tokens));
  // Token ids go through a ring of page-locked slices, one per queued chunk: a slice is rewritten only
  // after the host-to-device copy that reads it has completed (its event), so chunks queued back to
  // back without a wait (several work groups, wait_for_completion = false) never share staging memory.
  {
    const int slot = tok_ring_next;
    tok_ring_next = (tok_ring_next + 1) % kTokRing;
    if (tok_ring_used[slot]) B2_CUDA(cudaEventSynchronize(tok_ring_done[slot]));
    int* stage = pin_ints + (size_t)slot * t_pad;
    memcpy(stage, tokens, sizeof(int) * T);
    // the device-side id buffer is read by the first kernel of the chunk only; chunks are stream-ordered
    B2_CUDA(cudaMemcpyAsync(pf_tokens, stage, sizeof(int) * T, cudaMemcpyHostToDevice, stream));
    B2_CUDA(cudaEventRecord(tok_ring_done[slot], stream));
    tok_ring_used[slot] = true;
  }
  h2d_bytes += sizeof(int) * (size_t)T;
  int* err = &dargs.st->err;
  const int* ptab = page_table_dev + (size_t)active * pages_per_seq;     // the active session's pages
  const size_t sm_d = sizeof(float) * d.d;
  pf_embed_norm_kernel<<<T, kPfThreads, sm_d, stream>>>(pf_tokens, model->embed_rows, model->embed_scale,
                                                        model->layers_host[0].g_pre_attn, d.d, d.vocab, d.eps,
                                                        pf_xres, pf_h, err);
  ++launches;
  const int mode = prefill_gemm;
  const size_t attn_smem = sizeof(float) * ((size_t)(d.group() + 2) * d.hd + (size_t)8 * d.group() * (d.hd + 2));
  // split-K partials go to the partials buffer (8 x d floats per token); those of the QKV rows are summed by the append
  // kernel, but the CUDA-core attention reads whole rows, so it keeps one split
  int ks_q = 1, ks_o = 1, ks_d = 1;
  const int ch_q = gemm_chain(GemmRows::kNormed, d.d), ch_o = gemm_chain(GemmRows::kAttention, d.nq()), ch_d = gemm_chain(GemmRows::kGeglu, d.ffn);
  if (mode == B200LM_GEMM_TCGEN05) {
    if (attn_tc) ks_q = pick_ksplit(T, d.nqkv(), d.d, n_sms, std::max(1, 8 * d.d / d.nqkv()));
    ks_o = pick_ksplit(T, d.d, d.nq(), n_sms);
    ks_d = pick_ksplit(T, d.d, d.ffn, n_sms);
  }
  for (int li = 0; li < d.n_layers; ++li) {
    const LayerWeights& L = model->layers_host[li];
    const LayerGemmWeights& Gm = model->gemm_host[li];
    const float* cosT = model->rope_cos[L.is_global];
    const float* sinT = model->rope_sin[L.is_global];
    float* qkv_buf = ks_q > 1 ? pf_parts : pf_qkv;
    launch_gemm(stream, mode, tm_h, pf_h, L.wqkv, L.sqkv, Gm.wqkv, Gm.sqkv, T, d.nqkv(), d.d, ks_q, ch_q, false, qkv_buf,
                nullptr, err, &launches);
    __nv_bfloat16* qout = attn_tc ? pf_q : nullptr;
    if (d.kv_dtype == 0) launch_kv_append<float>(stream, d, T, qkv_buf, ks_q, start, ptab, L, cosT, sinT, kv_host[li], qout);
    else launch_kv_append<__nv_bfloat16>(stream, d, T, qkv_buf, ks_q, start, ptab, L, cosT, sinT, kv_host[li], qout);
    ++launches;
    if (attn_tc) {
      FaArgs fa{T, start, d.hq, d.hkv, d.window, L.is_global, ptab, pf_attn, model->attn_bound[li], err};
      const int TT = 128 / d.group();
      dim3 grid((T + TT - 1) / TT, d.hkv);
      if (d.hd == 256) launch_pdl(flash_prefill_tc_kernel<256>, grid, dim3(kFaThreads), FaSmem<256>::kTotal, stream, tm_q, tm_k[li], tm_vt[li], fa);
      else launch_pdl(flash_prefill_tc_kernel<128>, grid, dim3(kFaThreads), FaSmem<128>::kTotal, stream, tm_q, tm_k[li], tm_vt[li], fa);
      ++launches;
    } else {
    AttnJob j;
    memset(&j, 0, sizeof j);
    j.qkv = pf_qkv;
    j.pos = nullptr;
    j.pos0 = start;
    j.page_table = ptab;
    j.pages_per_seq = pages_per_seq;
    j.seq_stride = 0;
    j.is_global = L.is_global;
    j.nsplit = 1;
    j.appended = 1;
    j.g_q = L.g_q;
    j.g_k = L.g_k;
    j.cosT = cosT;
    j.sinT = sinT;
    j.kv = kv_host[li];
    j.out_bf16 = pf_attn;
    j.err = err;
    pf_attn_kernel<<<T * d.hkv, 256, attn_smem, stream>>>(d, j);
    ++launches;
    }
    launch_gemm(stream, mode, tm_attn, pf_attn, L.wo, L.so, Gm.wo, Gm.so, T, d.d, d.nq(), ks_o, ch_o, false, pf_parts,
                nullptr, err, &launches);
    if (tp_world > 1) tp_allreduce(pf_parts, (size_t)ks_o * T * d.d);
    launch_resid_norm(stream, pf_parts, ks_o, T, d, L.g_post_attn, L.g_pre_ffn, pf_xres, pf_h);
    ++launches;
    launch_gemm(stream, mode, tm_h, pf_h, L.wgu, L.sgu, Gm.wgu, Gm.sgu, T, 2 * d.ffn, d.d, 1, d.d, true, nullptr, pf_act,
                err, &launches);
    launch_gemm(stream, mode, tm_act, pf_act, L.wdown, L.sdown, Gm.wdown, Gm.sdown, T, d.d, d.ffn, ks_d, ch_d, false,
                pf_parts, nullptr, err, &launches);
    if (tp_world > 1) tp_allreduce(pf_parts, (size_t)ks_d * T * d.d);
    const float* g_next = li + 1 < d.n_layers ? model->layers_host[li + 1].g_pre_attn : nullptr;
    launch_resid_norm(stream, pf_parts, ks_d, T, d, L.g_post_ffn, g_next, pf_xres, pf_h);
    ++launches;
  }
  B2_CUDA(cudaGetLastError());
}

// llm_litert_compiled_model_executor.cc:157-276: a group of `len` ids runs the
// pending id (if any) followed by ids[0..len-2]; ids[len-1] becomes pending.
void Executor::prefill_group(const int* ids, int len) {
  std::vector<int> run;
  run.reserve(len);
  int start = current_step;
  for (int i = 0; i < len - 1;) {
    if (next_input_token != -1) {
      run.push_back(next_input_token);
      next_input_token = -1;
    } else {
      run.push_back(ids[i++]);
    }
    ++current_step;
  }
  next_input_token = ids[len - 1];
  if (!run.empty()) run_prefill_chunk(run.data(), (int)run.size(), start);
}

void Executor::prefill(const int* ids, int n, bool wait, const volatile int* cancel) {
  B2_CHECK(ids != nullptr, kInvalidArgument, "ids is null");
  B2_CHECK(n > 0, kInternal, "Prefill token ids must be non-empty.");
  B2_CUDA(cudaSetDevice(device));
  const ModelDims& d = model->dims;
  // Same bound the caller loop enforces before it reaches the executor
  // (runtime/core/pipeline.cc:249-255), checked before any work is queued.
  const int would_run = n - 1 + (next_input_token != -1 ? 1 : 0);
  B2_CHECK(current_step + would_run <= max_num_tokens, kInvalidArgument,
           "Input token ids are too long. Exceeding the maximum number of tokens allowed: " +
               std::to_string(current_step + would_run) + " > " + std::to_string(max_num_tokens));
  auto groups = plan_work_groups(d.buckets, d.n_buckets, n);
  last_plan = groups;
  int used = 0;
  for (auto& g : groups) {
    if (cancel && *cancel) throw Error{kCancelled, "Prefill cancelled."};
    prefill_group(ids + used, g.second);
    used += g.second;
  }
  B2_CHECK(used == n, kInternal, "Work groups not covering the entire prefill input.");
  if (wait) check_device_error("Prefill");
}

// -------------------------------------------------------------------- decode

// ncols sessions advance together, starting at `first_session` (default: the active one alone).
void Executor::launch_decode_steps(int nsteps, int ncols, int first_session) {
  const ModelDims& d = model->dims;
  const int ncta = n_sms;
  if (first_session < 0) first_session = active;
  if (decode_mode == B200LM_DECODE_WIDE) {
    launch_wide_steps(nsteps, ncols, first_session);
    return;
  }
  if (!chain) {
    DecodeArgs a = dargs;
    a.ncols = ncols;
    a.nterms = ncols * 3 <= kQCols ? 3 : kQCols / ncols;      // int8 terms per activation: 3, or 2 with 3-4 sessions
    a.page_table = page_table_dev + (size_t)first_session * pages_per_seq;
    // one CTA per (session, kv head, split)
    const int cap = std::max(1, ncta / (ncols * d.hkv));
    a.n_attn_splits_local = std::min(a.n_attn_splits_local, cap);
    a.n_attn_splits_global = std::min(a.n_attn_splits_global, cap);
    if (decode_mode == B200LM_DECODE_PHASE_KERNELS) {
      launch_phases(nsteps, a);
      return;
    }
    unsigned epoch0 = barrier_epoch;
    if (decode_mode == B200LM_DECODE_PERSISTENT) {
      int half = stream_half;
      void* params[] = {&a, &nsteps, &epoch0, &half};
      B2_CUDA(cudaLaunchCooperativeKernel(decode_stream_kernel_for(d), dim3(ncta), dim3(kStreamThreads), params,
                                          stream_smem, stream));
    } else {
      void* params[] = {&a, &nsteps, &epoch0};
      B2_CUDA(cudaLaunchCooperativeKernel((void*)decode_persistent_kernel, dim3(ncta), dim3(kDecThreads), params,
                                          dec_smem, stream));
    }
    barrier_epoch += (unsigned)nsteps * (unsigned)(5 * d.n_layers + 2) * (unsigned)ncta;
    launches += 1;
    return;
  }
  launch_chain(nsteps, ncols, first_session);
}

// The phases of the persistent kernel launched one by one, with the ranks' partial O and down outputs summed in between.
void Executor::launch_phases(int nsteps, const DecodeArgs& a) {
  const ModelDims& d = model->dims;
  for (int s = 0; s < nsteps; ++s) {
    for (int li = 0; li < d.n_layers; ++li)
      for (int ph = kPhQkv; ph <= kPhDown; ++ph) {
        decode_phase_kernel<<<n_sms, kDecThreads, dec_smem, stream>>>(a, ph, li);
        if (tp_world > 1 && ph == kPhOproj) tp_allreduce(a.opart, (size_t)a.o_slices * a.ncols * d.d);
        if (tp_world > 1 && ph == kPhDown) tp_allreduce(a.fpart, (size_t)a.down_slices * a.ncols * d.d);
      }
    decode_phase_kernel<<<n_sms, kDecThreads, dec_smem, stream>>>(a, kPhHead, 0);
    decode_phase_kernel<<<1, kDecThreads, dec_smem, stream>>>(a, kPhArgmax, n_sms);
  }
  B2_CUDA(cudaGetLastError());
  launches += (int64_t)nsteps * (5 * d.n_layers + 2);
}

// What `body` queues on `stream`, as a graph.  A caller's stream is not captured, but one made for that: the caller's may
// be the legacy default stream, which cannot be captured, or a blocking one, whose capture would make other threads' work
// on the default stream fail.  (Not for the executor's own stream: making and destroying one takes about 200 us.)
template <typename Body>
cudaGraph_t Executor::capture(const Body& body) {
  cudaStream_t rec = stream;
  cudaGraph_t graph = nullptr;
  if (!own_stream) B2_CUDA(cudaStreamCreateWithFlags(&rec, cudaStreamNonBlocking));
  std::swap(stream, rec);
  auto done = [&]() {
    std::swap(stream, rec);
    if (!own_stream) cudaStreamDestroy(rec);
  };
  try {
    B2_CUDA(cudaStreamBeginCapture(stream, cudaStreamCaptureModeThreadLocal));
    try {
      body();
    } catch (...) {
      if (cudaStreamEndCapture(stream, &graph) == cudaSuccess && graph) cudaGraphDestroy(graph);
      throw;
    }
    B2_CUDA(cudaStreamEndCapture(stream, &graph));
  } catch (...) {
    done();
    throw;
  }
  done();
  return graph;
}

// The chain of step kernels for sessions [first, first + ncols).  Under tensor parallelism
// the ranks' partial O and down outputs are summed between the kernels, launch by launch.
void Executor::launch_chain(int nsteps, int ncols, int first) {
  DecodeArgs a = dargs;
  a.ncols = ncols;
  a.nterms = ncols * 3 <= kQCols ? 3 : kQCols / ncols;      // int8 terms per activation: 3, or 2 with 3-4 sessions
  a.page_table = page_table_dev + (size_t)first * pages_per_seq;
  const LayerWeights* L = model->layers_host.data();
  if (tp_world > 1) {
    auto reduce = [](void* self, float* buf, size_t count) { static_cast<Executor*>(self)->tp_allreduce(buf, count); };
    for (int s = 0; s < nsteps; ++s) launches += step_launch(stream, a, step, L, kv_host.data(), reduce, this);
    return;
  }
  if (dargs.trace) {                          // a timeline is taken once: not worth a graph of its own
    for (int s = 0; s < nsteps; ++s) launches += step_launch(stream, a, step, L, kv_host.data(), nullptr, nullptr);
    return;
  }
  // Replaying the step as one graph saves 45 of 640 us (131 launches of the 1B model), but the host takes 75 us to capture
  // it, 270 to instantiate it and 220 to upload it, and the first call of every executor used to wait for all of that
  // (1102 us for the first DecodeLogits against 652 now).  So the steps start as plain launches, which take the host 430
  // us, and each part is done while the GPU runs one of them: an executor that decodes one step never makes a graph.
  StepGraph& g = step_graphs[std::make_pair(ncols, first)];
  for (int s = 0; s < nsteps; ++s) {
    if (g.steps >= 4 && g.exec) {
      B2_CUDA(cudaGraphLaunch(g.exec, stream));
      launches += 5 * model->dims.n_layers + 1;
      continue;
    }
    launches += step_launch(stream, a, step, L, kv_host.data(), nullptr, nullptr);
    ++g.steps;
    if (g.steps == 2) {
      g.graph = capture([&] { step_launch(stream, a, step, L, kv_host.data(), nullptr, nullptr); });
    } else if (g.steps == 3 && g.graph) {
      B2_CUDA(cudaGraphInstantiate(&g.exec, g.graph, 0));
      cudaGraphDestroy(g.graph);
      g.graph = nullptr;
    } else if (g.steps == 4 && g.exec) {
      B2_CUDA(cudaGraphUpload(g.exec, stream));
    }
  }
}

// One wide step for sessions [first, first + nb): the token rows of the GEMMs are the sessions.
void Executor::wide_step(int nb, int first) {
  const ModelDims& d = model->dims;
  int* err = &dargs.st->err;
  const int mode = B200LM_GEMM_TCGEN05;
  // key splits so that few sessions still fill the SMs with two CTAs each: one per (session, kv head, split)
  const int nsplit = std::max(1, std::min(kWideMaxSplits, 2 * n_sms / std::max(1, nb * d.hkv)));
  launch_pdl(pf_embed_norm_kernel, dim3(nb), dim3(kPfThreads), sizeof(float) * d.d, stream, wide.tok, model->embed_rows, model->embed_scale,
             model->layers_host[0].g_pre_attn, d.d, d.vocab, d.eps, pf_xres, pf_h, err);
  int64_t* nl = &launches;
  ++*nl;
  // split K so that the few token rows still spread the weight tiles over the SMs; the attention adds the QKV rows' parts
  const int ks_q = pick_ksplit(nb, d.nqkv(), d.d, n_sms, std::max(1, 8 * d.d / d.nqkv()));
  const int ks_o = pick_ksplit(nb, d.d, d.nq(), n_sms), ks_d = pick_ksplit(nb, d.d, d.ffn, n_sms);
  const int ch_q = gemm_chain(GemmRows::kNormed, d.d), ch_o = gemm_chain(GemmRows::kAttention, d.nq()), ch_d = gemm_chain(GemmRows::kGeglu, d.ffn);
  for (int li = 0; li < d.n_layers; ++li) {
    const LayerWeights& L = model->layers_host[li];
    const LayerGemmWeights& Gm = model->gemm_host[li];
    launch_gemm(stream, mode, tm_h, pf_h, L.wqkv, L.sqkv, Gm.wqkv, Gm.sqkv, nb, d.nqkv(), d.d, ks_q, ch_q, false,
                ks_q > 1 ? pf_parts : pf_qkv, nullptr, err, nl);
    WideAttnArgs wa{ks_q > 1 ? pf_parts : pf_qkv, wide.pos, page_table_dev + (size_t)first * pages_per_seq, pages_per_seq, L.is_global, nsplit, 0,
                    L.g_q, L.g_k, model->rope_cos[L.is_global], model->rope_sin[L.is_global], kv_host[li], wide_part, wide_ticket, pf_attn, err,
                    1, 0, nullptr, 2, ks_q, (size_t)nb * d.nqkv()};
    launch_wide_attn(stream, d, nb, smem_optin, wa);         // sums the projections' partials as it reads them
    ++*nl;
    launch_gemm(stream, mode, tm_attn, pf_attn, L.wo, L.so, Gm.wo, Gm.so, nb, d.d, d.nq(), ks_o, ch_o, false, pf_parts, nullptr, err, nl);
    launch_resid_norm(stream, pf_parts, ks_o, nb, d, L.g_post_attn, L.g_pre_ffn, pf_xres, pf_h);
    ++*nl;
    launch_gemm(stream, mode, tm_h, pf_h, L.wgu, L.sgu, Gm.wgu, Gm.sgu, nb, 2 * d.ffn, d.d, 1, d.d, true, nullptr, pf_act, err, nl);
    launch_gemm(stream, mode, tm_act, pf_act, L.wdown, L.sdown, Gm.wdown, Gm.sdown, nb, d.d, d.ffn, ks_d, ch_d, false, pf_parts, nullptr,
                err, nl);
    const float* g_next = li + 1 < d.n_layers ? model->layers_host[li + 1].g_pre_attn : model->g_final;
    launch_resid_norm(stream, pf_parts, ks_d, nb, d, L.g_post_ffn, g_next, pf_xres, pf_h);
    ++*nl;
  }
  launch_gemm(stream, mode, tm_h, pf_h, model->head_w, model->embed_scale, model->head_g, model->head_gs, nb, d.vocab, d.d, 1, d.d, false, dargs.logits,
              nullptr, err, nl);
  const int arg_parts = std::max(1, std::min(kWideArgParts, 2 * n_sms / nb));
  launch_pdl(wide_argmax_kernel, dim3(nb * arg_parts), dim3(kWideArgThreads), 0, stream, dargs.logits, d.vocab, nb, arg_parts, wide, dargs.step_tokens);
  ++*nl;
  B2_CUDA(cudaGetLastError());
}

void Executor::launch_wide_steps(int nsteps, int nb, int first) {
  B2_CHECK(nb >= 1 && nb <= kWideMax && first >= 0 && first + nb <= n_sessions, kInternal, "wide step outside the sessions");
  B2_CHECK(model->head_g != nullptr, kFailedPrecondition, "the wide decode mode needs the tensor-core GEMM weights");
  if (nsteps == 1) {                                 // a single step is not worth a capture
    wide_step(nb, first);
    return;
  }
  auto key = std::make_pair(nb, first);
  auto it = wide_graphs.find(key);
  if (it == wide_graphs.end()) {
    const int64_t before = launches;
    cudaGraph_t graph = capture([&] { wide_step(nb, first); });
    cudaGraphExec_t exec = nullptr;
    B2_CUDA(cudaGraphInstantiate(&exec, graph, 0));
    cudaGraphDestroy(graph);
    wide_per_step = launches - before;
    launches = before;
    it = wide_graphs.emplace(key, exec).first;
  }
  for (int s = 0; s < nsteps; ++s) B2_CUDA(cudaGraphLaunch(it->second, stream));
  launches += (int64_t)nsteps * wide_per_step;
}

void Executor::push_decode_state(const int* tokens, const int* pos, int ncols) {
  if (decode_mode == B200LM_DECODE_WIDE) {
    B2_CUDA(cudaStreamSynchronize(stream));        // the staging words of the previous call have been read
    for (int c = 0; c < ncols; ++c) {
      pin_wide[c] = tokens[c];
      pin_wide[kWideMax + c] = pos[c];
      pin_wide[2 * kWideMax + c] = pos[c];
    }
    B2_CUDA(cudaMemcpyAsync(wide.tok, pin_wide, sizeof(int) * 3 * kWideMax, cudaMemcpyHostToDevice, stream));
    h2d_bytes += 2 * sizeof(int) * (size_t)ncols;
    return;
  }
  DecodeState* ps = pin_state;
  memset(ps, 0, sizeof(DecodeState));
  for (int c = 0; c < ncols; ++c) {
    ps->token[c] = tokens[c];
    ps->pos[c] = pos[c];
  }
  // token, pos, out_token: the first three arrays; err / barrier / steps_done handled separately
  B2_CUDA(cudaMemcpyAsync(dargs.st, ps, offsetof(DecodeState, err), cudaMemcpyHostToDevice, stream));
  B2_CUDA(cudaMemsetAsync(&dargs.st->steps_done, 0, sizeof(int), stream));
  h2d_bytes += 2 * sizeof(int) * (size_t)ncols;
}

int Executor::take_decode_id(const int* id_or_null) {
  int id = next_input_token;
  if (id_or_null) id = *id_or_null;
  B2_CHECK(id != -1, kInvalidArgument, "No id available to be decoded.");
  next_input_token = -1;
  B2_CHECK(current_step < max_num_tokens, kInvalidArgument, "Maximum kv-cache size reached.");
  return id;
}

void Executor::decode_logits(const int* id_or_null, float* host_logits) {
  B2_CHECK(host_logits != nullptr, kInvalidArgument, "logits destination is null");
  B2_CUDA(cudaSetDevice(device));
  int id = take_decode_id(id_or_null);
  push_decode_state(&id, &current_step, 1);
  launch_decode_steps(1);
  const size_t nb = sizeof(float) * (size_t)model->dims.vocab;
  // a page-locked destination takes the copy directly; pageable memory goes through the pinned staging
  cudaPointerAttributes pa{};
  const bool direct = cudaPointerGetAttributes(&pa, host_logits) == cudaSuccess && pa.type == cudaMemoryTypeHost;
  if (!direct) cudaGetLastError();
  d2h_bytes += nb;
  if (direct) {
    B2_CUDA(cudaMemcpyAsync(host_logits, dargs.logits, nb, cudaMemcpyDeviceToHost, stream));
    check_device_error("DecodeLogits");
  } else {
    // In parts, so that one part's copy out of the staging runs under the next one's transfer: 1 MB is 20 us on the bus
    // and as much again and more in the host's memory.  A part below 64 KB would cost more in calls than it hides.
    const int parts = (int)std::min<size_t>(kLogitParts, std::max<size_t>(1, nb / (64 << 10)));
    const size_t per = (nb / parts + 63) / 64 * 64;
    queue_device_error();
    for (int p = 0; p < parts; ++p) {
      const size_t off = std::min(nb, p * per), len = p + 1 < parts ? std::min(per, nb - off) : nb - off;
      B2_CUDA(cudaMemcpyAsync(reinterpret_cast<unsigned char*>(pin_logits) + off, reinterpret_cast<const unsigned char*>(dargs.logits) + off, len,
                              cudaMemcpyDeviceToHost, stream));
      if (!logit_part[p]) B2_CUDA(cudaEventCreateWithFlags(&logit_part[p], cudaEventDisableTiming));
      B2_CUDA(cudaEventRecord(logit_part[p], stream));
    }
    for (int p = 0; p < parts; ++p) {
      const size_t off = std::min(nb, p * per), len = p + 1 < parts ? std::min(per, nb - off) : nb - off;
      B2_CUDA(cudaEventSynchronize(logit_part[p]));
      if (p == 0) raise_device_error("DecodeLogits");
      memcpy(reinterpret_cast<unsigned char*>(host_logits) + off, reinterpret_cast<const unsigned char*>(pin_logits) + off, len);
    }
  }
  ++current_step;
}

void Executor::decode_tokens(int nsteps, int* out_ids) {
  B2_CHECK(nsteps > 0, kInvalidArgument, "n_steps must be positive");
  B2_CUDA(cudaSetDevice(device));
  B2_CHECK(current_step + nsteps <= max_num_tokens, kInvalidArgument, "Maximum kv-cache size reached.");
  int id = take_decode_id(nullptr);
  push_decode_state(&id, &current_step, 1);
  launch_decode_steps(nsteps);
  int* dst = pin_steps;
  B2_CUDA(cudaMemcpyAsync(dst, dargs.step_tokens, sizeof(int) * (size_t)nsteps, cudaMemcpyDeviceToHost, stream));
  d2h_bytes += sizeof(int) * (size_t)nsteps;
  check_device_error("Decode");
  for (int s = 0; s < nsteps; ++s) {
    int t = dst[s];
    if (t < 0) t = 0;   // "The sampled token is casted to 0 to avoid crash."
    if (out_ids) out_ids[s] = t;
    next_input_token = t;
  }
  current_step += nsteps;
}

// All sessions take `nsteps` greedy steps together: one pass over the weights per step.
void Executor::decode_tokens_batch(int nsteps, int* out_ids) {
  B2_CHECK(nsteps > 0, kInvalidArgument, "n_steps must be positive");
  B2_CUDA(cudaSetDevice(device));
  const int keep = active;
  std::vector<int> tok(n_sessions), pos(n_sessions);
  for (int sn = 0; sn < n_sessions; ++sn) {        // validate every session before any state changes
    const int pending = sn == active ? next_input_token : parked[sn].next_input_token;
    const int step = sn == active ? current_step : parked[sn].current_step;
    B2_CHECK(pending != -1, kInvalidArgument, "No id available to be decoded (session " + std::to_string(sn) + ").");
    B2_CHECK(step + nsteps <= max_num_tokens, kInvalidArgument, "Maximum kv-cache size reached.");
  }
  if (step_cols < n_sessions) {                    // the step's kernels carry one session of this geometry at a time
    std::vector<int> ids(nsteps);
    for (int sn = 0; sn < n_sessions; ++sn) {
      select_session(sn);
      decode_tokens(nsteps, ids.data());
      for (int s = 0; out_ids && s < nsteps; ++s) out_ids[(size_t)s * n_sessions + sn] = ids[s];
    }
    select_session(keep);
    return;
  }
  for (int sn = 0; sn < n_sessions; ++sn) {
    select_session(sn);
    tok[sn] = take_decode_id(nullptr);
    pos[sn] = current_step;
  }
  push_decode_state(tok.data(), pos.data(), n_sessions);
  launch_decode_steps(nsteps, n_sessions, 0);
  int* dst = pin_steps;
  B2_CUDA(cudaMemcpyAsync(dst, dargs.step_tokens, sizeof(int) * (size_t)nsteps * n_sessions, cudaMemcpyDeviceToHost,
                          stream));
  d2h_bytes += sizeof(int) * (size_t)nsteps * n_sessions;
  check_device_error("Decode");
  for (int sn = 0; sn < n_sessions; ++sn) {
    select_session(sn);
    for (int s = 0; s < nsteps; ++s) {
      int t = dst[(size_t)s * n_sessions + sn];
      if (t < 0) t = 0;
      if (out_ids) out_ids[(size_t)s * n_sessions + sn] = t;
      next_input_token = t;
    }
    current_step += nsteps;
  }
  select_session(keep);
}

void Executor::trace_decode_step(int* out_id, long long* stamps, long long capacity, int* n_barriers, int* n_cta,
                                 int* khz) {
  const ModelDims& d = model->dims;
  B2_CHECK(chain || decode_mode == B200LM_DECODE_PERSISTENT || decode_mode == B200LM_DECODE_PERSISTENT_BASIC, kFailedPrecondition,
           "the wide decode mode and one kernel per phase have no timeline");
  B2_CUDA(cudaSetDevice(device));
  const int nb = 5 * d.n_layers + 2;
  const long long need = (long long)nb * n_sms * 10;     // 2 barrier stamps + 8 in-phase stamps
  B2_CHECK(stamps != nullptr && capacity >= need, kInvalidArgument,
           "stamps must hold " + std::to_string(need) + " int64 values");
  if (!trace_dev) trace_dev = reinterpret_cast<long long*>(alloc(sizeof(long long) * need, true));
  B2_CUDA(cudaMemsetAsync(trace_dev, 0, sizeof(long long) * need, stream));
  dargs.trace = trace_dev;
  dargs.trace_pts = trace_dev + (size_t)nb * n_sms * 2;
  dargs.trace_ctas = n_sms;
  try {
    decode_tokens(1, out_id);
  } catch (...) {
    dargs.trace = nullptr;
    dargs.trace_pts = nullptr;
    throw;
  }
  dargs.trace = nullptr;
  dargs.trace_pts = nullptr;
  B2_CUDA(cudaMemcpy(stamps, trace_dev, sizeof(long long) * need, cudaMemcpyDeviceToHost));
  *n_barriers = nb;
  *n_cta = n_sms;
  int rate = 0;
  B2_CUDA(cudaDeviceGetAttribute(&rate, cudaDevAttrClockRate, device));
  // the chain's kernels stamp nanoseconds: their CTAs move between SMs, whose cycle counters differ
  *khz = chain ? 1000000 : rate;
}

void Executor::reset() {
  current_step = 0;
  next_input_token = -1;
}

void Executor::select_session(int session) {
  B2_CHECK(session >= 0 && session < n_sessions, kInvalidArgument,
           "session " + std::to_string(session) + " out of range (the executor has " + std::to_string(n_sessions) + ")");
  if (session == active) return;
  parked[active] = SessionState{current_step, next_input_token, last_plan};
  current_step = parked[session].current_step;
  next_input_token = parked[session].next_input_token;
  last_plan = parked[session].last_plan;
  active = session;
}

void Executor::read_kv_row(int layer, int is_v, int kv_head, int pos, float* out, int* page, int* slot) {
  const ModelDims& d = model->dims;
  B2_CHECK(layer >= 0 && layer < d.n_layers && kv_head >= 0 && kv_head < d.hkv && pos >= 0 && pos < d.max_ctx,
           kInvalidArgument, "KV row index out of range");
  B2_CUDA(cudaSetDevice(device));
  B2_CUDA(cudaStreamSynchronize(stream));
  int pg = page_table_host[(size_t)active * pages_per_seq + pos / kPage], sl = pos % kPage;
  size_t off = (((size_t)pg * d.hkv + kv_head) * kPage + sl) * d.hd;
  const void* base = is_v ? kv_host[layer].v : kv_host[layer].k;
  if (d.kv_dtype == 0) {
    B2_CUDA(cudaMemcpy(out, reinterpret_cast<const float*>(base) + off, sizeof(float) * d.hd, cudaMemcpyDeviceToHost));
  } else {
    std::vector<__nv_bfloat16> tmp(d.hd);
    B2_CUDA(cudaMemcpy(tmp.data(), reinterpret_cast<const __nv_bfloat16*>(base) + off, 2 * d.hd, cudaMemcpyDeviceToHost));
    for (int i = 0; i < d.hd; ++i) out[i] = __bfloat162float(tmp[i]);
  }
  if (page) *page = pg;
  if (slot) *slot = sl;
}

}  // namespace b200lm

// ===================================================================== C ABI

using namespace b200lm;

struct B200LmExecutor {
  std::unique_ptr<Executor> impl;
};

static int fail(char** err, int code, const std::string& msg) {
  if (err) {
    *err = reinterpret_cast<char*>(malloc(msg.size() + 1));
    if (*err) memcpy(*err, msg.c_str(), msg.size() + 1);
  }
  return code;
}

#define B2_API_BEGIN \
  if (err) *err = nullptr; \
  try {
#define B2_API_END                                                     \
  }                                                                    \
  catch (const Error& e_) { return fail(err, e_.code, e_.msg); }       \
  catch (const std::exception& e_) { return fail(err, kInternal, e_.what()); } \
  catch (...) { return fail(err, kInternal, "unknown failure"); }      \
  return kOk;

static void require_gpu(int device) {
  int n = 0;
  cudaError_t r = cudaGetDeviceCount(&n);
  if (r != cudaSuccess || n <= 0) {
    cudaGetLastError();
    throw Error{kFailedPrecondition, "no CUDA device: this backend has no CPU fallback"};
  }
  B2_CHECK(device >= 0 && device < n, kInvalidArgument, "device ordinal out of range");
}

static B200LmConfig effective_config(const B200LmConfig* c) {
  B200LmConfig cfg;
  memset(&cfg, 0, sizeof cfg);
  if (c) memcpy(&cfg, c, std::min<size_t>(sizeof cfg, c->struct_size > 0 ? (size_t)c->struct_size : sizeof cfg));
  return cfg;
}

extern "C" {

int B200Lm_Create(const B200LmConfig* config, const void* bytes, uint64_t n_bytes, const char* path,
                  B200LmExecutor** out, char** err) {
  B2_API_BEGIN
  B2_CHECK(out != nullptr, kInvalidArgument, "out is null");
  *out = nullptr;
  B200LmConfig cfg = effective_config(config);
  std::vector<uint8_t> file;
  const uint8_t* p = reinterpret_cast<const uint8_t*>(bytes);
  if (!p) {
    B2_CHECK(path != nullptr, kInvalidArgument, "neither bytes nor a path were given");
    std::ifstream f(path, std::ios::binary | std::ios::ate);
    B2_CHECK(f.good(), kNotFound, std::string("cannot open ") + path);
    std::streamsize sz = f.tellg();
    f.seekg(0);
    file.resize((size_t)sz);
    f.read(reinterpret_cast<char*>(file.data()), sz);
    B2_CHECK(f.good(), kInternal, std::string("cannot read ") + path);
    p = file.data();
    n_bytes = (uint64_t)sz;
  }
  // Parse first: malformed input is reported as such even without a GPU.
  (void)locate_weights(p, (size_t)n_bytes);
  require_gpu(cfg.device);
  auto model = Model::load(p, (size_t)n_bytes, cfg.device, cfg.prefill_gemm != B200LM_GEMM_CHECK);
  auto h = new B200LmExecutor();
  try {
    h->impl = Executor::create(model, cfg);
  } catch (...) {
    delete h;
    throw;
  }
  *out = h;
  B2_API_END
}

int B200Lm_CreateShared(B200LmExecutor* owner, const B200LmConfig* config, B200LmExecutor** out, char** err) {
  B2_API_BEGIN
  B2_CHECK(owner && owner->impl && out, kInvalidArgument, "null handle");
  B200LmConfig cfg = effective_config(config);
  cfg.device = owner->impl->device;
  auto h = new B200LmExecutor();
  try {
    h->impl = Executor::create(owner->impl->model, cfg);
  } catch (...) {
    delete h;
    throw;
  }
  *out = h;
  B2_API_END
}

void B200Lm_Destroy(B200LmExecutor* e) { delete e; }

int B200Lm_Prefill(B200LmExecutor* e, const int32_t* ids, int32_t n, int32_t wait, const volatile int32_t* cancel,
                   char** err) {
  B2_API_BEGIN
  B2_CHECK(e && e->impl, kInvalidArgument, "null handle");
  e->impl->prefill(ids, n, wait != 0, cancel);
  B2_API_END
}

int B200Lm_DecodeLogits(B200LmExecutor* e, const int32_t* id, float* logits, char** err) {
  B2_API_BEGIN
  B2_CHECK(e && e->impl, kInvalidArgument, "null handle");
  e->impl->decode_logits(id, logits);
  B2_API_END
}

int B200Lm_DecodeToken(B200LmExecutor* e, int32_t* out_id, char** err) {
  B2_API_BEGIN
  B2_CHECK(e && e->impl && out_id, kInvalidArgument, "null argument");
  e->impl->decode_tokens(1, out_id);
  B2_API_END
}

int B200Lm_DecodeTokens(B200LmExecutor* e, int32_t n_steps, int32_t* out_ids, char** err) {
  B2_API_BEGIN
  B2_CHECK(e && e->impl, kInvalidArgument, "null handle");
  e->impl->decode_tokens(n_steps, out_ids);
  B2_API_END
}

int B200Lm_PrefillSession(B200LmExecutor* e, int32_t session, const int32_t* ids, int32_t n, int32_t wait_for_completion,
                          const volatile int32_t* cancel_or_null, char** err) {
  B2_API_BEGIN
  B2_CHECK(e && e->impl, kInvalidArgument, "null handle");
  e->impl->select_session(session);
  e->impl->prefill(ids, n, wait_for_completion != 0, reinterpret_cast<const volatile int*>(cancel_or_null));
  B2_API_END
}

int B200Lm_DecodeTokensBatch(B200LmExecutor* e, int32_t n_steps, int32_t* out_ids, char** err) {
  B2_API_BEGIN
  B2_CHECK(e && e->impl, kInvalidArgument, "null handle");
  e->impl->decode_tokens_batch(n_steps, out_ids);
  B2_API_END
}

int B200Lm_SelectSession(B200LmExecutor* e, int32_t session, char** err) {
  B2_API_BEGIN
  B2_CHECK(e && e->impl, kInvalidArgument, "null handle");
  e->impl->select_session(session);
  B2_API_END
}

int B200Lm_GetNumSessions(B200LmExecutor* e, int32_t* out, char** err) {
  B2_API_BEGIN
  B2_CHECK(e && e->impl && out, kInvalidArgument, "null argument");
  *out = e->impl->n_sessions;
  B2_API_END
}

int B200Lm_Reset(B200LmExecutor* e, char** err) {
  B2_API_BEGIN
  B2_CHECK(e && e->impl, kInvalidArgument, "null handle");
  e->impl->reset();
  B2_API_END
}

int B200Lm_GetVocabSize(B200LmExecutor* e, int32_t* out, char** err) {
  B2_API_BEGIN
  B2_CHECK(e && e->impl && out, kInvalidArgument, "null argument");
  *out = e->impl->model->dims.vocab;
  B2_API_END
}

int B200Lm_GetCurrentStep(B200LmExecutor* e, int32_t* out, char** err) {
  B2_API_BEGIN
  B2_CHECK(e && e->impl && out, kInvalidArgument, "null argument");
  *out = e->impl->current_step + (e->impl->next_input_token == -1 ? 0 : 1);
  B2_API_END
}

int B200Lm_GetMaxNumTokens(B200LmExecutor* e, int32_t* out, char** err) {
  B2_API_BEGIN
  B2_CHECK(e && e->impl && out, kInvalidArgument, "null argument");
  *out = e->impl->max_num_tokens;
  B2_API_END
}

int B200Lm_TpUniqueId(void* out, char** err) {
  B2_API_BEGIN
  B2_CHECK(out != nullptr, kInvalidArgument, "out is null");
  const NcclApi& nccl = NcclApi::get();
  NcclApi::UniqueId id;
  nccl.check(nccl.GetUniqueId(&id), "ncclGetUniqueId");
  memcpy(out, &id, sizeof id);
  B2_API_END
}

int B200Lm_TpAllReduceProbe(B200LmExecutor* e, int64_t count, int32_t iters, float* ms_out, char** err) {
  B2_API_BEGIN
  B2_CHECK(e && e->impl && ms_out && count > 0 && iters > 0, kInvalidArgument, "bad argument");
  Executor& x = *e->impl;
  B2_CHECK(x.tp_world > 1, kFailedPrecondition, "this executor is not tensor-parallel");
  B2_CUDA(cudaSetDevice(x.device));
  float* buf = nullptr;
  B2_CUDA(cudaMalloc(&buf, sizeof(float) * (size_t)count));
  B2_CUDA(cudaMemsetAsync(buf, 0, sizeof(float) * (size_t)count, x.stream));
  cudaEvent_t e0, e1;
  B2_CUDA(cudaEventCreate(&e0));
  B2_CUDA(cudaEventCreate(&e1));
  for (int i = 0; i < 3; ++i) x.tp_allreduce(buf, (size_t)count);
  B2_CUDA(cudaEventRecord(e0, x.stream));
  for (int i = 0; i < iters; ++i) x.tp_allreduce(buf, (size_t)count);
  B2_CUDA(cudaEventRecord(e1, x.stream));
  B2_CUDA(cudaEventSynchronize(e1));
  float ms = 0.f;
  B2_CUDA(cudaEventElapsedTime(&ms, e0, e1));
  *ms_out = ms / (float)iters;
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFree(buf);
  B2_API_END
}

int B200Lm_GetDecodeMode(B200LmExecutor* e, int32_t* out, char** err) {
  B2_API_BEGIN
  B2_CHECK(e && e->impl && out, kInvalidArgument, "null argument");
  *out = e->impl->decode_mode;
  B2_API_END
}

const char* B200Lm_BackendName(void) { return "B200 CUDA (sm_100a)"; }

int B200Lm_Synchronize(B200LmExecutor* e, char** err) {
  B2_API_BEGIN
  B2_CHECK(e && e->impl, kInvalidArgument, "null handle");
  B2_CUDA(cudaSetDevice(e->impl->device));
  e->impl->check_device_error("Synchronize");
  B2_API_END
}

int B200Lm_GetLastPrefillPlan(B200LmExecutor* e, int32_t* buckets, int32_t* lengths, int32_t capacity,
                              int32_t* n_groups, char** err) {
  B2_API_BEGIN
  B2_CHECK(e && e->impl && n_groups, kInvalidArgument, "null argument");
  const auto& plan = e->impl->last_plan;
  *n_groups = (int32_t)plan.size();
  for (int i = 0; i < (int)plan.size() && i < capacity; ++i) {
    if (buckets) buckets[i] = plan[i].first;
    if (lengths) lengths[i] = plan[i].second;
  }
  B2_API_END
}

int B200Lm_ReadKvRow(B200LmExecutor* e, int32_t layer, int32_t is_v, int32_t kv_head, int32_t pos, float* out_row,
                     int32_t* out_page, int32_t* out_slot, char** err) {
  B2_API_BEGIN
  B2_CHECK(e && e->impl && out_row, kInvalidArgument, "null argument");
  e->impl->read_kv_row(layer, is_v, kv_head, pos, out_row, out_page, out_slot);
  B2_API_END
}

int B200Lm_TraceDecodeStep(B200LmExecutor* e, int32_t* out_id, int64_t* stamps, int64_t capacity,
                           int32_t* n_barriers, int32_t* n_cta, int32_t* sm_clock_khz, char** err) {
  B2_API_BEGIN
  B2_CHECK(e && e->impl && out_id && n_barriers && n_cta && sm_clock_khz, kInvalidArgument, "null argument");
  e->impl->trace_decode_step(out_id, reinterpret_cast<long long*>(stamps), capacity, n_barriers, n_cta, sm_clock_khz);
  B2_API_END
}

int B200Lm_GetLaunchCount(B200LmExecutor* e, int64_t* out, char** err) {
  B2_API_BEGIN
  B2_CHECK(e && e->impl && out, kInvalidArgument, "null argument");
  *out = e->impl->launches;
  B2_API_END
}

}  // extern "C"

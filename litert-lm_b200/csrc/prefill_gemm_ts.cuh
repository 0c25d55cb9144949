// Int4 weight-only GEMM for prefill with the WEIGHTS as the tensor-core "A"
// operand held in tensor memory:
//
//   D[weight row][token] = sum_k W[row][k] * X[token][k]
//
// The int4 weight tile is expanded to bf16 in registers and written straight
// into TMEM (tcgen05.st); the activations are the K-major "B" operand, staged
// in shared memory by TMA.  Compared with expanding the weights into a shared
// memory tile this removes, per 64-wide k block, 16 KB of shared-memory writes
// and a 4 KB operand read per MMA, which is what bounded the shared-memory
// variant (an M128 N128 K16 MMA reading both operands from shared memory
// needs the full 128 B/clk of the SM by itself).
//
// The kernel is persistent: one CTA per SM (two with tiles of up to 64 tokens)
// walks a static list of output tiles (128 weight rows x NTOK tokens x one K split).  Lane i of the accumulator is
// weight row i, so the per-channel scale is one scalar per epilogue thread and
// a warp's store covers 32 consecutive output features of one token.  The
// epilogue warps first pull the whole accumulator into registers (at most 64
// values per thread, added to those of the tile's chains before) and hand it back, so the scaling / GeGLU and the global
// stores of one tile run under the main loop of the next.
//
// The accumulator cuts off what it adds instead of rounding it, so its error grows with the products it takes: 5.1e-6 of
// the result over K = 21504 in one (GeGLU rows, 2-norm against 64 bits), 3.6e-7 over eight of 2688.  So EPI 0 hands its
// accumulator over every `chain` stages and adds the parts in fp32 in the epilogue's registers.  With narrower tiles the other
// CTA or the expansion's slack fills the gap (1152 x 1024 over 1023 tokens in four chains 7.4 us, in one 7.2); at 256 tokens the
// tensor cores stand still for 0.45 us (2560 x 10240 over 1023 tokens in eight chains 59.5, in one 56.5).  Handing the
// accumulator over in two halves cost more: M128 N128 products take 106 cycles, not 64.  gemm_chain in executor.cu has the lengths.
//
// Three rings, each with its own depth, move two k blocks (128 k) at a time: the
// int4 blocks (from HBM, deep), the activation tiles (from L2, shallow) and the
// expanded weights in tensor memory.  A hand-over between two roles costs a few
// hundred cycles however little it covers.  A stage of two k blocks takes 1020
// cycles at 256 tokens, of which the products are 1024: tensor-bound.  It takes
// 720 at 64 tokens: the expansion's chain of waits, loads and stores.  (While the
// MMA role issued behind `lane == 0`, its 8 instructions took 810 cycles and a
// stage 1260 at any width: elect_one in prefill_ops.cuh.)
//
// The weights do not depend on the preceding kernel, so their stream and their
// expansion start before griddepcontrol.wait; narrow tiles take half of an SM's
// shared and tensor memory, which lets the next GEMM's CTA do that while this one
// works.
//
// A narrow tile's k block still costs a CTA its hand-overs, so two CTAs share an SM and fill each other's gaps.
// The expansion's reads of the int4 block (16 bytes a lane at a stride of 32) take 8.2 shared-memory wavefronts
// each, where 4 are the least.
//
// Warp roles: 0 = activation producer, 1 = TMEM owner + MMA issue, 2 = weight
// producer, 4.. = int4 expansion, then epilogue.
//
// TMEM columns: [0, NTOK) accumulator, then slots of 64 columns holding one
// expanded 128 x 128 weight tile each.
#pragma once
#include "prefill_ops.cuh"

namespace b200lm {

constexpr int kTsRows = 128;                        // weight rows per tile
constexpr int kTsKb = 2;                            // k blocks per stage
constexpr int kTsAcols = 32;                        // TMEM columns of one expanded 128 x 64 weight block
// Depth of the rings and warps per role by token width.  Narrow tiles: the bytes in flight that HBM wants sit in the
// weight ring (8 KB a stage), everything together stays within half an SM.  256 tokens: tensor-bound, all of the SM.
__host__ __device__ constexpr int ts_xs(int ntok) { return ntok >= 128 ? (ntok >= 256 ? 3 : 2) : 3; }
__host__ __device__ constexpr int ts_qs(int ntok) { return ntok >= 256 ? 3 : ntok == 128 ? 5 : ntok == 64 ? 7 : 10; }
__host__ __device__ constexpr int ts_ws(int ntok) { return ntok >= 256 ? 4 : ntok == 128 ? 2 : 3; }
__host__ __device__ constexpr int ts_tmem(int ntok) { return ntok >= 256 ? 512 : 256; }
__host__ __device__ constexpr int ts_deq_warps(int ntok) { return ntok >= 256 ? 4 : 8; }
__host__ __device__ constexpr int ts_epi_cols(int ntok) { return ntok < 64 ? ntok : 64; }      // token columns per epilogue warp
__host__ __device__ constexpr int ts_epi_warps(int ntok) { return 4 * (ntok / ts_epi_cols(ntok)); }
__host__ __device__ constexpr int ts_threads(int ntok) { return 32 * (4 + ts_deq_warps(ntok) + ts_epi_warps(ntok)); }
__host__ __device__ constexpr int ts_ctas_per_sm(int ntok) { return ntok <= 64 ? 2 : 1; }
__host__ __device__ constexpr int ts_smem(int ntok) {
  return ts_xs(ntok) * kTsKb * ntok * kGemmBK * 2 + ts_qs(ntok) * kTsKb * kGemmStageQ + 1024 + 512;
}
// EPI 0 adds its chains in registers, a sum per column and thread of the epilogue.  From 64 tokens on that is more than
// an even share of the registers, and the other warps give up some of theirs.
struct TsRegs { int launch, issue, expand, sum; };
__host__ __device__ constexpr TsRegs ts_regs(int ntok) { return ntok >= 256 ? TsRegs{80, 56, 72, 88} : ntok == 128 ? TsRegs{96, 56, 80, 128} : ntok == 64 ? TsRegs{64, 56, 56, 88} : TsRegs{}; }
__host__ __device__ constexpr bool ts_shares_add_up(int ntok) {
  const TsRegs r = ts_regs(ntok);
  return 4 * r.issue + ts_deq_warps(ntok) * r.expand + ts_epi_warps(ntok) * r.sum <= ts_threads(ntok) / 32 * r.launch;
}
static_assert(ts_shares_add_up(256) && ts_shares_add_up(128) && ts_shares_add_up(64), "a warp that asks for more registers than the block has waits for ever");
static_assert(ts_tmem(256) >= 256 + ts_ws(256) * kTsKb * kTsAcols && ts_tmem(128) >= 128 + ts_ws(128) * kTsKb * kTsAcols &&
                  ts_tmem(64) >= 64 + ts_ws(64) * kTsKb * kTsAcols, "TMEM budget");
static_assert(ts_ctas_per_sm(64) * ts_tmem(64) <= 512 && ts_smem(256) <= 227 * 1024 && 2 * (ts_smem(128) + 1024) <= 228 * 1024 && 2 * (ts_smem(64) + 1024) <= 228 * 1024 &&
                  2 * (ts_smem(32) + 1024) <= 228 * 1024, "shared memory budget");

// A operand in tensor memory, B through a shared-memory descriptor
__device__ __forceinline__ void umma_bf16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc,
                                             uint32_t accumulate) {
  asm volatile(
      "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}"
      ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// 16 consecutive 32-bit columns of this thread's TMEM lane
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

__device__ __forceinline__ float gelu_tanh_fast(float x) {
  const float c = 0.7978845608028654f;
  float y = c * (x + 0.044715f * x * x * x), t;
  asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(y));
  return 0.5f * x * (1.0f + t);
}

// Tile list: tile = (ks * t_tiles + t_tile) * n_tiles + n_tile; CTA c takes
// tiles c, c + gridDim.x, ...
struct TsTile {
  int n_tile, t_tile, ks;
};
__device__ __forceinline__ TsTile ts_tile(int tile, int n_tiles, int t_tiles) {
  TsTile t;
  t.n_tile = tile % n_tiles;
  int r = tile / n_tiles;
  t.t_tile = r % t_tiles;
  t.ks = r / t_tiles;
  return t;
}

// EC consecutive accumulator columns of this thread's lane
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
template <int EC>
__device__ __forceinline__ void ts_load_acc(uint32_t taddr, uint32_t (&v)[EC]) {
#pragma unroll
  for (int c = 0; c < EC; c += 16) tmem_ld16(taddr + c, v + c);
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// EPI 0: fp32 partials outF[ks][T][N], each the sum of its chains.  EPI 1: GeGLU; tile rows alternate
// gate (even) and up (odd) rows of one ffn feature, output bf16 outB[T][N/2].
//
// NTOK is the token width of a tile (the N of the MMA): whichever of 16 .. 256 the launcher finds cheapest for the token
// rows, several tiles with the last one ragged among them.  Narrow tiles fill more CTAs and cost less each in activation
// bytes and MMA time; wide ones expand the weights less often.  tmX must have a box of min(NTOK, 128) rows.
template <int EPI, int NTOK>
__global__ void __launch_bounds__(ts_threads(NTOK), ts_ctas_per_sm(NTOK))
gemm_w4_ts_kernel(const __grid_constant__ CUtensorMap tmX, GemmArgs g) {
  constexpr int D = ts_deq_warps(NTOK), E = ts_epi_warps(NTOK), EC = ts_epi_cols(NTOK);
  constexpr int XS = ts_xs(NTOK), QS = ts_qs(NTOK), WS = ts_ws(NTOK);
  constexpr int kXb = NTOK * kGemmBK * 2;           // activation bytes of a k block
  constexpr bool kShare = EPI == 0 && ts_regs(NTOK).launch > 0;
  extern __shared__ unsigned char gsm_raw[];
  unsigned char* gsm = reinterpret_cast<unsigned char*>(((uintptr_t)gsm_raw + 1023) & ~(uintptr_t)1023);
  unsigned char* sX = gsm;
  unsigned char* sQ = gsm + XS * kTsKb * kXb;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sQ + QS * kTsKb * kGemmStageQ);
  uint64_t* x_full = bars;                          // [XS] activation tiles landed
  uint64_t* x_empty = x_full + XS;                  // [XS] MMAs finished with them
  uint64_t* q_full = x_empty + XS;                  // [QS] int4 blocks landed
  uint64_t* q_empty = q_full + QS;                  // [QS] expansion has read them
  uint64_t* w_full = q_empty + QS;                  // [WS] expanded weights are in TMEM
  uint64_t* w_empty = w_full + WS;                  // [WS] MMAs finished with them
  uint64_t* acc_full = w_empty + WS;                // accumulator of a chain complete
  uint64_t* acc_empty = acc_full + 1;               // accumulator read out by the epilogue warps
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_full + 2);

  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int KB = g.K / kGemmBK;
  const int nkb = KB / g.ksplit;
  const int nst = (nkb + kTsKb - 1) / kTsKb;        // stages of a tile; the last may hold one k block
  const int n_tiles = (g.N + kTsRows - 1) / kTsRows;
  const int t_tiles = (g.T + NTOK - 1) / NTOK;
  const int total = n_tiles * t_tiles * g.ksplit;
  const int my_tiles = (int)blockIdx.x < total ? (total - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;

  // weight producer: one lane's state, started ahead of everything else
  int q_it = 0, q_li = 0, q_st = 0;
  auto q_issue = [&]() {                            // warp 2, lane 0
    const TsTile tl = ts_tile(blockIdx.x + q_li * gridDim.x, n_tiles, t_tiles);
    const int kb = q_st * kTsKb, nk = min(kTsKb, nkb - kb), s = q_it % QS;
    mbar_arrive_expect_tx(&q_full[s], (uint32_t)nk * kGemmStageQ);
    bulk_load_1d(sQ + s * kTsKb * kGemmStageQ, g.w + ((size_t)tl.n_tile * KB + (size_t)tl.ks * nkb + kb) * kGemmStageQ,
                 (uint32_t)nk * kGemmStageQ, &q_full[s]);
    ++q_it;
    if (++q_st == nst) { q_st = 0; ++q_li; }
  };
  if (threadIdx.x == 64) {
#pragma unroll 1
    for (int s = 0; s < QS; ++s) { mbar_init(&q_full[s], 1); mbar_init(&q_empty[s], 4); }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
#pragma unroll 1
    while (q_it < QS && q_li < my_tiles) q_issue();
  }
  if (threadIdx.x == 0) {
#pragma unroll 1
    for (int s = 0; s < XS; ++s) { mbar_init(&x_full[s], 1); mbar_init(&x_empty[s], 1); }
#pragma unroll 1
    for (int s = 0; s < WS; ++s) { mbar_init(&w_full[s], 4); mbar_init(&w_empty[s], 1); }
    mbar_init(acc_full, 1);
    mbar_init(acc_empty, E);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) tmem_alloc(tmem_slot, ts_tmem(NTOK));
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  const uint32_t tmem_w = tmem_base + NTOK;         // weight slots follow the accumulator columns
  // Ahead of the wait below: the next GEMM may fill its weight ring while this one still waits.  A kernel behind this one
  // that reads ahead of its own wait must read nothing that the two kernels before it write.
  pdl_launch_dependents();

  bool ok = true;                                   // none of this thread's waits has given up
  if constexpr (kShare) {
    if (warp < 4) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(ts_regs(NTOK).issue));
    else if (warp < 4 + D) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(ts_regs(NTOK).expand));
  }
  if (warp == 0) {
    // ---- activation producer: what it reads comes from the preceding kernel
    pdl_wait();
    int it = 0;
    const bool leader = elect_one();
#pragma unroll 1
    for (int li = 0; li < my_tiles && ok; ++li) {
      const TsTile tl = ts_tile(blockIdx.x + li * gridDim.x, n_tiles, t_tiles);
#pragma unroll 1
      for (int st = 0; st < nst && ok; ++st, ++it) {
        const int s = it % XS, n = it / XS, kb = st * kTsKb, nk = min(kTsKb, nkb - kb);
        if (n > 0) ok = __all_sync(0xffffffffu, mbar_wait(&x_empty[s], (n - 1) & 1, g.err));
        if (ok && leader) {
          mbar_arrive_expect_tx(&x_full[s], (uint32_t)(nk * kXb));
#pragma unroll 1
          for (int k = 0; k < nk; ++k)
#pragma unroll
            for (int h = 0; h < (NTOK + 127) / 128; ++h)
              tma_load_2d(sX + (s * kTsKb + k) * kXb + h * 128 * 128, &tmX, (tl.ks * nkb + kb + k) * kGemmBK, tl.t_tile * NTOK + h * 128,
                          &x_full[s]);
        }
        __syncwarp();
      }
    }
  } else if (warp == 1) {
    // ---- MMA issue
    const uint32_t idesc = umma_idesc_bf16(kTsRows, NTOK);
    int it = 0, nacc = 0;                            // stages, accumulators begun
    const bool leader = elect_one();
#pragma unroll 1
    for (int li = 0; li < my_tiles && ok; ++li) {
#pragma unroll 1
      for (int st = 0, left = 0; st < nst && ok; ++st, ++it, --left) {
        const bool first = left == 0;                // stage of a chain
        if (first) {
          left = EPI == 0 ? g.chain : nst;
          if (nacc > 0) ok = __all_sync(0xffffffffu, mbar_wait(acc_empty, (nacc - 1) & 1, g.err));
          ++nacc;
          if (!ok) break;
        }
        const int sx = it % XS, sw = it % WS, nk = min(kTsKb, nkb - st * kTsKb);
        ok = __all_sync(0xffffffffu, mbar_wait(&w_full[sw], (it / WS) & 1, g.err) && mbar_wait(&x_full[sx], (it / XS) & 1, g.err));
        if (!ok) break;
        tc_fence_after();
        if (leader) {
#pragma unroll
          for (int kb = 0; kb < kTsKb; ++kb) {
            if (kb >= nk) break;
            const uint64_t xd = umma_desc_sw128(smem_u32(sX + (sx * kTsKb + kb) * kXb));
#pragma unroll
            for (int k = 0; k < kGemmBK / 16; ++k)   // 16 bf16 along K per MMA: 8 TMEM columns, 32 bytes of X
              umma_bf16_ts(tmem_base, tmem_w + (sw * kTsKb + kb) * kTsAcols + k * 8, xd + (uint64_t)(k * 2), idesc, first && !(kb | k) ? 0u : 1u);
          }
          umma_commit(&w_empty[sw]);
          umma_commit(&x_empty[sx]);
          if (left == 1 || st + 1 == nst) umma_commit(acc_full);
        }
        __syncwarp();
      }
    }
  } else if (warp == 2) {
    // ---- weight producer, behind the first fills
    if (lane == 0) {
#pragma unroll 1
      while (q_li < my_tiles && ok) {
        ok = mbar_wait(&q_empty[q_it % QS], (q_it / QS - 1) & 1, g.err);
        if (ok) q_issue();
      }
    }
  } else if (warp >= 4 && warp < 4 + D) {
    // ---- int4 -> bf16 expansion into TMEM: this thread does its weight row's part of a stage.  Eight warps take
    // alternate stages in two groups of four, so that one group's waits run beside the other's expansion.
    const int quarter = warp & 3;                  // TMEM lanes 32*quarter .. +31 belong to this warp
    constexpr int kGroups = D / 4;
    const int group = (warp - 4) >> 2;
    const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
    const int iters = my_tiles * nst;
    const __nv_bfloat162 bias = __float2bfloat162_rn(136.0f);
#pragma unroll 1
    for (int it = group, st = group; it < iters && ok; it += kGroups, st += kGroups) {
#pragma unroll 1
      while (st >= nst) st -= nst;
      const int sq = it % QS, sw = it % WS, nk = min(kTsKb, nkb - st * kTsKb);
      ok = __all_sync(0xffffffffu, mbar_wait(&q_full[sq], (it / QS) & 1, g.err) && (it < WS || mbar_wait(&w_empty[sw], (it / WS - 1) & 1, g.err)));
      if (!ok) break;
      tc_fence_after();
      uint4 q[2 * kTsKb];                            // all of the row's part first: the stores below order what follows them
#pragma unroll
      for (int i = 0; i < 2 * kTsKb; ++i)
        if (i / 2 < nk) q[i] = reinterpret_cast<const uint4*>(sQ + (sq * kTsKb + i / 2) * kGemmStageQ + (quarter * 32 + lane) * 32)[i % 2];
#pragma unroll
      for (int i = 0; i < 2 * kTsKb; ++i) {
        if (i / 2 >= nk) break;
        const uint32_t qw[4] = {q[i].x, q[i].y, q[i].z, q[i].w};
        uint32_t r[16];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            uint32_t v = ((qw[j] >> (4 * k)) & 0x000F000Fu) | 0x43004300u;   // bf16(128 + nibble) pairs
            __nv_bfloat162 h = __hsub2(*reinterpret_cast<__nv_bfloat162*>(&v), bias);
            r[j * 4 + k] = *reinterpret_cast<uint32_t*>(&h);
          }
        }
        tmem_st16(tmem_w + lane_base + (sw * kTsKb + i / 2) * kTsAcols + i % 2 * 16, r);
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) { mbar_arrive(&w_full[sw]); mbar_arrive(&q_empty[sq]); }
    }
  } else if (warp >= 4 + D) {
    // ---- epilogue: this warp takes EC token columns of its 32 weight rows
    const int quarter = warp & 3;
    const int row = quarter * 32 + lane;
    const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
    const int c0 = ((warp - 4 - D) >> 2) * EC;
    if constexpr (kShare) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(ts_regs(NTOK).sum));
    int nacc = 0;
    pdl_wait();                                     // the outputs may still be read by an earlier kernel
#pragma unroll 1
    for (int li = 0; li < my_tiles && ok; ++li) {
      const TsTile tl = ts_tile(blockIdx.x + li * gridDim.x, n_tiles, t_tiles);
      const float sc = g.wscale[tl.n_tile * kTsRows + row];
      if constexpr (EPI == 0) {
        float sum[EC];
#pragma unroll
        for (int c = 0; c < EC; ++c) sum[c] = 0.f;
#pragma unroll 1
        for (int st = 0; st < nst; st += g.chain, ++nacc) {
          ok = __all_sync(0xffffffffu, mbar_wait(acc_full, nacc & 1, g.err));
          if (!ok) break;
          tc_fence_after();
#pragma unroll
          for (int c = 0; c < EC; c += 16) {
            uint32_t v[16];
            ts_load_acc<16>(tmem_base + lane_base + c0 + c, v);
#pragma unroll
            for (int i = 0; i < 16; ++i) sum[c + i] += __uint_as_float(v[i]);
          }
          tc_fence_before();                        // the accumulator is in registers: hand it back before the stores
          __syncwarp();
          if (lane == 0) mbar_arrive(acc_empty);
        }
        const int nrow = tl.n_tile * kTsRows + row, t0 = tl.t_tile * NTOK + c0;
        if (ok && nrow < g.N) {
          float* dst = g.outF + ((size_t)tl.ks * g.T + t0) * g.N + nrow;
#pragma unroll
          for (int c = 0; c < EC; ++c, dst += g.N)
            if (t0 + c < g.T) *dst = sum[c] * sc;
        }
      } else {
        ok = __all_sync(0xffffffffu, mbar_wait(acc_full, li & 1, g.err));
        if (!ok) break;
        tc_fence_after();
        constexpr int EH = NTOK <= 64 && EC > 32 ? 32 : EC;   // columns in registers at a time
#pragma unroll 1
        for (int ch = 0; ch < EC; ch += EH) {
          const int t0 = tl.t_tile * NTOK + c0 + ch;
          uint32_t v[EH];
          ts_load_acc<EH>(tmem_base + lane_base + c0 + ch, v);
          if (ch + EH == EC) {                      // the accumulator is in registers: hand it back before the stores
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(acc_empty);
          }
          const int F = g.N / 2;
          const int f = tl.n_tile * (kTsRows / 2) + (row >> 1);
          const bool odd = lane & 1;
          __nv_bfloat16* dst = g.outB + (size_t)(t0 + (odd ? 1 : 0)) * F + f;
          const int tlim = g.T - t0 - (odd ? 1 : 0);          // columns c (even) with c < tlim are stored
#pragma unroll
          for (int c = 0; c < EH; c += 2) {
            float a = __uint_as_float(v[c]) * sc, bb = __uint_as_float(v[c + 1]) * sc;
            float got = __shfl_xor_sync(0xffffffffu, odd ? a : bb, 1);
            float gate = odd ? got : a, up = odd ? bb : got;
            if (c < tlim && f < F) dst[(size_t)c * F] = __float2bfloat16(gelu_tanh_fast(gate) * up);
          }
        }
      }
    }
  }
  tc_fence_before();
  sync_after_waits(ok);
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, ts_tmem(NTOK));
  }
}

}  // namespace b200lm

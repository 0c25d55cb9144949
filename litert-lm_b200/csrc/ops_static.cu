// Allocation-free variant of the split-KV decode attention (see b200lm_ops.h,
// B200LmOps_AttentionDecodeStatic).  Compiled into the same translation unit
// as ops.cu, whose kernels it launches.
//
// The ordinary entry point allocates device memory for the split partials
// (m, l, unnormalised o per split) on every call.  Some hosts cannot do that:
// a caller that runs inside another runtime's execution callback, a real-time
// serving loop that forbids allocator calls after start-up, or a process whose
// device memory is fully budgeted up front.  For them the partials, the query
// positions and the error word live in ONE file-scope device array of fixed
// size.  Every GPU that loads this library carries that array until the
// process exits.
#include "../../include/b200lm_ops.h"
#include "attn_mma.cuh"
#include "attn_tc.cuh"
#include "common.cuh"
#include "decode_ops.cuh"
#include "page_map.h"
#include "prefill_ops.cuh"

#include <atomic>
#include <mutex>

namespace b200lm {

constexpr size_t kStaticScratchBytes = 8u << 20;          // 8 MiB per GPU
constexpr size_t kStaticHeaderBytes = 64u << 10;          // error word + query positions
constexpr int kStaticMaxQueries = (int)(kStaticHeaderBytes / 4) - 16;

// In HOST code this name is only a stand-in for the symbol: it is not a device
// address.  Host code gets the address with cudaGetSymbolAddress (below);
// device code may name the array directly.
static __device__ __align__(256) unsigned char g_attn_static_scratch[kStaticScratchBytes];

// Tickets of attn_shared_kernel (split_ticket.h), 128 KiB; zero whenever no call is on the GPU.
static __device__ unsigned g_attn_static_tickets[kTicketWords];

// Header layout: int[0] = error word (zero in the image, cleared by the status call that reports it), int[16 + i] =
// position of query i.
__global__ void static_scratch_prepare_kernel(int nq, int pos) {
  int* hdr = reinterpret_cast<int*>(g_attn_static_scratch);
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < nq) hdr[16 + i] = pos;
}

constexpr int kMaxDevices = 64;
struct StaticScratch {
  unsigned char* base;
  unsigned* tickets;
  int sms;
  int clusters[2];            // of attn_tc_kernel at head size 128 and 256
};
static StaticScratch g_static_scratch[kMaxDevices] = {};
static std::mutex g_static_scratch_mu;     // guards the per-device set-up below

// Device address of the array on `device` (which must be current).  Looked up
// once per device, under a lock: concurrent first calls do the set-up once.
static StaticScratch static_scratch_for(int device) {
  B2_CHECK(device >= 0 && device < kMaxDevices, kInvalidArgument, "device ordinal out of range");
  std::lock_guard<std::mutex> lock(g_static_scratch_mu);
  StaticScratch& s = g_static_scratch[device];
  if (!s.base) {
    void *p = nullptr, *t = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_attn_static_scratch);
    if (e == cudaSuccess) e = cudaGetSymbolAddress(&t, g_attn_static_tickets);
    if (e != cudaSuccess || p == nullptr || t == nullptr)
      throw Error{kInternal, std::string("cudaGetSymbolAddress(static scratch): ") + cudaGetErrorString(e)};
    // attribute change, not an allocation; done with the set-up so later calls only launch.  The limit is
    // raised to the largest shape the entry point accepts and never lowered by any other caller.
    raise_dyn_smem(attn_decode_kernel, sizeof(float) * ((size_t)(4 + 2) * 256 + (size_t)kDecWarps * 4 * (256 + 2)));
    B2_CUDA(cudaDeviceGetAttribute(&s.sms, cudaDevAttrMultiProcessorCount, device));
    s.clusters[0] = atc_prepare<128>();
    s.clusters[1] = atc_prepare<256>();
    (void)encode_tiled_fn();
    s.tickets = reinterpret_cast<unsigned*>(t);
    s.base = reinterpret_cast<unsigned char*>(p);
  }
  return s;
}

// Makes `device` current for the duration of a call and puts the caller's device back afterwards.
struct DeviceScope {
  int prev = -1;
  explicit DeviceScope(int device) {
    if (cudaGetDevice(&prev) != cudaSuccess) { cudaGetLastError(); prev = -1; }
    if (prev == device) prev = -1;            // already current: nothing to set, nothing to put back
    else B2_CUDA(cudaSetDevice(device));
  }
  ~DeviceScope() {
    if (prev >= 0) cudaSetDevice(prev);
  }
};

static int static_fail(char** err, int code, const std::string& msg) {
  if (err) {
    *err = reinterpret_cast<char*>(malloc(msg.size() + 1));
    if (*err) memcpy(*err, msg.c_str(), msg.size() + 1);
  }
  return code;
}

static void require_device(int device) {
  static std::atomic<int> known{0};           // the count does not change while a process runs
  int ndev = known.load(std::memory_order_relaxed);
  if (ndev <= 0) {
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev <= 0) {
      cudaGetLastError();
      throw Error{kFailedPrecondition, "no CUDA device: this backend has no CPU fallback"};
    }
    known.store(ndev, std::memory_order_relaxed);
  }
  B2_CHECK(device >= 0 && device < ndev, kInvalidArgument, "device ordinal out of range");
}

// Splits of a batch's queries whose partials the scratch holds.
static int scratch_splits(int batch, int hq, int hd) {
  const size_t per_split = (size_t)batch * hq * (hd + 2) * sizeof(float);
  return (int)std::min<size_t>(kTicketSplits, (kStaticScratchBytes - kStaticHeaderBytes) / per_split);
}

}  // namespace b200lm

using namespace b200lm;

extern "C" int B200LmOps_AttentionDecodeStatic(int32_t device, const float* q_dev, const void* k_pages_dev,
                                               const void* v_pages_dev, const int32_t* page_table_dev, int32_t batch,
                                               int32_t s, int32_t hq, int32_t hkv, int32_t hd, int32_t window,
                                               int32_t kv_bf16, int32_t nsplit, float* out_dev, void* stream,
                                               char** err) {
  if (err) *err = nullptr;
  try {
    B2_CHECK(q_dev && k_pages_dev && v_pages_dev && page_table_dev && out_dev, kInvalidArgument, "null pointer");
    B2_CHECK(batch > 0 && s > 0 && hq > 0 && hkv > 0 && hq % hkv == 0, kInvalidArgument, "bad shape");
    const int G = hq / hkv;
    B2_CHECK(G == 1 || G == 2 || G == 4, kUnimplemented, "GQA group size must be 1, 2 or 4");
    B2_CHECK(hd == 32 || hd == 64 || hd == 128 || hd == 256, kUnimplemented, "head_dim must be 32/64/128/256");
    B2_CHECK(nsplit >= 1 && nsplit <= kMaxSplits, kInvalidArgument, "nsplit out of range");
    B2_CHECK(batch <= kStaticMaxQueries, kInvalidArgument,
             "batch exceeds the static scratch: at most " + std::to_string(kStaticMaxQueries) + " queries");
    const size_t part_o_bytes = (size_t)batch * hkv * nsplit * G * hd * sizeof(float);
    const size_t part_ml_bytes = (size_t)batch * hkv * nsplit * G * 2 * sizeof(float);
    B2_CHECK(kStaticHeaderBytes + part_o_bytes + part_ml_bytes <= kStaticScratchBytes, kInvalidArgument,
             "split partials need " + std::to_string(part_o_bytes + part_ml_bytes) + " bytes; the static scratch holds " +
                 std::to_string(kStaticScratchBytes - kStaticHeaderBytes) + " (lower batch or nsplit)");
    require_device(device);
    DeviceScope scope(device);                                  // the caller's current device is restored on return
    const StaticScratch sc = static_scratch_for(device);        // first call on a device does the set-up
    unsigned char* scratch = sc.base;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    int* hdr = reinterpret_cast<int*>(scratch);
    float* part_o = reinterpret_cast<float*>(scratch + kStaticHeaderBytes);
    float* part_ml = reinterpret_cast<float*>(scratch + kStaticHeaderBytes + part_o_bytes);
    // Bulk copies and 16-byte accesses need aligned rows; buffers that are not go through the plain-load kernel.
    const uintptr_t align = (uintptr_t)q_dev | (uintptr_t)k_pages_dev | (uintptr_t)v_pages_dev | (uintptr_t)out_dev;
    if (align % 16 == 0) {
      AmArgs a{};
      a.q = q_dev;
      a.q_stride = (hq + 2 * hkv) * hd;
      a.k = k_pages_dev;
      a.v = v_pages_dev;
      a.page_table = page_table_dev;
      a.rows = batch * G;
      a.G = G;
      a.hkv = hkv;
      a.lo = window > 0 && window < s ? s - window : 0;
      a.k1 = s;
      a.qscale = 1.4426950408889634f / sqrtf((float)hd);
      a.out = out_dev;
      a.part_o = part_o;
      a.err = hdr;
      // the caller's nsplit sized the check above; what fits the scratch is this kernel's own limit
      const int cap = scratch_splits(batch, hq, hd);
      a.part_ml = part_o + (size_t)batch * hq * cap * hd;
      if (const int ns = kv_bf16 ? atc_splits(a, hd, sc.clusters[hd == 256], cap) : 0) {
        // the pages of a cache as [page][kv head x slot][hd]
        const cuuint64_t strides[2] = {(cuuint64_t)hd * 2, (cuuint64_t)hkv * kPage * hd * 2};
        const cuuint64_t dims[3] = {(cuuint64_t)hd, (cuuint64_t)hkv * kPage, map_pages(strides[1])};
        const cuuint32_t box[3] = {64, kAtcKeys, 1};
        const CUtensorMap tm_k = make_bf16_map(k_pages_dev, 3, dims, strides, box), tm_v = make_bf16_map(v_pages_dev, 3, dims, strides, box);
        if (hd == 256) launch_attn_tc<256>(st, tm_k, tm_v, a, ns);
        else launch_attn_tc<128>(st, tm_k, tm_v, a, ns);
      } else if (kv_bf16) launch_attn_shared_bf16(st, a, hd, device, sc.sms, cap, sc.tickets);
      else launch_attn_shared_f32(st, a, hd, device, sc.sms, cap, sc.tickets);
      return kOk;
    }
    static_scratch_prepare_kernel<<<(batch + 255) / 256, 256, 0, st>>>(batch, s - 1);
    B2_CUDA(cudaGetLastError());
    ModelDims dm{};
    dm.hq = hq; dm.hkv = hkv; dm.hd = hd; dm.d = 64; dm.ffn = 64;
    dm.window = window > 0 ? window : 1 << 30;
    dm.kv_dtype = kv_bf16 ? 1 : 0;
    dm.eps = 1e-6f;
    const int npages = (s + kPage - 1) / kPage;
    dm.max_ctx = npages * kPage;
    AttnJob j;
    memset(&j, 0, sizeof j);
    j.qkv = q_dev;                       // rows of (hq + 2 hkv) * hd floats; only the q part is read
    j.pos = hdr + 16;
    j.page_table = page_table_dev;
    j.pages_per_seq = npages;
    j.seq_stride = 0;
    j.is_global = window > 0 ? 0 : 1;
    j.nsplit = nsplit;
    j.appended = 1;
    j.kv.k = const_cast<void*>(k_pages_dev);
    j.kv.v = const_cast<void*>(v_pages_dev);
    j.part_o = part_o;
    j.part_ml = part_ml;
    j.err = hdr;
    const size_t smem_dec = sizeof(float) * ((size_t)(G + 2) * hd + (size_t)kDecWarps * G * (hd + 2));
    const int items = batch * hkv * nsplit;
    const int grid = items < sc.sms ? items : sc.sms;
    attn_decode_kernel<<<grid, kDecThreads, smem_dec, st>>>(dm, j, batch);
    B2_CUDA(cudaGetLastError());         // a rejected launch must not be followed by a combine of stale partials
    const int total = batch * hq * hd;
    attn_combine_kernel<<<(total + 255) / 256, 256, 0, st>>>(part_o, part_ml, batch, hq, hkv, hd, nsplit, out_dev);
    B2_CUDA(cudaGetLastError());
  } catch (const Error& e_) {
    return static_fail(err, e_.code, e_.msg);
  } catch (...) {
    return static_fail(err, kInternal, "unknown failure");
  }
  return kOk;
}

// What atc_splits answers for a call of this shape on this device.
extern "C" int B200LmOps_AttentionDecodeStaticClusters(int32_t device, int32_t batch, int32_t s, int32_t hq, int32_t hkv, int32_t hd,
                                                       int32_t window, int32_t kv_bf16, int32_t* clusters, char** err) {
  if (err) *err = nullptr;
  try {
    B2_CHECK(clusters, kInvalidArgument, "null pointer");
    B2_CHECK(batch > 0 && batch <= kStaticMaxQueries && s > 0 && hq > 0 && hkv > 0 && hq % hkv == 0 && hd > 0, kInvalidArgument, "bad shape");
    require_device(device);
    DeviceScope scope(device);
    const StaticScratch sc = static_scratch_for(device);
    AmArgs a{};
    a.rows = batch * (hq / hkv);
    a.hkv = hkv;
    a.lo = window > 0 && window < s ? s - window : 0;
    a.k1 = s;
    *clusters = kv_bf16 ? atc_splits(a, hd, sc.clusters[hd == 256], scratch_splits(batch, hq, hd)) : 0;
  } catch (const Error& e_) {
    return static_fail(err, e_.code, e_.msg);
  } catch (...) {
    return static_fail(err, kInternal, "unknown failure");
  }
  return kOk;
}

// Reads back the error word that the kernels of B200LmOps_AttentionDecodeStatic write into the static
// array (a query position outside the cache).  Waits for `stream`, allocates nothing.
extern "C" int B200LmOps_AttentionDecodeStaticStatus(int32_t device, void* stream, int32_t* device_error, char** err) {
  if (err) *err = nullptr;
  try {
    require_device(device);
    DeviceScope scope(device);
    (void)static_scratch_for(device);
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    int word = 0;
    B2_CUDA(cudaMemcpyFromSymbolAsync(&word, g_attn_static_scratch, sizeof(int), 0, cudaMemcpyDeviceToHost, st));
    B2_CUDA(cudaStreamSynchronize(st));
    if (device_error) *device_error = word;
    if (word != kDevOk) B2_CUDA(cudaMemsetAsync(static_scratch_for(device).base, 0, sizeof(int), st));   // the next call starts clean
    if (word == kDevBadPosition) throw Error{kInvalidArgument, "a query position lay outside the cache"};
    if (word == kDevBarrierTimeout) throw Error{kDeadlineExceeded, "a bounded device-side wait gave up"};
    if (word != kDevOk) throw Error{kInternal, "device error word " + std::to_string(word)};
  } catch (const Error& e_) {
    return static_fail(err, e_.code, e_.msg);
  } catch (...) {
    return static_fail(err, kInternal, "unknown failure");
  }
  return kOk;
}

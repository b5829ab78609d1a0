// Runtime services around the kernels: intermediate slots keyed by Guid (the device form of the
// managed Store/Restore pair), packed download / upload of many tensors (what SaveWeightsAndMoments
// needs), device introspection and CUDA-event timing brackets.
#include <array>
#include <cstring>
#include <map>
#include <mutex>

#include "common.cuh"

namespace prad {

using Guid = std::array<uint8_t, 16>;

struct Slot {
  std::vector<void*> ptrs;      // what Restore hands back
  std::vector<size_t> bytes;
  bool owns = false;            // copies made by the store (freed when the slot is dropped)
};

struct TimingBracket {
  char label[48];
  cudaEvent_t begin = nullptr, end = nullptr;
  int64_t launches0 = 0, launches1 = 0;
  bool closed = false;
};

// per-context runtime state; lives in a side table so that the context struct stays plain
struct RuntimeState {
  std::map<Guid, Slot> slots;
  std::vector<TimingBracket> brackets;
  int open_bracket = -1;
};

static std::mutex g_rt_mu;
static std::map<prad_ctx*, RuntimeState*> g_rt;

static RuntimeState* rt_of(prad_ctx* ctx) {
  std::lock_guard<std::mutex> lock(g_rt_mu);
  auto it = g_rt.find(ctx);
  if (it != g_rt.end()) return it->second;
  RuntimeState* r = new RuntimeState();
  g_rt[ctx] = r;
  return r;
}

static void free_slot(Slot& s) {
  if (s.owns)
    for (void* p : s.ptrs)
      if (p) cudaFree(p);
  s.ptrs.clear();
  s.bytes.clear();
}

static void free_brackets(RuntimeState* r) {
  for (TimingBracket& b : r->brackets) {
    if (b.begin) cudaEventDestroy(b.begin);
    if (b.end) cudaEventDestroy(b.end);
  }
  r->brackets.clear();
  r->open_bracket = -1;
}

// called by prad_shutdown
void runtime_destroy(prad_ctx* ctx) {
  RuntimeState* r = nullptr;
  {
    std::lock_guard<std::mutex> lock(g_rt_mu);
    auto it = g_rt.find(ctx);
    if (it == g_rt.end()) return;
    r = it->second;
    g_rt.erase(it);
  }
  for (auto& kv : r->slots) free_slot(kv.second);
  free_brackets(r);
  delete r;
}

static Guid guid_of(const void* p) {
  Guid g;
  memcpy(g.data(), p, 16);
  return g;
}

// ---- pipe-rate probes: register-resident arithmetic, no memory traffic; every thread keeps eight
// independent dependency chains so that the pipe's latency is covered
__global__ void __launch_bounds__(256)
probe_fp64_fma_kernel(double* __restrict__ out, int iters, double seed) {
  double acc[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) acc[j] = seed + (double)(threadIdx.x + j) * 1e-9;
  const double b = 0.99999999, c = 1e-9;
  for (int i = 0; i < iters; ++i) {
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j] = fma(acc[j], b, c);
  }
  double s = 0.0;
#pragma unroll
  for (int j = 0; j < 8; ++j) s += acc[j];
  out[(size_t)blockIdx.x * blockDim.x + threadIdx.x] = s;
}
__global__ void __launch_bounds__(256)
probe_fp32_fma_kernel(float* __restrict__ out, int iters, float seed) {
  float acc[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) acc[j] = seed + (float)(threadIdx.x + j) * 1e-6f;
  const float b = 0.999999f, c = 1e-6f;
  for (int i = 0; i < iters; ++i) {
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j] = fmaf(acc[j], b, c);
  }
  float s = 0.f;
#pragma unroll
  for (int j = 0; j < 8; ++j) s += acc[j];
  out[(size_t)blockIdx.x * blockDim.x + threadIdx.x] = s;
}
// mma.sync m8n8k4 f64: 8 x 8 x 4 x 2 = 512 flop per warp instruction, four independent accumulators
__global__ void __launch_bounds__(256)
probe_fp64_mma_kernel(double* __restrict__ out, int iters, double seed) {
  double c[4][2];
#pragma unroll
  for (int j = 0; j < 4; ++j) { c[j][0] = seed; c[j][1] = -seed; }
  const double a = 1.0 + (double)(threadIdx.x & 31) * 1e-9, b = 0.5;
  for (int i = 0; i < iters; ++i) {
#pragma unroll
    for (int j = 0; j < 4; ++j)
      asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                   : "+d"(c[j][0]), "+d"(c[j][1]) : "d"(a), "d"(b));
  }
  double s = 0.0;
#pragma unroll
  for (int j = 0; j < 4; ++j) s += c[j][0] + c[j][1];
  out[(size_t)blockIdx.x * blockDim.x + threadIdx.x] = s;
}

}  // namespace prad

using namespace prad;

extern "C" {

// ---------------------------------------------------------------- pipe rates
prad_status prad_measure_pipe_rate(prad_ctx* ctx, int pipe, double* out_tflops) {
  PRAD_CHECK_CTX(ctx);
  PRAD_NOT_CAPTURING(ctx, "prad_measure_pipe_rate");
  PRAD_REQUIRE(out_tflops && pipe >= 0 && pipe <= 2, PRAD_ERR_INVALID,
               "prad_measure_pipe_rate: pipe is 0 (FP64 FMA), 1 (FP64 MMA) or 2 (FP32 FMA)");
  const int blocks = ctx->sm_count * 8, threads = 256, iters = 1 << 14;
  prad_status s = ensure_stage(ctx, (size_t)blocks * threads * sizeof(double));
  if (s) return s;
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  PRAD_CUDA(cudaEventCreate(&e0));
  cudaError_t err = cudaEventCreate(&e1);
  if (err != cudaSuccess) { cudaEventDestroy(e0); set_error("prad_measure_pipe_rate: %s", cudaGetErrorString(err)); return PRAD_ERR_CUDA; }
  double best_ms = 1e30;
  for (int rep = 0; rep < 4; ++rep) {   // the first repetition warms the clocks up
    cudaEventRecord(e0, ctx->stream);
    if (pipe == 0) probe_fp64_fma_kernel<<<blocks, threads, 0, ctx->stream>>>((double*)ctx->stage, iters, 1.0 + rep);
    else if (pipe == 1) probe_fp64_mma_kernel<<<blocks, threads, 0, ctx->stream>>>((double*)ctx->stage, iters, 1.0 + rep);
    else probe_fp32_fma_kernel<<<blocks, threads, 0, ctx->stream>>>((float*)ctx->stage, iters, 1.0f + rep);
    ctx->launches++;
    cudaEventRecord(e1, ctx->stream);
    err = cudaEventSynchronize(e1);
    float ms = 0.f;
    if (err == cudaSuccess) err = cudaEventElapsedTime(&ms, e0, e1);
    if (err != cudaSuccess) break;
    if (rep > 0 && ms < best_ms) best_ms = ms;
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (err != cudaSuccess) { (void)cudaGetLastError(); set_error("prad_measure_pipe_rate: %s", cudaGetErrorString(err)); return PRAD_ERR_CUDA; }
  const double per_thread = pipe == 1 ? 4.0 * 512.0 / 32.0 : 8.0 * 2.0;   // flop per thread and iteration
  *out_tflops = per_thread * iters * (double)blocks * threads / (best_ms * 1e-3) / 1e12;
  return PRAD_OK;
}

// ---------------------------------------------------------------- intermediate slots
prad_status prad_slot_store(prad_ctx* ctx, const void* guid_16_bytes, const void* const* ptrs_host,
                            const size_t* bytes_host, int count, int copy) {
  PRAD_CHECK_CTX(ctx);
  PRAD_REQUIRE(guid_16_bytes && count >= 0 && (count == 0 || (ptrs_host && bytes_host)), PRAD_ERR_INVALID,
               "prad_slot_store: null guid or pointer list");
  if (copy) PRAD_NOT_CAPTURING(ctx, "prad_slot_store with copies");
  RuntimeState* r = rt_of(ctx);
  Slot fresh;
  fresh.owns = copy != 0;
  for (int i = 0; i < count; ++i) {
    void* p = const_cast<void*>(ptrs_host[i]);
    if (copy && p && bytes_host[i]) {
      void* q = nullptr;
      cudaError_t e = device_malloc(&q, bytes_host[i]);
      if (e != cudaSuccess) {
        (void)cudaGetLastError();
        free_slot(fresh);
        set_error("prad_slot_store: copy of %zu bytes could not be allocated: %s", bytes_host[i], cudaGetErrorString(e));
        return PRAD_ERR_OOM;
      }
      fresh.ptrs.push_back(q);
      fresh.bytes.push_back(bytes_host[i]);
      e = cudaMemcpyAsync(q, p, bytes_host[i], cudaMemcpyDeviceToDevice, ctx->stream);
      if (e != cudaSuccess) {
        free_slot(fresh);
        set_error("prad_slot_store: device copy failed: %s", cudaGetErrorString(e));
        return PRAD_ERR_CUDA;
      }
    } else {
      fresh.ptrs.push_back(copy ? nullptr : p);
      fresh.bytes.push_back(bytes_host[i]);
    }
  }
  // AddOrUpdate: a second store under the same id replaces the first
  auto it = r->slots.find(guid_of(guid_16_bytes));
  if (it != r->slots.end()) {
    if (it->second.owns) PRAD_CUDA(cudaStreamSynchronize(ctx->stream));   // a kernel may still read the old copies
    free_slot(it->second);
    it->second = std::move(fresh);
  } else {
    r->slots.emplace(guid_of(guid_16_bytes), std::move(fresh));
  }
  return PRAD_OK;
}

prad_status prad_slot_restore(prad_ctx* ctx, const void* guid_16_bytes, void** out_ptrs_host, int count) {
  PRAD_CHECK_CTX(ctx);
  PRAD_REQUIRE(guid_16_bytes && count >= 0 && (count == 0 || out_ptrs_host), PRAD_ERR_INVALID,
               "prad_slot_restore: null guid or output list");
  RuntimeState* r = rt_of(ctx);
  auto it = r->slots.find(guid_of(guid_16_bytes));
  PRAD_REQUIRE(it != r->slots.end(), PRAD_ERR_INVALID,
               "prad_slot_restore: nothing was stored under this id (KeyNotFoundException)");
  PRAD_REQUIRE((int)it->second.ptrs.size() == count, PRAD_ERR_SHAPE,
               "prad_slot_restore: the slot holds %d buffers, %d were asked for", (int)it->second.ptrs.size(), count);
  for (int i = 0; i < count; ++i) out_ptrs_host[i] = it->second.ptrs[i];
  return PRAD_OK;
}

prad_status prad_slot_drop(prad_ctx* ctx, const void* guid_16_bytes) {
  PRAD_CHECK_CTX(ctx);
  PRAD_NOT_CAPTURING(ctx, "prad_slot_drop");
  PRAD_REQUIRE(guid_16_bytes, PRAD_ERR_INVALID, "prad_slot_drop: null guid");
  RuntimeState* r = rt_of(ctx);
  auto it = r->slots.find(guid_of(guid_16_bytes));
  if (it == r->slots.end()) return PRAD_OK;
  if (it->second.owns) PRAD_CUDA(cudaStreamSynchronize(ctx->stream));
  free_slot(it->second);
  r->slots.erase(it);
  return PRAD_OK;
}

prad_status prad_slot_count(prad_ctx* ctx, int* out_count) {
  PRAD_CHECK_CTX(ctx);
  PRAD_REQUIRE(out_count, PRAD_ERR_INVALID, "prad_slot_count: null output");
  *out_count = (int)rt_of(ctx)->slots.size();
  return PRAD_OK;
}

// ---------------------------------------------------------------- packed transfers
prad_status prad_download_many(prad_ctx* ctx, void* dst_host, const void* const* srcs_host, const size_t* bytes_host,
                               int count) {
  PRAD_CHECK_CTX(ctx);
  PRAD_NOT_CAPTURING(ctx, "prad_download_many");
  PRAD_REQUIRE(count >= 0 && (count == 0 || (dst_host && srcs_host && bytes_host)), PRAD_ERR_INVALID,
               "prad_download_many: null pointer");
  char* out = (char*)dst_host;
  for (int i = 0; i < count; ++i) {
    PRAD_REQUIRE(srcs_host[i] || bytes_host[i] == 0, PRAD_ERR_INVALID, "prad_download_many: tensor %d is null", i);
    if (bytes_host[i]) PRAD_CUDA(cudaMemcpyAsync(out, srcs_host[i], bytes_host[i], cudaMemcpyDeviceToHost, ctx->stream));
    out += bytes_host[i];
  }
  PRAD_CUDA(cudaStreamSynchronize(ctx->stream));
  return gemm_tf32x3_check(ctx);
}

prad_status prad_upload_many(prad_ctx* ctx, void* const* dsts_host, const void* src_host, const size_t* bytes_host,
                             int count) {
  PRAD_CHECK_CTX(ctx);
  PRAD_NOT_CAPTURING(ctx, "prad_upload_many");
  PRAD_REQUIRE(count >= 0 && (count == 0 || (dsts_host && src_host && bytes_host)), PRAD_ERR_INVALID,
               "prad_upload_many: null pointer");
  const char* in = (const char*)src_host;
  for (int i = 0; i < count; ++i) {
    PRAD_REQUIRE(dsts_host[i] || bytes_host[i] == 0, PRAD_ERR_INVALID, "prad_upload_many: tensor %d is null", i);
    if (bytes_host[i]) PRAD_CUDA(cudaMemcpyAsync(dsts_host[i], in, bytes_host[i], cudaMemcpyHostToDevice, ctx->stream));
    in += bytes_host[i];
  }
  PRAD_CUDA(cudaStreamSynchronize(ctx->stream));   // the host block may be reused when the call returns
  return PRAD_OK;
}

// ---------------------------------------------------------------- introspection
prad_status prad_device_info(prad_ctx* ctx, prad_device_info_t* out) {
  PRAD_CHECK_CTX(ctx);
  PRAD_REQUIRE(out, PRAD_ERR_INVALID, "prad_device_info: null output");
  memset(out, 0, sizeof(*out));
  cudaDeviceProp p;
  PRAD_CUDA(cudaGetDeviceProperties(&p, ctx->device));
  size_t free_b = 0, total_b = 0;
  PRAD_CUDA(cudaMemGetInfo(&free_b, &total_b));
  out->device = ctx->device;
  out->sm_count = p.multiProcessorCount;
  out->cc_major = p.major;
  out->cc_minor = p.minor;
  out->l2_bytes = p.l2CacheSize;
  out->smem_per_block_optin = (int)p.sharedMemPerBlockOptin;
  int khz = 0;
  if (cudaDeviceGetAttribute(&khz, cudaDevAttrClockRate, ctx->device) == cudaSuccess) out->sm_clock_khz = khz;
  if (cudaDeviceGetAttribute(&khz, cudaDevAttrMemoryClockRate, ctx->device) == cudaSuccess) out->mem_clock_khz = khz;
  (void)cudaGetLastError();
  out->total_bytes = (uint64_t)total_b;
  out->free_bytes = (uint64_t)free_b;
  out->scratch_bytes = (uint64_t)(ctx->ws_bytes + ctx->stage_bytes + ctx->parts_bytes);
  strncpy(out->name, p.name, sizeof(out->name) - 1);
  return PRAD_OK;
}

prad_status prad_timing_begin(prad_ctx* ctx, const char* label) {
  PRAD_CHECK_CTX(ctx);
  PRAD_NOT_CAPTURING(ctx, "prad_timing_begin");
  RuntimeState* r = rt_of(ctx);
  PRAD_REQUIRE(r->open_bracket < 0, PRAD_ERR_INVALID, "prad_timing_begin: the previous bracket is still open");
  PRAD_REQUIRE(r->brackets.size() < 65536, PRAD_ERR_UNSUPPORTED,
               "prad_timing_begin: 65536 brackets are pending; read them with prad_get_timings");
  TimingBracket b;
  memset(b.label, 0, sizeof(b.label));
  if (label) strncpy(b.label, label, sizeof(b.label) - 1);
  PRAD_CUDA(cudaEventCreate(&b.begin));
  cudaError_t e = cudaEventCreate(&b.end);
  if (e != cudaSuccess) { cudaEventDestroy(b.begin); set_error("prad_timing_begin: %s", cudaGetErrorString(e)); return PRAD_ERR_CUDA; }
  b.launches0 = ctx->launches;
  e = cudaEventRecord(b.begin, ctx->stream);
  if (e != cudaSuccess) {
    cudaEventDestroy(b.begin); cudaEventDestroy(b.end);
    set_error("prad_timing_begin: %s", cudaGetErrorString(e));
    return PRAD_ERR_CUDA;
  }
  r->brackets.push_back(b);
  r->open_bracket = (int)r->brackets.size() - 1;
  return PRAD_OK;
}

prad_status prad_timing_end(prad_ctx* ctx) {
  PRAD_CHECK_CTX(ctx);
  RuntimeState* r = rt_of(ctx);
  PRAD_REQUIRE(r->open_bracket >= 0, PRAD_ERR_INVALID, "prad_timing_end: no bracket is open");
  TimingBracket& b = r->brackets[r->open_bracket];
  PRAD_CUDA(cudaEventRecord(b.end, ctx->stream));
  b.launches1 = ctx->launches;
  b.closed = true;
  r->open_bracket = -1;
  return PRAD_OK;
}

prad_status prad_get_timings(prad_ctx* ctx, prad_timing_t* out, int capacity, int* out_count) {
  PRAD_CHECK_CTX(ctx);
  PRAD_NOT_CAPTURING(ctx, "prad_get_timings");
  PRAD_REQUIRE(out_count && capacity >= 0 && (capacity == 0 || out), PRAD_ERR_INVALID, "prad_get_timings: bad argument");
  RuntimeState* r = rt_of(ctx);
  PRAD_REQUIRE(r->open_bracket < 0, PRAD_ERR_INVALID, "prad_get_timings: a bracket is still open");
  PRAD_CUDA(cudaStreamSynchronize(ctx->stream));
  const int n = (int)r->brackets.size();
  *out_count = n;
  for (int i = 0; i < n && i < capacity; ++i) {
    TimingBracket& b = r->brackets[i];
    float ms = 0.f;
    PRAD_CUDA(cudaEventElapsedTime(&ms, b.begin, b.end));
    memset(&out[i], 0, sizeof(out[i]));
    memcpy(out[i].label, b.label, sizeof(out[i].label));
    out[i].milliseconds = (double)ms;
    out[i].launches = b.launches1 - b.launches0;
  }
  if (capacity >= n) free_brackets(r);   // everything was handed over
  return gemm_tf32x3_check(ctx);
}

}  // extern "C"

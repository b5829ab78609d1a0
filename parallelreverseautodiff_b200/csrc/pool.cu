// Device memory of prad_alloc / prad_free: freed blocks are kept and handed out again.
//
// A program that follows the managed contract gets new matrices from every Forward and Backward and
// drops the old ones.  With one cudaMalloc per matrix and a stream wait plus cudaFree per drop (which
// waits for the whole device and unmaps the memory), a 512 x 784 x 256 double node took 2 - 3 ms
// around 0.11 ms of kernels, and a 64-image attention block 14 ms around 4.5 ms.
//
// Rules of the cache:
//  - blocks come in size classes (eight per power of two, multiples of 2 MiB from 64 MiB on) and go
//    back to the context that allocated them, whose stream orders their old work before their new work;
//  - work on the legacy default stream and on blocking streams that was enqueued before the free is
//    waited for as well (an event per cached block), as the cudaFree before it did;
//  - while a context shares its device with others of the process, blocks may be used by all of them: a
//    free notes how far every one's stream is, and a block is handed out again when all of that is done
//    (the host waits; the block that was freed first is taken), so that no context finds work pending on it;
//  - a block that another context frees, or that is freed while a prefetch copy is pending, while another
//    context records or on a context with data-parallel communication, takes the old path: wait and cudaFree;
//  - a prefetch, which runs beside the context's stream, into a block that came out of the cache starts
//    behind what that stream was given before, unless a fence or such a prefetch has seen to that already;
//  - nothing is taken from the cache while a launch sequence is recorded;
//  - the cache of a context is bounded (1/16 of the device memory; the block that was freed first
//    leaves first), and is given back when the context is shut down, when any allocation of this
//    process' contexts fails for lack of memory, or by the option "pool_bytes" = "0".
#include <deque>
#include <mutex>
#include <unordered_map>

#include "common.cuh"

namespace prad {

struct CachedBlock {
  void* p;
  size_t bytes;
  cudaEvent_t freed;   // on the legacy default stream
  std::vector<cudaEvent_t> users;   // on the context's stream and those of the others on its device, if there were any
};

struct DevicePool {
  std::unordered_map<size_t, std::vector<CachedBlock>> by_size;
  std::deque<void*> order;            // cached blocks, oldest first (entries of reused blocks are skipped)
  std::unordered_map<void*, size_t> cached;   // block -> size, for `order`
  std::vector<cudaEvent_t> spare;
  size_t held = 0, cap = 0;
  int64_t fences = 0;                 // how often the context's copy stream was put behind all of its stream's work
  bool recycled = false;              // a block with old work pending was handed out since
};

namespace {
// recycled: what the owner's `fences` was when the block came out of the cache with old work ahead of it on the owner's stream,
// -1 if there is none
struct Live { size_t bytes; prad_ctx* owner; int64_t recycled; };
std::mutex g_pool_mu;
std::unordered_map<void*, Live> g_live;       // every block prad_alloc handed out
std::vector<prad_ctx*> g_contexts;            // every context
std::vector<prad_ctx*> g_pools;               // contexts that have a cache

std::vector<prad_ctx*> others_on_device(const prad_ctx* ctx) {
  std::vector<prad_ctx*> out;
  for (prad_ctx* c : g_contexts)
    if (c != ctx && c->device == ctx->device) out.push_back(c);
  return out;
}
bool recording(cudaStream_t stream) {
  cudaStreamCaptureStatus s = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(stream, &s) == cudaSuccess) return s != cudaStreamCaptureStatusNone;
  (void)cudaGetLastError();
  return true;
}

size_t size_class(size_t bytes) {
  if (bytes <= 256) return 256;
  if (bytes >= ((size_t)64 << 20)) return (bytes + (((size_t)2 << 20) - 1)) & ~(((size_t)2 << 20) - 1);
  int top = 63 - __builtin_clzll((unsigned long long)bytes);
  size_t step = (size_t)1 << (top - 3);
  if (step < 256) step = 256;
  return (bytes + step - 1) / step * step;
}

DevicePool* pool_of(prad_ctx* ctx) {
  if (!ctx->pool) {
    ctx->pool = new DevicePool();
    ctx->pool->cap = ctx->total_mem / 16;
    g_pools.push_back(ctx);
  }
  return ctx->pool;
}

void drop_block(DevicePool* pool, const CachedBlock& b) {
  pool->held -= b.bytes;
  pool->cached.erase(b.p);
  pool->spare.push_back(b.freed);
  pool->spare.insert(pool->spare.end(), b.users.begin(), b.users.end());
  cudaFree(b.p);       // waits for the device: whatever still uses the block is done
}

// frees cached blocks, oldest first, until at most `keep` bytes are held
void shrink(prad_ctx* ctx, size_t keep) {
  DevicePool* pool = ctx->pool;
  if (!pool || pool->held <= keep) return;
  int before = 0;
  cudaGetDevice(&before);
  cudaSetDevice(ctx->device);
  while (pool->held > keep && !pool->order.empty()) {
    void* p = pool->order.front();
    pool->order.pop_front();
    auto it = pool->cached.find(p);
    if (it == pool->cached.end()) continue;
    auto& list = pool->by_size[it->second];
    for (size_t i = 0; i < list.size(); ++i)
      if (list[i].p == p) {
        const CachedBlock b = list[i];
        list.erase(list.begin() + i);
        drop_block(pool, b);
        break;
      }
  }
  cudaSetDevice(before);
}

cudaError_t malloc_or_release(void** out, size_t bytes) {
  cudaError_t e = cudaMalloc(out, bytes);
  if (e != cudaErrorMemoryAllocation) return e;
  (void)cudaGetLastError();
  for (prad_ctx* c : g_pools) shrink(c, 0);
  return cudaMalloc(out, bytes);
}
}  // namespace

prad_status pool_alloc(prad_ctx* ctx, size_t bytes, void** out) {
  const size_t want = size_class(bytes);
  std::unique_lock<std::mutex> lock(g_pool_mu);
  DevicePool* pool = pool_of(ctx);
  auto it = pool->by_size.find(want);
  if (!ctx->capturing && it != pool->by_size.end() && !it->second.empty()) {
    const bool alone = others_on_device(ctx).empty();
    const size_t at = alone ? it->second.size() - 1 : 0;      // the one freed last: likeliest in L2
    const CachedBlock b = std::move(it->second[at]);
    it->second.erase(it->second.begin() + at);
    pool->held -= b.bytes;
    pool->cached.erase(b.p);
    const bool idle = !alone || !b.users.empty();
    if (idle) {
      lock.unlock();
      PRAD_CUDA(cudaEventSynchronize(b.freed));
      for (cudaEvent_t e : b.users) PRAD_CUDA(cudaEventSynchronize(e));
      lock.lock();
    } else if (cudaEventQuery(b.freed) != cudaSuccess) {
      (void)cudaGetLastError();
      PRAD_CUDA(cudaStreamWaitEvent(ctx->stream, b.freed, 0));
    }
    pool->spare.push_back(b.freed);
    pool->spare.insert(pool->spare.end(), b.users.begin(), b.users.end());
    g_live[b.p] = {want, ctx, idle ? -1 : pool->fences};
    pool->recycled = pool->recycled || !idle;
    *out = b.p;
    return PRAD_OK;
  }
  const cudaError_t e = malloc_or_release(out, want);
  if (e != cudaSuccess) {
    (void)cudaGetLastError();
    *out = nullptr;
    set_error("prad_alloc(%zu bytes): %s", bytes, cudaGetErrorString(e));
    return e == cudaErrorMemoryAllocation ? PRAD_ERR_OOM : PRAD_ERR_CUDA;
  }
  g_live[*out] = {want, ctx, -1};
  return PRAD_OK;
}

prad_status pool_free(prad_ctx* ctx, void* p) {
  std::lock_guard<std::mutex> lock(g_pool_mu);
  auto it = g_live.find(p);
  if (it == g_live.end())
    for (prad_ctx* c : g_pools)
      PRAD_REQUIRE(!c->pool->cached.count(p), PRAD_ERR_CUDA, "prad_free: the block at %p was freed before", p);
  const size_t bytes = it == g_live.end() ? 0 : it->second.bytes;
  const bool own = it != g_live.end() && it->second.owner == ctx;
  if (it != g_live.end()) g_live.erase(it);
  DevicePool* pool = own ? pool_of(ctx) : nullptr;
  bool keep = own && bytes <= pool->cap / 4 && !ctx->copy_pending && !ctx->dp;
  std::vector<cudaStream_t> streams;           // of everybody who may use the block, where that is not this context alone
  for (const prad_ctx* c : others_on_device(ctx)) {
    streams.push_back(c->stream);
    keep = keep && !c->copy_pending && !c->dp && !recording(streams.back());
  }
  if (!streams.empty()) streams.push_back(ctx->stream);
  if (keep) {
    CachedBlock b{p, bytes, nullptr, {}};
    auto mark = [&](cudaStream_t stream, cudaEvent_t* out) {
      cudaError_t e = cudaSuccess;
      if (!pool->spare.empty()) {
        *out = pool->spare.back();
        pool->spare.pop_back();
      } else {
        e = cudaEventCreateWithFlags(out, cudaEventDisableTiming);
      }
      return e == cudaSuccess ? cudaEventRecord(*out, stream) : e;
    };
    cudaError_t e = mark(cudaStreamLegacy, &b.freed);
    b.users.assign(streams.size(), nullptr);
    for (size_t i = 0; i < streams.size() && e == cudaSuccess; ++i) e = mark(streams[i], &b.users[i]);
    if (e == cudaSuccess) {
      pool->by_size[bytes].push_back(b);
      pool->order.push_back(p);
      pool->cached[p] = bytes;
      pool->held += bytes;
      if (pool->order.size() > 2 * pool->cached.size() + 64) {      // forget the entries of reused blocks
        std::deque<void*> kept;
        std::unordered_map<void*, int> seen;
        for (auto r = pool->order.rbegin(); r != pool->order.rend(); ++r)
          if (pool->cached.count(*r) && seen[*r]++ == 0) kept.push_front(*r);
        pool->order.swap(kept);
      }
      shrink(ctx, pool->cap);
      return PRAD_OK;
    }
    (void)cudaGetLastError();
    b.users.push_back(b.freed);
    for (cudaEvent_t u : b.users)
      if (u) pool->spare.push_back(u);
  }
  PRAD_CUDA(cudaStreamSynchronize(ctx->stream));
  PRAD_CUDA(cudaFree(p));
  return PRAD_OK;
}

prad_status pool_before_prefetch(prad_ctx* ctx, void* dst, size_t bytes) {
  std::lock_guard<std::mutex> lock(g_pool_mu);
  DevicePool* pool = pool_of(ctx);
  if (!pool->recycled) return PRAD_OK;
  // (a block of another context has no old work pending: its owner is not alone, or is gone and had waited)
  auto pending = [&](const void* p, const Live& l) {
    return l.owner == ctx && l.recycled == pool->fences && (char*)p < (char*)dst + bytes && (char*)dst < (char*)p + l.bytes;
  };
  auto it = g_live.find(dst);
  bool wait = it != g_live.end() && pending(it->first, it->second);
  if (it == g_live.end() || it->second.bytes < bytes)        // inside a block
    for (const auto& kv : g_live) wait = wait || pending(kv.first, kv.second);
  if (!wait) return PRAD_OK;
  PRAD_CUDA(cudaEventRecord(ctx->copy_done, ctx->stream));
  PRAD_CUDA(cudaStreamWaitEvent(ctx->copy_stream, ctx->copy_done, 0));
  pool->fences++;
  pool->recycled = false;
  return PRAD_OK;
}
void pool_fenced(prad_ctx* ctx) {
  std::lock_guard<std::mutex> lock(g_pool_mu);
  DevicePool* pool = pool_of(ctx);
  pool->fences++;
  pool->recycled = false;
}

void pool_limit(prad_ctx* ctx, size_t cap) {
  std::lock_guard<std::mutex> lock(g_pool_mu);
  pool_of(ctx)->cap = cap;
  shrink(ctx, cap);
}

cudaError_t device_malloc(void** out, size_t bytes) {
  std::lock_guard<std::mutex> lock(g_pool_mu);
  return malloc_or_release(out, bytes);
}

// called by prad_init.  What the others on the device freed so far was kept on the understanding that they use their blocks
// alone: from here on none of those is handed out, and none they hold has old work pending.
void pool_enter(prad_ctx* ctx) {
  std::lock_guard<std::mutex> lock(g_pool_mu);
  for (prad_ctx* c : others_on_device(ctx)) {
    shrink(c, 0);
    if (!recording(c->stream)) cudaStreamSynchronize(c->stream);
    for (auto& kv : g_live)
      if (kv.second.owner == c) kv.second.recycled = -1;
  }
  g_contexts.push_back(ctx);
}
void pool_use_stream(prad_ctx* ctx, cudaStream_t stream) {
  std::lock_guard<std::mutex> lock(g_pool_mu);
  ctx->stream = stream;
}
cudaError_t pool_begin_capture(prad_ctx* ctx) {
  std::lock_guard<std::mutex> lock(g_pool_mu);
  return cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeRelaxed);
}

// called by prad_shutdown: cached blocks are freed, blocks still held by the caller stay valid
void pool_destroy(prad_ctx* ctx) {
  std::lock_guard<std::mutex> lock(g_pool_mu);
  for (size_t i = 0; i < g_contexts.size(); ++i)
    if (g_contexts[i] == ctx) { g_contexts.erase(g_contexts.begin() + i); break; }
  for (auto& kv : g_live)
    if (kv.second.owner == ctx) kv.second.owner = nullptr;
  if (!ctx->pool) return;
  shrink(ctx, 0);
  for (cudaEvent_t e : ctx->pool->spare) cudaEventDestroy(e);
  for (size_t i = 0; i < g_pools.size(); ++i)
    if (g_pools[i] == ctx) { g_pools.erase(g_pools.begin() + i); break; }
  delete ctx->pool;
  ctx->pool = nullptr;
}

}  // namespace prad

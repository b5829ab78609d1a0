// Embedding: gather of table rows and the ordered scatter-add of their gradients.
// (Compiled with -fmad=false.)
#include "act_math.cuh"
#include "common.cuh"

namespace prad {

template <typename T> struct EmbVec;
template <> struct EmbVec<float> { using type = float4; static constexpr int N = 4; };
template <> struct EmbVec<double> { using type = double2; static constexpr int N = 2; };

constexpr int EMB_THREADS = 256;
constexpr int EMB_WARPS = EMB_THREADS / 32;

// EmbeddingOperation.cs:56-60: out[i] = W[(int)input[i,0]].  One warp per row, four 128-bit loads in flight per lane
// (16384 rows of 512 floats: 20 -> 12 us against one element per thread).  `bad` receives 1 + an offending position.
template <typename T, bool VECTORS>
__global__ void __launch_bounds__(EMB_THREADS)
embedding_gather_kernel(const T* __restrict__ index_col, const T* __restrict__ W, T* __restrict__ out, int n, int vocab, int dim,
                        int* bad) {
  chain_begin();
  using V = typename std::conditional<VECTORS, typename EmbVec<T>::type, T>::type;
  const int lane = threadIdx.x & 31;
  const int vecs = VECTORS ? dim / EmbVec<T>::N : dim;
  for (int i = blockIdx.x * EMB_WARPS + (threadIdx.x >> 5); i < n; i += gridDim.x * EMB_WARPS) {
    const int idx = (int)index_col[i];
    if (idx < 0 || idx >= vocab) {  // the managed code would throw IndexOutOfRange
      if (lane == 0) *(volatile int*)bad = i + 1;
      continue;
    }
    const V* src = reinterpret_cast<const V*>(W + (int64_t)idx * dim);
    V* dst = reinterpret_cast<V*>(out + (int64_t)i * dim);
    for (int j0 = lane; j0 < vecs; j0 += 128) {
      V v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (j0 + 32 * u < vecs) v[u] = src[j0 + 32 * u];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (j0 + 32 * u < vecs) __stcs(dst + j0 + 32 * u, v[u]);
    }
  }
}

// ---- ordered scatter-add --------------------------------------------------------------------------------
// EmbeddingOperation.cs:69-76: dW[idx[i]][j] += dOut[i][j] for i = 0..n-1 IN THAT ORDER, bit for bit, without
// floating-point atomics; rows nobody hit become zeros.
//
// The positions are grouped by row first (a counting pass, a place for every row's list, a filling pass -- integer atomics,
// so a list arrives in any order), and whoever sums a row puts its list into input order: a warp ranks up to 32 positions
// against each other, a CTA sorts longer lists with a bitmap over the positions.  Then every row is read and written once.
// (With every CTA scanning the whole index column for its rows instead, a pass over 16384 indices of a 50000 x 512 table took
// 560 us, most of it for scanning; now 12 us for the grouping and 44 for the sums, 52 with a cold cache: the table's 102 MB are 16.)
// Rows of many hits are the commonest words of a text: the commonest of 16384 appears a thousand times, and its additions are
// a chain, so 32 vectors of such a row have a CTA to themselves whose eight teams of threads copy rows of dOut into a ring in
// shared memory, 48 rows ahead of the team that adds them (with 16 rows in flight in registers that one row took 150 us).  The
// ring is 32 KB because the CTAs of the other rows, which make up most of the pass, have room for it too.
constexpr int EMB_FEW = 32;                       // hits a warp orders by itself
constexpr int EMB_WINDOW = 65536;                 // positions of one bitmap
constexpr int EMB_LIST = 2048;                    // ordered positions handed to the summing loop at a time
constexpr int EMB_ROWS = 8;                       // table rows a warp takes at once
constexpr int EMB_GROUP = 32;                     // vectors of a row of many hits that a CTA takes
constexpr int EMB_CHUNK = 16, EMB_CHUNKS = 4;     // rows per step of the ring, steps in the ring

struct EmbPlan {
  int *count, *offset, *slot, *list, *hot;        // per row, per row, per position, per position, rows of many hits
  int* cursor;                                    // [0] list entries given away, [1] rows of many hits
};

template <typename T>
__global__ void __launch_bounds__(EMB_THREADS)
emb_count_kernel(const T* __restrict__ index_col, EmbPlan p, int n, int vocab, int* bad) {
  chain_begin();
  for (int i = blockIdx.x * EMB_THREADS + threadIdx.x; i < n; i += gridDim.x * EMB_THREADS) {
    const int idx = (int)index_col[i];
    if (idx < 0 || idx >= vocab) *(volatile int*)bad = i + 1;
    else p.slot[i] = atomicAdd(p.count + idx, 1);
  }
}
__global__ void __launch_bounds__(EMB_THREADS)
emb_place_kernel(EmbPlan p, int vocab) {
  chain_begin();
  const int v = blockIdx.x * EMB_THREADS + threadIdx.x, lane = threadIdx.x & 31;
  const int c = v < vocab ? p.count[v] : 0;
  int incl = c;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += u;
  }
  int base = 0;
  if (lane == 31 && incl) base = atomicAdd(p.cursor, incl);
  base = __shfl_sync(0xffffffffu, base, 31);
  if (v < vocab) p.offset[v] = base + incl - c;
  if (c > EMB_FEW) p.hot[atomicAdd(p.cursor + 1, 1)] = v;
}
template <typename T>
__global__ void __launch_bounds__(EMB_THREADS)
emb_fill_kernel(const T* __restrict__ index_col, EmbPlan p, int n, int vocab) {
  chain_begin();
  for (int i = blockIdx.x * EMB_THREADS + threadIdx.x; i < n; i += gridDim.x * EMB_THREADS) {
    const int idx = (int)index_col[i];
    if (idx >= 0 && idx < vocab) p.list[p.offset[idx] + p.slot[i]] = i;
  }
}

// Counting, places and filling of a small call in one cluster of eight CTAs, a cluster barrier between the passes: as a memset
// and three launches the grouping of 16384 positions took 15 us, most of it launches.
constexpr int EMB_PLAN_MOST = 1 << 17;            // positions and rows together
__device__ __forceinline__ void emb_plan_barrier() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
template <typename T>
__global__ void __cluster_dims__(8, 1, 1) __launch_bounds__(1024)
emb_plan_kernel(const T* __restrict__ index_col, EmbPlan p, int n, int vocab, int* bad) {
  constexpr int THREADS = 8 * 1024;
  const int t = blockIdx.x * 1024 + threadIdx.x, lane = threadIdx.x & 31;
  if (t < 2) p.cursor[t] = 0;
#pragma unroll 8
  for (int v = t; v < vocab; v += THREADS) p.count[v] = 0;
  emb_plan_barrier();
#pragma unroll 4
  for (int i = t; i < n; i += THREADS) {
    const int idx = (int)index_col[i];
    if (idx < 0 || idx >= vocab) *(volatile int*)bad = i + 1;
    else p.slot[i] = atomicAdd(p.count + idx, 1);
  }
  emb_plan_barrier();
  constexpr int K = 8;                            // rows per thread and trip: one atomic round trip for 65536 rows
  for (int v0 = t; v0 - lane < vocab; v0 += K * THREADS) {
    int c[K], total = 0;
#pragma unroll
    for (int k = 0; k < K; ++k) c[k] = v0 + k * THREADS < vocab ? __ldcg(p.count + v0 + k * THREADS) : 0;
#pragma unroll
    for (int k = 0; k < K; ++k) total += c[k];
    int incl = total;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += u;
    }
    int at = 0;
    if (lane == 31 && incl) at = atomicAdd(p.cursor, incl);
    at = __shfl_sync(0xffffffffu, at, 31) + incl - total;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int v = v0 + k * THREADS;
      if (v < vocab) p.offset[v] = at;
      at += c[k];
      if (c[k] > EMB_FEW) p.hot[atomicAdd(p.cursor + 1, 1)] = v;
    }
  }
  emb_plan_barrier();
#pragma unroll 4
  for (int i = t; i < n; i += THREADS) {
    const int idx = (int)index_col[i];
    if (idx >= 0 && idx < vocab) p.list[__ldcg(p.offset + idx) + p.slot[i]] = i;
  }
}

template <int BYTES> __device__ __forceinline__ void emb_copy(void* dst, const void* src) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  if constexpr (BYTES == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(d), "l"(src), "n"(BYTES) : "memory");
}

template <typename T, typename V> __device__ __forceinline__ void emb_add(V& acc, const V& x) {
  T* a = reinterpret_cast<T*>(&acc);
  const T* b = reinterpret_cast<const T*>(&x);
#pragma unroll
  for (int q = 0; q < (int)(sizeof(V) / sizeof(T)); ++q) a[q] = add_rn(a[q], b[q]);
}
template <typename T, typename V> __device__ __forceinline__ V emb_zero() {
  V v;
  T* a = reinterpret_cast<T*>(&v);
#pragma unroll
  for (int q = 0; q < (int)(sizeof(V) / sizeof(T)); ++q) a[q] = (T)0;
  return v;
}

// CTAs [0, hot_ctas) take (row of many hits, group of 32 vectors) pairs, the others eight table rows per warp.
template <typename T, bool VECTORS>
__global__ void __launch_bounds__(EMB_THREADS)
emb_sum_kernel(const T* __restrict__ dOut, T* __restrict__ dW, EmbPlan p, int n, int vocab, int dim, int hot_ctas) {
  chain_begin();
  using V = typename std::conditional<VECTORS, typename EmbVec<T>::type, T>::type;
  const int vecs = VECTORS ? dim / EmbVec<T>::N : dim;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  __shared__ int ordered[EMB_LIST];
  if ((int)blockIdx.x >= hot_ctas) {
    const int r0 = (((int)blockIdx.x - hot_ctas) * EMB_WARPS + w) * EMB_ROWS;
    int* mine = ordered + w * EMB_FEW;
    int cnt = 0, off = 0;
    if (lane < EMB_ROWS && r0 + lane < vocab) {
      cnt = p.count[r0 + lane];
      off = p.offset[r0 + lane];
    }
    for (int q = 0; q < EMB_ROWS && r0 + q < vocab; ++q) {
      const int c = __shfl_sync(0xffffffffu, cnt, q), o = __shfl_sync(0xffffffffu, off, q);
      if (c > EMB_FEW) continue;
      V* row = reinterpret_cast<V*>(dW + (int64_t)(r0 + q) * dim);
      if (c == 0) {
        for (int j = lane; j < vecs; j += 32) __stcs(row + j, emb_zero<T, V>());
        continue;
      }
      const int pos = lane < c ? p.list[o + lane] : 0x7fffffff;
      int rank = 0;
      for (int k = 0; k < c; ++k) rank += __shfl_sync(0xffffffffu, pos, k) < pos;
      __syncwarp();
      if (lane < c) mine[rank] = pos;
      __syncwarp();
      for (int j = lane; j < vecs; j += 32) {
        V acc = emb_zero<T, V>();
        for (int k0 = 0; k0 < c; k0 += 4) {
          V x[4];
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (k0 + u < c) x[u] = __ldcs(reinterpret_cast<const V*>(dOut + (int64_t)mine[k0 + u] * dim) + j);
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (k0 + u < c) emb_add<T, V>(acc, x[u]);
        }
        __stcs(row + j, acc);
      }
    }
    return;
  }
  __shared__ unsigned bits[EMB_WINDOW / 32];
  __shared__ int warp_sum[EMB_WARPS];
  constexpr int WORDS = EMB_WINDOW / 32 / EMB_THREADS;       // bitmap words per thread
  extern __shared__ __align__(16) unsigned char emb_smem[];
  V* ring = reinterpret_cast<V*>(emb_smem);                  // [EMB_CHUNKS][EMB_CHUNK][EMB_GROUP]
  constexpr int TEAMS = EMB_THREADS / EMB_GROUP;
  const int team = tid / EMB_GROUP, jl = tid % EMB_GROUP;
  const int groups = (vecs + EMB_GROUP - 1) / EMB_GROUP;
  const int64_t tasks = (int64_t)p.cursor[1] * groups;
  for (int64_t h = blockIdx.x; h < tasks; h += hot_ctas) {
    const int v = p.hot[h / groups], j = (int)(h % groups) * EMB_GROUP + jl;
    const int c = p.count[v], o = p.offset[v];
    const V* col = reinterpret_cast<const V*>(dOut) + j;
    V acc = emb_zero<T, V>();
    for (int w0 = 0; w0 < n; w0 += EMB_WINDOW) {
#pragma unroll
      for (int k = 0; k < WORDS; ++k) bits[k * EMB_THREADS + tid] = 0;
      __syncthreads();
      for (int k = tid; k < c; k += EMB_THREADS) {
        const int q = p.list[o + k] - w0;
        if (q >= 0 && q < EMB_WINDOW) atomicOr(bits + (q >> 5), 1u << (q & 31));
      }
      __syncthreads();
      int here = 0;
#pragma unroll
      for (int k = 0; k < WORDS; ++k) here += __popc(bits[tid * WORDS + k]);
      int incl = here;
#pragma unroll
      for (int s = 1; s < 32; s <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, incl, s);
        if (lane >= s) incl += u;
      }
      if (lane == 31) warp_sum[w] = incl;
      __syncthreads();
      int base = incl - here, total = 0;
#pragma unroll
      for (int k = 0; k < EMB_WARPS; ++k) {
        if (k < w) base += warp_sum[k];
        total += warp_sum[k];
      }
      for (int r0 = 0; r0 < total; r0 += EMB_LIST) {
        int rank = base - r0;
        for (int k = 0; k < WORDS; ++k)
          for (unsigned m = bits[tid * WORDS + k]; m; m &= m - 1, ++rank)
            if (rank >= 0 && rank < EMB_LIST) ordered[rank] = w0 + (tid * WORDS + k) * 32 + __ffs(m) - 1;
        __syncthreads();
        const int m = total - r0 < EMB_LIST ? total - r0 : EMB_LIST, steps = (m + EMB_CHUNK - 1) / EMB_CHUNK;
        auto fetch = [&](int step) {
          if (step < steps && j < vecs)
#pragma unroll
            for (int q = 0; q < EMB_CHUNK / TEAMS; ++q) {
              const int k = step * EMB_CHUNK + q * TEAMS + team;
              if (k < m)
                emb_copy<sizeof(V)>(ring + (step % EMB_CHUNKS * EMB_CHUNK + q * TEAMS + team) * EMB_GROUP + jl,
                                    col + (int64_t)ordered[k] * vecs);
            }
          asm volatile("cp.async.commit_group;" ::: "memory");
        };
        for (int i = 0; i < EMB_CHUNKS - 1; ++i) fetch(i);
        for (int i = 0; i < steps; ++i) {
          asm volatile("cp.async.wait_group %0;" ::"n"(EMB_CHUNKS - 2) : "memory");
          __syncthreads();                                   // chunk i is there; chunk i - 1 has been added
          fetch(i + EMB_CHUNKS - 1);
          if (team == 0) {
            const V* x = ring + i % EMB_CHUNKS * EMB_CHUNK * EMB_GROUP + jl;
            const int here2 = m - i * EMB_CHUNK < EMB_CHUNK ? m - i * EMB_CHUNK : EMB_CHUNK;
#pragma unroll 8
            for (int k = 0; k < here2; ++k) emb_add<T, V>(acc, x[k * EMB_GROUP]);
          }
        }
        __syncthreads();
      }
    }
    if (team == 0 && j < vecs) __stcs(reinterpret_cast<V*>(dW + (int64_t)v * dim) + j, acc);
  }
}

template <typename T>
static prad_status scatter_t(prad_ctx* ctx, const void* index_col, const void* dOut, void* dW, int n, int vocab, int dim, int* bad,
                             cudaEvent_t checked = nullptr) {
  const size_t words = 3 * (size_t)vocab + 2 * (size_t)n + 64;
  prad_status s = ensure_stage(ctx, words * sizeof(int));
  if (s) return s;
  EmbPlan p;
  p.cursor = (int*)ctx->stage;
  p.count = p.cursor + 64;
  p.offset = p.count + vocab;
  p.hot = p.offset + vocab;
  p.slot = p.hot + vocab;
  p.list = p.slot + n;
  const T* idx = (const T*)index_col;
  const bool small = (int64_t)n + vocab <= EMB_PLAN_MOST && n > 0;
  if (!small) PRAD_CUDA(cudaMemsetAsync(p.cursor, 0, (64 + (size_t)vocab) * sizeof(int), ctx->stream));
  if (small) {
    emb_plan_kernel<T><<<8, 1024, 0, ctx->stream>>>(idx, p, n, vocab, bad);
    PRAD_LAUNCHED(ctx);
    if (checked) PRAD_CUDA(cudaEventRecord(checked, ctx->stream));       // `bad` is known
  } else if (n > 0) {
    const int g = stream_grid(ctx, n, EMB_THREADS, 8);
    launch_chained(emb_count_kernel<T>, g, EMB_THREADS, 0, ctx->stream, idx, p, n, vocab, bad);
    PRAD_LAUNCHED(ctx);
    if (checked) PRAD_CUDA(cudaEventRecord(checked, ctx->stream));       // `bad` is known
    launch_chained(emb_place_kernel, (unsigned)ceil_div(vocab, EMB_THREADS), EMB_THREADS, 0, ctx->stream, p, vocab);
    PRAD_LAUNCHED(ctx);
    launch_chained(emb_fill_kernel<T>, g, EMB_THREADS, 0, ctx->stream, idx, p, n, vocab);
    PRAD_LAUNCHED(ctx);
  }
  const int hot = n > EMB_FEW ? 2 * ctx->sm_count : 0;
  const unsigned grid = (unsigned)(hot + ceil_div(vocab, EMB_WARPS * EMB_ROWS));
  // shared memory for the ring only where a row can have many hits
  if (dim % EmbVec<T>::N == 0 && (((uintptr_t)dOut | (uintptr_t)dW) & 15) == 0) {
    constexpr int ring = EMB_CHUNKS * EMB_CHUNK * EMB_GROUP * 16;
    s = allow_smem<emb_sum_kernel<T, true>>(ctx, ring);
    if (s) return s;
    launch_chained(emb_sum_kernel<T, true>, grid, EMB_THREADS, hot ? ring : 0, ctx->stream, (const T*)dOut, (T*)dW, p, n, vocab, dim, hot);
  } else {
    constexpr int ring = EMB_CHUNKS * EMB_CHUNK * EMB_GROUP * (int)sizeof(T);
    s = allow_smem<emb_sum_kernel<T, false>>(ctx, ring);
    if (s) return s;
    launch_chained(emb_sum_kernel<T, false>, grid, EMB_THREADS, hot ? ring : 0, ctx->stream, (const T*)dOut, (T*)dW, p, n, vocab, dim, hot);
  }
  PRAD_LAUNCHED(ctx);
  return PRAD_OK;
}

// Also used by the PRAD Tensor gather reverse: dW[idx[i]] += dOut[i] for i ascending; `bad` is an int the device can write
// that receives 1 + an offending position.
prad_status embedding_scatter_ordered(prad_ctx* ctx, prad_dtype dt, const void* index_col, const void* dOut,
                                      void* dW, int n, int vocab, int dim, int* bad) {
  return dt == PRAD_F32 ? scatter_t<float>(ctx, index_col, dOut, dW, n, vocab, dim, bad)
                        : scatter_t<double>(ctx, index_col, dOut, dW, n, vocab, dim, bad);
}

// The offending position of a call arrives in page-locked host memory, so the check costs the wait alone.
static prad_status check_bad_index(prad_ctx* ctx, const char* who, cudaEvent_t checked = nullptr) {
  if (checked) PRAD_CUDA(cudaEventSynchronize(checked));
  else PRAD_CUDA(cudaStreamSynchronize(ctx->stream));
  const int h = *(volatile int*)ctx->host_flag;
  PRAD_REQUIRE(h == 0, PRAD_ERR_INVALID, "%s: index at input row %d is outside [0, vocab)", who, h - 1);
  return PRAD_OK;
}

template <typename T>
static prad_status gather_t(prad_ctx* ctx, const void* index_col, const void* W, void* out, int n, int vocab, int dim) {
  const int grid = stream_grid(ctx, n, EMB_WARPS, 8);
  if (dim % EmbVec<T>::N == 0 && (((uintptr_t)W | (uintptr_t)out) & 15) == 0)
    launch_chained(embedding_gather_kernel<T, true>, grid, EMB_THREADS, 0, ctx->stream, (const T*)index_col, (const T*)W, (T*)out, n, vocab, dim, ctx->host_flag);
  else
    launch_chained(embedding_gather_kernel<T, false>, grid, EMB_THREADS, 0, ctx->stream, (const T*)index_col, (const T*)W, (T*)out, n, vocab, dim, ctx->host_flag);
  PRAD_LAUNCHED(ctx);
  return PRAD_OK;
}

}  // namespace prad

using namespace prad;

extern "C" {

prad_status prad_embedding_forward(prad_ctx* ctx, prad_dtype dt, const void* index_col,
                                   const void* W, void* out, int n, int vocab, int dim) {
  PRAD_CHECK_CTX(ctx);
  PRAD_REQUIRE(dtype_ok(dt) && n >= 0 && vocab >= 0 && dim >= 0, PRAD_ERR_INVALID,
               "prad_embedding_forward: bad argument");
  if (n == 0 || dim == 0) return PRAD_OK;
  PRAD_REQUIRE(index_col && W && out, PRAD_ERR_INVALID, "prad_embedding_forward: null pointer");
  PRAD_NOT_CAPTURING(ctx, "prad_embedding_forward");   // the index check reads a flag back
  *(volatile int*)ctx->host_flag = 0;
  prad_status s = dt == PRAD_F32 ? gather_t<float>(ctx, index_col, W, out, n, vocab, dim) : gather_t<double>(ctx, index_col, W, out, n, vocab, dim);
  return s ? s : check_bad_index(ctx, "prad_embedding_forward");
}

prad_status prad_embedding_backward(prad_ctx* ctx, prad_dtype dt, const void* index_col,
                                    const void* dOut, void* dW, int n, int vocab, int dim) {
  PRAD_CHECK_CTX(ctx);
  PRAD_REQUIRE(dtype_ok(dt) && n >= 0 && vocab >= 0 && dim >= 0, PRAD_ERR_INVALID,
               "prad_embedding_backward: bad argument");
  if (vocab == 0 || dim == 0) return PRAD_OK;
  PRAD_REQUIRE(dW && (n == 0 || (index_col && dOut)), PRAD_ERR_INVALID,
               "prad_embedding_backward: null pointer");
  PRAD_NOT_CAPTURING(ctx, "prad_embedding_backward");
  *(volatile int*)ctx->host_flag = 0;
  // the indices have been looked at once the first kernel is done: the caller need not wait for the sums
  if (!ctx->flag_read) PRAD_CUDA(cudaEventCreateWithFlags(&ctx->flag_read, cudaEventDisableTiming));
  prad_status s = dt == PRAD_F32 ? scatter_t<float>(ctx, index_col, dOut, dW, n, vocab, dim, ctx->host_flag, ctx->flag_read)
                                 : scatter_t<double>(ctx, index_col, dOut, dW, n, vocab, dim, ctx->host_flag, ctx->flag_read);
  return s || n == 0 ? s : check_bad_index(ctx, "prad_embedding_backward", ctx->flag_read);
}

}  // extern "C"

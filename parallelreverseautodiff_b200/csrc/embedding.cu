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

// Where a call's host code learns of an index outside the table: flag[0] receives 1 + an offending position, and flag[1] the call's
// ticket once every index has been looked at.  Both lie in page-locked host memory.
__device__ __forceinline__ void emb_bad(int* flag, int i) {
  *(volatile int*)flag = i + 1;
  __threadfence_system();
}
__device__ __forceinline__ void emb_all_checked(int* flag, int ticket) {
  __threadfence_system();
  *(volatile int*)(flag + 1) = ticket;
}

// EmbeddingOperation.cs:56-60: out[i] = W[(int)input[i,0]].  One warp per row, four 128-bit loads in flight per lane
// (16384 rows of 512 floats: 20 -> 12 us against one element per thread).  The first `checkers` CTAs look at all indices
// instead, so that the host is back 3 us after the kernel has started instead of waiting for its 9 us and the stream.
template <typename T, bool VECTORS>
__global__ void __launch_bounds__(EMB_THREADS)
embedding_gather_kernel(const T* __restrict__ index_col, const T* __restrict__ W, T* __restrict__ out, int n, int vocab, int dim,
                        int* flag, int ticket, int checkers, int* checked) {
  chain_begin();
  if ((int)blockIdx.x < checkers) {
#pragma unroll 8
    for (int64_t i = blockIdx.x * EMB_THREADS + threadIdx.x; i < n; i += checkers * EMB_THREADS) {      // (n up to the last int)
      const int idx = (int)index_col[i];
      if (idx < 0 || idx >= vocab) emb_bad(flag, (int)i);   // the managed code would throw IndexOutOfRange
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      __threadfence();
      if (atomicAdd(checked, 1) == checkers - 1) {     // the last one: the counter is ready for the next call
        *checked = 0;
        emb_all_checked(flag, ticket);
      }
    }
    return;
  }
  using V = typename std::conditional<VECTORS, typename EmbVec<T>::type, T>::type;
  const int lane = threadIdx.x & 31;
  const int vecs = VECTORS ? dim / EmbVec<T>::N : dim;
  for (int i = ((int)blockIdx.x - checkers) * EMB_WARPS + (threadIdx.x >> 5); i < n; i += ((int)gridDim.x - checkers) * EMB_WARPS) {
    const int idx = (int)index_col[i];
    if (idx < 0 || idx >= vocab) continue;
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
// The positions are grouped by row first (integer atomics, so a row's list arrives in any order) while the rest of the GPU writes
// zeros over the table.  Then only the rows that were hit are summed: whoever sums a row puts its list into input order, a warp by
// ranking up to 32 positions against each other, a CTA by a bitmap over the positions.  16384 word-like positions, a 50000 x 512
// float table: with a grouping of four passes by a cluster of eight CTAs and sums that wrote the zeros in the place of rows without
// hits, eight rows a warp one after another, gather and scatter took 82 us; now 62.  The scatter alone, evenly spread positions: 5962
// over 130 rows of 394 floats 38 -> 27 us, 8677 over 157 of 858 doubles 51 -> 37, two million over 50000 of 512 floats 46 200 -> 2100.
// A row of many hits is summed by a CTA, whose threads copy rows of dOut into a ring in shared memory ahead of those that add them, a
// value each.  Up to 256 hits a CTA takes 32 vectors of the row, and orders the list by comparing every position with every other.
// The commonest words of a text have more, the commonest of 16384 over a thousand, and their additions are a chain: a CTA takes 8
// vectors of such a row, with 192 rows of dOut on their way, and where one launch has grouped the positions the longest chains begin
// first.  (That row took 38 000 cycles, after two others, with the additions of four values per lane waiting for every read, and the
// whole pass waited for it.  With 8 vectors a task for all rows of many hits, 32768 positions over 500 rows of 1024 doubles took
// 1470 us, most of it for putting the same list into order 64 times and for finding it; now 139.)
constexpr int EMB_FEW = 32;                       // hits a warp orders by itself
constexpr int EMB_MANY = 256;                     // hits a CTA's threads order, one each
constexpr int EMB_POSITIONS = 32768;              // most positions of a small call: the bitmap that orders lists of more
constexpr int EMB_ROWS = 8;                       // table rows a warp takes at once where the table is walked
constexpr int EMB_LIST = 2048;                    // ordered positions handed to the summing loop at a time
constexpr int EMB_WIDE = 32, EMB_NARROW = 8;      // vectors of a row of many, of very many hits that a CTA takes
constexpr int EMB_STEP = 512, EMB_STEPS = 4;      // vectors per step of the ring, steps in the ring

// The rows with hits, in `segments` parts of `stride` entries: part q has few[q] rows of few hits from its front, and from its back
// very[q] rows of very many and then many[q] rows of many.  An entry's hits are list[offset .. offset + count), with count and offset
// by entry.  A large call has one part and count and offset by row; its rows of very many hits follow the part, and their lists in
// `ordered` are in input order.  It may walk the table row by row, zeros included, instead of the entries of few hits.
struct EmbPlan {
  int *count, *offset, *rows, *list;
  const int *few, *many, *very, *ordered;
  int segments, stride;
  bool large, walk;
};

// A large call: a counting pass, a place for every row's list, a filling pass, and a pass that orders the longest lists.  cursor[0]: list
// entries given away, and in the high word the rows of few hits; cursor[1]: rows of many, and of very many.  One atomic addition per
// warp for the places.
template <typename T>
__global__ void __launch_bounds__(EMB_THREADS)
emb_count_kernel(const T* __restrict__ index_col, EmbPlan p, int* __restrict__ slot, int n, int vocab, int* bad) {
  chain_begin();
  for (int i = blockIdx.x * EMB_THREADS + threadIdx.x; i < n; i += gridDim.x * EMB_THREADS) {
    const int idx = (int)index_col[i];
    if (idx < 0 || idx >= vocab) *(volatile int*)bad = i + 1;
    else slot[i] = atomicAdd(p.count + idx, 1);
  }
}
__global__ void __launch_bounds__(EMB_THREADS)
emb_place_kernel(EmbPlan p, unsigned long long* __restrict__ cursor, int vocab) {
  chain_begin();
  const int v = blockIdx.x * EMB_THREADS + threadIdx.x, lane = threadIdx.x & 31;
  const int c = v < vocab ? p.count[v] : 0, few = c > 0 && c <= EMB_FEW;
  int incl = c, rank = few;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, incl, o), r = __shfl_up_sync(0xffffffffu, rank, o);
    if (lane >= o) incl += u, rank += r;
  }
  unsigned long long at = 0;
  if (lane == 31 && incl) at = atomicAdd(cursor, ((unsigned long long)rank << 32) + incl);
  at = __shfl_sync(0xffffffffu, at, 31);
  if (v < vocab) p.offset[v] = (int)(unsigned)at + incl - c;
  if (few && !p.walk) p.rows[(int)(at >> 32) + rank - 1] = v;
  if (c > EMB_MANY) p.rows[p.stride + (int)(atomicAdd(cursor + 1, 1ull << 32) >> 32)] = v;
  else if (c > EMB_FEW) p.rows[p.stride - 1 - (int)(unsigned)atomicAdd(cursor + 1, 1ull)] = v;
}
template <typename T>
__global__ void __launch_bounds__(EMB_THREADS)
emb_fill_kernel(const T* __restrict__ index_col, EmbPlan p, const int* __restrict__ slot, int n, int vocab) {
  chain_begin();
  for (int i = blockIdx.x * EMB_THREADS + threadIdx.x; i < n; i += gridDim.x * EMB_THREADS) {
    const int idx = (int)index_col[i];
    if (idx >= 0 && idx < vocab) p.list[p.offset[idx] + slot[i]] = i;
  }
}

// The lists of more than EMB_MANY hits in input order, a row to a CTA: by a bitmap over a window of the positions after the other.  (As
// part of every task that sums 8 vectors of the row, 2^20 word-like positions of 512 floats had it done 16 times.)
constexpr int EMB_ORDER_THREADS = 1024, EMB_ORDER_WINDOW = 1 << 18;
__global__ void __launch_bounds__(EMB_ORDER_THREADS)
emb_order_kernel(EmbPlan p, int* __restrict__ ordered, int n) {
  chain_begin();
  constexpr int NT = EMB_ORDER_THREADS, WORDS = EMB_ORDER_WINDOW / 32 / NT;      // bitmap words per thread
  __shared__ unsigned bits[EMB_ORDER_WINDOW / 32];
  __shared__ int warp_sum[NT / 32];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, rows = *p.very;
  for (int r = blockIdx.x; r < rows; r += gridDim.x) {
    const int v = p.rows[p.stride + r], c = p.count[v];
    const int* list = p.list + p.offset[v];
    int* to = ordered + p.offset[v];
    for (int64_t w0 = 0; w0 < n; w0 += EMB_ORDER_WINDOW) {
#pragma unroll
      for (int k = 0; k < WORDS; ++k) bits[k * NT + tid] = 0;
      __syncthreads();
#pragma unroll 4
      for (int k = tid; k < c; k += NT) {
        const int64_t q = list[k] - w0;
        if (q >= 0 && q < EMB_ORDER_WINDOW) atomicOr(bits + (q >> 5), 1u << (q & 31));
      }
      __syncthreads();
      unsigned mine[WORDS];
      int set = 0;
#pragma unroll
      for (int k = 0; k < WORDS; ++k) {
        mine[k] = bits[tid * WORDS + k];
        set += __popc(mine[k]);
      }
      int incl = set;
#pragma unroll
      for (int s = 1; s < 32; s <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, incl, s);
        if (lane >= s) incl += u;
      }
      if (lane == 31) warp_sum[w] = incl;
      __syncthreads();
      int at = incl - set, total = 0;
#pragma unroll 8
      for (int k = 0; k < NT / 32; ++k) {
        if (k < w) at += warp_sum[k];
        total += warp_sum[k];
      }
#pragma unroll
      for (int k = 0; k < WORDS; ++k)
        for (unsigned m = mine[k]; m; m &= m - 1) to[at++] = (int)(w0 + (tid * WORDS + k) * 32 + __ffs(m) - 1);
      to += total;
      __syncthreads();
    }
  }
}

// A small call in one launch: each of `segments` CTAs reads all indices and groups those of its own rows in shared memory, and the
// indices below its rows say where its lists begin, so no CTA waits for another (as passes of a cluster over counts in L2 the
// grouping of 16384 positions took 12 us, and more beside the zeros that the other CTAs write meanwhile).
constexpr int EMB_PLAN_MOST = 1 << 17;            // positions and rows together
constexpr int EMB_SEGMENTS = 16, EMB_PLAN_THREADS = 1024;
template <typename T>
__global__ void __launch_bounds__(EMB_PLAN_THREADS)
emb_plan_kernel(const T* __restrict__ index_col, EmbPlan p, int* __restrict__ few, int* __restrict__ many, int* __restrict__ very, int n, int vocab, int* flag,
                int ticket, uint4* __restrict__ clear, int64_t clear_vecs) {
  chain_begin();
  constexpr int NT = EMB_PLAN_THREADS;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, q = blockIdx.x;
  if (q >= p.segments) {
    const int64_t stride = (int64_t)(gridDim.x - p.segments) * NT;
#pragma unroll 4
    for (int64_t i = (int64_t)(q - p.segments) * NT + tid; i < clear_vecs; i += stride) clear[i] = make_uint4(0, 0, 0, 0);
    return;
  }
  __shared__ int place[EMB_PLAN_MOST / EMB_SEGMENTS];        // of the CTA's rows: hits, then where the next one goes
  __shared__ int sums[5][NT / 32];
  __shared__ int totals[5];
  const int lo = q * p.stride, mine = vocab - lo < p.stride ? vocab - lo : p.stride;
  for (int v = tid; v < mine; v += NT) place[v] = 0;
  __syncthreads();
  int below = 0;
#pragma unroll 8
  for (int i = tid; i < n; i += NT) {
    const int idx = (int)index_col[i];
    if (idx < 0 || idx >= vocab) {
      if (q == 0) emb_bad(flag, i);
    } else if (idx < lo) {
      ++below;
    } else if (idx < lo + mine) {
      atomicAdd(place + idx - lo, 1);
    }
  }
  __syncthreads();
  if (q == 0 && tid == 0 && ticket) emb_all_checked(flag, ticket);
  // neighbouring rows to a thread; a scan over the threads of hits, rows of few, of many and of very many hits
  const int per = (mine + NT - 1) / NT, r0 = tid * per, r1 = r0 + per < mine ? r0 + per : mine;
  int v[5] = {below, 0, 0, 0, 0};
  for (int r = r0; r < r1; ++r) {
    const int c = place[r];
    v[1] += c;
    v[2] += c > 0 && c <= EMB_FEW;
    v[3] += c > EMB_FEW && c <= EMB_MANY;
    v[4] += c > EMB_MANY;
  }
  int incl[5];
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    incl[k] = v[k];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, incl[k], o);
      if (lane >= o) incl[k] += u;
    }
    if (lane == 31) sums[k][w] = incl[k];
  }
  __syncthreads();
  if (w < 5) {
    int x = sums[w][lane], y = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, y, o);
      if (lane >= o) y += u;
    }
    sums[w][lane] = y - x;
    if (lane == 31) totals[w] = y;
  }
  __syncthreads();
  int at = totals[0] + sums[1][w] + incl[1] - v[1], front = lo + sums[2][w] + incl[2] - v[2], back = lo + p.stride - 1 - (totals[4] + sums[3][w] + incl[3] - v[3]);
  int first = lo + p.stride - 1 - (sums[4][w] + incl[4] - v[4]);
  for (int r = r0; r < r1; ++r) {
    const int c = place[r];
    place[r] = at;
    if (c) {
      const int e = c <= EMB_FEW ? front++ : c <= EMB_MANY ? back-- : first--;
      p.rows[e] = lo + r;
      p.count[e] = c;
      p.offset[e] = at;
    }
    at += c;
  }
  if (tid == 0) {
    few[q] = totals[2];
    many[q] = totals[3];
    very[q] = totals[4];
  }
  __syncthreads();
#pragma unroll 8
  for (int i = tid; i < n; i += NT) {
    const int idx = (int)index_col[i];
    if (idx >= lo && idx < lo + mine) p.list[atomicAdd(place + idx - lo, 1)] = i;
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

// Adds GROUP vectors of the rows of dOut at `ordered[0 .. m)` to a value per thread: the CTA's threads copy steps of rows into the ring,
// EMB_STEPS - 1 ahead of the one whose values are added.  col: the thread's vector of row 0; `on`: whether the row has it.
template <typename T, typename V, int GROUP>
__device__ __forceinline__ void emb_add_rows(T& sum, const V* __restrict__ col, bool on, int vecs, const int* ordered, int m, V* ring) {
  constexpr int ROWS = EMB_STEP / GROUP, TEAMS = EMB_THREADS / GROUP, VALUES = GROUP * (int)(sizeof(V) / sizeof(T));
  const int tid = threadIdx.x, team = tid / GROUP, jl = tid % GROUP, steps = (m + ROWS - 1) / ROWS;
  auto fetch = [&](int step) {
    if (step < steps && on)
#pragma unroll
      for (int q = 0; q < ROWS / TEAMS; ++q) {
        const int k = step * ROWS + q * TEAMS + team;
        if (k < m) emb_copy<sizeof(V)>(ring + step % EMB_STEPS * EMB_STEP + (q * TEAMS + team) * GROUP + jl, col + (int64_t)ordered[k] * vecs);
      }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  for (int i = 0; i < EMB_STEPS - 1; ++i) fetch(i);
  for (int i = 0; i < steps; ++i) {
    asm volatile("cp.async.wait_group %0;" ::"n"(EMB_STEPS - 2) : "memory");
    __syncthreads();                                         // step i is there; step i - 1 has been added
    fetch(i + EMB_STEPS - 1);
    if (tid < VALUES) {
      // a value per thread, B rows read ahead of the B that are added (vectors by eight lanes, one after another: 50 cycles a row)
      const T* x = reinterpret_cast<const T*>(ring + i % EMB_STEPS * EMB_STEP) + tid;
      const int rows = m - i * ROWS < ROWS ? m - i * ROWS : ROWS;
      constexpr int B = sizeof(T) == 4 ? 16 : 8;
      int k = 0;
      if (rows >= B) {
        T y[B];
#pragma unroll
        for (int u = 0; u < B; ++u) y[u] = x[u * VALUES];
#pragma unroll 1
        for (k = B; k + B <= rows; k += B) {
          T z[B];
#pragma unroll
          for (int u = 0; u < B; ++u) z[u] = x[(k + u) * VALUES];
#pragma unroll
          for (int u = 0; u < B; ++u) sum = add_rn(sum, y[u]);
#pragma unroll
          for (int u = 0; u < B; ++u) y[u] = z[u];
        }
#pragma unroll
        for (int u = 0; u < B; ++u) sum = add_rn(sum, y[u]);
      }
      for (; k < rows; ++k) sum = add_rn(sum, x[k * VALUES]);
    }
  }
  __syncthreads();
}

// CTAs [0, hot_ctas) take (row of very many hits, 8 vectors) and then (row of many hits, 32 vectors) pairs, the warps of the others
// (row of few, 64 vectors) pairs, whose loads of four hits are in flight together.  Such a pair is a chain of three loads, so a warp
// reads the next pair's entry and list while it sums this one's (without that, the sums of the few took longer than those of the many).
// S: vectors of a row that a lane takes, 32 apart.  (A kernel for each way through the rows of few: together they do not fit 64 registers.)
template <typename T, bool VECTORS, bool WALK, int S>
__global__ void __launch_bounds__(EMB_THREADS, 4)
emb_sum_kernel(const T* __restrict__ dOut, T* __restrict__ dW, EmbPlan p, int vocab, int dim, int hot_ctas, int rows_per_warp) {
  chain_begin();
  using V = typename std::conditional<VECTORS, typename EmbVec<T>::type, T>::type;
  const int vecs = VECTORS ? dim / EmbVec<T>::N : dim;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  __shared__ int ordered[EMB_LIST];
  // lane q: entries of one kind in the parts up to q; entry g of the kind is the returned one of its part (all lanes ask for the same)
  auto up_to = [&](int here) {
    int x = here;
#pragma unroll
    for (int o = 1; o < EMB_SEGMENTS; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += u;
    }
    return x;
  };
  auto part_of = [&](int incl, int here, int g, int& nth) {
    const int q = __popc(__ballot_sync(0xffffffffu, lane < EMB_SEGMENTS && incl <= g));
    nth = g - __shfl_sync(0xffffffffu, incl - here, q);
    return q;
  };
  if ((int)blockIdx.x >= hot_ctas) {
    int* mine = ordered + w * EMB_FEW;
    const int blocks = (vecs + 32 * S - 1) / (32 * S);
    auto order = [&](int c, int pos) {
      int rank = 0;
      for (int k = 0; k < c; ++k) rank += __shfl_sync(0xffffffffu, pos, k) < pos;
      __syncwarp();
      if (lane < c) mine[rank] = pos;
      __syncwarp();
    };
    auto add = [&](int v, int c, int block) {
      const int j = block * (32 * S) + lane;
      V acc[S];
#pragma unroll
      for (int q = 0; q < S; ++q) acc[q] = emb_zero<T, V>();
      for (int k0 = 0; k0 < c; k0 += 4) {
        V x[4][S];
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (k0 + u < c) {
            const V* from = reinterpret_cast<const V*>(dOut + (int64_t)mine[k0 + u] * dim) + j;
#pragma unroll
            for (int q = 0; q < S; ++q)
              if (j + 32 * q < vecs) x[u][q] = __ldcs(from + 32 * q);
          }
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (k0 + u < c)
#pragma unroll
            for (int q = 0; q < S; ++q)
              if (j + 32 * q < vecs) emb_add<T, V>(acc[q], x[u][q]);
      }
      V* to = reinterpret_cast<V*>(dW + (int64_t)v * dim) + j;
#pragma unroll
      for (int q = 0; q < S; ++q)
        if (j + 32 * q < vecs) __stcs(to + 32 * q, acc[q]);
    };
    if constexpr (WALK) {
      const int64_t first = (((int64_t)blockIdx.x - hot_ctas) * EMB_WARPS + w) * rows_per_warp;
      if (first >= vocab) return;
      const int r0 = (int)first, rows = vocab - r0 < rows_per_warp ? vocab - r0 : rows_per_warp;
      const int cnt = lane < rows ? p.count[r0 + lane] : 0, off = lane < rows ? p.offset[r0 + lane] : 0;
      auto read = [&](int q) {
        const int c = __shfl_sync(0xffffffffu, cnt, q), o = __shfl_sync(0xffffffffu, off, q);
        return lane < c && c <= EMB_FEW ? p.list[o + lane] : 0x7fffffff;
      };
      int pos = read(0);
      for (int q = 0; q < rows; ++q) {
        const int c = __shfl_sync(0xffffffffu, cnt, q), next = read((q + 1) & 31);
        if (c <= EMB_FEW) {
          order(c, pos);
          for (int b = 0; b < blocks; ++b) add(r0 + q, c, b);
        }
        pos = next;
      }
      return;
    }
    const int here = lane < p.segments ? p.few[lane] : 0, incl = up_to(here), entries = __shfl_sync(0xffffffffu, incl, EMB_SEGMENTS - 1);
    const int64_t units = (int64_t)entries * blocks, stride = (int64_t)(gridDim.x - hot_ctas) * EMB_WARPS;
    auto of = [&](int64_t u, int& v, int& c, int& o) {
      int nth;
      const int q = part_of(incl, here, (int)(u / blocks), nth), e = q * p.stride + nth;
      v = p.rows[e];
      c = p.count[p.large ? v : e];
      o = p.offset[p.large ? v : e];
    };
    int64_t u0 = ((int64_t)blockIdx.x - hot_ctas) * EMB_WARPS + w;
    if (u0 >= units) return;
    int v, c, o, v1 = 0, c1 = 0, o1 = 0;
    of(u0, v, c, o);
    int pos = lane < c ? p.list[o + lane] : 0x7fffffff;
    if (u0 + stride < units) of(u0 + stride, v1, c1, o1);
    for (; u0 < units; u0 += stride) {
      int v2 = 0, c2 = 0, o2 = 0;
      if (u0 + 2 * stride < units) of(u0 + 2 * stride, v2, c2, o2);
      const int pos1 = lane < c1 ? p.list[o1 + lane] : 0x7fffffff;
      order(c, pos);
      add(v, c, (int)(u0 % blocks));
      v = v1; c = c1; o = o1; pos = pos1;
      v1 = v2; c1 = c2; o1 = o2;
    }
    return;
  }
  __shared__ unsigned bits[EMB_POSITIONS / 32];
  __shared__ int warp_sum[EMB_WARPS];
  constexpr int WORDS = EMB_POSITIONS / 32 / EMB_THREADS;       // bitmap words per thread
  extern __shared__ __align__(16) unsigned char emb_smem[];
  V* ring = reinterpret_cast<V*>(emb_smem);                  // [EMB_STEPS][rows of a step][vectors]
  const int very = lane < p.segments ? p.very[lane] : 0, many = lane < p.segments ? p.many[lane] : 0;
  const int many_up_to = up_to(many);
  const int narrow = (vecs + EMB_NARROW - 1) / EMB_NARROW, wide = (vecs + EMB_WIDE - 1) / EMB_WIDE;
  const int64_t narrow_tasks = (int64_t)__reduce_add_sync(0xffffffffu, very) * narrow;
  const int64_t tasks = narrow_tasks + (int64_t)__reduce_add_sync(0xffffffffu, many) * wide;
  // row g of very many hits: every part's first one, then the second ones and so on, for the parts have their largest rows first
  auto entry_of_very = [&](int g) {
    if (p.large) return p.stride + g;
    int lo = 0, hi = p.stride;                               // rounds before row g: lo <= k < hi
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (__reduce_add_sync(0xffffffffu, very < mid ? very : mid) <= g) lo = mid;
      else hi = mid;
    }
    g -= __reduce_add_sync(0xffffffffu, very < lo ? very : lo);
    unsigned with = __ballot_sync(0xffffffffu, very > lo);
    for (; g > 0; --g) with &= with - 1;
    return __ffs(with) * p.stride - 1 - lo;
  };
  for (int64_t h = blockIdx.x; h < tasks; h += hot_ctas) {
    const bool is_narrow = h < narrow_tasks;
    const int64_t h2 = is_narrow ? h : h - narrow_tasks;
    const int groups = is_narrow ? narrow : wide, first = (int)(h2 % groups) * (is_narrow ? EMB_NARROW : EMB_WIDE);
    int e;
    if (is_narrow) {
      e = entry_of_very((int)(h2 / groups));
    } else {
      int nth;
      const int q = part_of(many_up_to, many, (int)(h2 / groups), nth);
      e = (q + 1) * p.stride - 1 - nth - (p.large ? 0 : __shfl_sync(0xffffffffu, very, q));
    }
    const int v = p.rows[e], c = p.count[p.large ? v : e], o = p.offset[p.large ? v : e];
    T sum = (T)0;
    if (!is_narrow) {
      int* list = reinterpret_cast<int*>(bits);
      const int pos = tid < c ? p.list[o + tid] : 0x7fffffff;
      if (tid < c) list[tid] = pos;
      __syncthreads();
      if (w * 32 < c) {
        int rank = 0;
#pragma unroll 4
        for (int k = 0; k < c; ++k) rank += list[k] < pos;
        if (tid < c) ordered[rank] = pos;
      }
      __syncthreads();
      const int j = first + tid % EMB_WIDE;
      emb_add_rows<T, V, EMB_WIDE>(sum, reinterpret_cast<const V*>(dOut) + j, j < vecs, vecs, ordered, c, ring);
    } else {
      const int j = first + tid % EMB_NARROW;
      const V* col = reinterpret_cast<const V*>(dOut) + j;
      if (p.large) {
        for (int r0 = 0; r0 < c; r0 += EMB_LIST) {
          const int m = c - r0 < EMB_LIST ? c - r0 : EMB_LIST;
          for (int k = tid; k < m; k += EMB_THREADS) ordered[k] = p.ordered[o + r0 + k];
          __syncthreads();
          emb_add_rows<T, V, EMB_NARROW>(sum, col, j < vecs, vecs, ordered, m, ring);
        }
      } else {
#pragma unroll
        for (int k = 0; k < WORDS; ++k) bits[k * EMB_THREADS + tid] = 0;
        __syncthreads();
#pragma unroll 4
        for (int k = tid; k < c; k += EMB_THREADS) {
          const int q = p.list[o + k];
          atomicOr(bits + (q >> 5), 1u << (q & 31));
        }
        __syncthreads();
        int set = 0;
#pragma unroll
        for (int k = 0; k < WORDS; ++k) set += __popc(bits[tid * WORDS + k]);
        int incl = set;
#pragma unroll
        for (int s = 1; s < 32; s <<= 1) {
          const int u = __shfl_up_sync(0xffffffffu, incl, s);
          if (lane >= s) incl += u;
        }
        if (lane == 31) warp_sum[w] = incl;
        __syncthreads();
        int base = incl - set;
#pragma unroll
        for (int k = 0; k < EMB_WARPS; ++k)
          if (k < w) base += warp_sum[k];
        for (int r0 = 0; r0 < c; r0 += EMB_LIST) {
          int rank = base - r0;
          for (int k = 0; k < WORDS; ++k)
            for (unsigned m = bits[tid * WORDS + k]; m; m &= m - 1, ++rank)
              if (rank >= 0 && rank < EMB_LIST) ordered[rank] = (tid * WORDS + k) * 32 + __ffs(m) - 1;
          __syncthreads();
          emb_add_rows<T, V, EMB_NARROW>(sum, col, j < vecs, vecs, ordered, c - r0 < EMB_LIST ? c - r0 : EMB_LIST, ring);
        }
      }
    }
    const int64_t column = (int64_t)first * (sizeof(V) / sizeof(T)) + tid;
    if (tid < (is_narrow ? EMB_NARROW : EMB_WIDE) * (int)(sizeof(V) / sizeof(T)) && column < dim) dW[(int64_t)v * dim + column] = sum;
  }
}

// A small call's sixteen CTAs read all positions each, a large call's launches share them.  Word-like and evenly spread positions,
// 20000 rows of 64 floats: 8000 positions 17 and 14 us as a small call, 25 and 19 as a large one, 24000 31 and 23 against 32 and 18, 48000
// 57 and 35 against 46 and 19.  Over 2000 rows, too few to be walked: 32768 47 and 24 against 52 and 23, 48000 73 and 32 against 62 and 25.
//
// A large call walks a table that has rows for all of its warps, so that only rows without hits are cleared: 262144 positions over 200000
// rows of 512 floats take 177 us, 313 where the whole table is cleared first.  Clearing it is better where few rows have hits and a
// row is too short for a warp: 25000 positions, 200000 rows of 64 floats 42 against 44 us, 33000, two million of 16 floats 67 against 167;
// with 512 floats 110 against 100.
static int64_t emb_walk_warps(const prad_ctx* ctx) { return 4 * (int64_t)ctx->sm_count * EMB_WARPS; }
static bool emb_small(const prad_ctx* ctx, int n, int vocab) {
  return (int64_t)n + vocab <= EMB_PLAN_MOST && n <= (vocab < emb_walk_warps(ctx) ? EMB_POSITIONS : 20000);
}

// ticket: the call's, where `bad` is the context's flag; 0: `bad` is a plain int.  A large call writes no ticket: it records
// `checked` behind the kernel that looks at the indices.
template <typename T>
static prad_status scatter_t(prad_ctx* ctx, const void* index_col, const void* dOut, void* dW, int n, int vocab, int dim, int* bad,
                             int ticket = 0, cudaEvent_t checked = nullptr) {
  const int64_t table = (int64_t)vocab * dim * sizeof(T);
  if (n == 0) {
    PRAD_CUDA(cudaMemsetAsync(dW, 0, table, ctx->stream));
    return PRAD_OK;
  }
  const T* idx = (const T*)index_col;
  const int most = n < vocab ? n : vocab;        // rows that can have hits
  EmbPlan p;
  prad_status s;
  const bool small = emb_small(ctx, n, vocab);
  p.walk = !small && vocab >= emb_walk_warps(ctx) && (4 * (int64_t)n >= vocab || dim * sizeof(T) >= 512);
  if (small) {
    // sixteen segments, even of few rows: they share the additions to the rows' counters (30000 word-like and
    // evenly spread positions over 128 rows of 64 floats: 57 and 26 us, with one segment for them 66 and 37)
    p.segments = vocab < EMB_SEGMENTS ? vocab : EMB_SEGMENTS;
    p.stride = (int)ceil_div(vocab, p.segments);
    p.segments = (int)ceil_div(vocab, p.stride);
    p.large = false;
    const size_t all = (size_t)p.segments * p.stride;
    if ((s = ensure_stage(ctx, (64 + 3 * all + n) * sizeof(int)))) return s;
    int* head = (int*)ctx->stage;
    p.few = head;
    p.many = head + EMB_SEGMENTS;
    p.very = head + 2 * EMB_SEGMENTS;
    p.ordered = nullptr;
    p.count = head + 64;
    p.offset = p.count + all;
    p.rows = p.offset + all;
    p.list = p.rows + all;
    // a table that starts off a 16-byte boundary or lies over the indices is cleared by a launch of its own
    const bool apart = (const char*)index_col + n * sizeof(T) <= (const char*)dW || (const char*)dW + table <= (const char*)index_col;
    const bool beside = ((uintptr_t)dW & 15) == 0 && table % 16 == 0 && apart;
    const int64_t vecs = beside ? table / 16 : 0;
    int clearing = (int)ceil_div(vecs, 4 * EMB_PLAN_THREADS);
    if (clearing > 2 * ctx->sm_count - p.segments) clearing = 2 * ctx->sm_count - p.segments;
    launch_chained(emb_plan_kernel<T>, p.segments + clearing, EMB_PLAN_THREADS, 0, ctx->stream, idx, p, head, head + EMB_SEGMENTS, head + 2 * EMB_SEGMENTS, n, vocab, bad, ticket, (uint4*)dW, vecs);
    PRAD_LAUNCHED(ctx);
    if (!beside) PRAD_CUDA(cudaMemsetAsync(dW, 0, table, ctx->stream));
  } else {
    const int longest = n / (EMB_MANY + 1);      // rows that can have very many hits
    if ((s = ensure_stage(ctx, (64 + 2 * (size_t)vocab + most + longest + 2 * (size_t)n) * sizeof(int)))) return s;
    unsigned long long* cursor = (unsigned long long*)ctx->stage;
    p.few = (const int*)ctx->stage + 1;
    p.many = (const int*)ctx->stage + 2;
    p.very = (const int*)ctx->stage + 3;
    p.segments = 1;
    p.stride = most;
    p.large = true;
    p.count = (int*)ctx->stage + 64;
    p.offset = p.count + vocab;
    p.rows = p.offset + vocab;
    p.list = p.rows + most + longest;
    int* slot = p.list + n;
    p.ordered = slot;                            // which the filling pass has read by then
    PRAD_CUDA(cudaMemsetAsync(cursor, 0, (64 + (size_t)vocab) * sizeof(int), ctx->stream));
    const int g = stream_grid(ctx, n, EMB_THREADS, 8);
    launch_chained(emb_count_kernel<T>, g, EMB_THREADS, 0, ctx->stream, idx, p, slot, n, vocab, bad);
    PRAD_LAUNCHED(ctx);
    if (checked) PRAD_CUDA(cudaEventRecord(checked, ctx->stream));       // `bad` is known
    launch_chained(emb_place_kernel, (unsigned)ceil_div(vocab, EMB_THREADS), EMB_THREADS, 0, ctx->stream, p, cursor, vocab);
    PRAD_LAUNCHED(ctx);
    launch_chained(emb_fill_kernel<T>, g, EMB_THREADS, 0, ctx->stream, idx, p, slot, n, vocab);
    PRAD_LAUNCHED(ctx);
    if (longest > 0) {
      launch_chained(emb_order_kernel, (unsigned)(longest < 2 * ctx->sm_count ? longest : 2 * ctx->sm_count), EMB_ORDER_THREADS, 0, ctx->stream, p, slot, n);
      PRAD_LAUNCHED(ctx);
    }
    if (!p.walk) PRAD_CUDA(cudaMemsetAsync(dW, 0, table, ctx->stream));
  }
  // as many CTAs as can have work, and no more than two an SM for either kind of row: all of them run at once.  Where the table is
  // walked, the warps for all of its rows.
  const bool vectors = dim % EmbVec<T>::N == 0 && (((uintptr_t)dOut | (uintptr_t)dW) & 15) == 0;
  const int vecs = vectors ? dim / EmbVec<T>::N : dim;
  auto at_most = [&](int64_t wanted, int per_sm) { return (int)(wanted < (int64_t)per_sm * ctx->sm_count ? wanted : (int64_t)per_sm * ctx->sm_count); };
  const int hot = at_most(n / (EMB_FEW + 1) * ceil_div(vecs, EMB_WIDE) + n / (EMB_MANY + 1) * ceil_div(vecs, EMB_NARROW), 2);
  const int rows_per_warp = vocab < EMB_ROWS * emb_walk_warps(ctx) ? (int)ceil_div(vocab, emb_walk_warps(ctx)) : EMB_ROWS;
  const int64_t others = p.walk ? ceil_div(vocab, EMB_WARPS * rows_per_warp)
                                : at_most(ceil_div((int64_t)most * ceil_div(vecs, vecs > 32 ? 64 : 32), EMB_WARPS), hot ? 2 : 4);
  auto sum = [&](auto kernel, prad_status allowed, int ring) {       // shared memory for the ring only where a row can have many hits
    if (!allowed)
      launch_chained(kernel, (unsigned)(hot + others), EMB_THREADS, hot ? ring : 0, ctx->stream, (const T*)dOut, (T*)dW, p, vocab, dim, hot, rows_per_warp);
    return allowed;
  };
#define PRAD_EMB_SUM(VECTORS_, WALK_, S_)                                                                \
  do {                                                                                                   \
    constexpr int ring_ = EMB_STEPS * EMB_STEP * (VECTORS_ ? 16 : (int)sizeof(T));                       \
    s = sum(emb_sum_kernel<T, VECTORS_, WALK_, S_>, allow_smem<emb_sum_kernel<T, VECTORS_, WALK_, S_>>(ctx, ring_), ring_); \
  } while (0)
#define PRAD_EMB_SUM_OF(VECTORS_)                                                                        \
  do {                                                                                                   \
    if (p.walk && vecs > 32) PRAD_EMB_SUM(VECTORS_, true, 2);                                            \
    else if (p.walk) PRAD_EMB_SUM(VECTORS_, true, 1);                                                    \
    else if (vecs > 32) PRAD_EMB_SUM(VECTORS_, false, 2);                                                \
    else PRAD_EMB_SUM(VECTORS_, false, 1);                                                               \
  } while (0)
  if (vectors) PRAD_EMB_SUM_OF(true);
  else PRAD_EMB_SUM_OF(false);
#undef PRAD_EMB_SUM_OF
#undef PRAD_EMB_SUM
  if (s) return s;
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

// A call's flag words, cleared for it; every call has another ticket.
static int next_ticket(prad_ctx* ctx) {
  *(volatile int*)ctx->host_flag = 0;
  ctx->flag_ticket = ctx->flag_ticket < 0x7fffffff ? ctx->flag_ticket + 1 : 1;
  return ctx->flag_ticket;
}
static prad_status check_bad_index(prad_ctx* ctx, const char* who) {
  const int h = *(volatile int*)ctx->host_flag;
  PRAD_REQUIRE(h == 0, PRAD_ERR_INVALID, "%s: index at input row %d is outside [0, vocab)", who, h - 1);
  return PRAD_OK;
}
// Waits until the call's ticket is in host memory, which the kernel writes before its other work is done, so that the host is
// ahead of the GPU.  A stream that has stopped or come to its end without it ends the wait.
static prad_status wait_ticket(prad_ctx* ctx, const char* who, int ticket) {
  volatile int* arrived = ctx->host_flag + 1;
  for (unsigned polls = 1; *arrived != ticket; ++polls) {
    if (polls % 4096) continue;
    const cudaError_t e = cudaStreamQuery(ctx->stream);
    if (e == cudaErrorNotReady) continue;
    if (e == cudaSuccess && *arrived == ticket) break;
    (void)cudaGetLastError();
    PRAD_REQUIRE(false, PRAD_ERR_CUDA, "%s failed: %s", who, e == cudaSuccess ? "the indices were not looked at" : cudaGetErrorString(e));
  }
  std::atomic_thread_fence(std::memory_order_acquire);
  return check_bad_index(ctx, who);
}

template <typename T>
static prad_status gather_t(prad_ctx* ctx, const void* index_col, const void* W, void* out, int n, int vocab, int dim, int ticket) {
  const int grid = stream_grid(ctx, n, EMB_WARPS, 8);
  int checkers = (int)ceil_div(n, 8 * EMB_THREADS);        // eight loads in flight per thread
  if (checkers > ctx->sm_count) checkers = ctx->sm_count;
  const bool vectors = dim % EmbVec<T>::N == 0 && (((uintptr_t)W | (uintptr_t)out) & 15) == 0;
  auto launch = [&](int first, int rest) -> prad_status {
    launch_chained(vectors ? embedding_gather_kernel<T, true> : embedding_gather_kernel<T, false>, first + rest, EMB_THREADS, 0, ctx->stream,
                   (const T*)index_col, (const T*)W, (T*)out, n, vocab, dim, ctx->host_flag, ticket, first, ctx->tc_err + 48);
    PRAD_LAUNCHED(ctx);
    return PRAD_OK;
  };
  // rows written over the indices (a table of one column, in place): looked at before the first one is
  const char *i0 = (const char*)index_col, *o0 = (const char*)out;
  const bool over = i0 < o0 + (int64_t)n * dim * sizeof(T) && o0 < i0 + (int64_t)n * sizeof(T);
  if (!over) return launch(checkers, grid);
  const prad_status s = launch(checkers, 0);
  return s ? s : launch(0, grid);
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
  const int ticket = next_ticket(ctx);
  prad_status s = dt == PRAD_F32 ? gather_t<float>(ctx, index_col, W, out, n, vocab, dim, ticket)
                                 : gather_t<double>(ctx, index_col, W, out, n, vocab, dim, ticket);
  return s ? s : wait_ticket(ctx, "prad_embedding_forward", ticket);
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
  const int ticket = next_ticket(ctx);
  // the indices have been looked at once the first kernel is done: the caller need not wait for the sums
  if (!ctx->flag_read) PRAD_CUDA(cudaEventCreateWithFlags(&ctx->flag_read, cudaEventDisableTiming));
  prad_status s = dt == PRAD_F32 ? scatter_t<float>(ctx, index_col, dOut, dW, n, vocab, dim, ctx->host_flag, ticket, ctx->flag_read)
                                 : scatter_t<double>(ctx, index_col, dOut, dW, n, vocab, dim, ctx->host_flag, ticket, ctx->flag_read);
  if (s || n == 0) return s;
  if (emb_small(ctx, n, vocab)) return wait_ticket(ctx, "prad_embedding_backward", ticket);
  PRAD_CUDA(cudaEventSynchronize(ctx->flag_read));
  return check_bad_index(ctx, "prad_embedding_backward");
}

}  // extern "C"

// Runs a graph's walk as ONE kernel.
//
// What bounded it: an unrolled network from a JSON architecture is hundreds of operations on a few hundred values each.  An
// eight-step two-layer LSTM of 64 units is 1058 launches of 2 - 6 us per training step, 4.9 ms, for 25 MFLOP.
//
// Here the walk is recorded once as a list of primitive operations.  A level of the plan holds operations that depend on
// earlier levels only; chains of elementwise operations on the same elements (a gate's sum and activation, a cell update, the
// += of a shared weight's gradients over the time steps) share a level too, as a small program that keeps every value of one
// element in shared memory from its load to its store, and such a program computes the products that it reads, where they are
// small, for its own elements: a cell of an LSTM is one level instead of a level of products and one of programs.  One cluster of
// 16 CTAs runs the levels with the cluster's hardware barrier between them (no waiting loops, no other CTA to wait for).  What
// nothing waits for (weight gradients, outputs) comes as late as it can, and from the level on where that gains most the levels run
// on all SMs, as launches of their own.  A level is latency: a barrier (1.1 us), a program (1.7), operands from L2 (1.2), a chain of 64 additions (1.5).  So
// the pieces of a level -- 32, 64 or 256 elements, 256 or 1024 outputs -- are dealt to 32 workers when the plan is made, two to an
// SM, and a worker fetches its next program while it runs this one.  The eight-step two-layer LSTM of 64 units and 8 columns, both
// walks, losses and optimiser: 297 us with 22 levels each way and four workers of 64 registers (their spilled values went through
// L2 after every barrier, which emptied the L1), 160 us now.
//
// Values are those of the separate kernels bit for bit for elementwise operations and products (k ascending, product and sum
// rounded separately); row reductions and column sums add in double or in the same lane order.  (Compiled with -fmad=false.)
#include <algorithm>
#include <cstring>
#include <map>

#include "act_math.cuh"
#include "graph_plan.cuh"

namespace prad {
namespace gp {

constexpr int NT = 256;                   // threads of a worker
constexpr int WORKERS = 2;                // workers of a CTA: a piece is mostly latency, so two share an SM; up to 128 registers, no spills
constexpr int SLOTS = 64;                 // values of one element a program keeps
constexpr int MAX_INS = 96;
constexpr int MAX_DOTS = 16;              // products a program computes for its own elements
constexpr int MAX_TASKS = 64;             // copies their operands are cut into
constexpr int PROG_BYTES = 64 + SLOTS * 16 + MAX_INS * 24 + SLOTS * 16 + MAX_TASKS * 40 + MAX_DOTS * 24;
constexpr int WORK_BYTES = 88 * 1024;     // a worker's shared memory: the slots of its elements, or the operands of a product

// a piece of one worker
struct Item { uint32_t prog, bytes, chunk, barrier; };

// team: how many threads share an element's instructions: 8 (a piece is 32 elements then) where it has products, 4 or 1
// n_dot products of rows x dot_n outputs, ks values of k of their n_opd operands at a time, from work_at values on; dot_inv and
// Opd::inv divide by dot_n and Opd::most
struct Head { int32_t kind, n_load, n_ins, n_store; int64_t n; int32_t team, n_opd, n_dot, dot_n, most_k, ks, work_at; uint32_t dot_inv; };
struct Load { const void* p; uint32_t cols, slot; };        // cols: 0 = element i, else element i % cols
// phase: in the first instruction of a phase (instructions that do not touch one another's values), how many it has
struct Ins { uint8_t op, act, n_in, phase; uint8_t dst[2], pad2[2]; uint8_t src[8]; double scalar; };
constexpr uint8_t INS_FOLD = 64;          // ((src0 + src1) + src2) + ... in T: a run of dst += src
struct Store { void* p; uint32_t slot, pad; };
// An operand of a program's products.  kind 0: the piece's rows of an [M][K] matrix, 1: of a [K][M] one (X = M),
// 2: all columns of a [K][N] matrix, 3: of an [N][K] one (X = N); at: where it goes, behind work_at, as [row or column][k]
// (values k_lo .. k_hi of k: an operand is several tasks)
struct Opd { const void* p; int32_t kind, X, K, at, k_lo, k_hi, most, inv; };     // most: rows or columns of a piece
struct Dot { double alpha; int32_t K, slot, a_at, b_at; };
static_assert(sizeof(Head) == 56 && sizeof(Load) == 16 && sizeof(Ins) == 24 && sizeof(Store) == 16 && sizeof(Opd) == 40 && sizeof(Dot) == 24,
              "program layout");
struct ProductProg {
  Head h;                                                    // kind = PRIM_PRODUCT
  const void *A, *B;
  void* C;
  int64_t sA, sB, sC;
  double alpha;
  int32_t tA, tB, M, N, K, tm, tn, ks, tiles_n, tiles_mn, r;   // r: r x r outputs per thread
};
struct RowProg { Head h; const void* in[4]; void* out[3]; int64_t rows; int32_t cols, depth; double scalar; };

// The cluster meets, and what its threads wrote is visible to all of them: a CTA's stores are published by one fence of one
// thread behind a barrier of the CTA (a release by every thread took 1800 cycles, most of it 32 fences one after another).
__device__ __forceinline__ void cluster_barrier() {
  __syncthreads();
  if (threadIdx.x == 0) __threadfence();
  asm volatile("barrier.cluster.arrive.relaxed;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
template <int BYTES> __device__ __forceinline__ void copy_async(void* dst, const void* src) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(d), "l"(src), "n"(BYTES) : "memory");
}
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// a worker's threads meet
__device__ __forceinline__ void worker_sync() { asm volatile("bar.sync %0, %1;" ::"r"(1 + (int)(threadIdx.x / NT)), "n"(NT) : "memory"); }

// The start gradients of this run; most walks have few, and short arguments launch faster.
template <int N> struct StartTable { const void* p[N]; };
constexpr int FEW_STARTS = 64;
template <typename T, int N> __device__ __forceinline__ const T* source(const void* p, const StartTable<N>& starts) {
  const uint64_t a = (uint64_t)p;
  return (const T*)((a >> 62) == 1 ? starts.p[(a >> 40) & 0x3fffff] : p);
}

// ---- elementwise programs
// One instruction on one element; v[slot * stride] is the element's value in a slot.
template <typename T>
__device__ __forceinline__ void execute(const Ins& c, T* v, int stride) {
  const T a = v[c.src[0] * stride], s = (T)c.scalar;
  T r;
  switch (c.op) {
    case PRIM_ACT_FORWARD: r = act_value<T>((prad_act)c.act, a, s); break;
    case PRIM_ACT_BACKWARD: r = mul_rn(v[c.src[1] * stride], act_derivative<T>((prad_act)c.act, a, s)); break;
    case PRIM_ADD2: case PRIM_ADD_ROW: r = add_rn(a, v[c.src[1] * stride]); break;
    case PRIM_ADD3: r = add_rn(add_rn(a, v[c.src[1] * stride]), v[c.src[2] * stride]); break;
    case PRIM_MUL2: r = mul_rn(a, v[c.src[1] * stride]); break;
    case PRIM_MUL_BACKWARD: {              // a, b, dy -> dy b, dy a
      const T b = v[c.src[1] * stride], d = v[c.src[2] * stride];
      v[c.dst[1] * stride] = mul_rn(d, a);
      r = mul_rn(d, b);
      break;
    }
    case PRIM_SCALE: r = mul_rn(a, s); break;
    case PRIM_COPY: r = a; break;
    case INS_FOLD: {
      r = a;
      for (int q = 1; q < c.n_in; ++q) r = add_rn(r, v[c.src[q] * stride]);
      break;
    }
    default: {                             // PRIM_SUM: in list order, in double, cast once
      double acc = (double)a;
      for (int q = 1; q < c.n_in; ++q) acc += (double)v[c.src[q] * stride];
      r = (T)acc;
    }
  }
  v[c.dst[0] * stride] = r;
}

// ---- products: operands as [row][k] in shared memory
// rows of 16-byte vectors plus one: the rows of neighbouring threads fall into different banks
template <typename T> __host__ __device__ constexpr int product_pitch(int ks) {
  constexpr int VEC = 16 / (int)sizeof(T);
  return (ks + VEC - 1) / VEC * VEC + VEC;
}
// R x R sums over kc values of k, ascending, product and sum rounded separately; a thread's rows (columns) are `da` (`db`) values
// apart.  16-byte reads (with a read per value, reading was most of a piece), the next ones on their way while these are added.
template <typename T, int R>
__device__ __forceinline__ void multiply(const T* a, int da, const T* b, int db, int kc, T (&acc)[R][R]) {
  constexpr int VEC = 16 / (int)sizeof(T), G = R == 1 ? 2 : 1, KG = G * VEC;      // k at a time
  alignas(16) T x[R][KG], y[R][KG];
  auto fetch = [&](int k) {
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
      for (int g = 0; g < G; ++g) {
        *reinterpret_cast<uint4*>(&x[i][g * VEC]) = *reinterpret_cast<const uint4*>(a + i * da + k + g * VEC);
        *reinterpret_cast<uint4*>(&y[i][g * VEC]) = *reinterpret_cast<const uint4*>(b + i * db + k + g * VEC);
      }
  };
  int k = 0;
  if (kc >= KG) fetch(0);
#pragma unroll 1
  for (; k + KG <= kc; k += KG) {
    T pr[R][R][KG];
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
      for (int j = 0; j < R; ++j)
#pragma unroll
        for (int q = 0; q < KG; ++q) pr[i][j][q] = mul_rn(x[i][q], y[j][q]);
    if (k + 2 * KG <= kc) fetch(k + KG);
#pragma unroll
    for (int q = 0; q < KG; ++q)
#pragma unroll
      for (int i = 0; i < R; ++i)
#pragma unroll
        for (int j = 0; j < R; ++j) acc[i][j] = add_rn(acc[i][j], pr[i][j][q]);
  }
#pragma unroll 1
  for (; k < kc; ++k)
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
      for (int j = 0; j < R; ++j) acc[i][j] = add_rn(acc[i][j], mul_rn(a[i * da + k], b[j * db + k]));
}

// The worker copies ks values of k, from k0 on, of a program's operands.  The plan has cut them into tasks of about the same size,
// which the warps take in turn.  (A loop of all warps over all operands took longer than all the arithmetic: it is a chain of
// instructions per operand, not bytes, that takes the time.)
template <typename T, int N>
__device__ __forceinline__ void copy_program_operands(const Opd* op, int n_opd, T* work, int pitch, int row0, int k0, int ks,
                                                      const StartTable<N>& starts) {
  constexpr int VEC = 16 / (int)sizeof(T);
  const int lane = threadIdx.x & 31;
  for (int o = threadIdx.x % NT / 32; o < n_opd; o += NT / 32) {
    const Opd d = op[o];
    int k_lo = d.k_lo > k0 ? d.k_lo : k0, k_hi = d.k_hi < k0 + ks ? d.k_hi : k0 + ks;
    if (k_lo >= k_hi) continue;
    const int first = d.kind < 2 ? row0 : 0, left = d.X - first, count = left < d.most ? left : d.most;
    const T* g = source<T>(d.p, starts);
    T* s = work + d.at - k0;
    if (d.kind == 0 || d.kind == 3) {                        // [row][k]
      g += (int64_t)first * d.K;
      if (k_lo % VEC == 0 && k_hi % VEC == 0 && k0 % VEC == 0 && d.K % VEC == 0 && ((uintptr_t)g & 15) == 0) {
#pragma unroll 4
        for (int r = 0; r < count; ++r)
          for (int k = k_lo + lane * VEC; k < k_hi; k += 32 * VEC) {
            const uint32_t to = (uint32_t)__cvta_generic_to_shared(s + r * pitch + k);
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to), "l"(g + r * d.K + k) : "memory");
          }
      } else {
#pragma unroll 4
        for (int r = 0; r < count; ++r)
          for (int k = k_lo + lane; k < k_hi; k += 32) copy_async<sizeof(T)>(s + r * pitch + k, g + r * d.K + k);
      }
    } else {                                                 // [k][row]
      const int k_lane = lane * d.inv >> 16, r = lane - k_lane * d.most, step = 32 * d.inv >> 16;
      if (r < count && k_lane < step) {                      // (at most 32 rows; lanes beyond a whole number of k stay out)
        g += first + r;
        s += r * pitch;
#pragma unroll 4
        for (int k = k_lo + k_lane; k < k_hi; k += step) copy_async<sizeof(T)>(s + k, g + k * d.X);
      }
    }
  }
}

// A piece: 256 elements, one per thread, or 64 (32) elements with four (eight) threads each, which take the loads, the products,
// the instructions of a phase and the stores in turn (four gates' exponentials side by side instead of one after another).
template <typename T, int N>
__device__ void run_elementwise(const Head* h, int chunk, T* work, const StartTable<N>& starts) {
  const int tid = threadIdx.x % NT, team = h->team, n_dot = h->n_dot;
  // (a piece of 32: columns by the lanes' upper bits and rows by bits 0 and 4, so that reads of either operand of a product have
  // lane pairs one or two apart on one address: 2 cycles instead of 4)
  const int per = team == 8 ? NT / 8 : team == 4 ? NT / 4 : NT, q0 = team == 8 ? tid >> 5 : team == 4 ? tid >> 6 : 0;
  const int e = team == 8 ? (tid >> 1 & 15) | (tid & 1) << 4 : tid & (per - 1);
  const Load* ld = reinterpret_cast<const Load*>(h + 1);
  const Ins* ins = reinterpret_cast<const Ins*>(ld + h->n_load);
  const Store* st = reinterpret_cast<const Store*>(ins + h->n_ins);
  const int64_t i = (int64_t)chunk * per + e;
  const bool on = i < h->n;
  T* v = work + e;
  if (on)
    for (int k = q0; k < h->n_load; k += team)      // all on their way at once
      copy_async<sizeof(T)>(v + ld[k].slot * per, source<T>(ld[k].p, starts) + (ld[k].cols ? (uint32_t)i % ld[k].cols : (uint32_t)i));
  if (n_dot) {
    const Opd* op = reinterpret_cast<const Opd*>(st + h->n_store);
    const Dot* dots = reinterpret_cast<const Dot*>(op + h->n_opd);
    const int ks = h->ks, pitch = product_pitch<T>(ks), dot_n = h->dot_n, i0 = chunk * per, most = h->most_k;
    auto row_of = [&](int x) { return (int)((uint32_t)x * h->dot_inv >> 20); };      // x < 2048 + 32, dot_n <= 32
    const int row0 = row_of(i0), row = row_of(i0 + e), m = row - row0, c = i0 + e - row * dot_n;
    T* operands = work + h->work_at;
    for (int k0 = 0; k0 < most; k0 += ks) {
      if (k0) worker_sync();
      copy_program_operands<T>(op, h->n_opd, operands, pitch, row0, k0, ks, starts);
      copy_wait();
      worker_sync();
      if (on)
        for (int d = q0; d < n_dot; d += team) {
          const Dot& t = dots[d];
          const int kc = t.K - k0 < ks ? t.K - k0 : ks;
          if (kc <= 0) continue;
          T acc[1][1];
          acc[0][0] = k0 ? v[t.slot * per] : (T)0;
          multiply<T, 1>(operands + t.a_at + m * pitch, 0, operands + t.b_at + c * pitch, 0, kc, acc);
          v[t.slot * per] = k0 + ks < t.K ? acc[0][0] : mul_rn((T)t.alpha, acc[0][0]);
        }
    }
  } else {
    copy_wait();
  }
  if (team > 1) {
    worker_sync();
    for (int k0 = 0; k0 < h->n_ins;) {
      const int c = ins[k0].phase;
      if (on)
        for (int k = k0 + q0; k < k0 + c; k += team) execute<T>(ins[k], v, per);
      worker_sync();
      k0 += c;
    }
  } else if (on) {
    for (int k = 0; k < h->n_ins; ++k) execute<T>(ins[k], v, per);
  }
  if (on)
    for (int k = q0; k < h->n_store; k += team) ((T*)st[k].p)[i] = v[st[k].slot * per];
}

// ---- products of their own: a tm x tn tile, R x R outputs per thread, both operands of ks values of k in shared memory
// `rows` operand rows of kc values of k into s[row][pitch]; KC: memory is [row][k], otherwise [k][row] (rows a power of two)
template <typename T, bool KC>
__device__ __forceinline__ void copy_operand(T* s, int pitch, const T* g, int64_t ld, int row0, int X, int rows, int kc) {
  const int tid = threadIdx.x % NT, lane = tid & 31, warp = tid >> 5;
  if (KC) {
    constexpr int VEC = 16 / (int)sizeof(T);
    g += (int64_t)row0 * ld;
    const bool vec = kc % VEC == 0 && ld % VEC == 0 && ((uintptr_t)g & 15) == 0;
    for (int r = warp; r < rows && row0 + r < X; r += NT / 32)
      if (vec) {
        for (int k = lane * VEC; k < kc; k += 32 * VEC) {
          const uint32_t d = (uint32_t)__cvta_generic_to_shared(s + r * pitch + k);
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(g + (int64_t)r * ld + k) : "memory");
        }
      } else {
        for (int k = lane; k < kc; k += 32) copy_async<sizeof(T)>(s + r * pitch + k, g + (int64_t)r * ld + k);
      }
  } else {
    const int sh = 31 - __clz(rows), r = tid & (rows - 1);
    if (row0 + r < X)
      for (int k = tid >> sh; k < kc; k += NT >> sh) copy_async<sizeof(T)>(s + r * pitch + k, g + (int64_t)k * ld + row0 + r);
  }
}

template <typename T, int R, int N_STARTS>
__device__ void run_product(const ProductProg* p, int chunk, T* smem, const StartTable<N_STARTS>& starts) {
  const int tid = threadIdx.x % NT, tm = p->tm, tn = p->tn, ks = p->ks, K = p->K, M = p->M, N = p->N;
  const int bz = chunk / p->tiles_mn, t2 = chunk % p->tiles_mn;
  const int m0 = t2 / p->tiles_n * tm, n0 = t2 % p->tiles_n * tn;
  const T* A = source<T>(p->A, starts) + bz * p->sA;
  const T* B = source<T>(p->B, starts) + bz * p->sB;
  T* C = (T*)p->C + bz * p->sC;
  const int pa = product_pitch<T>(ks);
  T* As = smem;                              // [tm][pa]
  T* Bs = smem + tm * pa;                    // [tn][pa]
  const int tx = tn / R, ty = tm / R, mi = tid / tx, ni = tid % tx;
  const bool on = mi < ty;
  T acc[R][R];
#pragma unroll
  for (int i = 0; i < R; ++i)
#pragma unroll
    for (int j = 0; j < R; ++j) acc[i][j] = (T)0;
  for (int k0 = 0; k0 < K; k0 += ks) {
    const int kc = K - k0 < ks ? K - k0 : ks;
    if (k0) worker_sync();
    if (p->tA) copy_operand<T, false>(As, pa, A + (int64_t)k0 * M, M, m0, M, tm, kc);
    else copy_operand<T, true>(As, pa, A + k0, K, m0, M, tm, kc);
    if (p->tB) copy_operand<T, true>(Bs, pa, B + k0, K, n0, N, tn, kc);
    else copy_operand<T, false>(Bs, pa, B + (int64_t)k0 * N, N, n0, N, tn, kc);
    copy_wait();
    worker_sync();
    if (on) multiply<T, R>(As + mi * pa, ty * pa, Bs + ni * pa, tx * pa, kc, acc);
  }
  if (on)
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
      for (int j = 0; j < R; ++j) {
        const int m = m0 + mi + i * ty, n = n0 + ni + j * tx;
        if (m < M && n < N) C[(int64_t)m * N + n] = mul_rn((T)p->alpha, acc[i][j]);
      }
}

template <typename A> __device__ __forceinline__ A warp_sum(A v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
template <typename T> __device__ __forceinline__ T sine_exp(T x) { return (T)exp((double)(T)sin((double)x)); }

// ---- row-wise operations: one warp per row, eight rows per piece (the arithmetic of the kernels in rowops.cu); column sums
// and transposes: 256 outputs per piece
template <typename T, int N>
__device__ void run_rows(const RowProg* p, int chunk, const StartTable<N>& starts) {
  const int tid = threadIdx.x % NT, lane = tid & 31, cols = p->cols;
  const T* x = source<T>(p->in[0], starts);
  const T* in1 = source<T>(p->in[1], starts);
  T* out = (T*)p->out[0];
  if (p->h.kind == PRIM_COLUMN_SUM) {        // out[j] = scalar * sum of rows (scalar 1: as is)
    const int64_t j = (int64_t)chunk * NT + tid;
    if (j >= cols) return;
    double acc[8] = {};                      // eight chains, as many as the separate kernel has at the least
    for (int64_t r = 0; r < p->rows; r += 8) {
      T v[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) v[q] = r + q < p->rows ? x[(r + q) * cols + j] : (T)0;
#pragma unroll
      for (int q = 0; q < 8; ++q) acc[q] += (double)v[q];
    }
    out[j] = (T)sum_of_8(acc);
    return;
  }
  if (p->h.kind == PRIM_TRANSPOSE) {
    const int64_t e = (int64_t)chunk * NT + tid, per = p->rows * cols;
    if (e >= per * p->depth) return;
    const int64_t d = e / per, q = e % per, c = q / p->rows, r = q % p->rows;
    out[e] = x[d * per + r * cols + c];
    return;
  }
  const int64_t r = (int64_t)chunk * (NT / 32) + (tid >> 5);
  if (r >= p->rows) return;
  const T* xr = x + r * cols;
  T* yr = out + r * cols;
  switch (p->h.kind) {
    case PRIM_SOFTMAX: {
      T mx = -INFINITY;
      for (int j = lane; j < cols; j += 32) { const T v = xr[j]; mx = v > mx ? v : mx; }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) { const T u = __shfl_xor_sync(0xffffffffu, mx, o); mx = u > mx ? u : mx; }
      T sum = 0;
      for (int j = lane; j < cols; j += 32) sum += t_exp(sub_rn(xr[j], mx));
      sum = warp_sum(sum);
      for (int j = lane; j < cols; j += 32) yr[j] = div_rn(t_exp(sub_rn(xr[j], mx)), sum);
      break;
    }
    case PRIM_SOFTMAX_BACKWARD: {            // in: y, dy
      const T* dr = in1 + r * cols;
      T dot = 0;
      for (int j = lane; j < cols; j += 32) dot += mul_rn(dr[j], xr[j]);
      dot = warp_sum(dot);
      for (int j = lane; j < cols; j += 32) yr[j] = mul_rn(xr[j], sub_rn(dr[j], dot));
      break;
    }
    case PRIM_SINE_SOFTMAX: case PRIM_SINE_SOFTMAX_BACKWARD: {
      T m = 0;
      for (int j = lane; j < cols; j += 32) m += sine_exp<T>(xr[j]);
      m = warp_sum(m);
      for (int j = lane; j < cols; j += 32) {
        const T e = sine_exp<T>(xr[j]);
        if (p->h.kind == PRIM_SINE_SOFTMAX) {
          yr[j] = div_rn(e, add_rn(m, e));
        } else {
          const T num = mul_rn(mul_rn(m, e), (T)cos((double)xr[j])), s = add_rn(m, e);
          yr[j] = mul_rn(in1[r * cols + j], div_rn(num, mul_rn(s, s)));
        }
      }
      break;
    }
    case PRIM_LAYERNORM: {                   // out: y, mean, sigma
      double s = 0.0;
      for (int j = lane; j < cols; j += 32) s += (double)xr[j];
      s = warp_sum(s);
      const T mu = (T)(s / (double)cols);
      double v = 0.0;
      for (int j = lane; j < cols; j += 32) { const T d = sub_rn(xr[j], mu); v += (double)mul_rn(d, d); }
      v = warp_sum(v);
      const T sd = sqrt_rn(div_rn((T)v, (T)cols));
      if (lane == 0) { ((T*)p->out[1])[r] = mu; ((T*)p->out[2])[r] = sd; }
      const T den = add_rn(sd, sizeof(T) == 4 ? (T)1e-9f : (T)1e-9);
      for (int j = lane; j < cols; j += 32) yr[j] = div_rn(sub_rn(xr[j], mu), den);
      break;
    }
    case PRIM_LAYERNORM_BACKWARD: {          // in: x, mean, sigma, dy
      const T mu = in1[r], se = add_rn(source<T>(p->in[2], starts)[r], sizeof(T) == 4 ? (T)1e-9f : (T)1e-9);
      const T* dr = source<T>(p->in[3], starts) + r * cols;
      const T exp1 = mul_rn(sub_rn((T)1, div_rn((T)1, (T)cols)), div_rn((T)1, se));
      const T den = mul_rn((T)cols, mul_rn(mul_rn(se, se), se));
      for (int j = lane; j < cols; j += 32) {
        const T d = sub_rn(xr[j], mu);
        yr[j] = mul_rn(dr[j], sub_rn(exp1, div_rn(mul_rn(d, d), den)));
      }
      break;
    }
  }
}

constexpr int SMEM_BYTES = WORKERS * (2 * PROG_BYTES + WORK_BYTES);

template <typename T, int N>
__global__ void __launch_bounds__(WORKERS * NT)
walk_kernel(const unsigned char* __restrict__ blob, const Item* __restrict__ items, const int* __restrict__ first,
            const __grid_constant__ StartTable<N> starts) {
  chain_begin();
  extern __shared__ __align__(16) unsigned char gp_smem[];
  const int tid = threadIdx.x % NT, worker = blockIdx.x * WORKERS + threadIdx.x / NT;
  unsigned char* prog = gp_smem + (threadIdx.x / NT) * (2 * PROG_BYTES + WORK_BYTES);
  T* work = reinterpret_cast<T*>(prog + 2 * PROG_BYTES);
  items += first[worker];
  const int n = first[worker + 1] - first[worker];
  auto fetch = [&](const Item& it, int i) {
    for (uint32_t b = tid * 16; b < it.bytes; b += NT * 16) {
      const uint32_t d = (uint32_t)__cvta_generic_to_shared(prog + (i & 1) * PROG_BYTES + b);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(blob + it.prog + b) : "memory");
    }
  };
  Item cur{0, 0, 0, 0}, nxt{0, 0, 0, 0};
  if (n > 0) { cur = items[0]; fetch(cur, 0); }
  if (n > 1) nxt = items[1];
  for (int i = 0; i < n; ++i) {
    copy_wait();
    worker_sync();                           // this piece's program is here, the last piece is done with the working memory
    if (i + 1 < n) fetch(nxt, i + 1);
    Item later{0, 0, 0, 0};
    if (i + 2 < n) later = items[i + 2];
    if (cur.bytes) {
      const Head* h = reinterpret_cast<const Head*>(prog + (i & 1) * PROG_BYTES);
      const ProductProg* pp = reinterpret_cast<const ProductProg*>(h);
      if (h->kind <= PRIM_LAST_ELEMENTWISE) run_elementwise<T>(h, (int)cur.chunk, work, starts);
      else if (h->kind == PRIM_PRODUCT && pp->r == 1) run_product<T, 1>(pp, (int)cur.chunk, work, starts);
      else if (h->kind == PRIM_PRODUCT) run_product<T, 2>(pp, (int)cur.chunk, work, starts);
      else run_rows<T>(reinterpret_cast<const RowProg*>(h), (int)cur.chunk, starts);
    }
    if (cur.barrier) cluster_barrier();
    cur = nxt;
    nxt = later;
  }
}

}  // namespace gp

struct GraphPlan {
  // a launch: one cluster with barriers between the levels, or one level on all SMs
  struct Part { int ctas; bool cluster; const int* first; };
  int device = 0;
  prad_dtype dt = PRAD_F32;
  void* mem = nullptr;                       // [items][first item of each worker, part by part][blob]
  const unsigned char* blob = nullptr;
  const gp::Item* items = nullptr;
  std::vector<Part> parts;
  int products = 0;                          // that programs compute for themselves
  std::vector<std::pair<uintptr_t, uintptr_t>> written;      // where the operations write: ascending, without overlaps
};

void GraphPlanFree::operator()(GraphPlan* p) const {
  if (!p) return;
  if (p->mem) {
    cudaSetDevice(p->device);
    cudaFree(p->mem);                        // waits for a run that may still read it
  }
  delete p;
}

namespace gp {

static bool elementwise(const Prim& p) { return p.kind <= PRIM_LAST_ELEMENTWISE; }

// What an operation reads and writes.  `local`: value i of the operation touches element i of the buffer only.
// `fresh`: written by a product that a program computes for its own elements, ahead of whatever else the program does.
struct Access { uintptr_t lo, hi; bool write, local, fresh = false; };

static void accesses(const Prim& p, size_t es, std::vector<Access>& out) {
  out.clear();
  auto add = [&](const void* q, int64_t elems, bool write, bool local) {
    if (q && elems > 0) out.push_back({(uintptr_t)q, (uintptr_t)q + (size_t)elems * es, write, local});
  };
  if (elementwise(p)) {
    for (size_t i = 0; i < p.in.size(); ++i)
      if (p.kind == PRIM_ADD_ROW && i == 1) add(p.in[i], p.cols, false, false);
      else add(p.in[i], p.n, false, true);
    for (void* q : p.out) add(q, p.n, true, true);
    return;
  }
  if (p.kind == PRIM_PRODUCT) {
    add(p.in[0], (p.batch - 1) * p.sA + (int64_t)p.M * p.K, false, false);
    add(p.in[1], (p.batch - 1) * p.sB + (int64_t)p.K * p.N, false, false);
    add(p.out[0], (p.batch - 1) * p.sC + (int64_t)p.M * p.N, true, false);
    return;
  }
  const int64_t all = p.rows * p.cols * p.depth;
  switch (p.kind) {
    case PRIM_COLUMN_SUM: add(p.in[0], all, false, false); add(p.out[0], p.cols, true, false); return;
    case PRIM_LAYERNORM:
      add(p.in[0], all, false, false);
      add(p.out[0], all, true, false);
      add(p.out[1], p.rows, true, false);
      add(p.out[2], p.rows, true, false);
      return;
    case PRIM_LAYERNORM_BACKWARD:
      add(p.in[0], all, false, false);
      add(p.in[1], p.rows, false, false);
      add(p.in[2], p.rows, false, false);
      add(p.in[3], all, false, false);
      add(p.out[0], all, true, false);
      return;
    default:
      for (const void* q : p.in) add(q, all, false, false);
      add(p.out[0], all, true, false);
  }
}

// Memory as regions with their last writers and the readers since.  Accesses that overlap without being the same join their
// regions (gradient destinations that are parts of one buffer, say, only ever meet themselves).
struct Region {
  uintptr_t lo, hi;
  bool local;                                // every access so far was element-local to the same interval
  bool written;                              // by any operation
  std::vector<int> writers, readers;
};

// (buffer, columns of a row operand or 0): what has a place of its own in a program
using Place = std::pair<const void*, int>;

// An elementwise program in the making.
struct Group {
  int64_t n = 0;
  std::vector<int> ops;                      // ascending
  std::vector<Place> places;                 // of their operands, ascending
  int dots = 0, rows = 0, dot_n = 0;         // products taken along, rows of their operands, their columns
};

// Products that programs can compute for themselves.  A product of few outputs whose first reader is an elementwise operation on
// them needs no level of its own, with its barrier and its way through memory: dots[e] are the products that operation e takes
// along, fused[i] says that product i is one.  The product moves to the place of its reader, so nothing in between may write what
// it reads or touch what it writes.
//
// Which ones pay (us of both walks, losses and update of an LSTM of two layers and six steps, or as many as said; products as levels of
// their own, then inside programs): up to 2048 outputs, where several threads share an element -- 64 units and 8 columns 157, 129 in
// double and 142, 112 in float, 64 and 16 196, 130 and 172, 116, 32 and 32 148, 126 and 137, 115, 100 and 12 238, 186 and 222, 158, 30 and
// 20 over twelve steps of three layers 463, 309 and 260, 216, though 20 and 32 131, 154 and 124, 145, 48 and 11 165, 179 and 150, 154; a
// second operand of up to 16 KB, for every piece of 32 elements reads all its columns (with up to 8 KB 100 and 20 221, 160 and 12 249 in
// double, now 205 and 229); and operands that fit a worker's memory at once, or in two parts where nearly every SM of the cluster has
// a piece (150 and 3 335, 267, but 128 and 2 in two parts 244, as levels 192).  What a program will hold is known when it is complete: then
// everything is grouped once more without its products.
constexpr int DOT_COLUMNS = 32, DOT_LOOK = 256, DOT_OPERAND = 16 * 1024;
constexpr int64_t TEAM_ELEMENTS = 2048;      // up to here several threads can share an element
static bool dot_pays(const Prim& p, size_t es) {
  return p.kind == PRIM_PRODUCT && p.batch == 1 && p.K >= 1 && p.N >= 1 && p.N <= DOT_COLUMNS && (int64_t)p.M * p.N <= TEAM_ELEMENTS &&
         (int64_t)p.K * p.N * (int64_t)es <= DOT_OPERAND;
}
static void find_dots(const std::vector<Prim>& ops, size_t es, const std::vector<std::vector<Access>>& acc, const std::vector<char>& barred,
                      std::vector<std::vector<int>>& dots, std::vector<char>& fused) {
  const int N = (int)ops.size();
  auto meets = [](const Access& a, const Access& b) { return a.lo < b.hi && b.lo < a.hi; };
  for (int i = 0; i < N; ++i) {
    const Prim& p = ops[i];
    if (!dot_pays(p, es) || acc[i].size() != 3 || (!barred.empty() && barred[i])) continue;
    const Access &A = acc[i][0], &B = acc[i][1], &X = acc[i][2];
    if (meets(X, A) || meets(X, B)) continue;
    for (int e = i + 1; e < N && e <= i + DOT_LOOK; ++e) {
      bool touched = false, good = elementwise(ops[e]) && ops[e].n == (int64_t)p.M * p.N, harm = false;
      for (const Access& a : acc[e]) {
        if (meets(a, X)) {
          touched = true;
          good = good && !a.write && a.local && a.lo == X.lo && a.hi == X.hi;
        }
        harm = harm || (a.write && (meets(a, A) || meets(a, B)));
      }
      if (!touched && !harm) continue;
      int same = 0;                          // programs have one shape of product each
      for (int d : dots[e]) same += ops[d].N == p.N;
      if (touched && good && !harm && same == (int)dots[e].size()) {
        dots[e].push_back(i);
        fused[i] = 1;
      }
      break;
    }
  }
}

static Place place_of(const Prim& p, size_t k) { return {p.in[k], p.kind == PRIM_ADD_ROW && k == 1 ? p.cols : 0}; }
template <typename T> static int slot_limit(int64_t n) {
  return n <= TEAM_ELEMENTS ? SLOTS : std::min(SLOTS, WORK_BYTES / (NT * (int)sizeof(T)));
}
// operand rows a product in a program keeps in shared memory, at the most
constexpr int DOT_PIECE = NT / 8, DOT_ROWS = 320;
static int dot_rows(const Prim& p) { return (p.N <= DOT_PIECE && DOT_PIECE % p.N == 0 ? DOT_PIECE / p.N : (DOT_PIECE - 1) / p.N + 2) + p.N; }
// a program of one operation
static void program_of(const std::vector<Prim>& all, int i, const std::vector<int>& dots, Group& g) {
  g.n = all[i].n;
  g.ops.assign(1, i);
  g.places.clear();
  for (size_t k = 0; k < all[i].in.size(); ++k) g.places.push_back(place_of(all[i], k));
  for (void* q : all[i].out) g.places.push_back({q, 0});
  std::sort(g.places.begin(), g.places.end());
  g.places.erase(std::unique(g.places.begin(), g.places.end()), g.places.end());
  g.dots = g.rows = g.dot_n = 0;
  for (int d : dots) {
    ++g.dots;
    g.rows += dot_rows(all[d]);
    g.dot_n = all[d].N;
  }
}

// The operands of the products that a program takes along, and how many k of them fit beside its slots.
struct DotLayout {
  struct Operand { const void* p; int kind, X, K, rows; };
  std::vector<Operand> operands;
  std::vector<std::pair<int, int>> of;       // by product: the numbers of its two
  int rows = 0, most_k = 0, ks = 0, slot_values = 0;
};
template <typename T> static void dot_layout(const std::vector<Prim>& ops, const Group& g, const std::vector<std::vector<int>>& dots, DotLayout& l) {
  l.operands.clear();
  l.of.clear();
  l.rows = l.most_k = 0;
  auto operand = [&](const void* q, int kind, int X, int K, int rows) {
    for (size_t k = 0; k < l.operands.size(); ++k) {
      const auto& o = l.operands[k];
      if (o.p == q && o.kind == kind && o.X == X && o.K == K) return (int)k;
    }
    l.operands.push_back({q, kind, X, K, rows});
    l.rows += rows;
    return (int)l.operands.size() - 1;
  };
  for (int o : g.ops)
    for (int d : dots[o]) {
      const Prim& q = ops[d];
      const int a = operand(q.in[0], q.tA ? 1 : 0, q.M, q.K, dot_rows(q) - q.N);
      l.of.push_back({a, operand(q.in[1], q.tB ? 3 : 2, q.N, q.K, q.N)});
      l.most_k = std::max(l.most_k, q.K);
    }
  const int es = (int)sizeof(T);
  l.slot_values = ((int)g.places.size() * DOT_PIECE * es + 15) / 16 * 16 / es;
  l.ks = l.most_k;
  while (l.rows * product_pitch<T>(l.ks) * es > WORK_BYTES - l.slot_values * es) l.ks = (int)ceil_div(l.ks / 2, 8) * 8;
}

struct Piece { uint32_t prog, bytes, chunk; double cost; };

static int outputs(const Ins& c) { return c.op == PRIM_MUL_BACKWARD ? 2 : 1; }
static bool writes(const Ins& c, int slot) { return c.dst[0] == slot || (outputs(c) == 2 && c.dst[1] == slot); }
static bool reads(const Ins& c, int slot) {
  for (int k = 0; k < c.n_in; ++k)
    if (c.src[k] == slot) return true;
  return false;
}

// Appends an instruction; dst += src that continues a run (nothing in between has to do with it) joins that run's fold.
static void fold_into(std::vector<Ins>& ins, const Ins& c) {
  if (c.op == PRIM_ADD2 && c.src[0] == c.dst[0] && c.src[1] != c.dst[0])
    for (size_t y = ins.size(); y-- > 0;) {
      Ins& p = ins[y];
      if (p.dst[0] == c.dst[0] && (p.op == INS_FOLD || (p.op == PRIM_ADD2 && p.src[0] == p.dst[0] && p.src[1] != p.dst[0]))) {
        bool free = p.n_in < 8;
        for (size_t z = y + 1; z < ins.size() && free; ++z)
          for (int k = 1; k < p.n_in; ++k) free = free && !writes(ins[z], p.src[k]);
        if (!free) break;
        Ins joined = p;
        joined.op = INS_FOLD;
        joined.src[joined.n_in++] = c.src[1];
        ins.erase(ins.begin() + y);
        ins.push_back(joined);
        return;
      }
      if (writes(p, c.dst[0]) || reads(p, c.dst[0])) break;
    }
  ins.push_back(c);
}

// Sorts a program into phases: an instruction comes behind those whose values it reads or replaces.  Returns how many.
static int order_by_phase(std::vector<Ins>& ins) {
  std::vector<int> phase(ins.size(), 0);
  int phases = 0, written[SLOTS], read[SLOTS];               // by a slot: the first phase behind its writers, behind its readers
  std::fill(written, written + SLOTS, 0);
  std::fill(read, read + SLOTS, 0);
  for (size_t x = 0; x < ins.size(); ++x) {
    const Ins& c = ins[x];
    int ph = 0;
    for (int k = 0; k < c.n_in; ++k) ph = std::max(ph, written[c.src[k]]);
    for (int k = 0; k < outputs(c); ++k) ph = std::max(ph, std::max(written[c.dst[k]], read[c.dst[k]]));
    phase[x] = ph;
    for (int k = 0; k < c.n_in; ++k) read[c.src[k]] = std::max(read[c.src[k]], ph + 1);
    for (int k = 0; k < outputs(c); ++k) written[c.dst[k]] = ph + 1;
    phases = std::max(phases, ph + 1);
  }
  std::vector<Ins> sorted;
  for (int ph = 0; ph < phases; ++ph) {
    const size_t first = sorted.size();
    for (size_t x = 0; x < ins.size(); ++x)
      if (phase[x] == ph) sorted.push_back(ins[x]);
    sorted[first].phase = (uint8_t)(sorted.size() - first);
  }
  ins.swap(sorted);
  return phases;
}

// Time of an operation's own launch on the whole device, for comparison (us).
static double launch_cost(const Prim& p, int sms) {
  const double base = 2.6;
  if (p.kind == PRIM_PRODUCT) {
    const double outs = (double)p.M * p.N * p.batch;
    return base + p.K * 0.013 * std::max(1.0, outs / 256.0 / sms / 2.0);
  }
  const double n = elementwise(p) ? (double)p.n : (double)p.rows * p.cols * p.depth;
  return base + n / 400e3;
}

// One launch of a plan: its workers' lists.
struct Part { int ctas; bool cluster; std::vector<std::vector<Item>> lists; };

template <typename T> static void build(prad_ctx* ctx, const std::vector<Prim>& ops, int ctas, std::vector<unsigned char>& blob,
                                        std::vector<Part>& parts, std::vector<std::pair<uintptr_t, uintptr_t>>& written,
                                        double* est_us, double* launch_us, int* products, std::vector<char> barred = {}) {
  const size_t es = sizeof(T);
  const int N = (int)ops.size();
  std::vector<int> level(N, 0), group_of(N, -1);
  std::vector<Group> groups;
  std::map<uintptr_t, Region> mem;
  std::vector<std::vector<Access>> all_acc(N);
  std::vector<std::vector<int>> dots(N), after(N);           // after[d]: operations that wait for d
  std::vector<char> fused(N, 0);
  for (int i = 0; i < N; ++i) accesses(ops[i], es, all_acc[i]);
  find_dots(ops, es, all_acc, barred, dots, fused);
  std::vector<Access> acc;
  *launch_us = 0;
  int joins = 0;
  auto region_at = [&](const Access& a) -> Region& {
    auto it = mem.upper_bound(a.lo);
    if (it != mem.begin()) {
      auto p = std::prev(it);
      if (p->second.hi > a.lo) it = p;
    }
    if (it == mem.end() || it->first >= a.hi) return mem.emplace(a.lo, Region{a.lo, a.hi, true, false, {}, {}}).first->second;
    if (it->first == a.lo && it->second.hi == a.hi) return it->second;
    Region joined{a.lo, a.hi, false, false, {}, {}};      // overlaps: one region for all of them
    ++joins;
    while (it != mem.end() && it->first < a.hi) {
      joined.lo = std::min(joined.lo, it->first);
      joined.hi = std::max(joined.hi, it->second.hi);
      joined.written = joined.written || it->second.written;
      joined.writers.insert(joined.writers.end(), it->second.writers.begin(), it->second.writers.end());
      joined.readers.insert(joined.readers.end(), it->second.readers.begin(), it->second.readers.end());
      it = mem.erase(it);
    }
    const uintptr_t lo = joined.lo;
    return mem.emplace(lo, std::move(joined)).first->second;
  };
  std::vector<int> near, join;               // operations that one may share a program with, their programs
  Group one;
  std::vector<Place> united, both;
  std::vector<Region*> regions;              // of its accesses
  for (int i = 0; i < N; ++i) {
    *launch_us += launch_cost(ops[i], ctx->sm_count);
    if (fused[i]) continue;                  // with its reader
    acc.clear();
    for (int d : dots[i])
      for (Access a : all_acc[d]) {
        if (a.write) a.local = a.fresh = true;
        acc.push_back(a);
      }
    acc.insert(acc.end(), all_acc[i].begin(), all_acc[i].end());
    int lv = 0;
    near.clear();
    regions.clear();
    const int joins_before = joins;
    for (const Access& a : acc) {
      Region& r = region_at(a);
      regions.push_back(&r);
      auto depend = [&](int d) {
        if (d == i) return;
        const bool local = a.local && !a.fresh && r.local && elementwise(ops[i]) && elementwise(ops[d]) && ops[i].n == ops[d].n;
        lv = std::max(lv, local ? level[d] : level[d] + 1);
        if (local) near.push_back(d);
        if (after[d].empty() || after[d].back() != i) after[d].push_back(i);
      };
      for (int d : r.writers) depend(d);
      if (a.write)
        for (int d : r.readers) depend(d);
    }
    if (elementwise(ops[i])) {
      // join the programs of the local neighbours at this level, if one program can hold them all
      join.clear();
      for (int d : near)
        if (level[d] == lv && std::find(join.begin(), join.end(), group_of[d]) == join.end()) join.push_back(group_of[d]);
      program_of(ops, i, dots[i], one);
      if (!join.empty()) {
        size_t count = 1;
        int n_dot = one.dots, rows = one.rows, columns = one.dot_n;
        bool fits = true;
        united = one.places;
        for (int g : join) {
          const Group& o = groups[g];
          count += o.ops.size();
          n_dot += o.dots;
          rows += o.rows;
          fits = fits && (!o.dots || !columns || columns == o.dot_n);      // programs have one shape of product each
          if (o.dots) columns = o.dot_n;
          both.clear();
          std::set_union(united.begin(), united.end(), o.places.begin(), o.places.end(), std::back_inserter(both));
          united.swap(both);
        }
        if (fits && count <= MAX_INS && (int)united.size() <= slot_limit<T>(one.n) && n_dot <= MAX_DOTS && rows <= DOT_ROWS) {
          Group& g = groups[join[0]];
          for (size_t k = 1; k < join.size(); ++k) {
            Group& o = groups[join[k]];
            for (int op : o.ops) group_of[op] = join[0];
            const size_t mid = g.ops.size();
            g.ops.insert(g.ops.end(), o.ops.begin(), o.ops.end());
            std::inplace_merge(g.ops.begin(), g.ops.begin() + mid, g.ops.end());
            o = Group();
          }
          g.ops.push_back(i);
          g.places = united;
          g.dots = n_dot;
          g.rows = rows;
          g.dot_n = columns;
          group_of[i] = join[0];
        } else {
          ++lv;                              // a program of its own, behind a barrier
          join.clear();
        }
      }
      if (join.empty()) {
        group_of[i] = (int)groups.size();
        groups.push_back(one);
      }
    }
    level[i] = lv;
    for (size_t k = 0; k < acc.size(); ++k) {
      const Access& a = acc[k];
      Region& r = joins == joins_before ? *regions[k] : region_at(a);
      r.local = r.local && a.local;
      if (!a.write) { r.readers.push_back(i); continue; }
      r.written = true;
      if (r.lo == a.lo && r.hi == a.hi) { r.writers.clear(); r.readers.clear(); }
      r.writers.push_back(i);
    }
  }

  *products = (int)std::count(fused.begin(), fused.end(), 1);
  // once more without the products whose operands make a program go over k several times (dot_pays)
  DotLayout layout;
  bool again = false;
  for (const Group& g : groups) {
    if (!g.dots) continue;
    dot_layout<T>(ops, g, dots, layout);
    const int64_t passes = ceil_div(layout.most_k, layout.ks);
    if (passes == 1 || (passes == 2 && g.n > 14 * DOT_PIECE)) continue;
    barred.resize(N, 0);
    again = true;
    for (int o : g.ops)
      for (int d : dots[o])
        for (int i = 0; i < N; ++i) {
          const Prim &p = ops[d], &q = ops[i];
          if (q.kind == PRIM_PRODUCT && p.M == q.M && p.N == q.N && p.K == q.K && p.tA == q.tA && p.tB == q.tB) barred[i] = 1;
        }
  }
  if (again) {
    build<T>(ctx, ops, ctas, blob, parts, written, est_us, launch_us, products, std::move(barred));
    return;
  }

  for (const auto& m : mem)
    if (m.second.written) {
      if (!written.empty() && written.back().second == m.second.lo) written.back().second = m.second.hi;
      else written.emplace_back(m.second.lo, m.second.hi);
    }

  // As late as possible: what nothing waits for yet (the embedding of the next time steps, weight gradients and their sums,
  // outputs) would take workers from what the next level waits for.  Whole programs move, to the level before their first user.
  const int levels = N ? *std::max_element(level.begin(), level.end()) + 1 : 0;
  {
    auto unit = [&](int i) { return group_of[i] >= 0 ? groups[group_of[i]].ops.front() : i; };
    std::vector<int> order, latest(N, levels - 1);
    for (int i = 0; i < N; ++i)
      if (!fused[i] && unit(i) == i) order.push_back(i);
    std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return level[x] > level[y]; });
    std::vector<std::vector<int>> users(N);                  // of a unit: units behind it
    for (int d = 0; d < N; ++d)
      for (int i : after[d])
        if (unit(i) != unit(d)) users[unit(d)].push_back(unit(i));
    for (int u : order) {                                    // users have a higher level, so they have been here
      int lv = levels - 1;
      for (int v : users[u]) lv = std::min(lv, latest[v] - 1);
      latest[u] = lv;
    }
    // Of the rest, what may be anywhere between two levels goes where it prolongs a level least: the embeddings of all time steps
    // as early as they can be, or all as late, take workers from the cells.
    if (order.size() <= 500 && levels > 2) {
      const int workers = ctas * WORKERS;
      std::vector<double> times((size_t)levels * workers, 0.0), total(levels, 0.0), copy(workers);
      auto busy = [&](int lv) { return times.data() + (size_t)lv * workers; };       // ascending
      auto pieces_of = [&](int u, double* cost) {            // how many, and a piece's time
        const Prim& p = ops[u];
        int64_t n;
        if (group_of[u] >= 0) {
          const Group& g = groups[group_of[u]];
          int k = 0;
          for (int o : g.ops)
            for (int d : dots[o]) k = std::max(k, ops[d].K);
          const bool team = k || (g.n <= TEAM_ELEMENTS && g.ops.size() >= 4);
          n = ceil_div(g.n, k ? DOT_PIECE : team ? NT / 4 : NT);
          *cost = (k ? 1.8 + 0.02 * k : 1.0) + (team ? 0.25 * (double)std::min<size_t>(g.ops.size(), 7) : 0.3 * (double)g.ops.size());
        } else if (p.kind == PRIM_PRODUCT) {
          n = ceil_div((int64_t)p.M * p.N, p.K <= 32 && p.M > 16 && p.N > 16 ? 1024 : NT) * p.batch;
          *cost = 1.5 + 0.02 * p.K;
        } else {
          n = ceil_div(p.rows * p.depth, NT / 32);
          *cost = 2.0 + 0.1 * p.cols;
        }
        return std::min<int64_t>(n, 4 * workers);
      };
      auto add = [&](double* b, int64_t n, double cost) {    // every piece to whoever has least
        for (; n > 0 && b[workers - 1] - b[0] > cost; --n) {
          const double x = b[0] + cost;
          int k = 0;
          for (; k + 1 < workers && b[k + 1] < x; ++k) b[k] = b[k + 1];
          b[k] = x;
        }
        const int each = (int)(n / workers), more = (int)(n % workers);              // in turn from here on
        for (int k = 0; k < workers; ++k) b[k] += (each + (k < more)) * cost;
        std::rotate(b, b + more, b + workers);
      };
      auto longer = [&](int lv, int64_t n, double cost, double least) {              // by how much the level would be, if less than `least`
        const double* b = busy(lv);
        const double most = b[workers - 1], mean = (total[lv] + (double)n * cost) / workers;
        if (mean - most >= least) return least;
        std::copy(b, b + workers, copy.begin());
        add(copy.data(), n, cost);
        return std::max(0.0, copy[workers - 1] - most);
      };
      auto put = [&](int lv, int64_t n, double cost) {
        add(busy(lv), n, cost);
        total[lv] += (double)n * cost;
      };
      std::vector<int> lowest(N, 0);
      double cost;
      for (int u : order)
        if (level[u] == latest[u]) {
          const int64_t n = pieces_of(u, &cost);
          put(latest[u], n, cost);
        }
      for (size_t x = order.size(); x-- > 0;) {              // those with a lower level first
        const int u = order[x];
        if (lowest[u] < latest[u] && latest[u] < levels - 2) {
          const int64_t n = pieces_of(u, &cost);
          int best = latest[u];
          double least = 1e30;
          for (int lv = latest[u]; lv >= lowest[u] && least > 0; --lv) {
            const double more = longer(lv, n, cost, least);
            if (more < least - 1e-9) { least = more; best = lv; }
          }
          latest[u] = best;
          put(best, n, cost);
        }
        for (int v : users[u]) lowest[v] = std::max(lowest[v], latest[u] + 1);
      }
    }
    std::vector<int> moved(N);
    for (int i = 0; i < N; ++i) moved[i] = fused[i] ? 0 : latest[unit(i)];
    level.swap(moved);
  }

  // programs, and the pieces of every level
  std::vector<std::vector<Piece>> pieces(levels);
  auto put = [&](const void* p, size_t bytes) {
    const size_t at = blob.size();
    blob.resize(at + ((bytes + 15) & ~(size_t)15));
    memcpy(blob.data() + at, p, bytes);
    return (uint32_t)at;
  };
  for (int i = 0; i < N; ++i) {
    const Prim& p = ops[i];
    if (fused[i]) continue;
    if (elementwise(p)) {
      const Group& g = groups[group_of[i]];
      if (g.ops.front() != i) continue;
      std::vector<Load> loads;
      std::vector<Ins> ins;
      std::vector<Store> stores;
      int slot_of[SLOTS + 1], slots = 0;
      std::fill(slot_of, slot_of + SLOTS + 1, -1);
      auto slot = [&](const Place& at) -> int& { return slot_of[std::lower_bound(g.places.begin(), g.places.end(), at) - g.places.begin()]; };
      std::vector<int> taken;                // products, with their places
      for (int o : g.ops) {
        const Prim& q = ops[o];
        for (int d : dots[o]) {
          taken.push_back(d);
          slot(Place{ops[d].out[0], 0}) = slots;
          stores.push_back({ops[d].out[0], (uint32_t)slots++, 0});
        }
        Ins c;
        memset(&c, 0, sizeof(c));
        c.op = (uint8_t)q.kind;
        c.act = (uint8_t)q.act;
        c.n_in = (uint8_t)q.in.size();
        c.scalar = q.scalar;
        for (size_t k = 0; k < q.in.size(); ++k) {
          const Place at = place_of(q, k);
          int& it = slot(at);
          if (it < 0) {
            it = slots++;
            loads.push_back({at.first, (uint32_t)at.second, (uint32_t)it});
          }
          c.src[k] = (uint8_t)it;
        }
        for (size_t k = 0; k < q.out.size(); ++k) {
          int& it = slot(Place{q.out[k], 0});
          if (it < 0) it = slots++;
          c.dst[k] = (uint8_t)it;
          bool stored = false;
          for (const Store& s : stores) stored = stored || s.p == q.out[k];
          if (!stored) stores.push_back({q.out[k], (uint32_t)it, 0});
        }
        fold_into(ins, c);
      }
      const int phases = order_by_phase(ins);
      Head h{};
      h.kind = PRIM_ACT_FORWARD;
      h.n_load = (int)loads.size();
      h.n_ins = (int)ins.size();
      h.n_store = (int)stores.size();
      h.n = g.n;
      h.team = !taken.empty() ? NT / DOT_PIECE : g.n <= TEAM_ELEMENTS && (ins.size() >= 4 || slots > WORK_BYTES / (NT * (int)es)) ? 4 : 1;
      std::vector<Opd> opds;
      std::vector<Dot> dot;
      int most_k = 0;
      if (!taken.empty()) {
        dot_layout<T>(ops, g, dots, layout);
        for (const auto& o : layout.operands) opds.push_back({o.p, o.kind, o.X, o.K, 0, 0, o.K, o.rows, 65536 / o.rows + 1});
        for (size_t k = 0; k < taken.size(); ++k) {
          const Prim& q = ops[taken[k]];
          dot.push_back({q.scalar, q.K, slot(Place{q.out[0], 0}), layout.of[k].first, layout.of[k].second});
        }
        most_k = layout.most_k;
        h.ks = layout.ks;
        h.most_k = most_k;
        h.n_dot = (int)dot.size();
        h.dot_n = ops[taken[0]].N;
        h.dot_inv = (1u << 20) / h.dot_n + 1;
        h.work_at = layout.slot_values;
        int at = 0;
        for (size_t k = 0; k < opds.size(); ++k) {
          opds[k].at = at;
          at += layout.operands[k].rows * product_pitch<T>(h.ks);
        }
        for (Dot& t : dot) {
          t.a_at = opds[t.a_at].at;
          t.b_at = opds[t.b_at].at;
        }
        // operands of more than 256 copies are cut along k, while there is room for tasks; whole vectors of k
        const int copy_of[4] = {16, (int)es, (int)es, 16};
        std::vector<Opd> tasks;
        for (size_t k = 0; k < opds.size(); ++k) {
          const int copies = opds[k].most * opds[k].K * (int)es / copy_of[opds[k].kind];
          const int room = (MAX_TASKS - (int)tasks.size()) / (int)(opds.size() - k);
          const int cut = std::max(1, std::min(room, copies / 192));
          const int len = (int)ceil_div(ceil_div(opds[k].K, cut), 8) * 8;
          for (int lo = 0; lo < opds[k].K; lo += len) {
            tasks.push_back(opds[k]);
            tasks.back().k_lo = lo;
            tasks.back().k_hi = std::min(opds[k].K, lo + len);
          }
        }
        opds.swap(tasks);
      }
      h.n_opd = (int)opds.size();
      std::vector<unsigned char> prog(sizeof(Head) + loads.size() * sizeof(Load) + ins.size() * sizeof(Ins) + stores.size() * sizeof(Store) +
                                      opds.size() * sizeof(Opd) + dot.size() * sizeof(Dot));
      unsigned char* w = prog.data();
      memcpy(w, &h, sizeof(h)); w += sizeof(h);
      memcpy(w, loads.data(), loads.size() * sizeof(Load)); w += loads.size() * sizeof(Load);
      memcpy(w, ins.data(), ins.size() * sizeof(Ins)); w += ins.size() * sizeof(Ins);
      memcpy(w, stores.data(), stores.size() * sizeof(Store)); w += stores.size() * sizeof(Store);
      memcpy(w, opds.data(), opds.size() * sizeof(Opd)); w += opds.size() * sizeof(Opd);
      memcpy(w, dot.data(), dot.size() * sizeof(Dot));
      const uint32_t at = put(prog.data(), prog.size());
      double cost = 1.0 + 0.02 * (double)loads.size() / (double)h.team;
      if (!dot.empty())
        cost += 0.4 + most_k * (es == 8 ? 0.012 : 0.008) * (double)ceil_div((int64_t)dot.size(), h.team) + 0.6 * (double)(ceil_div(most_k, h.ks) - 1);
      if (h.team > 1) {
        cost += 0.25 * phases;
      } else {
        cost += 0.1 * (double)ins.size();
        for (const Ins& c : ins) cost += c.op == PRIM_ACT_FORWARD || c.op == PRIM_ACT_BACKWARD ? 0.3 : 0;
      }
      for (int64_t c = 0; c < ceil_div(g.n, NT / h.team); ++c) pieces[level[i]].push_back({at, (uint32_t)((prog.size() + 15) & ~(size_t)15), (uint32_t)c, cost});
      continue;
    }
    if (p.kind == PRIM_PRODUCT) {
      ProductProg q{};
      q.h.kind = PRIM_PRODUCT;
      q.A = p.in[0]; q.B = p.in[1]; q.C = p.out[0];
      q.sA = p.sA; q.sB = p.sB; q.sC = p.sC;
      q.alpha = p.scalar;
      q.tA = p.tA; q.tB = p.tB; q.M = p.M; q.N = p.N; q.K = p.K;
      // 32 x 32 outputs while that many are there and the chain is short (a weight gradient's outer products), else 256
      q.r = p.K <= 32 && p.M > 16 && p.N > 16 ? 2 : 1;
      if (q.r == 1) {
        q.tn = p.N > 8 ? 16 : p.N > 4 ? 8 : p.N > 2 ? 4 : p.N > 1 ? 2 : 1;
        q.tm = std::min(NT / q.tn, 64);
      } else {
        q.tm = q.tn = 32;
      }
      q.ks = p.K;
      while ((q.tm + q.tn) * product_pitch<T>(q.ks) * (int)es > WORK_BYTES) q.ks = (q.ks + 1) / 2;
      q.tiles_n = (int)ceil_div(p.N, q.tn);
      q.tiles_mn = (int)ceil_div(p.M, q.tm) * q.tiles_n;
      const uint32_t at = put(&q, sizeof(q));
      const double cost = 1.2 + p.K * (es == 8 ? 0.017 : 0.012) * (q.r == 2 ? 2 : 1) + 0.6 * (double)(ceil_div(p.K, q.ks) - 1);
      for (int64_t c = 0; c < (int64_t)q.tiles_mn * p.batch; ++c) pieces[level[i]].push_back({at, (uint32_t)((sizeof(q) + 15) & ~(size_t)15), (uint32_t)c, cost});
      continue;
    }
    RowProg q{};
    q.h.kind = p.kind;
    for (size_t k = 0; k < p.in.size(); ++k) q.in[k] = p.in[k];
    for (size_t k = 0; k < p.out.size(); ++k) q.out[k] = p.out[k];
    q.rows = p.rows; q.cols = p.cols; q.depth = p.depth;
    q.scalar = p.scalar;
    int64_t chunks;
    double cost;
    if (p.kind == PRIM_COLUMN_SUM) { chunks = ceil_div(p.cols, NT); cost = 0.8 + 0.15 * (double)p.rows; }
    else if (p.kind == PRIM_TRANSPOSE) { chunks = ceil_div(p.rows * p.cols * p.depth, NT); cost = 0.9; }
    else { q.rows = p.rows * p.depth; chunks = ceil_div(q.rows, NT / 32); cost = 2.0 + 0.1 * (double)p.cols; }
    const uint32_t at = put(&q, sizeof(q));
    for (int64_t c = 0; c < chunks; ++c) pieces[level[i]].push_back({at, (uint32_t)((sizeof(q) + 15) & ~(size_t)15), (uint32_t)c, cost});
  }

  // Deal the pieces of a level to the workers of `c` CTAs, the longest first to whoever has least (and to another SM before the
  // same one again); worker k of the dealing order is number k / c of CTA k % c.  Returns the time of the busiest.
  auto deal = [&](int lv, int c, std::vector<std::vector<Item>>& lists) {
    if (pieces[lv].size() <= (size_t)c * WORKERS) {          // one each
      for (int k = 0; k < (int)pieces[lv].size(); ++k) {
        const Piece& p = pieces[lv][k];
        lists[k % c * WORKERS + k / c].push_back({p.prog, p.bytes, p.chunk, 0});
      }
      return pieces[lv].empty() ? 0.0 : pieces[lv][0].cost;
    }
    std::vector<std::pair<double, int>> heap;                // least busy first
    for (int k = 0; k < c * WORKERS; ++k) heap.push_back({0.0, k});
    auto later = [](const std::pair<double, int>& x, const std::pair<double, int>& y) { return x > y; };
    auto give = [&](std::pair<double, int>& to, const Piece& p) {
      to.first += p.cost;
      lists[to.second % c * WORKERS + to.second / c].push_back({p.prog, p.bytes, p.chunk, 0});
    };
    const std::vector<Piece>& all = pieces[lv];
    for (auto& l : lists) l.reserve(l.size() + all.size() / (size_t)(c * WORKERS) + 1);
    for (size_t k = 0; k < all.size();) {
      size_t end = k + 1;                                    // pieces of one cost, many: in turn, once nobody is a piece ahead
      while (end < all.size() && all[end].cost == all[k].cost) ++end;
      if (end - k > 16) {
        std::sort(heap.begin(), heap.end());                 // (a heap too)
        if (heap.back().first - heap[0].first <= all[k].cost) {
          for (size_t at = 0; k < end; ++k, at = at + 1 == heap.size() ? 0 : at + 1) give(heap[at], all[k]);
          std::make_heap(heap.begin(), heap.end(), later);
          continue;
        }
      }
      for (; k < end; ++k) {
        std::pop_heap(heap.begin(), heap.end(), later);
        give(heap.back(), all[k]);
        std::push_heap(heap.begin(), heap.end(), later);
      }
    }
    double most = 0;
    for (const auto& w : heap) most = std::max(most, w.first);
    return most;
  };
  for (auto& lv : pieces) std::stable_sort(lv.begin(), lv.end(), [](const Piece& a, const Piece& b) { return a.cost > b.cost; });
  // The last levels run on all SMs, a launch each (its program's way into every SM and the launch: 2.8 us more than a level of the
  // cluster), from the level on where that gains most: a level of many pieces may be followed by one that loses by it.  (Ended at the first
  // level from behind that would gain less than 6 us, twenty elementwise operations on 128 x 128 floats took 40 us backward, and
  // a step of three layers of 128 units, 16 columns, twelve time steps, double, 1246; now 21 and 469.)
  int narrow = levels;
  double gained = 0, most_gained = 0;
  for (int lv = levels; lv-- > 0;) {
    const std::vector<Piece>& level_pieces = pieces[lv];
    if (level_pieces.empty()) continue;
    const double longest = level_pieces.front().cost;
    double all = 0;
    for (const Piece& p : level_pieces) all += p.cost;
    auto time = [&](int workers) {
      if (longest == level_pieces.back().cost) return (double)ceil_div((int64_t)level_pieces.size(), workers) * longest;
      return std::max(longest, all / workers);
    };
    gained += time(ctas * WORKERS) - time(ctx->sm_count * WORKERS) - 2.8;
    if (gained > most_gained) {
      most_gained = gained;
      narrow = lv;
    }
  }
  *est_us = 4.0;
  if (narrow > 0) {
    Part part{ctas, true, {}};
    part.lists.assign(ctas * WORKERS, {});
    for (int lv = 0; lv < narrow; ++lv) {
      std::vector<size_t> before(part.lists.size());
      for (size_t c = 0; c < before.size(); ++c) before[c] = part.lists[c].size();
      *est_us += 0.8 + deal(lv, ctas, part.lists);
      for (size_t c = 0; c < before.size(); ++c) {           // a barrier behind every level
        if (part.lists[c].size() == before[c]) part.lists[c].push_back({0, 0, 0, 1});
        else part.lists[c].back().barrier = 1;
      }
    }
    parts.push_back(std::move(part));
  }
  for (int lv = narrow; lv < levels; ++lv) {
    if (pieces[lv].empty()) continue;
    Part part{ctx->sm_count, false, {}};
    part.lists.assign(ctx->sm_count * WORKERS, {});
    *est_us += 3.0 + deal(lv, ctx->sm_count, part.lists);
    parts.push_back(std::move(part));
  }
}

// 16 CTAs if the device runs such a cluster of this kernel, else 8, else none
template <typename T> static cudaError_t reserve(void) {
  cudaError_t e = cudaSuccess;
  auto one = [&](auto* kernel) {
    if (e == cudaSuccess) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  };
  one(walk_kernel<T, FEW_STARTS>);
  one(walk_kernel<T, MOST_STARTS>);
  return e;
}
template <typename T> static int cluster_ctas(prad_ctx* ctx) {
  static std::atomic<int> known[64];
  std::atomic<int>& k = known[ctx->device & 63];
  int n = k.load(std::memory_order_acquire);
  if (n) return n - 1;
  n = 0;
  const cudaError_t e = reserve<T>();
  for (int cs : {16, 8}) {
    if (e != cudaSuccess || n) break;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = cs;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3((unsigned)cs);
    cfg.blockDim = dim3(WORKERS * NT);
    cfg.dynamicSmemBytes = SMEM_BYTES;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int fit = 0;
    if (cudaOccupancyMaxActiveClusters(&fit, walk_kernel<T, FEW_STARTS>, &cfg) == cudaSuccess && fit > 0) n = cs;
    else (void)cudaGetLastError();
  }
  if (e != cudaSuccess) (void)cudaGetLastError();
  k.store(n + 1, std::memory_order_release);
  return n;
}

template <typename T> static GraphPlanPtr build_plan(prad_ctx* ctx, prad_dtype dt, const std::vector<Prim>& ops) {
  if (ops.size() < 3 || ops.size() > 20000) return nullptr;
  const int ctas = cluster_ctas<T>(ctx);
  if (!ctas) return nullptr;
  // an operation that deserves the whole device makes the walk one for separate launches
  for (const Prim& p : ops) {
    if (p.kind == PRIM_PRODUCT && (p.K < 1 || (double)p.M * p.N * p.K * p.batch > 4e6)) return nullptr;
    if (elementwise(p) ? p.n > 65536 : p.kind != PRIM_PRODUCT && (double)p.rows * p.cols * p.depth > 65536) return nullptr;
    if (p.in.size() > 8) return nullptr;
  }
  std::vector<unsigned char> blob;
  std::vector<Part> parts;
  double est = 0, launches = 0;
  std::vector<std::pair<uintptr_t, uintptr_t>> written;      // where the operations write: ascending, without overlaps
  int products = 0;
  build<T>(ctx, ops, ctas, blob, parts, written, &est, &launches, &products);
  if (est >= launches) return nullptr;
  std::vector<Item> items;
  std::vector<int> first;
  for (auto& part : parts) {
    for (auto& l : part.lists) {
      first.push_back((int)items.size());
      items.insert(items.end(), l.begin(), l.end());
    }
    first.push_back((int)items.size());
  }
  const size_t items_bytes = items.size() * sizeof(Item), first_bytes = (first.size() * sizeof(int) + 15) & ~(size_t)15;
  std::vector<unsigned char> host(items_bytes + first_bytes + blob.size());
  memcpy(host.data(), items.data(), items_bytes);
  memcpy(host.data() + items_bytes, first.data(), first.size() * sizeof(int));
  memcpy(host.data() + items_bytes + first_bytes, blob.data(), blob.size());
  GraphPlanPtr plan(new GraphPlan());
  plan->device = ctx->device;
  plan->dt = dt;
  if (device_malloc(&plan->mem, host.size()) != cudaSuccess ||
      cudaMemcpyAsync(plan->mem, host.data(), host.size(), cudaMemcpyHostToDevice, ctx->stream) != cudaSuccess ||
      cudaStreamSynchronize(ctx->stream) != cudaSuccess) {
    (void)cudaGetLastError();
    return nullptr;
  }
  plan->written = std::move(written);
  plan->products = products;
  plan->items = (const Item*)plan->mem;
  const int* at = (const int*)((const unsigned char*)plan->mem + items_bytes);
  for (const auto& part : parts) {
    plan->parts.push_back({part.ctas, part.cluster, at});
    at += part.lists.size() + 1;
  }
  plan->blob = (const unsigned char*)plan->mem + items_bytes + first_bytes;
  return plan;
}

}  // namespace gp

GraphPlanPtr graph_plan_build(prad_ctx* ctx, prad_dtype dt, const std::vector<Prim>& ops) {
  return dt == PRAD_F32 ? gp::build_plan<float>(ctx, dt, ops) : gp::build_plan<double>(ctx, dt, ops);
}

int graph_plan_products(const GraphPlan* plan) { return plan->products; }

bool graph_plan_writes(const GraphPlan* plan, const void* p, size_t bytes) {
  const uintptr_t lo = (uintptr_t)p, hi = lo + bytes;
  auto it = std::upper_bound(plan->written.begin(), plan->written.end(), std::make_pair(lo, ~(uintptr_t)0));
  return (it != plan->written.begin() && std::prev(it)->second > lo) || (it != plan->written.end() && it->first < hi);
}

template <typename T, int N>
static prad_status run_walk(prad_ctx* ctx, const GraphPlan* plan, const void* const* starts, int count) {
  gp::StartTable<N> table;
  for (int i = 0; i < count; ++i) table.p[i] = starts[i];
  for (const GraphPlan::Part& part : plan->parts) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = part.ctas;
    at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
    cfg.gridDim = dim3((unsigned)part.ctas);
    cfg.blockDim = dim3(gp::WORKERS * gp::NT);
    cfg.dynamicSmemBytes = gp::SMEM_BYTES;
    cfg.stream = ctx->stream;
    cfg.attrs = at;
    cfg.numAttrs = part.cluster ? 2 : 1;
    PRAD_CUDA(cudaLaunchKernelEx(&cfg, gp::walk_kernel<T, N>, plan->blob, plan->items, part.first, table));
    PRAD_LAUNCHED(ctx);
  }
  return PRAD_OK;
}

prad_status graph_plan_run(prad_ctx* ctx, GraphPlan* plan, const void* const* starts, int count) {
  const bool few = count <= gp::FEW_STARTS;
  if (plan->dt == PRAD_F32)
    return few ? run_walk<float, gp::FEW_STARTS>(ctx, plan, starts, count) : run_walk<float, MOST_STARTS>(ctx, plan, starts, count);
  return few ? run_walk<double, gp::FEW_STARTS>(ctx, plan, starts, count) : run_walk<double, MOST_STARTS>(ctx, plan, starts, count);
}

}  // namespace prad

// Runs a graph's walk as ONE kernel.
//
// What bounded it: an unrolled network from a JSON architecture is hundreds of operations on a few hundred values each.  An
// eight-step two-layer LSTM of 64 units is 1058 launches of 2 - 6 us per training step, 4.9 ms, for 25 MFLOP.
//
// Here the walk is recorded once as a list of primitive operations.  A level of the plan holds operations that depend on
// earlier levels only; chains of elementwise operations on the same elements (a gate's sum and activation, a cell update, the
// += of a shared weight's gradients over the time steps) share a level too, as a small program that keeps every value of one
// element in shared memory from its load to its store.  One cluster of 16 CTAs runs the levels with the cluster's hardware
// barrier between them (no waiting loops, no other CTA to wait for).  A level is latency: a barrier, a program, loads from L2,
// a chain of 64 additions.  So the pieces of a level -- 64 or 256 elements, 256 or 1024 outputs -- are dealt to 64 workers when
// the plan is made, four to an SM, and a worker fetches its next program while it runs this one. 
// (One worker per SM took 240 us per walk of that LSTM, four take 150 us.)
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
constexpr int WORKERS = 4;                // workers of a CTA: a piece is mostly latency, so several share an SM
constexpr int SLOTS = 64;                 // values of one element a program keeps
constexpr int MAX_INS = 96;
constexpr int PROG_BYTES = 32 + SLOTS * 16 + MAX_INS * 24 + SLOTS * 16;
constexpr int WORK_BYTES = 44 * 1024;     // a worker's shared memory: the slots of its elements, or the operands of a product

// a piece of one worker
struct Item { uint32_t prog, bytes, chunk, barrier; };

// team: 4 where four threads share an element's instructions (a piece is 64 elements then), else 1
struct Head { int32_t kind, n_load, n_ins, n_store; int64_t n; int64_t team; };
struct Load { const void* p; uint32_t cols, slot; };        // cols: 0 = element i, else element i % cols
// phase: in the first instruction of a phase (instructions that do not touch one another's values), how many it has
struct Ins { uint8_t op, act, n_in, phase; uint8_t dst[2], pad2[2]; uint8_t src[8]; double scalar; };
constexpr uint8_t INS_FOLD = 64;          // ((src0 + src1) + src2) + ... in T: a run of dst += src
struct Store { void* p; uint32_t slot, pad; };
static_assert(sizeof(Head) == 32 && sizeof(Load) == 16 && sizeof(Ins) == 24 && sizeof(Store) == 16, "program layout");
struct ProductProg {
  Head h;                                                    // kind = PRIM_PRODUCT
  const void *A, *B;
  void* C;
  int64_t sA, sB, sC;
  double alpha;
  int32_t tA, tB, M, N, K, tm, tn, ks, tiles_n, tiles_mn, r;   // r: r x r outputs per thread
};
struct RowProg { Head h; const void* in[4]; void* out[3]; int64_t rows; int32_t cols, depth; double scalar; };

__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
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

// A piece: 256 elements, one per thread, or 64 elements with four threads each, which take the loads, the instructions of a
// phase and the stores in turn (four gates' exponentials side by side instead of one after another).
template <typename T, int N>
__device__ void run_elementwise(const Head* h, int chunk, T* v, const StartTable<N>& starts) {
  const int tid = threadIdx.x % NT, team = (int)h->team;
  const int per = NT / team, e = tid % per, q0 = tid / per;
  const Load* ld = reinterpret_cast<const Load*>(h + 1);
  const Ins* ins = reinterpret_cast<const Ins*>(ld + h->n_load);
  const Store* st = reinterpret_cast<const Store*>(ins + h->n_ins);
  const int64_t i = (int64_t)chunk * per + e;
  const bool on = i < h->n;
  v += e;
  if (on)
    for (int k = q0; k < h->n_load; k += team)      // all on their way at once
      copy_async<sizeof(T)>(v + ld[k].slot * per, source<T>(ld[k].p, starts) + (ld[k].cols ? i % ld[k].cols : i));
  copy_wait();
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

// ---- products: a tm x tn tile, R x R outputs per thread, both operands of ks values of k in shared memory
// rows of 16-byte vectors plus one: the rows of neighbouring threads fall into different banks
template <typename T> __host__ __device__ constexpr int product_pitch(int ks) {
  constexpr int VEC = 16 / (int)sizeof(T);
  return (ks + VEC - 1) / VEC * VEC + VEC;
}
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
    if (on) {
      const T* a = As + mi * pa;
      const T* b = Bs + ni * pa;
      T x[R][R], y[R][R];
      auto products = [&](T (&d)[R][R], int k) {
        T av[R], bv[R];
#pragma unroll
        for (int i = 0; i < R; ++i) { av[i] = a[i * ty * pa + k]; bv[i] = b[i * tx * pa + k]; }
#pragma unroll
        for (int i = 0; i < R; ++i)
#pragma unroll
          for (int j = 0; j < R; ++j) d[i][j] = mul_rn(av[i], bv[j]);
      };
      auto sums = [&](const T (&d)[R][R]) {
#pragma unroll
        for (int i = 0; i < R; ++i)
#pragma unroll
          for (int j = 0; j < R; ++j) acc[i][j] = add_rn(acc[i][j], d[i][j]);
      };
      // the products of the next k are formed ahead of the sums of this one
      products(x, 0);
      int k = 1;
#pragma unroll 4
      for (; k + 1 < kc; k += 2) {
        products(y, k);
        sums(x);
        products(x, k + 1);
        sums(y);
      }
      if (k < kc) {
        products(y, k);
        sums(x);
        sums(y);
      } else {
        sums(x);
      }
    }
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
  extern __shared__ __align__(16) unsigned char gp_smem[];
  const int tid = threadIdx.x % NT, worker = blockIdx.x * WORKERS + threadIdx.x / NT;
  unsigned char* prog = gp_smem + (threadIdx.x / NT) * (2 * PROG_BYTES + WORK_BYTES);
  T* work = reinterpret_cast<T*>(prog + 2 * PROG_BYTES);
  items += first[worker];
  const int n = first[worker + 1] - first[worker];
  auto fetch = [&](const Item& it, int i) {
    for (uint32_t b = tid * 8; b < it.bytes; b += NT * 8) copy_async<8>(prog + (i & 1) * PROG_BYTES + b, blob + it.prog + b);
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
  int device = 0, ctas = 0;
  prad_dtype dt = PRAD_F32;
  void* mem = nullptr;                       // [items][first item of each worker][blob]
  const unsigned char* blob = nullptr;
  const gp::Item* items = nullptr;
  const int* first = nullptr;
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
struct Access { uintptr_t lo, hi; bool write, local; };

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

// An elementwise program in the making.
struct Group {
  int64_t n = 0;
  std::vector<int> ops;                      // ascending
};

// (buffer, columns of a row operand or 0): what has a place of its own in a program
using Place = std::pair<const void*, int>;
static Place place_of(const Prim& p, size_t k) { return {p.in[k], p.kind == PRIM_ADD_ROW && k == 1 ? p.cols : 0}; }
constexpr int64_t TEAM_ELEMENTS = 2048;      // up to here four threads can share an element
template <typename T> static int slot_limit(int64_t n) {
  return n <= TEAM_ELEMENTS ? SLOTS : std::min(SLOTS, WORK_BYTES / (NT * (int)sizeof(T)));
}
static int places(const std::vector<Prim>& all, const std::vector<int>& ops) {
  std::vector<Place> seen;
  for (int o : ops) {
    for (size_t k = 0; k < all[o].in.size(); ++k) seen.push_back(place_of(all[o], k));
    for (void* q : all[o].out) seen.push_back({q, 0});
  }
  std::sort(seen.begin(), seen.end());
  return (int)(std::unique(seen.begin(), seen.end()) - seen.begin());
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
  int phases = 0;
  for (size_t x = 0; x < ins.size(); ++x) {
    for (size_t y = 0; y < x; ++y) {
      bool after = false;
      for (int k = 0; k < ins[x].n_in; ++k) after = after || writes(ins[y], ins[x].src[k]);
      for (int k = 0; k < outputs(ins[x]); ++k) after = after || writes(ins[y], ins[x].dst[k]) || reads(ins[y], ins[x].dst[k]);
      if (after) phase[x] = std::max(phase[x], phase[y] + 1);
    }
    phases = std::max(phases, phase[x] + 1);
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

template <typename T> static void build(prad_ctx* ctx, const std::vector<Prim>& ops, int ctas, std::vector<unsigned char>& blob,
                                        std::vector<std::vector<Item>>& lists, std::vector<std::pair<uintptr_t, uintptr_t>>& written,
                                        double* est_us, double* launch_us) {
  const size_t es = sizeof(T);
  const int N = (int)ops.size();
  std::vector<int> level(N, 0), group_of(N, -1);
  std::vector<Group> groups;
  std::map<uintptr_t, Region> mem;
  std::vector<Access> acc;
  *launch_us = 0;
  auto region_at = [&](const Access& a) -> Region& {
    auto it = mem.upper_bound(a.lo);
    if (it != mem.begin()) {
      auto p = std::prev(it);
      if (p->second.hi > a.lo) it = p;
    }
    if (it == mem.end() || it->first >= a.hi) return mem.emplace(a.lo, Region{a.lo, a.hi, true, false, {}, {}}).first->second;
    if (it->first == a.lo && it->second.hi == a.hi) return it->second;
    Region joined{a.lo, a.hi, false, false, {}, {}};      // overlaps: one region for all of them
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
  for (int i = 0; i < N; ++i) {
    *launch_us += launch_cost(ops[i], ctx->sm_count);
    accesses(ops[i], es, acc);
    int lv = 0;
    std::vector<int> near;                   // operations this one may share a program with
    for (const Access& a : acc) {
      Region& r = region_at(a);
      auto depend = [&](int d) {
        if (d == i) return;
        const bool local = a.local && r.local && elementwise(ops[i]) && elementwise(ops[d]) && ops[i].n == ops[d].n;
        lv = std::max(lv, local ? level[d] : level[d] + 1);
        if (local) near.push_back(d);
      };
      for (int d : r.writers) depend(d);
      if (a.write)
        for (int d : r.readers) depend(d);
    }
    if (elementwise(ops[i])) {
      // join the programs of the local neighbours at this level, if one program can hold them all
      Group merged;
      merged.n = ops[i].n;
      std::vector<int> join;
      for (int d : near)
        if (level[d] == lv && std::find(join.begin(), join.end(), group_of[d]) == join.end()) join.push_back(group_of[d]);
      for (int g : join) merged.ops.insert(merged.ops.end(), groups[g].ops.begin(), groups[g].ops.end());
      std::sort(merged.ops.begin(), merged.ops.end());
      merged.ops.push_back(i);
      if (!join.empty() && ((int)merged.ops.size() > MAX_INS || places(ops, merged.ops) > slot_limit<T>(merged.n))) {
        ++lv;                                // a program of its own, behind a barrier
        join.clear();
        merged.ops.assign(1, i);
      }
      for (int g : join) groups[g].ops.clear();
      const int id = (int)groups.size();
      for (int o : merged.ops) group_of[o] = id;
      groups.push_back(std::move(merged));
    }
    level[i] = lv;
    for (const Access& a : acc) {
      Region& r = region_at(a);
      r.local = r.local && a.local;
      if (!a.write) { r.readers.push_back(i); continue; }
      r.written = true;
      if (r.lo == a.lo && r.hi == a.hi) { r.writers.clear(); r.readers.clear(); }
      r.writers.push_back(i);
    }
  }

  for (const auto& m : mem)
    if (m.second.written) {
      if (!written.empty() && written.back().second == m.second.lo) written.back().second = m.second.hi;
      else written.emplace_back(m.second.lo, m.second.hi);
    }

  // programs, and the pieces of every level
  const int levels = N ? *std::max_element(level.begin(), level.end()) + 1 : 0;
  std::vector<std::vector<Piece>> pieces(levels);
  auto put = [&](const void* p, size_t bytes) {
    const size_t at = blob.size();
    blob.resize(at + ((bytes + 15) & ~(size_t)15));
    memcpy(blob.data() + at, p, bytes);
    return (uint32_t)at;
  };
  for (int i = 0; i < N; ++i) {
    const Prim& p = ops[i];
    if (elementwise(p)) {
      const Group& g = groups[group_of[i]];
      if (g.ops.front() != i) continue;
      std::vector<Load> loads;
      std::vector<Ins> ins;
      std::vector<Store> stores;
      std::map<Place, int> slot;
      int slots = 0;
      for (int o : g.ops) {
        const Prim& q = ops[o];
        Ins c;
        memset(&c, 0, sizeof(c));
        c.op = (uint8_t)q.kind;
        c.act = (uint8_t)q.act;
        c.n_in = (uint8_t)q.in.size();
        c.scalar = q.scalar;
        for (size_t k = 0; k < q.in.size(); ++k) {
          const Place at = place_of(q, k);
          auto it = slot.find(at);
          if (it == slot.end()) {
            it = slot.emplace(at, slots++).first;
            loads.push_back({at.first, (uint32_t)at.second, (uint32_t)it->second});
          }
          c.src[k] = (uint8_t)it->second;
        }
        for (size_t k = 0; k < q.out.size(); ++k) {
          auto it = slot.find(Place{q.out[k], 0});
          if (it == slot.end()) it = slot.emplace(Place{q.out[k], 0}, slots++).first;
          c.dst[k] = (uint8_t)it->second;
          bool stored = false;
          for (const Store& s : stores) stored = stored || s.p == q.out[k];
          if (!stored) stores.push_back({q.out[k], (uint32_t)it->second, 0});
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
      h.team = g.n <= TEAM_ELEMENTS && (ins.size() >= 4 || slots > WORK_BYTES / (NT * (int)es)) ? 4 : 1;
      std::vector<unsigned char> prog(sizeof(Head) + loads.size() * sizeof(Load) + ins.size() * sizeof(Ins) + stores.size() * sizeof(Store));
      unsigned char* w = prog.data();
      memcpy(w, &h, sizeof(h)); w += sizeof(h);
      memcpy(w, loads.data(), loads.size() * sizeof(Load)); w += loads.size() * sizeof(Load);
      memcpy(w, ins.data(), ins.size() * sizeof(Ins)); w += ins.size() * sizeof(Ins);
      memcpy(w, stores.data(), stores.size() * sizeof(Store));
      const uint32_t at = put(prog.data(), prog.size());
      double cost = 1.0 + 0.02 * (double)loads.size() / (double)h.team;
      if (h.team > 1) {
        cost += 0.35 * phases;
      } else {
        cost += 0.1 * (double)ins.size();
        for (const Ins& c : ins) cost += c.op == PRIM_ACT_FORWARD || c.op == PRIM_ACT_BACKWARD ? 0.3 : 0;
      }
      for (int64_t c = 0; c < ceil_div(g.n, NT / h.team); ++c) pieces[level[i]].push_back({at, (uint32_t)((prog.size() + 7) & ~(size_t)7), (uint32_t)c, cost});
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
      for (int64_t c = 0; c < (int64_t)q.tiles_mn * p.batch; ++c) pieces[level[i]].push_back({at, (uint32_t)((sizeof(q) + 7) & ~(size_t)7), (uint32_t)c, cost});
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
    for (int64_t c = 0; c < chunks; ++c) pieces[level[i]].push_back({at, (uint32_t)((sizeof(q) + 7) & ~(size_t)7), (uint32_t)c, cost});
  }

  // deal the pieces of a level to the workers, the longest first to whoever has least (and to another SM before the same one
  // again); a barrier behind every level
  const int workers = ctas * WORKERS;
  lists.assign(workers, {});
  *est_us = 4.0;
  std::vector<double> busy(workers);         // worker k of the dealing order is number k / ctas of CTA k % ctas
  for (int lv = 0; lv < levels; ++lv) {
    std::stable_sort(pieces[lv].begin(), pieces[lv].end(), [](const Piece& a, const Piece& b) { return a.cost > b.cost; });
    std::fill(busy.begin(), busy.end(), 0.0);
    std::vector<size_t> before(workers);
    for (int c = 0; c < workers; ++c) before[c] = lists[c].size();
    for (const Piece& p : pieces[lv]) {
      const int k = (int)(std::min_element(busy.begin(), busy.end()) - busy.begin());
      busy[k] += p.cost;
      lists[k % ctas * WORKERS + k / ctas].push_back({p.prog, p.bytes, p.chunk, 0});
    }
    for (int c = 0; c < workers; ++c) {
      if (lists[c].size() == before[c]) lists[c].push_back({0, 0, 0, 1});
      else lists[c].back().barrier = 1;
    }
    *est_us += 0.8 + *std::max_element(busy.begin(), busy.end());
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
  std::vector<std::vector<Item>> lists;
  double est = 0, launches = 0;
  std::vector<std::pair<uintptr_t, uintptr_t>> written;      // where the operations write: ascending, without overlaps
  build<T>(ctx, ops, ctas, blob, lists, written, &est, &launches);
  if (est >= launches) return nullptr;
  std::vector<Item> items;
  std::vector<int> first;
  for (auto& l : lists) {
    first.push_back((int)items.size());
    items.insert(items.end(), l.begin(), l.end());
  }
  first.push_back((int)items.size());
  const size_t items_bytes = items.size() * sizeof(Item), first_bytes = (first.size() * sizeof(int) + 15) & ~(size_t)15;
  std::vector<unsigned char> host(items_bytes + first_bytes + blob.size());
  memcpy(host.data(), items.data(), items_bytes);
  memcpy(host.data() + items_bytes, first.data(), first.size() * sizeof(int));
  memcpy(host.data() + items_bytes + first_bytes, blob.data(), blob.size());
  GraphPlanPtr plan(new GraphPlan());
  plan->device = ctx->device;
  plan->ctas = ctas;
  plan->dt = dt;
  if (device_malloc(&plan->mem, host.size()) != cudaSuccess ||
      cudaMemcpyAsync(plan->mem, host.data(), host.size(), cudaMemcpyHostToDevice, ctx->stream) != cudaSuccess ||
      cudaStreamSynchronize(ctx->stream) != cudaSuccess) {
    (void)cudaGetLastError();
    return nullptr;
  }
  plan->written = std::move(written);
  plan->items = (const Item*)plan->mem;
  plan->first = (const int*)((const unsigned char*)plan->mem + items_bytes);
  plan->blob = (const unsigned char*)plan->mem + items_bytes + first_bytes;
  return plan;
}

}  // namespace gp

GraphPlanPtr graph_plan_build(prad_ctx* ctx, prad_dtype dt, const std::vector<Prim>& ops) {
  return dt == PRAD_F32 ? gp::build_plan<float>(ctx, dt, ops) : gp::build_plan<double>(ctx, dt, ops);
}

bool graph_plan_writes(const GraphPlan* plan, const void* p, size_t bytes) {
  const uintptr_t lo = (uintptr_t)p, hi = lo + bytes;
  auto it = std::upper_bound(plan->written.begin(), plan->written.end(), std::make_pair(lo, ~(uintptr_t)0));
  return (it != plan->written.begin() && std::prev(it)->second > lo) || (it != plan->written.end() && it->first < hi);
}

template <typename T, int N>
static prad_status run_walk(prad_ctx* ctx, const cudaLaunchConfig_t& cfg, const GraphPlan* plan, const void* const* starts, int count) {
  gp::StartTable<N> table;
  for (int i = 0; i < count; ++i) table.p[i] = starts[i];
  PRAD_CUDA(cudaLaunchKernelEx(&cfg, gp::walk_kernel<T, N>, plan->blob, plan->items, plan->first, table));
  PRAD_LAUNCHED(ctx);
  return PRAD_OK;
}

prad_status graph_plan_run(prad_ctx* ctx, GraphPlan* plan, const void* const* starts, int count) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = plan->ctas;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3((unsigned)plan->ctas);
  cfg.blockDim = dim3(gp::WORKERS * gp::NT);
  cfg.dynamicSmemBytes = gp::SMEM_BYTES;
  cfg.stream = ctx->stream;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  const bool few = count <= gp::FEW_STARTS;
  if (plan->dt == PRAD_F32)
    return few ? run_walk<float, gp::FEW_STARTS>(ctx, cfg, plan, starts, count) : run_walk<float, MOST_STARTS>(ctx, cfg, plan, starts, count);
  return few ? run_walk<double, gp::FEW_STARTS>(ctx, cfg, plan, starts, count) : run_walk<double, MOST_STARTS>(ctx, cfg, plan, starts, count);
}

}  // namespace prad

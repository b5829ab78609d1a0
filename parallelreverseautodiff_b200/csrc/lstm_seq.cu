// A whole LSTM sequence per launch: the recurrent part of Forward and of backpropagation through time.
//
// What bounded it: one time step is a 32 x 1024 product over k = 256 and a handful of elementwise operations on 32 x 256
// values, and the next step needs all of it.  As 16 launches forward and 2 backward per step, a 64-step sequence took
// 5.1 ms of kernels and 8 ms with the calls that launch them; the arithmetic of a step is 1 us.
//
// Here the batch is cut into tiles of at most 5 rows, and a CLUSTER of CTAs owns one tile for all time steps: CTA r of the
// cluster owns JJ hidden units (all four gates of them), keeps their rows of the recurrent weights in shared memory from the
// first step to the last, and hands what it computed in a step (h_t forward, the four dpre_t backward) to its cluster
// neighbours' shared memory with one bulk copy each, which the receiver waits for on an mbarrier.  Clusters never talk to
// each other, so there is no grid-wide wait and any number of batch tiles can run, in turns if need be.  Two exchange
// buffers suffice: a neighbour sends step t + 1 only after it has everybody's step t.
//
// Arithmetic is that of the separate operations, rounding for rounding: k ascending, one accumulator, product and sum rounded
// separately (hidden units beyond the matrix are zeros, which change no sum); one rounding per managed operation in the cell.
// Every wait is bounded: a CTA that gives up raises the context's flag (PRAD_ERR_TIMEOUT at the next prad_sync) and runs
// on without waiting.  (Compiled with -fmad=false.)
#include "act_math.cuh"
#include "common.cuh"

namespace prad {
namespace lstm {

constexpr int WAIT_LIMIT = 1 << 18;  // polls

__device__ __forceinline__ uint32_t saddr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint32_t cluster_rank() { uint32_t r; asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ uint32_t cluster_size() { uint32_t r; asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ uint32_t in_cta(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ void mbar_init(uint32_t bar) { asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar)); }
__device__ __forceinline__ void mbar_expect(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.b32 %0, 1, 0, p;\n\t}"
      : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
  return ok != 0;
}
__device__ __forceinline__ void push(uint32_t dst, uint32_t src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(dst), "r"(src), "r"(bytes), "r"(bar) : "memory");
}

template <typename T, int N> __device__ __forceinline__ void lds16(const T* p, T (&v)[N]) {
  static_assert(N * sizeof(T) == 16, "16 bytes");
  *reinterpret_cast<uint4*>(v) = *reinterpret_cast<const uint4*>(p);
}

// JP: hidden units per CTA, padded; BB: batch rows of a tile; NG: gate matrices in the exchange buffer (1: h, 4: dpre)
template <typename T, int JP, int BB, int NG>
struct Tile {
  static constexpr int VEC = 16 / sizeof(T);
  static constexpr int TR = BB == 4 ? 2 : BB, TC = BB == 4 ? 2 : 1;    // outputs per multiplying thread: rows x columns
  static constexpr int COLS = 4 * JP;                                   // (gate, hidden unit)
  static constexpr int BLOCK = NG * BB * JP;                            // what one CTA hands over per step
  static constexpr int G = JP / VEC;                                     // 16-byte groups of k per block
  static constexpr int DEPTH = G % 4 == 0 ? 4 : G % 3 == 0 ? 3 : 2;     // groups in registers
  // Forward: a thread per gate value (their exponentials are most of a step outside the product), backward: per cell
  static constexpr int MUL = (COLS + 31) / 32 * 32;                      // the first warps multiply, those behind do the cell
  static constexpr int CELL = ((NG == 1 ? COLS : JP) * BB + 31) / 32 * 32;
  static constexpr int NT = MUL + CELL;
  static_assert(JP % VEC == 0 && G % DEPTH == 0 && COLS <= MUL && BB * JP <= CELL, "tile");
  static int pitch(int cs) { const int v = cs * JP / VEC; return (v % 2 ? v : v + 1) * VEC; }   // of a column's weights
  static size_t smem(int cs) {
    return 128 + sizeof(T) * ((size_t)COLS * pitch(cs) + 2 * (size_t)cs * BLOCK + 2 * BLOCK + (size_t)BB * COLS * (NG == 1 ? 2 : 1));
  }

  T *u, *buf, *src, *res;
  uint32_t bar;                       // two mbarriers
  int cs, ps, rank, ct;
  bool dead = false;

  __device__ Tile(unsigned char* smem) {
    cs = (int)cluster_size();
    rank = (int)cluster_rank();
    const int v = cs * JP / VEC;
    ps = (v % 2 ? v : v + 1) * VEC;
    bar = saddr(smem);
    u = reinterpret_cast<T*>(smem + 128);
    buf = u + COLS * ps;
    src = buf + 2 * cs * BLOCK;
    res = src + 2 * BLOCK;
    ct = threadIdx.x;
  }
  __device__ void begin() {
    if (threadIdx.x == 0) {
      mbar_init(bar);
      mbar_init(bar + 8);
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int i = threadIdx.x; i < 2 * BLOCK; i += NT) src[i] = (T)0;    // padding stays zero
    cluster_barrier();
  }
  // exchange e (0, 1, ...): everything in src[e & 1] goes to every CTA of the cluster, this one included.  Called by the
  // cell threads after they have written it.
  __device__ void send(int e) {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    cell_sync();
    const uint32_t b = bar + 8 * (e & 1), bytes = BLOCK * sizeof(T);
    const int r = (int)threadIdx.x - MUL;
    if (r == 0) mbar_expect(b, (uint32_t)cs * bytes);
    if (r < cs) push(in_cta(saddr(buf + ((e & 1) * cs + rank) * BLOCK), (uint32_t)r), saddr(src + (e & 1) * BLOCK), bytes, in_cta(b, (uint32_t)r));
  }
  __device__ void cell_sync() { asm volatile("bar.sync 1, %0;" ::"n"(CELL) : "memory"); }
  __device__ void wait(int e, int* err) {
    if (dead) return;
    for (int i = 0; i < WAIT_LIMIT; ++i)
      if (mbar_try(bar + 8 * (e & 1), (uint32_t)(e >> 1) & 1)) return;
    dead = true;
    atomicExch(err, 1);
  }

  // res[row][column] = sum over k ascending of (exchanged row) * (weight column)
  __device__ void multiply(int e) {
    if (ct >= COLS) return;
    int row0, col0;
    if (BB == 4) {
      const int q = ct % (2 * JP);
      row0 = ct / (2 * JP) * 2;
      col0 = q / (JP / 2) * JP + q % (JP / 2);
    } else {
      row0 = 0;
      col0 = ct;
    }
    const int gate = NG == 1 ? 0 : col0 / JP;
    const T* ap = buf + (e & 1) * cs * BLOCK + (gate * BB + row0) * JP;
    const T* up = u + col0 * ps;
    constexpr int CSTEP = JP / 2;      // a thread's second column is of the same gate
    // DEPTH - 1 groups of k are on their way from shared memory while one is multiplied (a group is 16 cycles of double
    // arithmetic, half of what a load takes), and the products of the next k are formed before the sums of this one.  What
    // is read behind the last block is memory that is there and never used.
    T acc[TR][TC], pr[TR][TC];
    alignas(16) T a[DEPTH][TR][VEC], b[DEPTH][TC][VEC];
#pragma unroll
    for (int g = 0; g < DEPTH - 1; ++g) {
#pragma unroll
      for (int i = 0; i < TR; ++i) lds16(ap + g * VEC + i * JP, a[g][i]);
#pragma unroll
      for (int j = 0; j < TC; ++j) lds16(up + g * VEC + j * CSTEP * ps, b[g][j]);
    }
#pragma unroll
    for (int i = 0; i < TR; ++i)
#pragma unroll
      for (int j = 0; j < TC; ++j) {
        acc[i][j] = (T)0;
        pr[i][j] = mul_rn(a[0][i][0], b[0][j][0]);
      }
    for (int p = 0; p < cs; ++p) {
#pragma unroll
      for (int g = 0; g < G; ++g) {
        constexpr int D1 = DEPTH - 1;
        const T* an = g + D1 < G ? ap + (g + D1) * VEC : ap + BLOCK + (g + D1 - G) * VEC;
#pragma unroll
        for (int i = 0; i < TR; ++i) lds16(an + i * JP, a[(g + D1) % DEPTH][i]);
#pragma unroll
        for (int j = 0; j < TC; ++j) lds16(up + (g + D1) * VEC + j * CSTEP * ps, b[(g + D1) % DEPTH][j]);
        const int h = g % DEPTH, h1 = (g + 1) % DEPTH;
#pragma unroll
        for (int kk = 0; kk < VEC; ++kk) {
          T pn[TR][TC];
#pragma unroll
          for (int i = 0; i < TR; ++i)
#pragma unroll
            for (int j = 0; j < TC; ++j)
              pn[i][j] = kk + 1 < VEC ? mul_rn(a[h][i][kk + 1], b[h][j][kk + 1]) : mul_rn(a[h1][i][0], b[h1][j][0]);
#pragma unroll
          for (int i = 0; i < TR; ++i)
#pragma unroll
            for (int j = 0; j < TC; ++j) {
              acc[i][j] = add_rn(acc[i][j], pr[i][j]);
              pr[i][j] = pn[i][j];
            }
        }
      }
      ap += BLOCK;
      up += JP;
    }
#pragma unroll
    for (int i = 0; i < TR; ++i)
#pragma unroll
      for (int j = 0; j < TC; ++j) res[(row0 + i) * COLS + col0 + j * CSTEP] = acc[i][j];
  }
};

template <typename T> struct ForwardArgs {
  int steps, batch, nh, jj;
  const T* U;            // four nh x nh matrices [gate][unit][k]
  const T* b[4];
  T* pre;                // four (steps * batch) x nh matrices, W x on entry, the pre-activations on exit
  T* gate[4];
  T *C, *tanhC, *H, *Hprev, *FC, *IG;
  int* err;
};

template <typename T, int JP, int BB>
__global__ void __launch_bounds__(Tile<T, JP, BB, 1>::NT)
forward_kernel(const __grid_constant__ ForwardArgs<T> p) {
  using L = Tile<T, JP, BB, 1>;
  extern __shared__ __align__(128) unsigned char lstm_smem[];
  L s(lstm_smem);
  const int nh = p.nh;
  const int64_t plane = (int64_t)p.steps * p.batch * nh;
  const int kp = s.cs * JP;
  for (int i = threadIdx.x; i < L::COLS * kp; i += L::NT) {     // this CTA's rows of U_g
    const int c = i / kp, k = i % kp, q = k % JP, unit = s.rank * p.jj + c % JP, kg = k / JP * p.jj + q;
    T v = (T)0;
    if (c % JP < p.jj && unit < nh && q < p.jj && kg < nh) v = p.U[((int64_t)(c / JP) * nh + unit) * nh + kg];
    s.u[c * s.ps + k] = v;
  }
  s.begin();
  const int q = (int)threadIdx.x - L::MUL;
  const bool cell_thread = q >= 0;
  // as a gate thread: row q / COLS, column q % COLS
  const int grow = q / L::COLS, gcol = q % L::COLS, gate = gcol / JP, gunit = s.rank * p.jj + gcol % JP;
  const int tile0 = (int)(blockIdx.x / s.cs) * BB;
  const bool gate_on = cell_thread && grow < BB && gcol % JP < p.jj && gunit < nh && tile0 + grow < p.batch;
  // as a cell thread: row q / JP, hidden unit q % JP
  const int row = q / JP, jl = q % JP, unit = s.rank * p.jj + jl;
  const bool cell = cell_thread && row < BB && jl < p.jj && unit < nh && tile0 + row < p.batch;
  const T bias = gate_on ? p.b[gate][gunit] : (T)0;
  T* gates = s.res + BB * L::COLS;
  T c_prev = (T)0;

  for (int t = 0; t < p.steps; ++t) {
    const int64_t gat = ((int64_t)t * p.batch + tile0 + grow) * nh + gunit;
    T pre = gate_on ? p.pre[gate * plane + gat] : (T)0;
    if (t > 0 && !cell_thread) {
      s.wait(t - 1, p.err);
      s.multiply(t - 1);
    }
    __syncthreads();
    if (gate_on) {
      if (t > 0) pre = add_rn(pre, s.res[grow * L::COLS + gcol]);
      pre = add_rn(pre, bias);
      p.pre[gate * plane + gat] = pre;
      const T v = act_value<T>(gate == 2 ? PRAD_ACT_TANH : PRAD_ACT_SIGMOID, pre, (T)0);      // i, f, g, o
      gates[grow * L::COLS + gcol] = v;
      p.gate[gate][gat] = v;
    }
    if (cell_thread) s.cell_sync();
    if (cell) {
      const int64_t at = ((int64_t)t * p.batch + tile0 + row) * nh + unit;
      const T* v = gates + row * L::COLS + jl;
      const T ig = mul_rn(v[0], v[2 * JP]), fc = t > 0 ? mul_rn(v[JP], c_prev) : (T)0;
      const T c = add_rn(fc, ig), tc = act_value<T>(PRAD_ACT_TANH, c, (T)0), h = mul_rn(v[3 * JP], tc);
      c_prev = c;
      s.src[(t & 1) * L::BLOCK + row * JP + jl] = h;
      p.IG[at] = ig;
      p.FC[at] = fc;
      p.C[at] = c;
      p.tanhC[at] = tc;
      p.H[at] = h;
      if (t == 0) p.Hprev[at] = (T)0;
      if (t + 1 < p.steps) p.Hprev[at + (int64_t)p.batch * nh] = h;
    }
    if (cell_thread && t + 1 < p.steps) s.send(t);
  }
  cluster_barrier();        // nobody leaves while a neighbour may still write here
}

template <typename T> struct BackwardArgs {
  int steps, batch, nh, jj;
  const T* U;
  const T *H, *Y, *tanhC, *C;
  const T* gate[4];
  T loss_scale;
  T* dpre;               // four (steps * batch) x nh matrices
  int* err;
};

template <typename T, int JP, int BB>
__global__ void __launch_bounds__(Tile<T, JP, BB, 4>::NT)
backward_kernel(const __grid_constant__ BackwardArgs<T> p) {
  using L = Tile<T, JP, BB, 4>;
  extern __shared__ __align__(128) unsigned char lstm_smem[];
  L s(lstm_smem);
  const int nh = p.nh;
  const int64_t plane = (int64_t)p.steps * p.batch * nh;
  const int kp = s.cs * JP;
  for (int i = threadIdx.x; i < L::COLS * kp; i += L::NT) {     // this CTA's columns of U_g; neighbouring threads: neighbouring columns
    const int jl = i % JP, k = i / JP % kp, g = i / (JP * kp), q = k % JP, unit = s.rank * p.jj + jl, kg = k / JP * p.jj + q;
    T v = (T)0;
    if (jl < p.jj && unit < nh && q < p.jj && kg < nh) v = p.U[((int64_t)g * nh + kg) * nh + unit];
    s.u[(g * JP + jl) * s.ps + k] = v;
  }
  s.begin();
  const int e = (int)threadIdx.x - L::MUL, row = e / JP, jl = e % JP, unit = s.rank * p.jj + jl;
  const int brow = (int)(blockIdx.x / s.cs) * BB + row;
  const bool cell_thread = e >= 0, cell = cell_thread && row < BB && jl < p.jj && unit < nh && brow < p.batch;
  T dc_next = (T)0;

  for (int t = p.steps - 1; t >= 0; --t) {
    const int x = p.steps - 1 - t;                            // exchanges so far
    const int64_t at = ((int64_t)t * p.batch + brow) * nh + unit;
    T h, y, gi, gf, gg, go, tc, c_prev = (T)0;
    if (cell) {
      h = p.H[at]; y = p.Y[at];
      gi = p.gate[0][at]; gf = p.gate[1][at]; gg = p.gate[2][at]; go = p.gate[3][at];
      tc = p.tanhC[at];
      if (t > 0) c_prev = p.C[at - (int64_t)p.batch * nh];
    }
    if (x > 0 && !cell_thread) {
      s.wait(x - 1, p.err);
      s.multiply(x - 1);
    }
    __syncthreads();
    if (cell) {
      // the chain of lstm_cell_backward_kernel: loss gradient plus the four recurrent gradients in gate order, ...
      T dh = mul_rn(p.loss_scale, sub_rn(h, y));
      if (x > 0)
#pragma unroll
        for (int g = 0; g < 4; ++g) dh = add_rn(dh, s.res[row * L::COLS + g * JP + jl]);
      const T d_o = mul_rn(dh, tc), d_tc = mul_rn(dh, go);
      const T dc_a = mul_rn(d_tc, sub_rn((T)1, mul_rn(tc, tc)));
      const T dc = x > 0 ? add_rn(dc_a, dc_next) : dc_a;
      const T d_i = mul_rn(dc, gg), d_g = mul_rn(dc, gi), d_f = t > 0 ? mul_rn(dc, c_prev) : (T)0;
      dc_next = mul_rn(dc, gf);
      T d[4];
      d[0] = mul_rn(d_i, mul_rn(gi, sub_rn((T)1, gi)));
      d[1] = mul_rn(d_f, mul_rn(gf, sub_rn((T)1, gf)));
      d[2] = mul_rn(d_g, sub_rn((T)1, mul_rn(gg, gg)));
      d[3] = mul_rn(d_o, mul_rn(go, sub_rn((T)1, go)));
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        s.src[(x & 1) * L::BLOCK + (g * BB + row) * JP + jl] = d[g];
        p.dpre[g * plane + at] = d[g];
      }
    }
    if (cell_thread && t > 0) s.send(x);
  }
  cluster_barrier();
}

// ---- host side: which tile, launch --------------------------------------------------------------------------
// Padded hidden units per CTA (8, 12 or 16; float 8 or 16: two 16-byte groups at a time) and CTAs per cluster (a power of
// two, at most 16 -- above 8 needs the device's consent): as few padded k as the clusters allow, and on a tie the smaller
// CTAs, i.e. the larger cluster.  Up to 256 hidden units.  (That tie is not measured: 56 float units run on eight CTAs, 1.9 us per
// step, where their weights would fit one.)
struct Plan { int jp = 0, cs = 0, jj = 0; };
template <typename T> static Plan plan_of(int nh) {
  Plan best;
  int best_k = 0;
  for (int jp : {8, 12, 16}) {
    if (sizeof(T) == 4 && jp == 12) continue;
    for (int cs = 1; cs <= 16; cs *= 2) {
      if (cs * jp < nh) continue;
      if (!best.jp || cs * jp < best_k) { best.jp = jp; best.cs = cs; best.jj = (int)ceil_div(nh, cs); best_k = cs * jp; }
      break;
    }
  }
  return best;
}

// Clusters of this kernel that fit the device at once; 0 if none does.  Asked once per kernel, cluster size and device.  (A kernel
// serves several cluster sizes, and what it may use of shared memory is a property of the kernel: the most there is, for all.)
constexpr int MOST_SMEM = 227 * 1024;
template <auto Kernel> static int clusters_at_once(prad_ctx* ctx, int cs, int nt, size_t smem) {
  static std::atomic<int> known[64][5];
  int lg = 0;
  while ((1 << lg) < cs) ++lg;
  std::atomic<int>& k = known[ctx->device & 63][lg];
  int n = k.load(std::memory_order_acquire);
  if (n) return n - 1;
  n = 0;
  cudaError_t e = cudaFuncSetAttribute(Kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, MOST_SMEM);
  if (e == cudaSuccess && cs > 8) e = cudaFuncSetAttribute(Kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e == cudaSuccess) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = cs;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3((unsigned)cs);
    cfg.blockDim = dim3((unsigned)nt);
    cfg.dynamicSmemBytes = smem;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    e = cudaOccupancyMaxActiveClusters(&n, Kernel, &cfg);
  }
  if (e != cudaSuccess) { (void)cudaGetLastError(); n = 0; }
  k.store(n + 1, std::memory_order_release);
  return n;
}

template <auto Kernel, typename Args>
static prad_status launch(prad_ctx* ctx, int cs, int nt, size_t smem, int tiles, const Args& args) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = cs;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3((unsigned)(cs * tiles));
  cfg.blockDim = dim3((unsigned)nt);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = ctx->stream;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  PRAD_CUDA(cudaLaunchKernelEx(&cfg, Kernel, args));
  PRAD_LAUNCHED(ctx);
  ctx->tc_pending_check = true;
  return PRAD_OK;
}

// The batch tile.  A step takes a cluster little longer for four rows than for one (double, 256 units: 3.5 .. 5.7 us), and a
// B200 runs 7 clusters of 16 at once, 15 of 8: so the smallest tile with which all clusters run at once, or else the tile with the
// fewest turns.  Tiles have 1, 2, 4 or 5 rows (five serve 35 rows at once on those 7 clusters; three run as four, which a step
// hardly feels; more than five are not instantiated).  PRAD_ERR_UNSUPPORTED: more turns than one launch per operation is worth, or
// too many hidden units for a cluster's shared memory.
constexpr int MAX_TURNS = 8;
template <typename T, bool FORWARD, int JP, typename Args>
static prad_status run_jp(prad_ctx* ctx, const Plan& pl, Args& a) {
  constexpr int NG = FORWARD ? 1 : 4;
  const int B = a.batch;
  a.jj = pl.jj;
  int rows = 0, turns = 0;
#define PRAD_LSTM_TILE(BB_, DO)                                                                                        \
  do {                                                                                                                 \
    constexpr auto K = [] {                                                                                            \
      if constexpr (FORWARD) return &forward_kernel<T, JP, BB_>;                                                       \
      else return &backward_kernel<T, JP, BB_>;                                                                        \
    }();                                                                                                               \
    using L = Tile<T, JP, BB_, NG>;                                                                                    \
    const size_t smem = L::smem(pl.cs);                                                                                \
    const int tiles = (int)ceil_div(B, BB_);                                                                           \
    DO;                                                                                                                \
  } while (0)
#define PRAD_LSTM_WEIGH(BB_)                                                                                           \
  PRAD_LSTM_TILE(BB_, {                                                                                                \
    const int fit = smem <= MOST_SMEM ? clusters_at_once<K>(ctx, pl.cs, L::NT, smem) : 0;                             \
    const int n = fit > 0 ? (int)ceil_div(tiles, fit) : 0;                                                             \
    if (n && (!turns || n < turns)) { turns = n; rows = BB_; }                                                         \
  })
#define PRAD_LSTM_RUN(BB_) \
  PRAD_LSTM_TILE(BB_, if (rows == BB_) return launch<K>(ctx, pl.cs, L::NT, smem, tiles, a))
  PRAD_LSTM_WEIGH(1);
  PRAD_LSTM_WEIGH(2);
  PRAD_LSTM_WEIGH(4);
  PRAD_LSTM_WEIGH(5);
  if (!turns || turns > MAX_TURNS) return PRAD_ERR_UNSUPPORTED;
  PRAD_LSTM_RUN(1);
  PRAD_LSTM_RUN(2);
  PRAD_LSTM_RUN(4);
  PRAD_LSTM_RUN(5);
#undef PRAD_LSTM_RUN
#undef PRAD_LSTM_WEIGH
#undef PRAD_LSTM_TILE
  return PRAD_ERR_UNSUPPORTED;
}

template <typename T, bool FORWARD, typename Args> static prad_status run(prad_ctx* ctx, Args& a) {
  const Plan pl = plan_of<T>(a.nh);
  if (pl.jp == 8) return run_jp<T, FORWARD, 8>(ctx, pl, a);
  if (pl.jp == 16) return run_jp<T, FORWARD, 16>(ctx, pl, a);
  if constexpr (sizeof(T) == 8)
    if (pl.jp == 12) return run_jp<T, FORWARD, 12>(ctx, pl, a);
  return PRAD_ERR_UNSUPPORTED;
}

}  // namespace lstm

#define L_TRY(call)                \
  do {                             \
    prad_status s_ = (call);       \
    if (s_ != PRAD_OK) return s_;  \
  } while (0)

template <typename T>
static prad_status lstm_forward_t(prad_ctx* ctx, prad_dtype dt, int steps, int batch, int nh, const void* U, const void* const* b,
                                  void* pre, void* const* gate, void* C, void* tanhC, void* H, void* Hprev, void* FC, void* IG) {
  lstm::ForwardArgs<T> a;
  a.steps = steps; a.batch = batch; a.nh = nh; a.jj = 0;
  a.U = (const T*)U;
  for (int g = 0; g < 4; ++g) { a.b[g] = (const T*)b[g]; a.gate[g] = (T*)gate[g]; }
  a.pre = (T*)pre;
  a.C = (T*)C; a.tanhC = (T*)tanhC; a.H = (T*)H; a.Hprev = (T*)Hprev; a.FC = (T*)FC; a.IG = (T*)IG;
  a.err = ctx->tc_err;
  const prad_status st = lstm::run<T, true>(ctx, a);
  if (st != PRAD_ERR_UNSUPPORTED) return st;
  // more hidden units than a cluster holds: one launch per operation
  const int64_t plane = (int64_t)steps * batch * nh, n = (int64_t)batch * nh;
  const prad_act act[4] = {PRAD_ACT_SIGMOID, PRAD_ACT_SIGMOID, PRAD_ACT_TANH, PRAD_ACT_SIGMOID};
  L_TRY(prad_zero(ctx, Hprev, (size_t)n * sizeof(T)));
  for (int t = 0; t < steps; ++t) {
    auto step = [&](void* m) { return (T*)m + t * n; };
    if (t > 0) {
      GemmEpilogue e;
      L_TRY(gemm_dispatch(ctx, dt, false, true, batch, nh, nh, 1.0, step(Hprev), nh, U, nh, 1.0, step(pre), nh, 4, 0,
                          (int64_t)nh * nh, plane, e));
    }
    for (int g = 0; g < 4; ++g) {
      T* p = step(pre) + g * plane;
      L_TRY(prad_add_broadcast_forward(ctx, dt, p, b[g], p, batch, nh));
      L_TRY(prad_act_forward(ctx, dt, act[g], p, step(gate[g]), n, 0.0));
    }
    L_TRY(prad_hadamard_forward(ctx, dt, step(gate[0]), step(gate[2]), step(IG), n));
    if (t > 0) L_TRY(prad_hadamard_forward(ctx, dt, step(gate[1]), step(C) - n, step(FC), n));
    else L_TRY(prad_zero(ctx, FC, (size_t)n * sizeof(T)));
    L_TRY(prad_add_forward(ctx, dt, step(FC), step(IG), nullptr, step(C), n));
    L_TRY(prad_act_forward(ctx, dt, PRAD_ACT_TANH, step(C), step(tanhC), n, 0.0));
    L_TRY(prad_hadamard_forward(ctx, dt, step(gate[3]), step(tanhC), step(H), n));
    if (t + 1 < steps) L_TRY(prad_copy(ctx, step(Hprev) + n, step(H), (size_t)n * sizeof(T)));
  }
  return PRAD_OK;
}

template <typename T>
static prad_status lstm_backward_t(prad_ctx* ctx, prad_dtype dt, int steps, int batch, int nh, const void* U, const void* H,
                                   const void* Y, double loss_scale, const void* const* gate, const void* tanhC, const void* C,
                                   void* dpre, void* scratch) {
  lstm::BackwardArgs<T> a;
  a.steps = steps; a.batch = batch; a.nh = nh; a.jj = 0;
  a.U = (const T*)U;
  a.H = (const T*)H; a.Y = (const T*)Y; a.tanhC = (const T*)tanhC; a.C = (const T*)C;
  for (int g = 0; g < 4; ++g) a.gate[g] = (const T*)gate[g];
  a.loss_scale = (T)loss_scale;
  a.dpre = (T*)dpre;
  a.err = ctx->tc_err;
  const prad_status st = lstm::run<T, false>(ctx, a);
  if (st != PRAD_ERR_UNSUPPORTED) return st;
  const int64_t plane = (int64_t)steps * batch * nh, n = (int64_t)batch * nh;
  T* rec = (T*)scratch;              // four recurrent gradients, then two buffers of dc (.) f in turn
  const void* contrib[4] = {rec, rec + n, rec + 2 * n, rec + 3 * n};
  const void* dc_next = nullptr;
  for (int t = steps - 1; t >= 0; --t) {
    auto at = [&](const void* m) { return (const void*)((const T*)m + t * n); };
    const void* g[4] = {at(gate[0]), at(gate[1]), at(gate[2]), at(gate[3])};
    T* d = (T*)dpre + t * n;
    void* dp[4] = {d, d + plane, d + 2 * plane, d + 3 * plane};
    void* dc_prev = t > 0 ? (void*)(rec + (4 + (t & 1)) * n) : nullptr;
    L_TRY(prad_lstm_cell_backward(ctx, dt, n, at(H), at(Y), loss_scale, contrib, t + 1 < steps ? 4 : 0, dc_next, g, at(tanhC),
                                  t > 0 ? (const void*)((const T*)C + (t - 1) * n) : nullptr, dp, dc_prev));
    dc_next = dc_prev;
    if (t > 0) {
      GemmEpilogue e;
      L_TRY(gemm_dispatch(ctx, dt, false, false, batch, nh, nh, 1.0, d, nh, U, nh, 0.0, rec, nh, 4, plane, (int64_t)nh * nh, n, e));
    }
  }
  return PRAD_OK;
}

}  // namespace prad

using namespace prad;

static prad_status check_lists4(const char* who, const void* const* list) {
  PRAD_REQUIRE(list && list[0] && list[1] && list[2] && list[3], PRAD_ERR_INVALID, "%s: a gate's pointer is null", who);
  return PRAD_OK;
}

extern "C" prad_status prad_lstm_forward(prad_ctx* ctx, prad_dtype dt, int steps, int batch, int hidden, const void* U,
                                         const void* const* bias_ifgo_host, void* pre, void* const* gates_ifgo_host, void* C,
                                         void* tanh_c, void* H, void* H_prev, void* FC, void* IG) {
  PRAD_CHECK_CTX(ctx);
  PRAD_REQUIRE(dtype_ok(dt) && steps >= 0 && batch >= 0 && hidden >= 0, PRAD_ERR_INVALID, "prad_lstm_forward: bad dtype or size");
  if (steps == 0 || batch == 0 || hidden == 0) return PRAD_OK;
  PRAD_REQUIRE(U && pre && C && tanh_c && H && H_prev && FC && IG, PRAD_ERR_INVALID, "prad_lstm_forward: null pointer");
  L_TRY(check_lists4("prad_lstm_forward", bias_ifgo_host));
  L_TRY(check_lists4("prad_lstm_forward", gates_ifgo_host));
  return dt == PRAD_F32
             ? lstm_forward_t<float>(ctx, dt, steps, batch, hidden, U, bias_ifgo_host, pre, gates_ifgo_host, C, tanh_c, H, H_prev, FC, IG)
             : lstm_forward_t<double>(ctx, dt, steps, batch, hidden, U, bias_ifgo_host, pre, gates_ifgo_host, C, tanh_c, H, H_prev, FC, IG);
}

extern "C" prad_status prad_lstm_backward(prad_ctx* ctx, prad_dtype dt, int steps, int batch, int hidden, const void* U,
                                          const void* H, const void* target, double loss_scale, const void* const* gates_ifgo_host,
                                          const void* tanh_c, const void* C, void* dpre, void* scratch) {
  PRAD_CHECK_CTX(ctx);
  PRAD_REQUIRE(dtype_ok(dt) && steps >= 0 && batch >= 0 && hidden >= 0, PRAD_ERR_INVALID, "prad_lstm_backward: bad dtype or size");
  if (steps == 0 || batch == 0 || hidden == 0) return PRAD_OK;
  PRAD_REQUIRE(U && H && target && tanh_c && C && dpre && scratch, PRAD_ERR_INVALID, "prad_lstm_backward: null pointer");
  L_TRY(check_lists4("prad_lstm_backward", gates_ifgo_host));
  return dt == PRAD_F32 ? lstm_backward_t<float>(ctx, dt, steps, batch, hidden, U, H, target, loss_scale, gates_ifgo_host, tanh_c, C, dpre, scratch)
                        : lstm_backward_t<double>(ctx, dt, steps, batch, hidden, U, H, target, loss_scale, gates_ifgo_host, tanh_c, C, dpre, scratch);
}

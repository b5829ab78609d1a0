// FP64 GEMM on the tensor cores (DMMA): C = alpha*op(A)*op(B) + beta*C with
// mma.sync.aligned.m8n8k4.row.col.f64 tiles.  tcgen05.mma has no FP64 kind, so double
// precision stays on the warp-level MMA path.
//
// What bounds it: an m8n8k4 takes a scheduler's tensor pipe 16 cycles (37 TFLOP/s with every SM full), so the pipe is easy to
// feed -- a 32 x 32 warp tile reads 8 fragments per 16 MMAs -- as long as the feeding is off its path.  A CTA owns a 64 x 64
// tile: four warps multiply (32 x 32 each, 32 accumulators per thread), two copy (cp.async, four stages of 16 k), and two
// such CTAs share an SM, so one's tile store and first loads hide behind the other's MMAs and the last wave is counted in
// 64 x 64 tiles.  The output leaves through shared memory: one copy of the epilogue code, whole rows.
// 2048 x 1000 over k = 1536 (NN) 233 us, its backward pair (NT, TN) in one launch 421 us; before, 128 x 128 tiles with one CTA
// per SM or 64 x 64 tiles staged through registers took 346 us and 430 + 292 us.  4096^3: 33.4 TFLOP/s (26.7 before), 0.90 of
// the pipe; 2048 x 1024 over k = 128: 28 us (52).
//
// The summation order inside a DMMA differs from the managed code's sequential loop, so this variant is held to the
// tolerance, not to bit equality; "auto" uses it only for large products and keeps the bit-exact kernel for everything else.
#include "gemm_simt.cuh"

namespace prad {
namespace dm {

constexpr int BM = 64, BN = 64, BK = 16, STAGES = 4, NT = 128, NC = 64, THREADS = NT + NC;
// Fragment reads (8 rows x 4 k of doubles) are free of bank conflicts with rows 4 doubles further apart than a multiple of 16.
template <bool KC> using Operand = OperandTile<double, BM, BK, NC, KC, 4>;
constexpr int STAGE = Operand<true>::SIZE > Operand<false>::SIZE ? Operand<true>::SIZE : Operand<false>::SIZE;
constexpr int SMEM = STAGES * 2 * STAGE * (int)sizeof(double);
static_assert(SMEM >= BM * BN * (int)sizeof(double), "the epilogue stages a whole output tile there");

__device__ __forceinline__ void mma(double& d0, double& d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(d0), "+d"(d1) : "d"(a), "d"(b));
}
// fragment element (mn, k) of a tile in either layout
template <bool KC> __device__ __forceinline__ double frag(const double* tile, int mn, int k) {
  return KC ? tile[mn * Operand<true>::PITCH + k] : tile[k * Operand<false>::PITCH + mn];
}

// One product, or `slices` of them: slice s multiplies k in [s k_slice, (s + 1) k_slice) into its own M x N block of C
// (blocks sC apart, the slices of a batch entry one after the other).
struct Problem {
  Product<double> p;
  int slices, k_slice;
};

template <bool TA, bool TB>
__device__ __forceinline__ void tile_of(const Problem& pr, int tile, double* smem) {
  const Product<double>& p = pr.p;
  constexpr bool A_KC = !TA, B_KC = TB;
  const int tid = threadIdx.x;
  const int64_t bz = tile / p.tiles_mn;
  const int t2 = tile % p.tiles_mn;
  const int m0 = t2 / p.tiles_n * BM, n0 = t2 % p.tiles_n * BN;
  const int64_t bat = bz / pr.slices, k0 = (bz - bat * pr.slices) * (int64_t)pr.k_slice;
  const int K = (int)(p.K - k0 < pr.k_slice ? p.K - k0 : pr.k_slice);
  double* As = smem;
  double* Bs = smem + STAGES * STAGE;
  const int ktiles = (K + BK - 1) / BK;
  const int lane = tid & 31, warp = tid >> 5;
  const int wm = (warp >> 1 & 1) * 32, wn = (warp & 1) * 32;
  const int g = lane >> 2, q = lane & 3;

  double acc[4][4][2];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;

  if (tid >= NT) {
    const int ct = tid - NT;
    Operand<A_KC> la;
    Operand<B_KC> lb;
    la.begin(p.A + bat * p.sA + (A_KC ? k0 : k0 * p.lda), p.lda, m0, p.M, p.vecA, ct);
    lb.begin(p.B + bat * p.sB + (B_KC ? k0 : k0 * p.ldb), p.ldb, n0, p.N, p.vecB, ct);
    const bool vecA = p.vecA, vecB = p.vecB;
    int k_left = K;
    auto stage = [&](int s) {
      if (k_left > 0) {
        la.load(As + s * STAGE, k_left, vecA);
        lb.load(Bs + s * STAGE, k_left, vecB);
      }
      k_left -= BK;
      cp_async_commit();
    };
    for (int s = 0; s < STAGES - 1; ++s) stage(s);
    cp_async_wait<STAGES - 2>();
    __syncthreads();
    int nxt = STAGES - 1;
    for (int kt = 0; kt < ktiles; ++kt) {
      stage(nxt);
      cp_async_wait<STAGES - 2>();
      __syncthreads();
      nxt = nxt + 1 == STAGES ? 0 : nxt + 1;
    }
    cp_async_wait<0>();
  } else {
    __syncthreads();
    int cur = 0;
    for (int kt = 0; kt < ktiles; ++kt) {
      const double* as = As + cur * STAGE;
      const double* bs = Bs + cur * STAGE;
      double a[2][4], b[2][4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[0][i] = frag<A_KC>(as, wm + i * 8 + g, q);
#pragma unroll
      for (int j = 0; j < 4; ++j) b[0][j] = frag<B_KC>(bs, wn + j * 8 + g, q);
#pragma unroll
      for (int k4 = 0; k4 < BK / 4; ++k4) {
        const int h = k4 & 1;
        if (k4 + 1 < BK / 4) {
#pragma unroll
          for (int i = 0; i < 4; ++i) a[h ^ 1][i] = frag<A_KC>(as, wm + i * 8 + g, (k4 + 1) * 4 + q);
#pragma unroll
          for (int j = 0; j < 4; ++j) b[h ^ 1][j] = frag<B_KC>(bs, wn + j * 8 + g, (k4 + 1) * 4 + q);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) mma(acc[i][j][0], acc[i][j][1], a[h][i], b[h][j]);
      }
      __syncthreads();
      cur = cur + 1 == STAGES ? 0 : cur + 1;
    }
    // rows wm + i*8 + g, columns wn + j*8 + 2q + {0,1}
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j)
        *reinterpret_cast<double2*>(smem + (wm + i * 8 + g) * BN + wn + j * 8 + 2 * q) = make_double2(acc[i][j][0], acc[i][j][1]);
  }
  __syncthreads();
  const EpiParams<double>& epi = p.epi;
  double* C = p.C + bz * p.sC;
  const double* saved = epi.saved ? epi.saved + bz * p.sC : nullptr;
  double* z_out = epi.z_out ? epi.z_out + bz * p.sC : nullptr;
  const bool plain = p.beta == 0.0 && !epi.bias && !epi.z_out && epi.act == PRAD_ACT_NONE && epi.dact == PRAD_ACT_NONE;
  if (plain && p.vecC && n0 + BN <= p.N) {
    for (int e = tid; e < BM * BN / 2; e += THREADS) {
      const int m = m0 + e / (BN / 2), n = n0 + e % (BN / 2) * 2;
      if (m >= p.M) break;
      double2 v = *reinterpret_cast<const double2*>(smem + 2 * e);
      v.x *= p.alpha;
      v.y *= p.alpha;
      *reinterpret_cast<double2*>(C + (int64_t)m * p.ldc + n) = v;
    }
    return;
  }
#pragma unroll 1
  for (int e = tid; e < BM * BN; e += THREADS) {
    const int m = m0 + e / BN, n = n0 + e % BN;
    if (m >= p.M || n >= p.N) continue;
    const int64_t off = (int64_t)m * p.ldc + n;
    double v = p.alpha * smem[e];
    if (p.beta != 0.0) v = fma(p.beta, C[off], v);
    if (epi.bias) v += epi.bias[n];
    if (z_out) z_out[off] = v;
    if (epi.act != PRAD_ACT_NONE) v = act_value<double>((prad_act)epi.act, v, epi.act_alpha);
    if (epi.dact != PRAD_ACT_NONE) v = mul_rn(v, act_derivative<double>((prad_act)epi.dact, saved[off], epi.act_alpha));
    C[off] = v;
  }
}

template <bool TA, bool TB>
__global__ void __launch_bounds__(THREADS, 2)
gemm_kernel(const __grid_constant__ Problem p) {
  chain_begin();
  extern __shared__ __align__(16) double dmma_smem[];
  tile_of<TA, TB>(p, blockIdx.x, dmma_smem);
}

// dA = dC*B^T and dB = A^T*dC of one Backward (see gemm_simt_backward_kernel)
__global__ void __launch_bounds__(THREADS, 2)
backward_kernel(const __grid_constant__ Problem nt, const __grid_constant__ Problem tn, int tn_first, int first_tiles) {
  chain_begin();
  extern __shared__ __align__(16) double dmma_smem[];
  const bool first = (int)blockIdx.x < first_tiles;
  const int local = first ? blockIdx.x : blockIdx.x - first_tiles;
  if (first == (tn_first != 0)) tile_of<true, false>(tn, local, dmma_smem);
  else tile_of<false, true>(nt, local, dmma_smem);
}

// C = alpha * (P_0 + P_1 + ...) + beta * C, slices added in order; P_s are dense M x N.
__global__ void __launch_bounds__(256)
combine_kernel(const double* __restrict__ part, int splits, int64_t mn, int N, double* __restrict__ C, int64_t ldc, int64_t sC,
               double alpha, double beta) {
  chain_begin();
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  part += (int64_t)blockIdx.y * splits * mn;      // blockIdx.y = batch
  C += (int64_t)blockIdx.y * sC;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < mn; i += stride) {
    double acc = part[i];
    for (int s = 1; s < splits; ++s) acc = __dadd_rn(acc, part[(int64_t)s * mn + i]);
    const int64_t off = (i / N) * ldc + (i % N);
    double v = __dmul_rn(alpha, acc);
    if (beta != 0.0) v = (beta == 1.0) ? __dadd_rn(C[off], v) : fma(beta, C[off], v);
    C[off] = v;
  }
}

// Slices of a k: two CTAs on every SM, slices of at least 128 (256 beyond sixteen, which the ordered pass would feel).
static int slices_of(const prad_ctx* ctx, int64_t tiles, int K) {
  if (tiles * 2 > ctx->sm_count || K < 512) return 1;
  const int most = K / 128 < 16 ? K / 128 : (K / 256 > 16 ? K / 256 : 16);
  const int64_t S = 2 * ctx->sm_count / tiles;
  return (int)(S < most ? S : most);
}
// One launch for both products of a Backward: where the longest tile (and a short one on the same SM, when there are more tiles
// than SMs), or all of them spread over the SMs, takes less than the two products one after the other with their slices.  In
// units of k per SM; a launch's ramp is about 64, the ordered pass 96.  512 x 512 over 512: 41 -> 27 us; 1024 x 512 over 256,
// where one tile of k = 1024 would outlast everything, stays at 37 us in two launches (57 in one).
static bool one_launch(const prad_ctx* ctx, int M, int K, int N) {
  const int64_t tA = ceil_div(M, BM) * ceil_div(K, BN), tB = ceil_div(K, BM) * ceil_div(N, BN);
  const int64_t both = (tA * N + tB * M) / ctx->sm_count, lo = N < M ? N : M, hi = N < M ? M : N;
  const int64_t chain = hi + (tA + tB > ctx->sm_count ? lo : 0);
  auto alone = [&](int64_t tiles, int k) {
    const int S = slices_of(ctx, tiles, k);
    return ceil_div(k, S) * ceil_div(tiles * S, ctx->sm_count) + (S > 1 ? 96 : 0);
  };
  return (both > chain ? both : chain) <= alone(tA, N) + alone(tB, M) + 64;
}

static prad_status set_problem(Problem& pr, const Product<double>& p, int batch, int64_t* tiles) {
  pr.p = p;
  pr.slices = 1;
  pr.k_slice = p.K;
  pr.p.tiles_n = (int)ceil_div(p.N, BN);
  const int64_t mn = ceil_div(p.M, BM) * pr.p.tiles_n;
  *tiles = mn * batch;
  PRAD_REQUIRE(*tiles <= 0x3fffffff, PRAD_ERR_UNSUPPORTED, "gemm dmma: too many tiles for one launch");
  pr.p.tiles_mn = (int)mn;
  return PRAD_OK;
}

static prad_status launch(prad_ctx* ctx, bool tA, bool tB, const Problem& pr, int64_t tiles) {
  prad_status st;
#define PRAD_DMMA(TA_, TB_)                                                                        \
  do {                                                                                             \
    if ((st = allow_smem<gemm_kernel<TA_, TB_>>(ctx, SMEM))) return st;                            \
    launch_chained(gemm_kernel<TA_, TB_>, (unsigned)tiles, THREADS, SMEM, ctx->stream, pr);                    \
  } while (0)
  if (!tA && !tB) PRAD_DMMA(false, false);
  else if (!tA && tB) PRAD_DMMA(false, true);
  else if (tA && !tB) PRAD_DMMA(true, false);
  else PRAD_DMMA(true, true);
#undef PRAD_DMMA
  PRAD_LAUNCHED(ctx);
  return PRAD_OK;
}

}  // namespace dm

prad_status gemm_f64_dmma(prad_ctx* ctx, bool tA, bool tB, int M, int N, int K, double alpha,
                          const void* A, int lda, const void* B, int ldb, double beta, void* C,
                          int ldc, int batch, int64_t sA, int64_t sB, int64_t sC,
                          const GemmEpilogue& e, bool probe_only) {
  const bool forced = ctx->gemm_f64 == GemmF64::Dmma;
  const bool big = (int64_t)M * N * K * batch >= ((int64_t)1 << 27) && M >= 32 && N >= 32;
  if (!(forced || big) || K < 1) return PRAD_ERR_UNSUPPORTED;
  if (probe_only) return PRAD_OK;
  dm::Problem pr;
  int64_t tiles = 0;
  prad_status st = dm::set_problem(pr, make_product<double>(M, N, K, alpha, A, lda, B, ldb, beta, C, ldc, sA, sB, sC, e), batch, &tiles);
  if (st) return st;
  // Few output tiles and a long k (the time-batched weight gradients of an LSTM: 256 x 128 outputs over k = 2048 in a batch of
  // four are 32 tiles): k is cut into slices that run as further tiles into scratch, and an ordered pass adds them.
  const bool plain = !e.bias && !e.z_out && e.act == PRAD_ACT_NONE && e.dact == PRAD_ACT_NONE;
  // The sum over a batch (sC = 0) is that with the batch entries as further slices.
  const bool sum = batch > 1 && sC == 0;
  if (int S = plain ? dm::slices_of(ctx, tiles, K) : 1; S > 1 || (plain && sum)) {
    const int k_slice = (int)(ceil_div(ceil_div(K, S), dm::BK) * dm::BK);
    S = (int)ceil_div(K, k_slice);
    if (S > 1 || sum) {
      const int64_t mn = (int64_t)M * N;
      st = ensure_parts(ctx, (size_t)batch * S * mn * sizeof(double));
      if (st) return sum ? PRAD_ERR_UNSUPPORTED : st;     // (a sum also goes product by product)
      double* part = (double*)ctx->parts;
      pr.slices = S;
      pr.k_slice = k_slice;
      pr.p.alpha = 1.0;
      pr.p.beta = 0.0;
      pr.p.C = part;
      pr.p.ldc = N;
      pr.p.sC = mn;
      pr.p.vecC = N % 2 == 0 && mn % 2 == 0;
      if ((st = dm::launch(ctx, tA, tB, pr, tiles * S))) return st;
      const int cg = stream_grid(ctx, mn, 256, 8);
      launch_chained(dm::combine_kernel, dim3((unsigned)cg, sum ? 1u : (unsigned)batch), 256, 0, ctx->stream, part, sum ? S * batch : S, mn, N, (double*)C, ldc, sC, alpha, beta);
      PRAD_LAUNCHED(ctx);
      return PRAD_OK;
    }
  }
  return dm::launch(ctx, tA, tB, pr, tiles);
}

bool gemm_f64_dmma_one_launch(prad_ctx* ctx, int M, int K, int N) { return dm::one_launch(ctx, M, K, N); }

// dA (M x K) = dC (M x N) * B^T (.) act'(saved)  and  dB (K x N) = scale * A^T * dC [+ dB] of a product both of whose
// gradients belong on the tensor cores, in one launch
prad_status gemm_f64_dmma_backward(prad_ctx* ctx, const void* A, const void* B, const void* dC, void* dA, void* dB, int M, int K, int N,
                                   bool accumulate_dB, double dB_scale, const GemmEpilogue& e_dA) {
  dm::Problem nt, tn;
  int64_t n_nt = 0, n_tn = 0;
  prad_status st = dm::set_problem(nt, make_product<double>(M, K, N, 1.0, dC, N, B, N, 0.0, dA, K, 0, 0, 0, e_dA), 1, &n_nt);
  if (!st)
    st = dm::set_problem(tn, make_product<double>(K, N, M, dB_scale, A, K, dC, N, accumulate_dB ? 1.0 : 0.0, dB, N, 0, 0, 0, GemmEpilogue()),
                         1, &n_tn);
  if (!st) st = allow_smem<dm::backward_kernel>(ctx, dm::SMEM);
  if (st) return st;
  const int tn_first = tn.p.K >= nt.p.K;      // the longer tiles start first
  launch_chained(dm::backward_kernel, (unsigned)(n_nt + n_tn), dm::THREADS, dm::SMEM, ctx->stream, nt, tn, tn_first, (int)(tn_first ? n_tn : n_nt));
  PRAD_LAUNCHED(ctx);
  return PRAD_OK;
}

}  // namespace prad

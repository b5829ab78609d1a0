// SIMT GEMM family (FP32 FMA / FP64 DFMA): C = alpha*op(A)*op(B) + beta*C, row-major,
// any M/N/K, strided-batched, with the fused epilogues of the backward path.
//
// This is the always-available variant: every product in the storage precision, k ascending,
// either with separately rounded multiply and add (EXACT: bit-identical to the managed
// code's sequential `+=` loop, the default) or with FMA accumulation (twice the rate), for
// all transpose forms the backward needs
//   NN  C = A*B          MatrixMultiplyOperation.Forward   (MatrixMultiplyOperation.cs:50-80)
//   NT  dA = dC*B^T      MatrixMultiplyOperation.Backward  (:94-104)
//   TN  dB = A^T*dC      MatrixMultiplyOperation.Backward  (:110-120)
//
// What bounds it: one output is one chain of K dependent additions (4 cycles each in float, 8 in double), a multiply-add
// is two instructions (35.5 TFLOP/s float, 18.4 TFLOP/s double with every SM full), and a thread's fragments come out of
// shared memory at 128 bytes per cycle and SM: with TM x TN outputs per thread a tile needs (TM + TN) / (TM TN) values per
// multiply-add.  Products below 2^27 multiply-adds leave an SM one or two small tiles, a warp its scheduler to itself, so
// nothing may ever wait for something that could have been started before:
//  - k advances through a ring of shared-memory stages filled with cp.async by warps of their own (the address
//    arithmetic of the copies took the multiplying warps 8 of 26 cycles per k);
//  - the fragments of the next 16 bytes of k are read while these are multiplied;
//  - the products of the next k are formed before the sums of this one (26 -> 16 cycles per k in float, 49 -> 25 in double
//    for a 16 x 16 tile).
// 256 x 512 over k = 784: float 47 -> 14.5 us, double (as 512 x 256) 39 -> 21 us, against one register-staged tile ahead.
//
// Each operand keeps the orientation it has in global memory -- [row][k] when k is contiguous, [k][row] when the row index
// is -- because a copy cannot transpose.  A thread reads its fragments as 128-bit vectors along whichever is contiguous:
// rows of a [row][k] tile are one 16-byte slot further apart than they need to be, so the rows of neighbouring threads
// fall into different banks.
#pragma once

#include "gemm_tiles.cuh"

namespace prad {

__device__ __forceinline__ void cp_async16(void* dst, const void* src, int src_bytes) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(src_bytes) : "memory");
}
template <int BYTES> __device__ __forceinline__ void cp_async_one(void* dst, const void* src, int src_bytes) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(d), "l"(src), "n"(BYTES), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// One operand's ROWS x BK tile in shared memory.  KC: k is contiguous in memory, layout [row][k]; otherwise [k][row].
template <typename T, int ROWS, int BK, int NT, bool KC, int PAD = 16 / sizeof(T)>
struct OperandTile {
  static constexpr int VEC = 16 / sizeof(T);
  static constexpr int PITCH = (KC ? BK : ROWS) + PAD;
  static constexpr int FAST = KC ? BK : ROWS, SLOW = KC ? ROWS : BK;
  static constexpr int SIZE = SLOW * PITCH;

  // A thread's part of the copies: chunks of VEC elements (or single elements where a row does not start at a 16-byte
  // boundary) STEP rows of memory apart.  The source pointer moves on by one stage with every load.
  const T* base;      // somewhere readable, for copies of nothing
  const T* src;
  int64_t ld, advance;
  int s, f, limit;    // slow and fast index inside the tile; limit of the index that is not k
  __device__ __forceinline__ void begin(const T* __restrict__ p, int64_t ld_, int row0, int X, bool vec, int tid) {
    const int per_row = vec ? FAST / VEC : FAST;
    s = tid / per_row;
    f = tid % per_row * (vec ? VEC : 1);
    ld = ld_;
    base = p;
    src = p + (KC ? (int64_t)(row0 + s) * ld + f : (int64_t)s * ld + row0 + f);
    advance = KC ? BK : (int64_t)BK * ld;
    limit = KC ? X - row0 : X - row0 - f;
  }
  // copies the tile at k0 and moves on; elements outside the matrix become zero
  __device__ __forceinline__ void load(T* tile, int k_left, bool vec) {      // k_left = K - k0
    T* dst = tile + s * PITCH + f;
    if (vec) {
      constexpr int STEP = NT / (FAST / VEC);
      static_assert(NT % (FAST / VEC) == 0, "threads of a copy");
#pragma unroll
      for (int it = 0; it < (SLOW + STEP - 1) / STEP; ++it) {
        if (SLOW % STEP != 0 && s + it * STEP >= SLOW) break;
        const bool row_ok = s + it * STEP < (KC ? limit : k_left);
        int left = KC ? k_left - f : limit;
        left = row_ok && left > 0 ? (left < VEC ? left : VEC) : 0;
        cp_async16(dst + it * STEP * PITCH, left ? src + (int64_t)it * STEP * ld : base, left * (int)sizeof(T));
      }
    } else {
      constexpr int STEP = NT >= FAST ? NT / FAST : 1, SPAN = NT < FAST ? NT : FAST;   // threads along a row
      static_assert(NT % FAST == 0 || FAST % NT == 0, "threads of a copy");
      const T* q = src;
      const int64_t step = STEP * ld;
      const int slow_left = (KC ? limit : k_left) - s, fast_left = KC ? k_left - f : limit;
#pragma unroll 8
      for (int it = 0; it < (SLOW + STEP - 1) / STEP; ++it) {
        if (SLOW % STEP != 0 && s + it * STEP >= SLOW) break;
#pragma unroll
        for (int o = 0; o < FAST; o += SPAN) {
          const bool ok = it * STEP < slow_left && o < fast_left;
          cp_async_one<sizeof(T)>(dst + it * STEP * PITCH + o, ok ? q + o : base, ok ? (int)sizeof(T) : 0);
        }
        q += step;
      }
    }
    src += advance;
  }
};

// W consecutive elements from shared memory (W elements are W * sizeof(T) bytes and aligned to that, at most 16)
template <typename T, int W> __device__ __forceinline__ void lds_vec(const T* p, T (&v)[W]) {
  if constexpr (W * sizeof(T) == 16) {
    *reinterpret_cast<uint4*>(v) = *reinterpret_cast<const uint4*>(p);
  } else if constexpr (W * sizeof(T) == 8) {
    *reinterpret_cast<uint2*>(v) = *reinterpret_cast<const uint2*>(p);
  } else {
    static_assert(W == 1, "fragments are 1, 2 or 4 elements");
    v[0] = p[0];
  }
}

// The fragment of TR rows x KV k values that one thread multiplies, and which rows of the tile they are.
template <typename T, int ROWS, int BK, int NT, bool KC, int TR>
struct Fragment {
  using Tile = OperandTile<T, ROWS, BK, NT, KC>;
  static constexpr int KV = 16 / sizeof(T);              // k values per step
  static constexpr int THREADS = ROWS / TR;               // threads along this dimension
  static constexpr int W = KC ? 1 : (TR < KV ? TR : KV);  // consecutive rows a thread owns
  static __device__ __forceinline__ int row(int t, int i) { return (i / W) * (THREADS * W) + t * W + i % W; }
  static __device__ __forceinline__ void read(const T* tile, int t, int k, T (&v)[TR][KV]) {
    if constexpr (KC) {
#pragma unroll
      for (int i = 0; i < TR; ++i) lds_vec<T, KV>(tile + (t + i * THREADS) * Tile::PITCH + k, v[i]);
    } else {
#pragma unroll
      for (int kk = 0; kk < KV; ++kk)
#pragma unroll
        for (int c = 0; c < TR / W; ++c) {
          alignas(16) T w[W];
          lds_vec<T, W>(tile + (k + kk) * Tile::PITCH + c * (THREADS * W) + t * W, w);
#pragma unroll
          for (int q = 0; q < W; ++q) v[c * W + q][kk] = w[q];
        }
    }
  }
};

// one product of a launch
template <typename T> struct Product {
  int M, N, K;
  T alpha, beta;
  const T *A, *B;
  T* C;
  int64_t lda, ldb, ldc, sA, sB, sC;
  bool vecA, vecB, vecC;
  int tiles_n, tiles_mn;       // column tiles, tiles of one batch entry
  EpiParams<T> epi;
};

// tile shapes: BM x BN outputs, TM x TN per thread, BK k per stage, NC threads that copy
template <typename T, int BM_, int BN_, int BK_, int TM_, int TN_, int STAGES_, int NC_>
struct TileShape {
  static constexpr int BM = BM_, BN = BN_, BK = BK_, TM = TM_, TN = TN_, STAGES = STAGES_;
  static constexpr int NT = (BM / TM) * (BN / TN);      // threads that multiply
  static constexpr int NC = NC_;
  static constexpr int THREADS = NT + NC;
  // either layout of either operand
  static constexpr int STAGE_A = OperandTile<T, BM, BK, NC, true>::SIZE > OperandTile<T, BM, BK, NC, false>::SIZE
                                     ? OperandTile<T, BM, BK, NC, true>::SIZE : OperandTile<T, BM, BK, NC, false>::SIZE;
  static constexpr int STAGE_B = OperandTile<T, BN, BK, NC, true>::SIZE > OperandTile<T, BN, BK, NC, false>::SIZE
                                     ? OperandTile<T, BN, BK, NC, true>::SIZE : OperandTile<T, BN, BK, NC, false>::SIZE;
  static constexpr int SMEM = STAGES * (STAGE_A + STAGE_B) * (int)sizeof(T);
  static_assert(SMEM >= BM * BN * (int)sizeof(T), "the epilogue stages a whole output tile there");
};

template <typename T, typename S, bool TA, bool TB, bool EXACT>
__device__ __forceinline__ void product_tile(const Product<T>& p, int tile, T* smem) {
  constexpr int NT = S::NT, BK = S::BK, TM = S::TM, TN = S::TN, STAGES = S::STAGES;
  // op(A) is M x K: memory has k contiguous when !TA.  op(B) is K x N: memory has k contiguous when TB.
  using FA = Fragment<T, S::BM, BK, S::NC, !TA, TM>;
  using FB = Fragment<T, S::BN, BK, S::NC, TB, TN>;
  constexpr int KV = FA::KV;
  constexpr int WX = S::BN / TN / 8;             // a warp is 4 x 8 threads
  static_assert(S::BN / TN % 8 == 0 && S::BM / TM % 4 == 0 && BK % KV == 0, "tile shape");
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // Neighbouring lanes share a column and lanes two apart share a row: a 128-bit read of shared memory takes 2 cycles instead of 4
  // where lane pairs one apart, or all pairs two apart, read the same address.
  const int tx = (warp % WX) * 8 + (lane >> 1 & 7), ty = (warp / WX) * 4 + ((lane & 1) | (lane >> 4 << 1));
  const int64_t bz = tile / p.tiles_mn;
  const int t2 = tile % p.tiles_mn;
  const int m0 = t2 / p.tiles_n * S::BM, n0 = t2 % p.tiles_n * S::BN;
  T* As = smem;
  T* Bs = smem + STAGES * S::STAGE_A;

  T acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = (T)0;

  const int ktiles = (p.K + BK - 1) / BK;
  if (tid >= NT) {
    const int ct = tid - NT;
    const bool vecA = p.vecA, vecB = p.vecB;
    typename FA::Tile la;
    typename FB::Tile lb;
    la.begin(p.A + bz * p.sA, p.lda, m0, p.M, vecA, ct);
    lb.begin(p.B + bz * p.sB, p.ldb, n0, p.N, vecB, ct);
    int k_left = p.K;                            // k of the next stage to be asked for and beyond
    auto stage = [&](int s) {
      if (k_left > 0) {
        la.load(As + s * S::STAGE_A, k_left, vecA);
        lb.load(Bs + s * S::STAGE_B, k_left, vecB);
      }
      k_left -= BK;
      cp_async_commit();
    };
    for (int s = 0; s < STAGES - 1; ++s) stage(s);
    cp_async_wait<STAGES - 2>();                 // the first stage has landed
    __syncthreads();
    int nxt = STAGES - 1;
    for (int kt = 0; kt < ktiles; ++kt) {        // while stage kt is multiplied: its predecessor's place is free
      stage(nxt);
      cp_async_wait<STAGES - 2>();               // stage kt + 1 has landed
      __syncthreads();
      nxt = nxt + 1 == STAGES ? 0 : nxt + 1;
    }
    cp_async_wait<0>();
  } else {
    __syncthreads();
    int cur = 0;
    for (int kt = 0; kt < ktiles; ++kt) {
      const T* as = As + cur * S::STAGE_A;
      const T* bs = Bs + cur * S::STAGE_B;
      // two values of k are on their way at any time: the fragments of the next KV values are read, and the products
      // of the next k are formed, while the products of this k are added (an addition that waited for its own product
      // would stall a warp that has its scheduler to itself)
      alignas(16) T a[2][TM][KV], b[2][TN][KV];
      T pr[TM][TN];
      FA::read(as, ty, 0, a[0]);
      FB::read(bs, tx, 0, b[0]);
#pragma unroll
      for (int k = 0; k < BK; ++k) {
        const int g = k / KV, h = g & 1, kk = k % KV;
        if (kk == 0 && g + 1 < BK / KV) {
          FA::read(as, ty, (g + 1) * KV, a[h ^ 1]);
          FB::read(bs, tx, (g + 1) * KV, b[h ^ 1]);
        }
        // EXACT: round the product, then the sum, as `Output[i][j] += a * b` does in the
        // managed code (k ascending), so the result is bit-identical to that loop
        if constexpr (EXACT) {
          if (k == 0) {
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
              for (int j = 0; j < TN; ++j) pr[i][j] = mul_rn(a[0][i][0], b[0][j][0]);
          }
          T pn[TM][TN];
          if (k + 1 < BK) {
            const int h1 = ((k + 1) / KV) & 1, k1 = (k + 1) % KV;
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
              for (int j = 0; j < TN; ++j) pn[i][j] = mul_rn(a[h1][i][k1], b[h1][j][k1]);
          }
#pragma unroll
          for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) {
              acc[i][j] = add_rn(acc[i][j], pr[i][j]);
              if (k + 1 < BK) pr[i][j] = pn[i][j];
            }
        } else {
#pragma unroll
          for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) acc[i][j] = fma(a[h][i][kk], b[h][j][kk], acc[i][j]);
        }
      }
      __syncthreads();
      cur = cur + 1 == STAGES ? 0 : cur + 1;
    }
  }

  // alpha * acc + beta * C
  T* C = p.C + bz * p.sC;
  constexpr int W = FB::W;                       // consecutive columns of a thread
  const EpiParams<T>& epi = p.epi;
  const bool plain = !epi.bias && !epi.z_out && epi.act == PRAD_ACT_NONE && epi.dact == PRAD_ACT_NONE;
  T* staged = smem;                              // [BM][BN]
  if (tid < NT) {
#pragma unroll
    for (int i = 0; i < TM; ++i) {
      const int ml = FA::row(ty, i), m = m0 + ml;
      if (m >= p.M) continue;
#pragma unroll
      for (int c = 0; c < TN / W; ++c) {
        const int nl = FB::row(tx, c * W), n = n0 + nl;
        if (n >= p.N) continue;
        const int64_t off = (int64_t)m * p.ldc + n;
        alignas(16) T out[W];
#pragma unroll
        for (int q = 0; q < W; ++q) {
          T v = mul_rn(p.alpha, acc[i][c * W + q]);
          if (p.beta != (T)0 && (W == 1 || n + q < p.N)) {
            const T old = C[off + q];
            v = (p.beta == (T)1) ? add_rn(old, v) : fma(p.beta, old, v);
          }
          out[q] = v;
        }
        if (!plain) {
#pragma unroll
          for (int q = 0; q < W; ++q) staged[ml * S::BN + nl + q] = out[q];
        } else if (W > 1 && p.vecC && n + W <= p.N) {
          if constexpr (W * sizeof(T) == 16) *reinterpret_cast<uint4*>(C + off) = *reinterpret_cast<const uint4*>(out);
          else if constexpr (W * sizeof(T) == 8) *reinterpret_cast<uint2*>(C + off) = *reinterpret_cast<const uint2*>(out);
        } else {
#pragma unroll
          for (int q = 0; q < W; ++q)
            if (W == 1 || n + q < p.N) C[off + q] = out[q];
        }
      }
    }
  }
  if (plain) return;
  // bias, pre-activation copy and activation: one copy of that code for all outputs, row by row out of shared memory
  __syncthreads();
  const T* saved = epi.saved ? epi.saved + bz * p.sC : nullptr;
  T* z_out = epi.z_out ? epi.z_out + bz * p.sC : nullptr;
#pragma unroll 1
  for (int e = tid; e < S::BM * S::BN; e += S::THREADS) {
    const int m = m0 + e / S::BN, n = n0 + e % S::BN;
    if (m >= p.M || n >= p.N) continue;
    const int64_t off = (int64_t)m * p.ldc + n;
    T v = staged[e];
    if (epi.bias) v = add_rn(v, epi.bias[n]);
    if (z_out) z_out[off] = v;
    if (epi.act != PRAD_ACT_NONE) v = act_value<T>((prad_act)epi.act, v, epi.act_alpha);
    if (epi.dact != PRAD_ACT_NONE) v = mul_rn(v, act_derivative<T>((prad_act)epi.dact, saved[off], epi.act_alpha));
    C[off] = v;
  }
}

template <typename T, typename S, bool TA, bool TB, bool EXACT>
__global__ void __launch_bounds__(S::THREADS)
gemm_simt_kernel(const __grid_constant__ Product<T> p) {
  chain_begin();
  extern __shared__ __align__(16) unsigned char simt_smem[];
  product_tile<T, S, TA, TB, EXACT>(p, blockIdx.x, reinterpret_cast<T*>(simt_smem));
}

// ---- many small products ----------------------------------------------------------------------
// A strided batch of products whose whole output is at most 64 x 64 (the per-window, per-head
// attention products Q K^T, P V and their four backward forms: 49 x 49 x 32 and 49 x 32 x 49).  The
// 64 x 64 tile of the kernel above would spend more than half of its multiply-adds on rows, columns
// and k beyond the matrices, and at these sizes the arithmetic, not the memory, is what takes the
// time.  Here a CTA owns one product and has just the threads its output needs (4 x 4 outputs per
// thread, rounded up to whole warps); both operands of up to KC values of k sit in shared memory in
// k-major order, so a thread reads one 4-vector of each per k.  Same arithmetic per output element
// as above (k ascending, one accumulator), hence bit-identical results.
template <typename T> __device__ __forceinline__ void load4(const T* p, T (&v)[4]);
template <> __device__ __forceinline__ void load4<float>(const float* p, float (&v)[4]) {
  const float4 t = *reinterpret_cast<const float4*>(p);
  v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
}
template <> __device__ __forceinline__ void load4<double>(const double* p, double (&v)[4]) {
  const double2 t = *reinterpret_cast<const double2*>(p), u = *reinterpret_cast<const double2*>(p + 2);
  v[0] = t.x; v[1] = t.y; v[2] = u.x; v[3] = u.y;
}

// one operand chunk into shared memory as [k][XP]: X operand rows (M or N; columns X..XP-1 are zero-filled),
// kc values of k starting at k0.  KMAJOR: memory is [K][X] (x contiguous), otherwise [X][K].  A warp takes
// every nw-th memory row, its lanes consecutive elements of it (at most 64: two trips); the loads of eight rows
// are issued before the first of them is stored, so that a thread has up to sixteen loads in flight.
template <typename T, bool KMAJOR>
__device__ __forceinline__ void load_small_operand(T* __restrict__ s, int XP, const T* __restrict__ g, int64_t ld, int X,
                                                   int k0, int kc, int warp, int lane, int nw) {
  constexpr int U = 8;
  const int rows = KMAJOR ? kc : XP;          // memory rows of the chunk (rows X..XP-1 of the [X][K] form are zeros)
  const int cols = KMAJOR ? XP : kc;          // elements taken from each
  const int rows_valid = KMAJOR ? kc : X, cols_valid = KMAJOR ? X : kc;
  const T* base = KMAJOR ? g + (int64_t)k0 * ld : g + k0;
  for (int r0 = warp; r0 < rows; r0 += nw * U) {
    T v[U][2];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int r = r0 + u * nw;
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        const int c = lane + 32 * t;
        v[u][t] = (r < rows_valid && c < cols_valid) ? base[(int64_t)r * ld + c] : (T)0;
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int r = r0 + u * nw;
      if (r >= rows) break;
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        const int c = lane + 32 * t;
        if (c < cols) s[KMAJOR ? r * XP + c : c * XP + r] = v[u][t];
      }
    }
  }
}

template <typename T, bool TA, bool TB, bool EXACT>
__global__ void __launch_bounds__(256)
gemm_small_kernel(int M, int N, int K, int KC, int MP, int NP, T alpha, const T* __restrict__ A, int64_t lda,
                  const T* __restrict__ B, int64_t ldb, T beta, T* __restrict__ C, int64_t ldc, int64_t sA, int64_t sB,
                  int64_t sC, bool vecC) {
  extern __shared__ __align__(16) unsigned char small_smem[];
  T* As = reinterpret_cast<T*>(small_smem);   // [KC][MP]
  T* Bs = As + KC * MP;                        // [KC][NP]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nw = blockDim.x >> 5;
  const int txn = NP >> 2;
  const int tx = tid % txn, ty = tid / txn;
  const bool active = ty < (MP >> 2);
  const int64_t bz = blockIdx.x;
  A += bz * sA;
  B += bz * sB;
  C += bz * sC;

  T acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = (T)0;

  for (int k0 = 0; k0 < K; k0 += KC) {
    const int kc = K - k0 < KC ? K - k0 : KC;
    if (k0) __syncthreads();
    load_small_operand<T, TA>(As, MP, A, lda, M, k0, kc, warp, lane, nw);     // op(A) is M x K: k-major memory when TA
    load_small_operand<T, !TB>(Bs, NP, B, ldb, N, k0, kc, warp, lane, nw);    // op(B) is K x N: k-major memory unless TB
    __syncthreads();
    if (active) {
      const T* ap = As + 4 * ty;
      const T* bp = Bs + 4 * tx;
#pragma unroll 4
      for (int k = 0; k < kc; ++k) {
        T a[4], b[4];
        load4<T>(ap + k * MP, a);
        load4<T>(bp + k * NP, b);
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            if (EXACT) acc[i][j] = add_rn(acc[i][j], mul_rn(a[i], b[j]));
            else acc[i][j] = fma(a[i], b[j], acc[i][j]);
          }
      }
    }
  }
  if (!active) return;
  const int n = 4 * tx;
  const bool full = vecC && n + 4 <= N;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int m = 4 * ty + i;
    if (m >= M) continue;
    const int64_t off = (int64_t)m * ldc + n;
    T out[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      T v = mul_rn(alpha, acc[i][q]);
      if (beta != (T)0 && n + q < N) {
        const T old = C[off + q];
        v = (beta == (T)1) ? add_rn(old, v) : fma(beta, old, v);
      }
      out[q] = v;
    }
    if (full) {
      if constexpr (sizeof(T) == 4) {
        *reinterpret_cast<float4*>(C + off) = make_float4(out[0], out[1], out[2], out[3]);
      } else {
        *reinterpret_cast<double2*>(C + off) = make_double2(out[0], out[1]);
        *reinterpret_cast<double2*>(C + off + 2) = make_double2(out[2], out[3]);
      }
    } else {
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (n + q < N) C[off + q] = out[q];
    }
  }
}

template <typename T>
static prad_status launch_small(prad_ctx* ctx, bool exact, bool tA, bool tB, int M, int N, int K, T alpha, const T* A,
                                int64_t lda, const T* B, int64_t ldb, T beta, T* C, int64_t ldc, int batch, int64_t sA,
                                int64_t sB, int64_t sC) {
  const int MP = (M + 3) & ~3, NP = (N + 3) & ~3;
  const int kc_max = sizeof(T) == 4 ? 64 : 32;                  // at most 32 KB of shared memory
  const int KC = K < kc_max ? K : kc_max;
  int nt = (MP / 4) * (NP / 4);
  nt = (nt + 31) & ~31;
  if (nt < 64) nt = 64;
  const size_t smem = (size_t)KC * (MP + NP) * sizeof(T);
  const bool vC = (((uintptr_t)C & 15) == 0) && ldc % 4 == 0 && sC % 4 == 0;
#define PRAD_SMALL_LAUNCH(TA_, TB_)                                                                          \
  do {                                                                                                       \
    if (exact)                                                                                               \
      gemm_small_kernel<T, TA_, TB_, true><<<(unsigned)batch, nt, smem, ctx->stream>>>(                     \
          M, N, K, KC, MP, NP, alpha, A, lda, B, ldb, beta, C, ldc, sA, sB, sC, vC);                         \
    else                                                                                                     \
      gemm_small_kernel<T, TA_, TB_, false><<<(unsigned)batch, nt, smem, ctx->stream>>>(                    \
          M, N, K, KC, MP, NP, alpha, A, lda, B, ldb, beta, C, ldc, sA, sB, sC, vC);                         \
  } while (0)
  if (!tA && !tB) PRAD_SMALL_LAUNCH(false, false);
  else if (!tA && tB) PRAD_SMALL_LAUNCH(false, true);
  else if (tA && !tB) PRAD_SMALL_LAUNCH(true, false);
  else PRAD_SMALL_LAUNCH(true, true);
#undef PRAD_SMALL_LAUNCH
  PRAD_LAUNCHED(ctx);
  return PRAD_OK;
}

template <typename T> static bool aligned16(const void* p) { return ((uintptr_t)p & 15) == 0; }

// Small tiles, of which an SM has one or two: the copies' instructions are spread over all four schedulers, for the four multiplying
// warps meet after every stage and wait for the slowest (512 x 784 x 256 in double, forward and backward, 67 us with copying warps
// on two schedulers, 59 on four).  Where an operand's rows do not start at 16-byte boundaries (SmallOdd) there are twice or four
// times as many copies, and four warps of them get in the way: a double step of 887 x 98-217-217-217-9 takes 301 us with them,
// 212 with two.  So do they in float where an SM has more than four tiles (256 x 784 x 512, backward, 4.05 tiles an SM: 25.5 us with
// four, 23.2 with two; 128 x 784 x 512, 3.4 tiles: 14.3 and 15.0), for one less of the larger CTAs has room there.  (A Small without the
// element-wise copies that it does not need is no better: 256 x 784 x 512 in double 24.0 instead of 19.3 us.)
// Double: stages of 32 k, for half the barriers and half the ends of rows (that step took 350 us with 16), but of 16 (SmallShort), with
// as many values on their way, for one product whose last stage of 32 would be zeros for a sixteenth of the work: 512 x 33 x 512 4.8
// and 4.15 us, 184 x 80 x 1008 6.1 and 5.7, 1000 x 100 x 1000 21.5 and 20.1, but 176 x 144 x 656 5.4 and 5.8.  For the two products of a
// Backward longer stages are the better ones all the same (41 x 230 x 896 13.2 and 14.4), and for 16 x 16 tiles in a network's step
// (500 x 33-128-128-10 from the host 108 and 122).
template <typename T> struct SimtShapes;
template <> struct SimtShapes<float> {
  using Tiny = TileShape<float, 16, 16, 32, 2, 2, 4, 64>;
  using Small = TileShape<float, 32, 32, 32, 4, 2, 4, 128>;
  using SmallOdd = TileShape<float, 32, 32, 32, 4, 2, 4, 64>;
  using SmallShort = SmallOdd;
  using Wide = TileShape<float, 64, 32, 32, 4, 4, 3, 64>;
  using Medium = TileShape<float, 64, 64, 32, 4, 4, 3, 64>;
  using Large = TileShape<float, 128, 128, 16, 8, 8, 4, 64>;
};
template <> struct SimtShapes<double> {
  using Tiny = TileShape<double, 16, 16, 32, 2, 2, 4, 64>;
  using Small = TileShape<double, 32, 32, 32, 4, 2, 3, 128>;
  using SmallOdd = TileShape<double, 32, 32, 32, 4, 2, 3, 64>;
  using SmallShort = TileShape<double, 32, 32, 16, 4, 2, 6, 64>;
  using Wide = TileShape<double, 64, 32, 16, 4, 4, 3, 64>;
  using Medium = TileShape<double, 64, 64, 16, 4, 4, 3, 64>;
  using Large = Medium;
};

// Two products of one launch, dA = dC*B^T and dB = A^T*dC of one MatrixMultiplyOperation.Backward: neither reads what the
// other writes, and together they leave fewer SMs idle than one after the other.
template <typename T, typename S, bool EXACT>
__global__ void __launch_bounds__(S::THREADS)
gemm_simt_backward_kernel(const __grid_constant__ Product<T> nt, const __grid_constant__ Product<T> tn, int tn_first, int first_tiles) {
  chain_begin();
  extern __shared__ __align__(16) unsigned char simt_smem[];
  T* smem = reinterpret_cast<T*>(simt_smem);
  const int tile = blockIdx.x;
  const bool first = tile < first_tiles;
  const int local = first ? tile : tile - first_tiles;
  if (first == (tn_first != 0)) product_tile<T, S, true, false, EXACT>(tn, local, smem);
  else product_tile<T, S, false, true, EXACT>(nt, local, smem);
}

template <typename T, typename S>
static prad_status set_tiles(Product<T>& p, int batch, int64_t* all) {
  p.tiles_n = (int)ceil_div(p.N, S::BN);
  const int64_t mn = ceil_div(p.M, S::BM) * p.tiles_n;
  *all = mn * batch;
  PRAD_REQUIRE(*all <= 0x3fffffff, PRAD_ERR_UNSUPPORTED, "gemm: too many tiles for one launch");
  p.tiles_mn = (int)mn;
  return PRAD_OK;
}

template <typename T, typename S>
static prad_status launch_shape(prad_ctx* ctx, bool exact, bool tA, bool tB, int batch, Product<T> p) {
  int64_t all = 0;
  prad_status ts = set_tiles<T, S>(p, batch, &all);
  if (ts) return ts;
#define PRAD_GEMM_LAUNCH(TA_, TB_, EX_)                                                            \
  do {                                                                                             \
    prad_status st_ = allow_smem<gemm_simt_kernel<T, S, TA_, TB_, EX_>>(ctx, S::SMEM);             \
    if (st_) return st_;                                                                           \
    launch_chained(gemm_simt_kernel<T, S, TA_, TB_, EX_>, (unsigned)all, S::THREADS, S::SMEM, ctx->stream, p);      \
  } while (0)
#define PRAD_GEMM_FORM(TA_, TB_)                       \
  do {                                                 \
    if (exact) PRAD_GEMM_LAUNCH(TA_, TB_, true);       \
    else PRAD_GEMM_LAUNCH(TA_, TB_, false);            \
  } while (0)
  if (!tA && !tB) PRAD_GEMM_FORM(false, false);
  else if (!tA && tB) PRAD_GEMM_FORM(false, true);
  else if (tA && !tB) PRAD_GEMM_FORM(true, false);
  else PRAD_GEMM_FORM(true, true);
#undef PRAD_GEMM_FORM
#undef PRAD_GEMM_LAUNCH
  PRAD_LAUNCHED(ctx);
  return PRAD_OK;
}

template <typename T, typename S>
static prad_status launch_backward(prad_ctx* ctx, bool exact, Product<T> nt, Product<T> tn) {
  int64_t n_nt = 0, n_tn = 0;
  prad_status st = set_tiles<T, S>(nt, 1, &n_nt);
  if (!st) st = set_tiles<T, S>(tn, 1, &n_tn);
  if (st) return st;
  const int tn_first = tn.K >= nt.K;             // the longer chains start first
  const unsigned grid = (unsigned)(n_nt + n_tn);
  const int first = (int)(tn_first ? n_tn : n_nt);
  if (exact) {
    if ((st = allow_smem<gemm_simt_backward_kernel<T, S, true>>(ctx, S::SMEM))) return st;
    launch_chained(gemm_simt_backward_kernel<T, S, true>, grid, S::THREADS, S::SMEM, ctx->stream, nt, tn, tn_first, first);
  } else {
    if ((st = allow_smem<gemm_simt_backward_kernel<T, S, false>>(ctx, S::SMEM))) return st;
    launch_chained(gemm_simt_backward_kernel<T, S, false>, grid, S::THREADS, S::SMEM, ctx->stream, nt, tn, tn_first, first);
  }
  PRAD_LAUNCHED(ctx);
  return PRAD_OK;
}

// Which tile shape.  A CTA that has its SM to itself takes `alone` cycles per k (its chain of additions, and the shared
// memory's 128 bytes per cycle), n CTAs of one SM take n * `shared`: measured for the exact variants on products of
// 128^2 x 2048, 256 x 512 x 784, 1024^2 x 120 and 2048^2 x 31, with the lanes, copies and stages of that time (16 x 16 alone takes
// 14.5 and 23 since).  With the shapes that they choose, 69 other sizes of either type are as fast as with those kernels or faster, but for
// those named at SimtShapes; where the shapes would cross now has not been measured.  The estimate is the busiest SM's time; the 24 stands for
// filling the stages and writing the tile.  Small tiles win while there are fewer tiles than SMs, large ones once
// every SM has several.
struct ShapeCost { int bm, bn; double alone, shared; };
template <typename T> struct ShapeCosts;
template <> struct ShapeCosts<float> {
  static constexpr ShapeCost c[5] = {{16, 16, 15.5, 10.5}, {32, 32, 34, 28}, {64, 32, 57, 49}, {64, 64, 98, 93}, {128, 128, 340, 330}};
};
template <> struct ShapeCosts<double> {
  static constexpr ShapeCost c[4] = {{16, 16, 25, 15.3}, {32, 32, 54, 45.5}, {64, 32, 92, 87}, {64, 64, 163, 163}};
};
struct ProductSize { int64_t M, N, K, batch; };
template <typename T> static int pick_shape(const prad_ctx* ctx, const ProductSize* p, int count) {
  int best = 0;
  double best_cost = 0;
  for (int s = 0; s < (int)(sizeof(ShapeCosts<T>::c) / sizeof(ShapeCost)); ++s) {
    const ShapeCost& c = ShapeCosts<T>::c[s];
    double tiles = 0, work = 0, longest = 0;
    for (int i = 0; i < count; ++i) {
      const double t = (double)(ceil_div(p[i].M, c.bm) * ceil_div(p[i].N, c.bn) * p[i].batch), k = (double)p[i].K + 24;
      tiles += t;
      work += t * k;
      if (k > longest) longest = k;
    }
    const double per_sm = (double)ceil_div((int64_t)tiles, ctx->sm_count);       // CTAs of the busiest SM
    double cost = per_sm * (work / tiles) * c.shared;
    if (longest * c.alone > cost) cost = longest * c.alone;
    if (s == 0 || cost < best_cost) { best = s; best_cost = cost; }
  }
  return best;
}

// The two rules of SimtShapes: whether small tiles are copied by four warps, and in stages of 16 k.
template <typename T> static bool four_copying_warps(const prad_ctx* ctx, const ProductSize* p, int count) {
  int64_t tiles = 0;
  for (int i = 0; i < count; ++i) tiles += ceil_div(p[i].M, 32) * ceil_div(p[i].N, 32) * p[i].batch;
  return sizeof(T) == 8 || tiles <= 4 * (int64_t)ctx->sm_count;
}
template <typename T> static bool short_stages(int64_t K) { return sizeof(T) == 8 && 16 * (ceil_div(K, 32) * 32) > 17 * (ceil_div(K, 16) * 16); }

template <typename T>
static Product<T> make_product(int M, int N, int K, double alpha, const void* A, int64_t lda, const void* B, int64_t ldb, double beta,
                               void* C, int64_t ldc, int64_t sA, int64_t sB, int64_t sC, const GemmEpilogue& e) {
  constexpr int VEC = VecOf<T>::N;
  Product<T> p;
  p.M = M; p.N = N; p.K = K;
  p.alpha = (T)alpha; p.beta = (T)beta;
  p.A = (const T*)A; p.B = (const T*)B; p.C = (T*)C;
  p.lda = lda; p.ldb = ldb; p.ldc = ldc;
  p.sA = sA; p.sB = sB; p.sC = sC;
  p.vecA = aligned16<T>(A) && lda % VEC == 0 && sA % VEC == 0;
  p.vecB = aligned16<T>(B) && ldb % VEC == 0 && sB % VEC == 0;
  p.vecC = aligned16<T>(C) && ldc % VEC == 0 && sC % VEC == 0;
  p.epi = EpiParams<T>{(const T*)e.bias, (T*)e.z_out, (int)e.act, (int)e.dact, (const T*)e.saved, (T)e.act_alpha};
  return p;
}

template <typename T>
prad_status gemm_simt(prad_ctx* ctx, bool exact, bool tA, bool tB, int M, int N, int K,
                      double alpha, const void* A, int lda, const void* B, int ldb, double beta,
                      void* C, int ldc, int batch, int64_t sA, int64_t sB, int64_t sC,
                      const GemmEpilogue& e) {
  // a batch of products no larger than one small tile each, enough of them to fill the machine by themselves
  const bool plain = !e.bias && !e.z_out && e.act == PRAD_ACT_NONE && e.dact == PRAD_ACT_NONE;
  if (plain && M <= 64 && N <= 64 && K >= 1 && batch >= ctx->sm_count && ctx->gemm_small)
    return launch_small<T>(ctx, exact, tA, tB, M, N, K, (T)alpha, (const T*)A, lda, (const T*)B, ldb, (T)beta, (T*)C, ldc,
                           batch, sA, sB, sC);
  const Product<T> p = make_product<T>(M, N, K, alpha, A, lda, B, ldb, beta, C, ldc, sA, sB, sC, e);
  const ProductSize size{M, N, K, batch};
  using Shapes = SimtShapes<T>;
  switch (pick_shape<T>(ctx, &size, 1)) {
    case 0: return launch_shape<T, typename Shapes::Tiny>(ctx, exact, tA, tB, batch, p);
    case 1:
      if (short_stages<T>(K)) return launch_shape<T, typename Shapes::SmallShort>(ctx, exact, tA, tB, batch, p);
      return p.vecA && p.vecB && four_copying_warps<T>(ctx, &size, 1) ? launch_shape<T, typename Shapes::Small>(ctx, exact, tA, tB, batch, p)
                                                                      : launch_shape<T, typename Shapes::SmallOdd>(ctx, exact, tA, tB, batch, p);
    case 2: return launch_shape<T, typename Shapes::Wide>(ctx, exact, tA, tB, batch, p);
    case 3: return launch_shape<T, typename Shapes::Medium>(ctx, exact, tA, tB, batch, p);
    default: return launch_shape<T, typename Shapes::Large>(ctx, exact, tA, tB, batch, p);
  }
}

// dA (M x K) = dC (M x N) * B^T (.) act'(saved)  and  dB (K x N) = scale * A^T * dC [+ dB], in one launch
template <typename T>
prad_status gemm_simt_backward(prad_ctx* ctx, bool exact, const void* A, const void* B, const void* dC, void* dA, void* dB, int M,
                               int K, int N, bool accumulate_dB, double dB_scale, const GemmEpilogue& e_dA) {
  const Product<T> nt = make_product<T>(M, K, N, 1.0, dC, N, B, N, 0.0, dA, K, 0, 0, 0, e_dA);
  const Product<T> tn = make_product<T>(K, N, M, dB_scale, A, K, dC, N, accumulate_dB ? 1.0 : 0.0, dB, N, 0, 0, 0, GemmEpilogue());
  const ProductSize size[2] = {{M, K, N, 1}, {K, N, M, 1}};
  using Shapes = SimtShapes<T>;
  switch (pick_shape<T>(ctx, size, 2)) {
    case 0: return launch_backward<T, typename Shapes::Tiny>(ctx, exact, nt, tn);
    case 1:
      return nt.vecA && nt.vecB && tn.vecA && tn.vecB && four_copying_warps<T>(ctx, size, 2)
                 ? launch_backward<T, typename Shapes::Small>(ctx, exact, nt, tn)
                 : launch_backward<T, typename Shapes::SmallOdd>(ctx, exact, nt, tn);
    case 2: return launch_backward<T, typename Shapes::Wide>(ctx, exact, nt, tn);
    case 3: return launch_backward<T, typename Shapes::Medium>(ctx, exact, nt, tn);
    default: return launch_backward<T, typename Shapes::Large>(ctx, exact, nt, tn);
  }
}

}  // namespace prad

// Windowed self-attention: per (window, head)  S = scale Q K^T,  P = softmax(S),  O = P V, and its Backward, each as one
// kernel over the [tokens x 3 dim] QKV matrix in place.
//
// What bounded it: as strided-batched products and softmax passes (six launches forward, thirteen backward for three heads)
// the 49 x 49 scores of 12288 (window, head) pairs went to memory and back three to five times, and the products were bound by
// shared-memory reads with 4 x 4 outputs per thread: 443 us forward, 740 us backward for 64 images of 64 windows.
//
// Here 64 threads own one pair: an 8 x 8 grid with T x T scores per thread (rows and columns eight apart, T = ceil(window / 8):
// 7 for 49 tokens, 14 reads of shared memory per 49 multiply-adds), a row's scores in eight neighbouring lanes, so the softmax is
// three shuffles.  P is written once (the Backward reads it); the scores and their gradients never leave the SM.  Backward:
// dV = P^T dO first, then dP = dO V^T in registers and dS = P (.) (dP - rowsum(dP (.) P)) over P's place, then K and Q over V's and
// dO's places and dQ = scale dS K, dK = scale dS^T Q -- 30 KB per pair, seven or eight pairs per SM.  193 us forward and 295 us
// backward, three quarters of the issue slots used, half of them by multiply-adds.
// Sums are fused multiply-adds, k ascending (the separate products round product and sum; both within the tolerance of the
// composition they replace: BatchMatrixMultiplyOperation, MatrixMultiplyScalarOperation, SoftmaxOperation.cs:53-109).
#include "act_math.cuh"
#include "common.cuh"

namespace prad {
namespace wa {

constexpr int NT = 64;

template <int T, int HD> struct Shape {
  static constexpr int ROWS = 8 * T;             // padded tokens
  static constexpr int PQ = HD + 4;              // pitch of Q, K, V, dO rows
  static constexpr int C = HD / 8;               // columns per thread of the token x head outputs
};
__host__ __device__ inline int score_pitch(int ws) {     // a multiple of four, rows in different 16-byte banks
  const int v = (ws + 3) / 4;
  return (v % 2 ? v : v + 1) * 4;
}
template <int T, int HD> static int smem_floats(int ws, bool backward) {
  using S = Shape<T, HD>;
  const int score = (S::ROWS + 1) * score_pitch(ws) + 64, tile = S::ROWS * S::PQ;
  if (backward) return 2 * tile + score;
  return tile + (score > 2 * tile ? score : 2 * tile);       // forward: P takes Q's and K's place
}

// ws rows of HD floats (pitch ld) into s; rows up to 8 T are zero-filled
template <int T, int HD>
__device__ __forceinline__ void load_rows(float* s, const float* __restrict__ g, int64_t ld, int ws) {
  using S = Shape<T, HD>;
  constexpr int V = HD / 4;
#pragma unroll
  for (int it = 0; it < (S::ROWS * V + NT - 1) / NT; ++it) {
    const int e = threadIdx.x + it * NT, r = e / V, c = e % V * 4;
    if (S::ROWS * V % NT != 0 && r >= S::ROWS) break;
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(s + r * S::PQ + c);
    const bool on = r < ws;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(on ? g + (int64_t)r * ld + c : g), "r"(on ? 16 : 0) : "memory");
  }
}
__device__ __forceinline__ void landed() {
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
}

// acc[i][j] += sum_k a[i * 8 + ty][k] * b[j * 8 + tx][k], k < HD
template <int T, int HD>
__device__ __forceinline__ void scores(const float* a, const float* b, int ty, int tx, float (&acc)[T][T]) {
  constexpr int PQ = Shape<T, HD>::PQ;
#pragma unroll 2
  for (int k = 0; k < HD; k += 4) {
    float4 x[T], y[T];
#pragma unroll
    for (int i = 0; i < T; ++i) x[i] = *reinterpret_cast<const float4*>(a + (i * 8 + ty) * PQ + k);
#pragma unroll
    for (int j = 0; j < T; ++j) y[j] = *reinterpret_cast<const float4*>(b + (j * 8 + tx) * PQ + k);
#pragma unroll
    for (int i = 0; i < T; ++i)
#pragma unroll
      for (int j = 0; j < T; ++j)
        acc[i][j] = fmaf(x[i].w, y[j].w, fmaf(x[i].z, y[j].z, fmaf(x[i].y, y[j].y, fmaf(x[i].x, y[j].x, acc[i][j]))));
  }
}
template <int C> __device__ __forceinline__ void read_cols(const float* p, float (&v)[C]) {
  if constexpr (C == 2) {
    const float2 t = *reinterpret_cast<const float2*>(p);
    v[0] = t.x; v[1] = t.y;
  } else {
#pragma unroll
    for (int q = 0; q < C; q += 4) {
      const float4 t = *reinterpret_cast<const float4*>(p + q);
      v[q] = t.x; v[q + 1] = t.y; v[q + 2] = t.z; v[q + 3] = t.w;
    }
  }
}
// acc[i][c] += sum_k s[i * 8 + ty][k] * b[k][tx * C + c], k < ws rounded up to 4 (the columns of s beyond ws are zero)
template <int T, int HD>
__device__ __forceinline__ void weigh_rows(const float* s, int ps, const float* b, int ws, int ty, int tx, float (&acc)[T][HD / 8]) {
  constexpr int PQ = Shape<T, HD>::PQ, C = HD / 8;
  for (int k = 0; k < ws; k += 4) {
    float4 x[T];
#pragma unroll
    for (int i = 0; i < T; ++i) x[i] = *reinterpret_cast<const float4*>(s + (i * 8 + ty) * ps + k);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      float y[C];
      read_cols<C>(b + (k + q) * PQ + tx * C, y);
#pragma unroll
      for (int i = 0; i < T; ++i) {
        const float xv = q == 0 ? x[i].x : q == 1 ? x[i].y : q == 2 ? x[i].z : x[i].w;
#pragma unroll
        for (int c = 0; c < C; ++c) acc[i][c] = fmaf(xv, y[c], acc[i][c]);
      }
    }
  }
}
// acc[j][c] += sum_i s[i][j * 8 + ty] * b[i][tx * C + c], i < ws
template <int T, int HD>
__device__ __forceinline__ void weigh_cols(const float* s, int ps, const float* b, int ws, int ty, int tx, float (&acc)[T][HD / 8]) {
  constexpr int PQ = Shape<T, HD>::PQ, C = HD / 8;
#pragma unroll 2
  for (int i = 0; i < ws; ++i) {
    float x[T], y[C];
#pragma unroll
    for (int j = 0; j < T; ++j) x[j] = s[i * ps + j * 8 + ty];
    read_cols<C>(b + i * PQ + tx * C, y);
#pragma unroll
    for (int j = 0; j < T; ++j)
#pragma unroll
      for (int c = 0; c < C; ++c) acc[j][c] = fmaf(x[j], y[c], acc[j][c]);
  }
}
template <int T, int HD>
__device__ __forceinline__ void store_rows(float* __restrict__ g, int64_t ld, int ws, int ty, int tx, float alpha, const float (&acc)[T][HD / 8]) {
  constexpr int C = HD / 8;
#pragma unroll
  for (int i = 0; i < T; ++i) {
    const int r = i * 8 + ty;
    if (r >= ws) continue;
    float* p = g + (int64_t)r * ld + tx * C;
    if constexpr (C == 2) {
      *reinterpret_cast<float2*>(p) = make_float2(alpha * acc[i][0], alpha * acc[i][1]);
    } else {
#pragma unroll
      for (int q = 0; q < C; q += 4)
        *reinterpret_cast<float4*>(p + q) = make_float4(alpha * acc[i][q], alpha * acc[i][q + 1], alpha * acc[i][q + 2], alpha * acc[i][q + 3]);
    }
  }
}
template <int R, int C> __device__ __forceinline__ void clear(float (&a)[R][C]) {
#pragma unroll
  for (int i = 0; i < R; ++i)
#pragma unroll
    for (int j = 0; j < C; ++j) a[i][j] = 0.f;
}

template <int T, int HD>
__global__ void __launch_bounds__(NT)
forward_kernel(const float* __restrict__ qkv, float* __restrict__ P, float* __restrict__ out, int ws, int heads, float scale) {
  chain_begin();
  using S = Shape<T, HD>;
  extern __shared__ __align__(16) float wa_smem[];
  const int dim = heads * HD, ps = score_pitch(ws), ty = threadIdx.x >> 3, tx = threadIdx.x & 7;
  const int w = blockIdx.x / heads, h = blockIdx.x % heads;
  float *v = wa_smem, *q = v + S::ROWS * S::PQ, *k = q + S::ROWS * S::PQ, *s = q;
  const float* base = qkv + (int64_t)w * ws * 3 * dim + h * HD;
  load_rows<T, HD>(q, base, 3 * dim, ws);
  load_rows<T, HD>(k, base + dim, 3 * dim, ws);
  load_rows<T, HD>(v, base + 2 * dim, 3 * dim, ws);
  landed();
  {
    float a[T][T];
    clear(a);
    scores<T, HD>(q, k, ty, tx, a);
    __syncthreads();                                         // Q and K are done with
#pragma unroll
    for (int i = 0; i < T; ++i) {
      float mx = -INFINITY, sum = 0.f;
#pragma unroll
      for (int j = 0; j < T; ++j) {
        a[i][j] = j * 8 + tx < ws ? scale * a[i][j] : -INFINITY;
        mx = fmaxf(mx, a[i][j]);
      }
#pragma unroll
      for (int o = 1; o < 8; o <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
#pragma unroll
      for (int j = 0; j < T; ++j) {
        a[i][j] = t_exp(a[i][j] - mx);
        sum += a[i][j];
      }
#pragma unroll
      for (int o = 1; o < 8; o <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      const int r = i * 8 + ty;
      const float inv = div_rn(1.f, sum);
#pragma unroll
      for (int j = 0; j < T; ++j)
        if (j * 8 + tx < ps) s[r * ps + j * 8 + tx] = a[i][j] * inv;              // zero beyond the window
    }
    for (int c = T * 8 + tx; c < ps; c += 8)
      for (int i = 0; i < T; ++i) s[(i * 8 + ty) * ps + c] = 0.f;
  }
  __syncthreads();
  float* Pg = P + (int64_t)blockIdx.x * ws * ws;
  for (int r = threadIdx.x >> 5; r < ws; r += NT / 32)
    for (int c = threadIdx.x & 31; c < ws; c += 32) Pg[r * ws + c] = s[r * ps + c];
  float o[T][S::C];
  clear(o);
  weigh_rows<T, HD>(s, ps, v, ws, ty, tx, o);
  store_rows<T, HD>(out + (int64_t)w * ws * dim + h * HD, dim, ws, ty, tx, 1.f, o);
}

template <int T, int HD>
__global__ void __launch_bounds__(NT)
backward_kernel(const float* __restrict__ qkv, const float* __restrict__ P, const float* __restrict__ d_out, float* __restrict__ d_qkv,
                int ws, int heads, float scale) {
  chain_begin();
  using S = Shape<T, HD>;
  extern __shared__ __align__(16) float wa_smem[];
  const int dim = heads * HD, ps = score_pitch(ws), ty = threadIdx.x >> 3, tx = threadIdx.x & 7;
  const int w = blockIdx.x / heads, h = blockIdx.x % heads;
  float *x = wa_smem, *y = x + S::ROWS * S::PQ, *s = y + S::ROWS * S::PQ;
  const int64_t at = (int64_t)w * ws * 3 * dim + h * HD;
  load_rows<T, HD>(x, d_out + (int64_t)w * ws * dim + h * HD, dim, ws);
  load_rows<T, HD>(y, qkv + at + 2 * dim, 3 * dim, ws);
  const float* Pg = P + (int64_t)blockIdx.x * ws * ws;
  for (int r = threadIdx.x >> 5; r < S::ROWS; r += NT / 32)
    for (int c = threadIdx.x & 31; c < ps; c += 32) {
      const bool on = r < ws && c < ws;
      const uint32_t d = (uint32_t)__cvta_generic_to_shared(s + r * ps + c);
      asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(on ? Pg + r * ws + c : Pg), "r"(on ? 4 : 0) : "memory");
    }
  landed();
  {
    float a[T][S::C];
    clear(a);
    weigh_cols<T, HD>(s, ps, x, ws, ty, tx, a);              // dV = P^T dO
    store_rows<T, HD>(d_qkv + at + 2 * dim, 3 * dim, ws, ty, tx, 1.f, a);
  }
  {
    float a[T][T];
    clear(a);
    scores<T, HD>(x, y, ty, tx, a);                          // dP = dO V^T
    __syncthreads();                                         // dV has read all of P, and dO and V are done with
    load_rows<T, HD>(x, qkv + at, 3 * dim, ws);              // Q
    load_rows<T, HD>(y, qkv + at + dim, 3 * dim, ws);        // K
#pragma unroll
    for (int i = 0; i < T; ++i) {
      float p[T], dot = 0.f;
#pragma unroll
      for (int j = 0; j < T; ++j) {
        p[j] = j * 8 + tx < ws ? s[(i * 8 + ty) * ps + j * 8 + tx] : 0.f;
        dot = fmaf(a[i][j], p[j], dot);
      }
#pragma unroll
      for (int o = 1; o < 8; o <<= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
#pragma unroll
      for (int j = 0; j < T; ++j)
        if (j * 8 + tx < ws) s[(i * 8 + ty) * ps + j * 8 + tx] = p[j] * (a[i][j] - dot);     // dS
    }
  }
  landed();
  {
    float a[T][S::C];
    clear(a);
    weigh_rows<T, HD>(s, ps, y, ws, ty, tx, a);              // dQ = scale dS K
    store_rows<T, HD>(d_qkv + at, 3 * dim, ws, ty, tx, scale, a);
  }
  {
    float a[T][S::C];
    clear(a);
    weigh_cols<T, HD>(s, ps, x, ws, ty, tx, a);              // dK = scale dS^T Q
    store_rows<T, HD>(d_qkv + at + dim, 3 * dim, ws, ty, tx, scale, a);
  }
}

struct Call {
  bool backward;
  const float *qkv, *P_in, *d_out;
  float *P, *out, *d_qkv;
  int windows, ws, heads;
  float scale;
};

template <int T, int HD> static prad_status launch(prad_ctx* ctx, const Call& c) {
  const int smem = smem_floats<T, HD>(c.ws, c.backward) * (int)sizeof(float);
  const unsigned grid = (unsigned)(c.windows * c.heads);
  constexpr int most = 100 * 1024;
  prad_status st = c.backward ? allow_smem<backward_kernel<T, HD>>(ctx, most) : allow_smem<forward_kernel<T, HD>>(ctx, most);
  if (st) return st;
  if (c.backward) launch_chained(backward_kernel<T, HD>, grid, NT, smem, ctx->stream, c.qkv, c.P_in, c.d_out, c.d_qkv, c.ws, c.heads, c.scale);
  else launch_chained(forward_kernel<T, HD>, grid, NT, smem, ctx->stream, c.qkv, c.P, c.out, c.ws, c.heads, c.scale);
  PRAD_LAUNCHED(ctx);
  return PRAD_OK;
}
// T = ceil(window / 8), or the next height there is: T = 1, 3 and 6 are not instantiated, so windows of 17 .. 24 and 41 .. 48 tokens
// work on the scores of 32 and 56 (4096 windows, three heads of 32: 62 us forward with 24 tokens, 71 with 32; 186 with 48, 193 with
// 49, 108 with 40).
template <int HD> static prad_status pick(prad_ctx* ctx, const Call& c) {
  const int t = (c.ws + 7) / 8;
  if (t <= 2) return launch<2, HD>(ctx, c);
  if (t <= 4) return launch<4, HD>(ctx, c);
  if (t <= 5) return launch<5, HD>(ctx, c);
  if (t <= 7) return launch<7, HD>(ctx, c);
  return launch<8, HD>(ctx, c);
}
static prad_status run(prad_ctx* ctx, const char* who, prad_dtype dt, int head_dim, const Call& c) {
  PRAD_REQUIRE(c.windows >= 0 && c.ws > 0 && c.heads > 0 && head_dim > 0, PRAD_ERR_SHAPE, "%s: bad shape", who);
  PRAD_REQUIRE(dt == PRAD_F32 && c.ws <= 64 && (head_dim == 16 || head_dim == 32 || head_dim == 64), PRAD_ERR_UNSUPPORTED,
               "%s: float windows of at most 64 tokens with heads of 16, 32 or 64 columns", who);
  PRAD_REQUIRE((int64_t)c.windows * c.heads <= 0x7fffffff, PRAD_ERR_UNSUPPORTED, "%s: too many windows", who);
  if (c.windows == 0) return PRAD_OK;
  return head_dim == 16 ? pick<16>(ctx, c) : head_dim == 32 ? pick<32>(ctx, c) : pick<64>(ctx, c);
}
static bool aligned(const void* p) { return p && ((uintptr_t)p & 15) == 0; }

}  // namespace wa
}  // namespace prad

using namespace prad;

extern "C" prad_status prad_window_attention_forward(prad_ctx* ctx, prad_dtype dt, const void* qkv, void* P, void* out, int windows,
                                                     int window, int heads, int head_dim, double scale) {
  PRAD_CHECK_CTX(ctx);
  PRAD_REQUIRE(windows == 0 || (wa::aligned(qkv) && P && wa::aligned(out)), PRAD_ERR_INVALID,
               "prad_window_attention_forward: null or unaligned pointer");
  wa::Call c{false, (const float*)qkv, nullptr, nullptr, (float*)P, (float*)out, nullptr, windows, window, heads, (float)scale};
  return wa::run(ctx, "prad_window_attention_forward", dt, head_dim, c);
}
extern "C" prad_status prad_window_attention_backward(prad_ctx* ctx, prad_dtype dt, const void* qkv, const void* P, const void* d_out,
                                                      void* d_qkv, int windows, int window, int heads, int head_dim, double scale) {
  PRAD_CHECK_CTX(ctx);
  PRAD_REQUIRE(windows == 0 || (wa::aligned(qkv) && P && wa::aligned(d_out) && wa::aligned(d_qkv)), PRAD_ERR_INVALID,
               "prad_window_attention_backward: null or unaligned pointer");
  wa::Call c{true, (const float*)qkv, (const float*)P, (const float*)d_out, nullptr, nullptr, (float*)d_qkv, windows, window, heads, (float)scale};
  return wa::run(ctx, "prad_window_attention_backward", dt, head_dim, c);
}

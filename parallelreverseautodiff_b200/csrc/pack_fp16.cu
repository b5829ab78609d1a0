// Packing kernels of the FP16-piece operand form (pack_fp16.cuh) and the C ABI around packed operands.
//
// One kernel produces either orientation, or both in a single pass over the source, and the source may
// be an activation evaluated on the fly (forward value, or upstream gradient times derivative): the
// operand of the next product is written where the values are born instead of being stored as FP32,
// read back, searched for its maxima and converted.  All of it is HBM-bound streaming.
//
// A CTA (256 threads = 8 warps) owns a tile of TR rows x TC columns.
//   Pass 1, one tile row per warp and trip: 128-bit loads, the activation, the optional FP32 copy; the
//   row block's maximum is a warp reduction, so the by-rows pieces of that row block are written at
//   once from registers; the values also go to a shared-memory stash (float4 stores) and every thread
//   keeps the running maximum of its columns.
//   Pass 2 (only for the by-columns form): column maxima are combined in shared memory, then each lane
//   takes one column and 32 consecutive k of it from the stash (consecutive lanes read consecutive
//   words: no bank conflicts) and writes one whole 128-byte line of pieces.
// TR is the by-columns block length, TC the by-rows block length.
#include <atomic>
#include <type_traits>

#include "act_math.cuh"
#include "pack_fp16.cuh"

namespace prad {

namespace pk {

__device__ __forceinline__ float pow2f(int e) { return __int_as_float((e + 127) << 23); }

// power-of-two shift that brings a block whose largest |x| has bit pattern `absbits` into [2^14, 2^15)
__device__ __forceinline__ int shift_of(uint32_t absbits) {
  const int e = (int)((absbits >> 23) & 0xffu);
  if (e == 0 || e == 255) return 0;              // all zero / denormal, or Inf / NaN present: unscaled
  const int s = 14 - (e - 127);
  return s > PACK_SHIFT_MAX ? PACK_SHIFT_MAX : (s < PACK_SHIFT_MIN ? PACK_SHIFT_MIN : s);
}
__device__ __forceinline__ void pieces(float xs, __half& p0, __half& p1) {
  p0 = __float2half_rn(xs);
  p1 = __float2half_rn(xs - __half2float(p0));   // the difference is exact in FP32
}
__device__ __forceinline__ uint32_t absbits(float x) { return __float_as_uint(fabsf(x)); }

// the four values at (r, c .. c+3) of the source, zero outside the matrix; writes the FP32 copy
__device__ __forceinline__ void fetch4(const PackSource& s, bool vec, int64_t r, int c, int R, int C, float (&v)[4]) {
  v[0] = v[1] = v[2] = v[3] = 0.f;
  if (r >= R || c >= C) return;
  const int64_t off = r * s.ld + c;
  float a[4] = {0.f, 0.f, 0.f, 0.f}, d[4] = {0.f, 0.f, 0.f, 0.f}, tg[4] = {0.f, 0.f, 0.f, 0.f};
  const bool full = vec && c + 4 <= C;
  if (full) {
    const float4 t = __ldcs(reinterpret_cast<const float4*>(s.x + off));
    a[0] = t.x; a[1] = t.y; a[2] = t.z; a[3] = t.w;
    if (s.kind >= 2) {
      const float4 u = __ldcs(reinterpret_cast<const float4*>(s.dy + off));
      d[0] = u.x; d[1] = u.y; d[2] = u.z; d[3] = u.w;
    }
    if (s.kind == 3) {
      const float4 u = __ldcs(reinterpret_cast<const float4*>(s.target + off));
      tg[0] = u.x; tg[1] = u.y; tg[2] = u.z; tg[3] = u.w;
    }
  } else {
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (c + q < C) {
        a[q] = s.x[off + q];
        if (s.kind >= 2) d[q] = s.dy[off + q];
        if (s.kind == 3) tg[q] = s.target[off + q];
      }
  }
  if (s.kind == 3) {     // MeanSquaredErrorLossOperation.Backward: scale * (output - target)
#pragma unroll
    for (int q = 0; q < 4; ++q) d[q] = mul_rn(s.loss_scale, sub_rn(d[q], tg[q]));
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    if (c + q >= C) continue;
    if (s.kind == 0) v[q] = a[q];
    else if (s.kind == 1) v[q] = act_value<float>((prad_act)s.act, a[q], s.act_alpha);
    else v[q] = mul_rn(d[q], act_derivative<float>((prad_act)s.act, a[q], s.act_alpha));
  }
  if (s.out) {
    if (full) __stcs(reinterpret_cast<float4*>(s.out + off), make_float4(v[0], v[1], v[2], v[3]));
    else {
#pragma unroll
      for (int q = 0; q < 4; ++q) if (c + q < C) s.out[off + q] = v[q];
    }
  }
}

// ---------------------------------------------------------------- fast path: interior 128 x 128 tiles
// The same two passes for tiles that lie completely inside the matrix, with 16-byte aligned operands and
// 128-long blocks: no bounds tests, the operation fixed at compile time, conversions two values at a
// time (cvt.rn.f16x2.f32).  OP: 0 plain; 1 / 2 / 3 forward GELU / LeakyReLU / any activation;
// 4 / 5 / 6 backward likewise; 7 / 8 mean-squared-error gradient times the GELU / any derivative;
// 9 / 10 / 11 are 1 / 4 / 7 (the GELU cases) in short arithmetic, chosen when no FP32 copy is written;
// 12 / 13 LayerNormalization of x / of x + dy, 14 its Backward plus the residual path's gradient (a warp has the whole row).
//
// Short arithmetic: the copy-less result exists only as pieces of 22 significant bits, so the GELU terms
// are contracted into fused multiply-adds and tanh is 1 - 2 / (1 + 2^(2 log2(e) u)) with the hardware's
// exp2 and reciprocal approximations (absolute error about 3e-7, of the order of the pieces' own
// rounding).  With an FP32 copy the arithmetic is the stand-alone activation kernels', operation by
// operation, so that the copy is bit-identical to theirs.
__device__ __forceinline__ void pieces2(float x0, float x1, __half2& p0, __half2& p1) {
  p0 = __floats2half2_rn(x0, x1);
  const float2 b = __half22float2(p0);
  p1 = __floats2half2_rn(x0 - b.x, x1 - b.y);      // the differences are exact in FP32
}
__device__ __forceinline__ float tanh_short(float u) {
  float t, r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(t) : "f"(u * 2.885390081777927f));    // e^(2u); inf / 0 at the ends
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(t + 1.0f));
  return fmaf(-2.0f, r, 1.0f);
}
__device__ __forceinline__ float gelu_inner_short(float x, float x2) {
  return x * fmaf(x2, 0.7978845f * 0.044715f, 0.7978845f);
}
__device__ __forceinline__ float gelu_value_short(float x) {
  const float b = tanh_short(gelu_inner_short(x, x * x));
  return x * fmaf(0.5f, b, 0.5f);
}
__device__ __forceinline__ float gelu_derivative_short(float x) {
  const float x2 = x * x;
  const float b = tanh_short(gelu_inner_short(x, x2));
  const float omb2 = fmaf(-b, b, 1.0f);
  const float d = fmaf(x2, 0.7978845f * (0.044715f * 3.0f), 0.7978845f);
  return fmaf(0.5f * x, fmaf(omb2 * omb2, d, b), fmaf(0.5f, b, 0.5f));
}
template <int OP>
__device__ __forceinline__ float apply_op(const PackSource& s, float a, float d, float tg) {
  if (OP == 0) return a;
  if (OP == 1) return gelu_value<float>(a);
  if (OP == 2) return a > 0.f ? a : mul_rn(s.act_alpha, a);
  if (OP == 3) return act_value<float>((prad_act)s.act, a, s.act_alpha);
  if (OP == 9) return gelu_value_short(a);
  if (OP == 7 || OP == 8 || OP == 11) d = mul_rn(s.loss_scale, sub_rn(d, tg));
  if (OP == 4 || OP == 7) return mul_rn(d, gelu_derivative<float>(a));
  if (OP == 10 || OP == 11) return d * gelu_derivative_short(a);
  if (OP == 5) return mul_rn(d, a > 0.f ? 1.f : s.act_alpha);
  return mul_rn(d, act_derivative<float>((prad_act)s.act, a, s.act_alpha));
}

// Stash: the tile's values as floats, [128 k][128 columns] without padding; the float4 of columns 4q..4q+3
// of tile row k sits in slot q ^ ((k >> 2) & 7) of its row.  Pass 1 stores whole float4 (any permutation of
// slots is conflict-free); in pass 2 a lane reads four consecutive k of one column and the eight lanes that
// share a column quad read eight different slot positions: 32 different banks.
//
// EDGE: tiles that the matrix fills only in part (C is a multiple of four, so whole float4 lie inside or outside): columns
// from C and rows from R on read as zeros, pieces are written up to the padded k of either form and for existing operand rows
// only.
//
// Column sums (a bias gradient) cost the second pass sixteen additions per lane and quad: the values are in shared memory anyway,
// and a pass of their own over a 200704 x 384 gradient takes 72 us.
// The sums over the lanes of U values at once: with two, the halves of the warp take one each after the first exchange, which is
// seven exchanges instead of ten, and two rows' chains run side by side (a LayerNorm pass waits for little else).
template <int U> __device__ __forceinline__ void lane_sums(double (&v)[U]) {
  if constexpr (U == 1) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
  } else {
    const bool high = (threadIdx.x & 16) != 0;
    double t = (high ? v[1] : v[0]) + __shfl_xor_sync(0xffffffffu, high ? v[0] : v[1], 16);
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    v[0] = __shfl_sync(0xffffffffu, t, 0);
    v[1] = __shfl_sync(0xffffffffu, t, 16);
  }
}
// LayerNormalizationOperation.cs:56-85 on U rows whose four values at a column each lane holds
template <int U>
__device__ __forceinline__ void layernorm_rows(float (&v)[U][4], bool inside, int C, float (&mu)[U], float (&sd)[U]) {
  double s[U], t[U];
#pragma unroll
  for (int u = 0; u < U; ++u) s[u] = inside ? ((double)v[u][0] + (double)v[u][1]) + ((double)v[u][2] + (double)v[u][3]) : 0.0;
  lane_sums<U>(s);
#pragma unroll
  for (int u = 0; u < U; ++u) {
    mu[u] = (float)(s[u] / (double)C);
    t[u] = 0.0;
#pragma unroll
    for (int q = 0; q < 4; ++q) { v[u][q] = sub_rn(v[u][q], mu[u]); t[u] += (double)mul_rn(v[u][q], v[u][q]); }
    if (!inside) t[u] = 0.0;
  }
  lane_sums<U>(t);
#pragma unroll
  for (int u = 0; u < U; ++u) {
    sd[u] = sqrt_rn(div_rn((float)t[u], (float)C));
    const float den = add_rn(sd[u], 1e-9f);
#pragma unroll
    for (int q = 0; q < 4; ++q) v[u][q] = div_rn(v[u][q], den);
  }
}
template <int OP, bool ROWS, bool COLS, int NT, bool EDGE>
__global__ void __launch_bounds__(NT, NT == 512 ? 2 : (OP == 0 ? 5 : 3))
pack_fast_kernel(PackSource src, PackedForm fr, PackedForm fc, int tile_r0, int tile_c0, int R, int C) {
  chain_begin();
  constexpr int T = 128, U = OP == 14 ? 1 : 2, NW = NT / 32, NB = T / NW / U;      // NW warps, each takes every NW-th tile row
  constexpr bool HAS_DY = OP >= 4 && OP != 9 && OP != 12, HAS_TG = OP == 7 || OP == 8 || OP == 11 || OP == 14;
  extern __shared__ float stash[];       // [T][T] when COLS
  __shared__ unsigned colmax[T];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rtile = tile_r0 + blockIdx.y;
  const int64_t r0 = (int64_t)rtile * T;
  const int ctile = tile_c0 + blockIdx.x;
  const int c0 = ctile * T, c = c0 + lane * 4;
  const bool inside = !EDGE || c < C;                  // this lane's four columns exist
  if (COLS && threadIdx.x < T) colmax[threadIdx.x] = 0;
  uint32_t cm[4] = {0, 0, 0, 0};
  // pass 1: the loads of the next two tile rows are in flight while the current two are converted
  float4 a[2][U], d[2][U], tg[2][U];
  auto load = [&](int buf, int b) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t r = r0 + warp + NW * (b * U + u), off = r * src.ld + c;
      if (EDGE && (!inside || r >= R)) {
        a[buf][u] = d[buf][u] = tg[buf][u] = make_float4(0.f, 0.f, 0.f, 0.f);
        continue;
      }
      a[buf][u] = __ldcs(reinterpret_cast<const float4*>(src.x + off));
      if (HAS_DY) d[buf][u] = __ldcs(reinterpret_cast<const float4*>(src.dy + off));
      if (HAS_TG) tg[buf][u] = __ldcs(reinterpret_cast<const float4*>(src.target + off));
    }
  };
  load(0, 0);
#pragma unroll
  for (int b = 0; b < NB; ++b) {
    const int cur = b & 1;
    if (b + 1 < NB) load(cur ^ 1, b + 1);
    float v_of[U][4];
    if constexpr (OP == 12 || OP == 13) {
      float mu[U], sd[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int64_t r = r0 + warp + NW * (b * U + u);
        float (&v)[4] = v_of[u];
        v[0] = a[cur][u].x; v[1] = a[cur][u].y; v[2] = a[cur][u].z; v[3] = a[cur][u].w;
        if constexpr (OP == 13) {
          v[0] = add_rn(v[0], d[cur][u].x); v[1] = add_rn(v[1], d[cur][u].y);
          v[2] = add_rn(v[2], d[cur][u].z); v[3] = add_rn(v[3], d[cur][u].w);
          if (inside && (!EDGE || r < R)) __stcs(reinterpret_cast<float4*>(src.out + r * src.ld + c), make_float4(v[0], v[1], v[2], v[3]));
        }
      }
      layernorm_rows<U>(v_of, inside, C, mu, sd);
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int64_t r = r0 + warp + NW * (b * U + u);
        if (lane == 0 && (!EDGE || r < R)) { src.mean[r] = mu[u]; src.sigma[r] = sd[u]; }
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int tr = warp + NW * (b * U + u);
      const int64_t r = r0 + tr;
      const bool row = !EDGE || r < R;
      float (&v)[4] = v_of[u];
      if constexpr (OP == 12 || OP == 13) {
      } else if constexpr (OP == 14) {
        // LayerNormalizationOperation.cs:88-112, then the sum of the two paths
        const float mu = row ? src.mean[r] : 0.f, se = add_rn(row ? src.sigma[r] : 1.f, 1e-9f);
        const float exp1 = mul_rn(sub_rn(1.f, div_rn(1.f, (float)C)), div_rn(1.f, se));
        const float rden = div_rn(1.f, mul_rn((float)C, mul_rn(mul_rn(se, se), se)));      // (as layernorm_backward_flat)
        const float x4[4] = {a[cur][u].x, a[cur][u].y, a[cur][u].z, a[cur][u].w}, d4[4] = {d[cur][u].x, d[cur][u].y, d[cur][u].z, d[cur][u].w};
        const float g4[4] = {tg[cur][u].x, tg[cur][u].y, tg[cur][u].z, tg[cur][u].w};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float t = sub_rn(x4[q], mu);
          v[q] = add_rn(g4[q], mul_rn(d4[q], sub_rn(exp1, mul_rn(mul_rn(t, t), rden))));
        }
      } else {
        v[0] = apply_op<OP>(src, a[cur][u].x, HAS_DY ? d[cur][u].x : 0.f, HAS_TG ? tg[cur][u].x : 0.f);
        v[1] = apply_op<OP>(src, a[cur][u].y, HAS_DY ? d[cur][u].y : 0.f, HAS_TG ? tg[cur][u].y : 0.f);
        v[2] = apply_op<OP>(src, a[cur][u].z, HAS_DY ? d[cur][u].z : 0.f, HAS_TG ? tg[cur][u].z : 0.f);
        v[3] = apply_op<OP>(src, a[cur][u].w, HAS_DY ? d[cur][u].w : 0.f, HAS_TG ? tg[cur][u].w : 0.f);
      }
      if (EDGE && !(inside && row)) v[0] = v[1] = v[2] = v[3] = 0.f;      // an activation of zero need not be zero
      if (((OP >= 1 && OP <= 8) || OP == 14) && src.out && inside && row)
        __stcs(reinterpret_cast<float4*>(src.out + r * src.ld + c), make_float4(v[0], v[1], v[2], v[3]));
      uint32_t m = 0;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const uint32_t bits = absbits(v[q]);
        m = max(m, bits);
        if (COLS) cm[q] = max(cm[q], bits);
      }
      if (COLS)
        *reinterpret_cast<float4*>(&stash[tr * T + ((lane ^ ((tr >> 2) & 7)) << 2)]) = make_float4(v[0], v[1], v[2], v[3]);
      if (ROWS) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
        const int sh = shift_of(m);
        const float scale = pow2f(sh);
        if (lane == 0 && row) fr.blk[(int64_t)ctile * fr.rows_ld + r] = pow2f(-sh);
        __half2 p0[2], p1[2];
        pieces2(v[0] * scale, v[1] * scale, p0[0], p1[0]);
        pieces2(v[2] * scale, v[3] * scale, p0[1], p1[1]);
        __half* dst = fr.h + r * fr.pitch + (int64_t)(c >> 5) * 64 + (c & 31);
        if (!EDGE || (row && c < fr.kp)) {                 // the row is padded with zeros up to kp and ends there
          *reinterpret_cast<uint2*>(dst) = *reinterpret_cast<const uint2*>(p0);
          *reinterpret_cast<uint2*>(dst + 32) = *reinterpret_cast<const uint2*>(p1);
        }
      }
    }
  }
  if (!COLS) return;
  __syncthreads();
#pragma unroll
  for (int q = 0; q < 4; ++q)
    if (cm[q] != 0) atomicMax(&colmax[lane * 4 + q], cm[q]);
  __syncthreads();
  // pass 2: a warp owns 32 / NW quads of columns; per quad and 32-k group, lane (cc, g) converts k 4g..4g+3 of
  // column cc of the quad, and the eight lanes of a column write 64 contiguous bytes of h0 and 64 of h1:
  // whole sectors, four lines per store instruction.
  const int cc = lane & 3, g = lane >> 2;
#pragma unroll 1
  for (int quad = warp * (32 / NW); quad < (warp + 1) * (32 / NW); ++quad) {
    const int tc = quad * 4 + cc;                    // column inside the tile
    if (EDGE && c0 + quad * 4 >= C) break;           // no operand rows from here on (whole quads: C is a multiple of 4)
    const int sh = shift_of(colmax[tc]);
    const float scale = pow2f(sh);
    if (g == 0) fc.blk[(int64_t)rtile * fc.rows_ld + c0 + tc] = pow2f(-sh);
    const float* sp = stash + (4 * g) * T + (((quad ^ g) << 2) | cc);      // (k >> 2) & 7 == g for k = 32 kg + 4g + i
    __half* dst = fc.h + (int64_t)(c0 + tc) * fc.pitch + (r0 >> 5) * 64 + 4 * g;
    double sum = 0.0;
#pragma unroll
    for (int kg = 0; kg < 4; ++kg) {
      const float x0 = sp[(kg * 32) * T], x1 = sp[(kg * 32 + 1) * T], x2 = sp[(kg * 32 + 2) * T], x3 = sp[(kg * 32 + 3) * T];
      if (src.colsum) sum += ((double)x0 + (double)x1) + ((double)x2 + (double)x3);
      if (EDGE && r0 + kg * 32 >= fc.kp) continue;
      __half2 p0[2], p1[2];
      pieces2(x0 * scale, x1 * scale, p0[0], p1[0]);
      pieces2(x2 * scale, x3 * scale, p0[1], p1[1]);
      *reinterpret_cast<uint2*>(dst + kg * 64) = *reinterpret_cast<const uint2*>(p0);
      *reinterpret_cast<uint2*>(dst + kg * 64 + 32) = *reinterpret_cast<const uint2*>(p1);
    }
    if (src.colsum) {
#pragma unroll
      for (int o = 4; o < 32; o <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      if (g == 0) src.colsum[(int64_t)rtile * C + c0 + tc] = sum;
    }
  }
}

// out[c] = sum of the partial column sums, in a fixed order: 32 warps share the rows of 32 columns
__global__ void __launch_bounds__(1024)
column_sum_kernel(const double* __restrict__ part, float* __restrict__ out, int rows, int C) {
  chain_begin();
  __shared__ double sm[32][33];
  constexpr int U = 12;                 // loads in flight per thread: 1568 partial rows are four trips
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, c = blockIdx.x * 32 + lane;
  double acc = 0.0;
  if (c < C)
    for (int r0 = w; r0 < rows; r0 += 32 * U) {
      double v[U];
#pragma unroll
      for (int u = 0; u < U; ++u) v[u] = r0 + 32 * u < rows ? part[(int64_t)(r0 + 32 * u) * C + c] : 0.0;
#pragma unroll
      for (int u = 0; u < U; ++u) acc += v[u];
    }
  sm[w][lane] = acc;
  __syncthreads();
  if (w == 0 && c < C) {
    double t = 0.0;
#pragma unroll
    for (int k = 0; k < 32; ++k) t += sm[k][lane];
    out[c] = (float)t;
  }
}

// R x C matrix: whole tiles, then the last column of tiles, then the last row of tiles
template <int OP, bool ROWS, bool COLS>
static prad_status launch_fast(prad_ctx* ctx, const PackSource& src, const PackedForm& fr, const PackedForm& fc, int R, int C) {
  const unsigned tr = (unsigned)(R / 128), tc = (unsigned)(C / 128), er = R % 128 != 0, ec = C % 128 != 0;
  PRAD_REQUIRE(tr + er <= 65535, PRAD_ERR_UNSUPPORTED, "operand packing: too many row tiles (%u)", tr + er);
  // with a stash (64 KB per tile) two CTAs of 16 warps hide the loads better than three of 8
  constexpr int NT = COLS ? 512 : 256;
  const int smem = COLS ? 128 * 128 * (int)sizeof(float) : 0;
  if (COLS) {
    static std::atomic<uint64_t> done{0};
    const uint64_t bit = 1ull << (ctx->device & 63);
    if (!(done.load(std::memory_order_acquire) & bit)) {
      cudaError_t e = cudaFuncSetAttribute(pack_fast_kernel<OP, ROWS, COLS, NT, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
      if (e == cudaSuccess)
        e = cudaFuncSetAttribute(pack_fast_kernel<OP, ROWS, COLS, NT, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
      if (e != cudaSuccess) {
        (void)cudaGetLastError();
        set_error("operand packing: cannot reserve %d bytes of shared memory: %s", smem, cudaGetErrorString(e));
        return PRAD_ERR_CUDA;
      }
      done.fetch_or(bit, std::memory_order_release);
    }
  }
  auto launch = [&](auto edge, unsigned x, unsigned y, unsigned r0, unsigned c0) -> prad_status {
    if (x == 0 || y == 0) return PRAD_OK;
    launch_chained(pack_fast_kernel<OP, ROWS, COLS, NT, decltype(edge)::value>, dim3(x, y), NT, smem, ctx->stream, src, fr, fc, (int)r0, (int)c0, R, C);
    PRAD_LAUNCHED(ctx);
    return PRAD_OK;
  };
  prad_status s = launch(std::false_type(), tc, tr, 0, 0);
  if (!s) s = launch(std::true_type(), ec, tr, 0, tc);
  if (!s) s = launch(std::true_type(), tc + ec, er, tr, 0);
  return s;
}
template <int OP>
static prad_status launch_fast_forms(prad_ctx* ctx, const PackSource& src, const PackedForm& fr, const PackedForm& fc, int R, int C) {
  if (fr.h && fc.h) return launch_fast<OP, true, true>(ctx, src, fr, fc, R, C);
  if (fr.h) return launch_fast<OP, true, false>(ctx, src, fr, fc, R, C);
  return launch_fast<OP, false, true>(ctx, src, fr, fc, R, C);
}
// which compile-time operation serves this source
static int fast_op_of(const PackSource& s) {
  if (s.kind == 0) return 0;
  if (s.kind == 4) return s.dy ? 13 : 12;
  if (s.kind == 5) return 14;
  const bool gelu = s.act == PRAD_ACT_GELU, leaky = s.act == PRAD_ACT_LEAKY_RELU;
  if (gelu && !s.out) return s.kind == 1 ? 9 : (s.kind == 2 ? 10 : 11);
  if (s.kind == 1) return gelu ? 1 : (leaky ? 2 : 3);
  if (s.kind == 2) return gelu ? 4 : (leaky ? 5 : 6);
  return gelu ? 7 : 8;
}

template <int TR, int TC>
__global__ void __launch_bounds__(256)
pack_tile_kernel(PackSource src, bool vec, int R, int C, PackedForm fr, PackedForm fc) {
  chain_begin();
  constexpr int W = TC / 128;            // float4 per lane and tile row
  constexpr int STRIDE = TC + 4;         // stash pitch in floats (16-byte multiple; see pass 2)
  constexpr int U = 4;                   // tile rows a warp loads before it starts converting
  extern __shared__ float stash[];       // [TR][STRIDE], only with a by-columns form
  __shared__ unsigned colmax[TC];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int r0 = blockIdx.y * TR, c0 = blockIdx.x * TC;
  const bool want_rows = fr.h != nullptr, want_cols = fc.h != nullptr;
  for (int i = threadIdx.x; i < TC; i += 256) colmax[i] = 0;

  uint32_t cm[W][4];
#pragma unroll
  for (int w = 0; w < W; ++w)
#pragma unroll
    for (int q = 0; q < 4; ++q) cm[w][q] = 0;

  // ---------------------------------------------------------------- pass 1
  for (int it0 = 0; it0 < TR / 8; it0 += U) {
    float v[U][W][4];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t r = (int64_t)r0 + warp + 8 * (it0 + u);
#pragma unroll
      for (int w = 0; w < W; ++w) fetch4(src, vec, r, c0 + lane * 4 + 128 * w, R, C, v[u][w]);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int tr = warp + 8 * (it0 + u);
      const int64_t r = (int64_t)r0 + tr;
      uint32_t m = 0;
#pragma unroll
      for (int w = 0; w < W; ++w)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const uint32_t b = absbits(v[u][w][q]);
          m = max(m, b);
          cm[w][q] = max(cm[w][q], b);
        }
      if (want_cols) {
#pragma unroll
        for (int w = 0; w < W; ++w)
          *reinterpret_cast<float4*>(&stash[tr * STRIDE + lane * 4 + 128 * w]) =
              make_float4(v[u][w][0], v[u][w][1], v[u][w][2], v[u][w][3]);
      }
      if (want_rows && r < R) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
        const int sh = shift_of(m);
        const float scale = pow2f(sh);
        if (lane == 0) fr.blk[(int64_t)(c0 / TC) * fr.rows_ld + r] = pow2f(-sh);
        __half* drow = fr.h + r * fr.pitch;
#pragma unroll
        for (int w = 0; w < W; ++w) {
          const int c = c0 + lane * 4 + 128 * w;
          if (c >= fr.kp) continue;                  // beyond the padded row (kp is a multiple of 32 >= C)
          __align__(8) __half p0[4];
          __align__(8) __half p1[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) pieces(v[u][w][q] * scale, p0[q], p1[q]);
          __half* d = drow + (int64_t)(c >> 5) * 64 + (c & 31);
          *reinterpret_cast<uint2*>(d) = *reinterpret_cast<uint2*>(p0);
          *reinterpret_cast<uint2*>(d + 32) = *reinterpret_cast<uint2*>(p1);
        }
      }
    }
  }
  if (!want_cols) return;

  // ---------------------------------------------------------------- pass 2
  __syncthreads();     // colmax cleared by everybody's first statement, stash complete
#pragma unroll
  for (int w = 0; w < W; ++w)
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (cm[w][q] != 0) atomicMax(&colmax[lane * 4 + 128 * w + q], cm[w][q]);
  __syncthreads();
  if (src.colsum && threadIdx.x < TC && c0 + (int)threadIdx.x < C) {
    double t = 0.0;
    for (int r = 0; r < TR; ++r) t += (double)stash[r * STRIDE + threadIdx.x];
    src.colsum[(int64_t)blockIdx.y * C + c0 + threadIdx.x] = t;
  }
  constexpr int CG = TC / 32, KG = TR / 32;
  for (int item = warp; item < CG * KG; item += 8) {
    const int cg = item % CG, kg = item / CG;
    const int col = c0 + cg * 32 + lane;             // operand row of the by-columns form
    const int64_t kbase = (int64_t)r0 + kg * 32;     // first k of this 32-group
    if (col >= C || kbase >= fc.kp) continue;
    const int sh = shift_of(colmax[cg * 32 + lane]);
    const float scale = pow2f(sh);
    if (kg == 0) fc.blk[(int64_t)(r0 / TR) * fc.rows_ld + col] = pow2f(-sh);
    __align__(16) __half p0[32];
    __align__(16) __half p1[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) pieces(stash[(kg * 32 + j) * STRIDE + cg * 32 + lane] * scale, p0[j], p1[j]);
    __half* d = fc.h + (int64_t)col * fc.pitch + (kbase >> 5) * 64;     // one 128-byte line: h0 | h1
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      reinterpret_cast<uint4*>(d)[j] = reinterpret_cast<const uint4*>(p0)[j];
      reinterpret_cast<uint4*>(d + 32)[j] = reinterpret_cast<const uint4*>(p1)[j];
    }
  }
}

// ---------------------------------------------------------------- small plain matrices, one form
// A weight matrix of a narrow layer (96 x 384) is three 128 x 128 tiles: on three CTAs of the kernel above, one round trip to
// memory after another, it took 15 us.  Here a CTA takes one 128-k block of 8 operand rows (by rows: a warp per row) or of
// 32 operand rows (by columns: its lanes are the rows, its warps share the k), every load in flight at once: 4 us.
__global__ void __launch_bounds__(256)
pack_small_rows_kernel(const float* __restrict__ x, int64_t ld, PackedForm f) {
  chain_begin();
  const int lane = threadIdx.x & 31;
  const int64_t r = (int64_t)blockIdx.y * 8 + (threadIdx.x >> 5);
  const int c0 = blockIdx.x * 128 + lane * 4;
  if (r >= f.rows) return;
  float v[4];
  uint32_t m = 0;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    v[q] = c0 + q < f.k ? x[r * ld + c0 + q] : 0.f;
    m = max(m, absbits(v[q]));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
  const int sh = shift_of(m);
  const float scale = pow2f(sh);
  if (lane == 0) f.blk[(int64_t)blockIdx.x * f.rows_ld + r] = pow2f(-sh);
  if (c0 >= f.kp) return;
  __half2 p0[2], p1[2];
  pieces2(v[0] * scale, v[1] * scale, p0[0], p1[0]);
  pieces2(v[2] * scale, v[3] * scale, p0[1], p1[1]);
  __half* d = f.h + r * f.pitch + (int64_t)(c0 >> 5) * 64 + (c0 & 31);
  *reinterpret_cast<uint2*>(d) = *reinterpret_cast<const uint2*>(p0);
  *reinterpret_cast<uint2*>(d + 32) = *reinterpret_cast<const uint2*>(p1);
}
__global__ void __launch_bounds__(256)
pack_small_cols_kernel(const float* __restrict__ x, int64_t ld, PackedForm f) {
  chain_begin();
  __shared__ uint32_t part[8][33];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t r = (int64_t)blockIdx.y * 32 + lane;        // operand row = matrix column
  const int64_t k0 = (int64_t)blockIdx.x * 128 + w * 16;
  float v[16];
  uint32_t m = 0;
#pragma unroll
  for (int q = 0; q < 16; ++q) {
    v[q] = r < f.rows && k0 + q < f.k ? x[(k0 + q) * ld + r] : 0.f;
    m = max(m, absbits(v[q]));
  }
  part[w][lane] = m;
  __syncthreads();
#pragma unroll
  for (int q = 0; q < 8; ++q) m = max(m, part[q][lane]);
  if (r >= f.rows) return;
  const int sh = shift_of(m);
  const float scale = pow2f(sh);
  if (w == 0) f.blk[(int64_t)blockIdx.x * f.rows_ld + r] = pow2f(-sh);
  if (k0 >= f.kp) return;                                   // kp is a multiple of 32
  __half2 p0[8], p1[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) pieces2(v[2 * q] * scale, v[2 * q + 1] * scale, p0[q], p1[q]);
  __half* d = f.h + r * f.pitch + (k0 >> 5) * 64 + (k0 & 31);
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    reinterpret_cast<uint4*>(d)[q] = reinterpret_cast<const uint4*>(p0)[q];
    reinterpret_cast<uint4*>(d + 32)[q] = reinterpret_cast<const uint4*>(p1)[q];
  }
}
static prad_status launch_small(prad_ctx* ctx, const PackSource& src, const PackedForm* by_rows, const PackedForm* by_cols) {
  if (by_rows) {
    launch_chained(pack_small_rows_kernel, dim3((unsigned)by_rows->nchunk, (unsigned)ceil_div(by_rows->rows, 8)), 256, 0, ctx->stream, src.x, src.ld, *by_rows);
    PRAD_LAUNCHED(ctx);
  }
  if (by_cols) {
    launch_chained(pack_small_cols_kernel, dim3((unsigned)by_cols->nchunk, (unsigned)ceil_div(by_cols->rows, 32)), 256, 0, ctx->stream, src.x, src.ld, *by_cols);
    PRAD_LAUNCHED(ctx);
  }
  return PRAD_OK;
}

template <int TR, int TC>
static prad_status launch_pack(prad_ctx* ctx, const PackSource& src, bool vec, int R, int C, const PackedForm& fr,
                               const PackedForm& fc) {
  const int smem = fc.h ? TR * (TC + 4) * (int)sizeof(float) : 0;
  if (smem > 48 * 1024) {
    static std::atomic<uint64_t> done{0};
    const uint64_t bit = 1ull << (ctx->device & 63);
    if (!(done.load(std::memory_order_acquire) & bit)) {
      const cudaError_t e = cudaFuncSetAttribute(pack_tile_kernel<TR, TC>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
      if (e != cudaSuccess) {
        (void)cudaGetLastError();
        set_error("operand packing: cannot reserve %d bytes of shared memory: %s", smem, cudaGetErrorString(e));
        return PRAD_ERR_CUDA;
      }
      done.fetch_or(bit, std::memory_order_release);
    }
  }
  // the tiles cover the padded extents: rows up to the by-columns kp, columns up to the by-rows kp
  const int64_t rows_cover = fc.h ? (fc.kp > R ? fc.kp : R) : R;
  const int64_t cols_cover = fr.h ? (fr.kp > C ? fr.kp : C) : C;
  dim3 grid((unsigned)ceil_div(cols_cover, TC), (unsigned)ceil_div(rows_cover, TR));
  PRAD_REQUIRE(grid.y <= 65535, PRAD_ERR_UNSUPPORTED, "operand packing: too many row tiles (%u)", grid.y);
  launch_chained(pack_tile_kernel<TR, TC>, grid, 256, smem, ctx->stream, src, vec, R, C, fr, fc);
  PRAD_LAUNCHED(ctx);
  return PRAD_OK;
}

}  // namespace pk

prad_status pack_fp16(prad_ctx* ctx, const PackSource& src, int R, int C, const PackedForm* by_rows,
                      const PackedForm* by_cols) {
  if (R <= 0 || C <= 0 || (!by_rows && !by_cols)) return PRAD_OK;
  PackedForm none;
  bool vec = (src.ld % 4 == 0) && (((uintptr_t)src.x & 15) == 0) && (!src.dy || ((uintptr_t)src.dy & 15) == 0) &&
             (!src.out || ((uintptr_t)src.out & 15) == 0) && (!src.target || ((uintptr_t)src.target & 15) == 0);
  if (by_rows) {
    PRAD_REQUIRE(by_rows->rows == R && by_rows->k == C && (by_rows->chunk == 128 || by_rows->chunk == 256), PRAD_ERR_SHAPE,
                 "operand packing: the by-rows form does not fit a %d x %d matrix", R, C);
  }
  if (by_cols) {
    PRAD_REQUIRE(by_cols->rows == C && by_cols->k == R && (by_cols->chunk == 128 || by_cols->chunk == 256), PRAD_ERR_SHAPE,
                 "operand packing: the by-columns form does not fit a %d x %d matrix", R, C);
  }
  const int tc = by_rows ? by_rows->chunk : 128, tr = by_cols ? by_cols->chunk : 128;
  // fewer 128 x 128 tiles than a quarter of the SMs: small CTAs, even at the price of reading the matrix once per form
  if (src.kind == 0 && !src.out && !src.colsum && tr == 128 && tc == 128 && ceil_div(R, 128) * ceil_div(C, 128) * 4 <= ctx->sm_count)
    return pk::launch_small(ctx, src, by_rows, by_cols);
  PRAD_REQUIRE(src.kind < 4 || (tr == 128 && tc == 128), PRAD_ERR_UNSUPPORTED, "operand packing: LayerNormalization needs 128-long blocks");
  if (tr == 256 && tc == 256) {
    // a 256 x 256 tile does not fit in shared memory: one pass per form (the FP32 copy is written by the first)
    PackSource again = src;
    if (src.out) { again = PackSource(); again.kind = 0; again.x = src.out; again.ld = src.ld; again.colsum = src.colsum; }
    PackSource first = src;
    first.colsum = nullptr;
    prad_status s = pk::launch_pack<128, 256>(ctx, first, vec, R, C, *by_rows, none);
    if (s) return s;
    return pk::launch_pack<256, 128>(ctx, again, vec, R, C, none, *by_cols);
  }
  const PackedForm& fr = by_rows ? *by_rows : none;
  const PackedForm& fc = by_cols ? *by_cols : none;
  if (tr == 256) return pk::launch_pack<256, 128>(ctx, src, vec, R, C, fr, fc);
  if (tc == 256) return pk::launch_pack<128, 256>(ctx, src, vec, R, C, fr, fc);
  // 128-long blocks of a matrix in whole float4: the specialised kernel
  if (vec && C % 4 == 0) {
    switch (pk::fast_op_of(src)) {
      case 0: return pk::launch_fast_forms<0>(ctx, src, fr, fc, R, C);
      case 1: return pk::launch_fast_forms<1>(ctx, src, fr, fc, R, C);
      case 2: return pk::launch_fast_forms<2>(ctx, src, fr, fc, R, C);
      case 3: return pk::launch_fast_forms<3>(ctx, src, fr, fc, R, C);
      case 4: return pk::launch_fast_forms<4>(ctx, src, fr, fc, R, C);
      case 5: return pk::launch_fast_forms<5>(ctx, src, fr, fc, R, C);
      case 6: return pk::launch_fast_forms<6>(ctx, src, fr, fc, R, C);
      case 7: return pk::launch_fast_forms<7>(ctx, src, fr, fc, R, C);
      case 8: return pk::launch_fast_forms<8>(ctx, src, fr, fc, R, C);
      case 9: return pk::launch_fast_forms<9>(ctx, src, fr, fc, R, C);
      case 10: return pk::launch_fast_forms<10>(ctx, src, fr, fc, R, C);
      case 12: return pk::launch_fast<12, true, true>(ctx, src, fr, fc, R, C);
      case 13: return pk::launch_fast<13, true, true>(ctx, src, fr, fc, R, C);
      case 14: return pk::launch_fast<14, true, true>(ctx, src, fr, fc, R, C);
      default: return pk::launch_fast_forms<11>(ctx, src, fr, fc, R, C);
    }
  }
  PRAD_REQUIRE(src.kind < 4, PRAD_ERR_UNSUPPORTED, "operand packing: LayerNormalization needs rows of whole, aligned float4 and 128-long blocks");
  return pk::launch_pack<128, 128>(ctx, src, vec, R, C, fr, fc);
}

}  // namespace prad

// ---------------------------------------------------------------- C ABI
struct prad_packed {
  prad_ctx* ctx = nullptr;
  int rows = 0, cols = 0;
  prad::PackedForm by_rows, by_cols;   // h == nullptr when the form was not requested
  bool filled = false;
  float* column_sums = nullptr;        // where the column sums of what is packed go
  uint32_t magic = 0x50414b44u;        // "PAKD"
};

using namespace prad;

namespace prad {
static bool packed_ok(const prad_packed* p) { return p && p->magic == 0x50414b44u && ctx_ok(p->ctx); }
#define PRAD_CHECK_PACKED(p, who)                                                                  \
  PRAD_REQUIRE(prad::packed_ok(p), PRAD_ERR_INVALID, who ": the packed operand is null or destroyed")

static void free_form(prad_ctx* ctx, PackedForm& f) {
  if (f.h) pool_free(ctx, f.h);
  if (f.blk) pool_free(ctx, f.blk);
  f.h = nullptr;
  f.blk = nullptr;
}
static prad_status alloc_form(prad_ctx* ctx, PackedForm& f) {
  prad_status s = pool_alloc(ctx, f.h_bytes() ? f.h_bytes() : 16, (void**)&f.h);
  if (!s) s = pool_alloc(ctx, f.blk_bytes() ? f.blk_bytes() : 16, (void**)&f.blk);
  if (s) {
    free_form(ctx, f);
    return s;
  }
  PRAD_CUDA(cudaMemsetAsync(f.blk, 0, f.blk_bytes(), ctx->stream));     // rows beyond the matrix keep exponent 0
  return PRAD_OK;
}
// block length of a packed object unless the caller names one: 128 (one pass writes both forms from a
// 128 x 128 tile, three CTAs per SM), or 256 when the option "tc_chunk_k" asks for at least that
static int chunk_of(prad_ctx* ctx) { return ctx->tc_chunk_k >= 256 && ctx->tc_chunk_k_set ? 256 : 128; }
}  // namespace prad

extern "C" {

prad_status prad_packed_create(prad_ctx* ctx, int rows, int cols, int forms, int block_rows_form, int block_cols_form,
                               prad_packed** out) {
  PRAD_CHECK_CTX(ctx);
  PRAD_NOT_CAPTURING(ctx, "prad_packed_create");
  PRAD_REQUIRE(out && rows > 0 && cols > 0 && (forms & 3) != 0 && (forms & ~3) == 0, PRAD_ERR_INVALID,
               "prad_packed_create: bad shape, forms must be PRAD_PACK_ROWS, PRAD_PACK_COLS or both");
  auto block_ok = [](int b) { return b == 0 || b == 128 || b == 256; };
  PRAD_REQUIRE(block_ok(block_rows_form) && block_ok(block_cols_form), PRAD_ERR_INVALID,
               "prad_packed_create: a block length is 0 (automatic), 128 or 256");
  prad_packed* p = new prad_packed();
  p->ctx = ctx;
  p->rows = rows;
  p->cols = cols;
  // both forms of one operand get different block lengths when both are wanted, so that one pass can
  // write them (a 256 x 256 tile does not fit in shared memory): the contraction over the batch (by
  // columns) keeps the long blocks
  const int chunk = chunk_of(ctx);
  prad_status s = PRAD_OK;
  if (forms & PRAD_PACK_ROWS) {
    const int b = block_rows_form ? block_rows_form : chunk;
    p->by_rows = packed_form_shape(rows, cols, b);
    s = alloc_form(ctx, p->by_rows);
  }
  if (!s && (forms & PRAD_PACK_COLS)) {
    p->by_cols = packed_form_shape(cols, rows, block_cols_form ? block_cols_form : chunk);
    s = alloc_form(ctx, p->by_cols);
  }
  if (s) {
    free_form(ctx, p->by_rows);
    free_form(ctx, p->by_cols);
    delete p;
    return s;
  }
  *out = p;
  return PRAD_OK;
}

prad_status prad_packed_destroy(prad_packed* p) {
  PRAD_CHECK_PACKED(p, "prad_packed_destroy");
  PRAD_CHECK_CTX(p->ctx);
  PRAD_NOT_CAPTURING(p->ctx, "prad_packed_destroy");
  free_form(p->ctx, p->by_rows);
  free_form(p->ctx, p->by_cols);
  p->magic = 0;
  delete p;
  return PRAD_OK;
}

static prad_status pack_into(prad_packed* p, PackSource src) {
  const int part_rows = p->column_sums ? (int)ceil_div(p->rows, p->by_cols.chunk) : 0;
  if (part_rows) {
    prad_status w = ensure_workspace(p->ctx, (size_t)part_rows * p->cols * sizeof(double));
    if (w) return w;
    src.colsum = (double*)p->ctx->ws;
  }
  prad_status s = pack_fp16(p->ctx, src, p->rows, p->cols, p->by_rows.h ? &p->by_rows : nullptr,
                            p->by_cols.h ? &p->by_cols : nullptr);
  if (s) return s;
  p->filled = true;
  if (part_rows) {
    launch_chained(pk::column_sum_kernel, (unsigned)ceil_div(p->cols, 32), 1024, 0, p->ctx->stream, src.colsum, p->column_sums, part_rows, p->cols);
    PRAD_LAUNCHED(p->ctx);
  }
  return PRAD_OK;
}

prad_status prad_packed_column_sums(prad_packed* p, void* out) {
  PRAD_CHECK_PACKED(p, "prad_packed_column_sums");
  PRAD_REQUIRE(!out || p->by_cols.h, PRAD_ERR_INVALID, "prad_packed_column_sums: the object has no by-columns form");
  p->column_sums = (float*)out;
  return PRAD_OK;
}

prad_status prad_layernorm_pack(prad_packed* p, const void* x, const void* residual, void* sum, void* mean, void* stdv) {
  PRAD_CHECK_PACKED(p, "prad_layernorm_pack");
  PRAD_CHECK_CTX(p->ctx);
  PRAD_REQUIRE(x && mean && stdv && (residual != nullptr) == (sum != nullptr), PRAD_ERR_INVALID, "prad_layernorm_pack: null pointer");
  PRAD_REQUIRE(p->cols <= 128 && p->by_rows.h && p->by_cols.h, PRAD_ERR_UNSUPPORTED,
               "prad_layernorm_pack: rows of at most 128 columns, both forms");
  PackSource src;
  src.kind = 4;
  src.x = (const float*)x;
  src.dy = (const float*)residual;
  src.out = (float*)sum;
  src.mean = (float*)mean;
  src.sigma = (float*)stdv;
  src.ld = p->cols;
  return pack_into(p, src);
}

prad_status prad_layernorm_backward_pack(prad_packed* p, const void* x, const void* mean, const void* stdv, const void* dy,
                                         const void* residual, void* dx) {
  PRAD_CHECK_PACKED(p, "prad_layernorm_backward_pack");
  PRAD_CHECK_CTX(p->ctx);
  PRAD_REQUIRE(x && mean && stdv && dy && residual && dx, PRAD_ERR_INVALID, "prad_layernorm_backward_pack: null pointer");
  PRAD_REQUIRE(p->cols <= 128 && p->by_rows.h && p->by_cols.h, PRAD_ERR_UNSUPPORTED,
               "prad_layernorm_backward_pack: rows of at most 128 columns, both forms");
  PackSource src;
  src.kind = 5;
  src.x = (const float*)x;
  src.dy = (const float*)dy;
  src.target = (const float*)residual;
  src.out = (float*)dx;
  src.mean = const_cast<float*>((const float*)mean);
  src.sigma = const_cast<float*>((const float*)stdv);
  src.ld = p->cols;
  return pack_into(p, src);
}

prad_status prad_pack(prad_packed* p, const void* x, int64_t ld) {
  PRAD_CHECK_PACKED(p, "prad_pack");
  PRAD_CHECK_CTX(p->ctx);
  PRAD_REQUIRE(x && ld >= p->cols, PRAD_ERR_INVALID, "prad_pack: null matrix or a pitch smaller than its row length");
  PackSource src;
  src.kind = 0;
  src.x = (const float*)x;
  src.ld = ld;
  return pack_into(p, src);
}

prad_status prad_act_forward_pack(prad_packed* p, prad_act act, const void* x, void* y, double act_alpha) {
  PRAD_CHECK_PACKED(p, "prad_act_forward_pack");
  PRAD_CHECK_CTX(p->ctx);
  PRAD_REQUIRE(x && act >= PRAD_ACT_NONE && act <= PRAD_ACT_AMPLIFIED_SIGMOID, PRAD_ERR_INVALID,
               "prad_act_forward_pack: null input or unknown activation");
  PackSource src;
  src.kind = act == PRAD_ACT_NONE ? 0 : 1;
  src.x = (const float*)x;
  src.out = (float*)y;
  src.ld = p->cols;
  src.act = (int)act;
  src.act_alpha = (float)act_alpha;
  if (src.kind == 0 && y && y != x) PRAD_CUDA(cudaMemcpyAsync(y, x, (size_t)p->rows * p->cols * sizeof(float), cudaMemcpyDeviceToDevice, p->ctx->stream));
  if (src.kind == 0) src.out = nullptr;
  return pack_into(p, src);
}

prad_status prad_act_backward_pack(prad_packed* p, prad_act act, const void* saved, const void* dy, void* dx,
                                   double act_alpha) {
  PRAD_CHECK_PACKED(p, "prad_act_backward_pack");
  PRAD_CHECK_CTX(p->ctx);
  PRAD_REQUIRE(dy && act >= PRAD_ACT_NONE && act <= PRAD_ACT_AMPLIFIED_SIGMOID && (saved || act == PRAD_ACT_NONE),
               PRAD_ERR_INVALID, "prad_act_backward_pack: null input or unknown activation");
  PackSource src;
  if (act == PRAD_ACT_NONE) {
    src.kind = 0;
    src.x = (const float*)dy;
    if (dx && dx != dy) PRAD_CUDA(cudaMemcpyAsync(dx, dy, (size_t)p->rows * p->cols * sizeof(float), cudaMemcpyDeviceToDevice, p->ctx->stream));
  } else {
    src.kind = 2;
    src.x = (const float*)saved;
    src.dy = (const float*)dy;
    src.out = (float*)dx;
  }
  src.ld = p->cols;
  src.act = (int)act;
  src.act_alpha = (float)act_alpha;
  return pack_into(p, src);
}

prad_status prad_mse_act_backward_pack(prad_packed* p, prad_act act, const void* saved, const void* output, const void* target,
                                       int64_t rows_total, void* dx, double act_alpha) {
  PRAD_CHECK_PACKED(p, "prad_mse_act_backward_pack");
  PRAD_CHECK_CTX(p->ctx);
  PRAD_REQUIRE(output && target && rows_total >= 1 && act >= PRAD_ACT_NONE && act <= PRAD_ACT_AMPLIFIED_SIGMOID &&
                   (saved || act == PRAD_ACT_NONE),
               PRAD_ERR_INVALID, "prad_mse_act_backward_pack: null input, bad row count or unknown activation");
  PackSource src;
  src.kind = 3;
  src.x = (const float*)(act == PRAD_ACT_NONE ? output : saved);   // any readable tensor when there is no activation
  src.dy = (const float*)output;
  src.target = (const float*)target;
  src.loss_scale = 2.0f / (float)(rows_total * p->cols);
  src.out = (float*)dx;
  src.ld = p->cols;
  src.act = (int)act;
  src.act_alpha = (float)act_alpha;
  return pack_into(p, src);
}

prad_status prad_gemm_packed(prad_ctx* ctx, const prad_packed* A, int form_a, const prad_packed* B, int form_b,
                             double alpha, double beta, void* C, int64_t ldc, const void* bias) {
  PRAD_CHECK_CTX(ctx);
  PRAD_CHECK_PACKED(A, "prad_gemm_packed");
  PRAD_CHECK_PACKED(B, "prad_gemm_packed");
  PRAD_REQUIRE(A->ctx == ctx && B->ctx == ctx, PRAD_ERR_INVALID, "prad_gemm_packed: an operand belongs to another context");
  PRAD_REQUIRE((form_a == PRAD_PACK_ROWS || form_a == PRAD_PACK_COLS) && (form_b == PRAD_PACK_ROWS || form_b == PRAD_PACK_COLS),
               PRAD_ERR_INVALID, "prad_gemm_packed: a form is PRAD_PACK_ROWS or PRAD_PACK_COLS");
  const PackedForm& a = form_a == PRAD_PACK_ROWS ? A->by_rows : A->by_cols;
  const PackedForm& b = form_b == PRAD_PACK_ROWS ? B->by_rows : B->by_cols;
  PRAD_REQUIRE(a.h && b.h, PRAD_ERR_INVALID, "prad_gemm_packed: the operand was created without the requested form");
  PRAD_REQUIRE(A->filled && B->filled, PRAD_ERR_INVALID, "prad_gemm_packed: an operand has not been packed yet");
  PRAD_REQUIRE(a.k == b.k, PRAD_ERR_SHAPE, "Input 1 columns do not match Input 2 rows");
  PRAD_REQUIRE(a.chunk == b.chunk, PRAD_ERR_SHAPE,
               "prad_gemm_packed: the operands were packed with different block lengths (%d and %d)", a.chunk, b.chunk);
  PRAD_REQUIRE(C && ldc >= b.rows, PRAD_ERR_INVALID, "prad_gemm_packed: null result or a pitch smaller than its row length");
  return gemm_fp16x3_packed(ctx, a, b, (float)alpha, (float)beta, (float*)C, ldc, (const float*)bias);
}

prad_status prad_packed_shape(const prad_packed* p, int* rows, int* cols, int* forms, int* chunk_rows_form,
                              int* chunk_cols_form) {
  PRAD_CHECK_PACKED(p, "prad_packed_shape");
  if (rows) *rows = p->rows;
  if (cols) *cols = p->cols;
  if (forms) *forms = (p->by_rows.h ? PRAD_PACK_ROWS : 0) | (p->by_cols.h ? PRAD_PACK_COLS : 0);
  if (chunk_rows_form) *chunk_rows_form = p->by_rows.chunk;
  if (chunk_cols_form) *chunk_cols_form = p->by_cols.chunk;
  return PRAD_OK;
}

}  // extern "C"

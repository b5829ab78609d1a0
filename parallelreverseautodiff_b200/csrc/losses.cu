// Loss values and loss gradients (MSE, categorical cross-entropy), Swish, SwigLU and BatchNormalization.
// (Compiled with -fmad=false.)
#include "act_math.cuh"
#include "common.cuh"
#include "reduce.cuh"

namespace prad {

template <typename T> struct Eps15;
template <> struct Eps15<float> { __device__ static float v() { return 1e-15f; } };   // lite PradTools.Epsilon
template <> struct Eps15<double> { __device__ static double v() { return 1e-15; } };  // PradTools.Epsilon

constexpr int LOSS_THREADS = 256;

// kind 0: MSE term (o-t)^2 (MeanSquaredErrorLossOperation.cs:50-55)
// kind 1: CCE term -t*log(o+eps) (CategoricalCrossEntropyLossOperation.cs:53-59)
template <typename T> __device__ __forceinline__ T loss_term(T o, T t, int kind) {
  if (kind == 0) {
    const T d = sub_rn(o, t);
    return mul_rn(d, d);
  }
  return mul_rn(-t, t_log(add_rn(o, Eps15<T>::v())));
}
template <typename T>
__global__ void __launch_bounds__(LOSS_THREADS)
loss_partial_kernel(const T* __restrict__ o, const T* __restrict__ t, double* __restrict__ partial,
                    int64_t n, int kind) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  double acc = 0.0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    acc += (double)loss_term<T>(o[i], t[i], kind);
  }
  double s = block_sum_d<LOSS_THREADS>(acc);
  if (threadIdx.x == 0) partial[blockIdx.x] = s;
}
// A small loss in one launch: one CTA adds every term.
constexpr int LOSS_SMALL_THREADS = 1024, LOSS_SMALL = 16 * LOSS_SMALL_THREADS;
template <typename T>
__global__ void __launch_bounds__(LOSS_SMALL_THREADS)
loss_small_kernel(const T* __restrict__ o, const T* __restrict__ t, T* loss, int n, int kind, T divisor) {
  chain_begin();
  double acc = 0.0;
  for (int i = threadIdx.x; i < n; i += LOSS_SMALL_THREADS) acc += (double)loss_term<T>(o[i], t[i], kind);
  const double s = block_sum_d<LOSS_SMALL_THREADS>(acc);
  if (threadIdx.x == 0) loss[0] = div_rn((T)s, divisor);
}
template <typename T>
__global__ void loss_final_kernel(const double* __restrict__ partial, int nblocks, T* loss,
                                  T divisor) {
  if (threadIdx.x == 0 && blockIdx.x == 0) {
    double s = 0.0;
    for (int b = 0; b < nblocks; ++b) s += partial[b];
    loss[0] = div_rn((T)s, divisor);
  }
}

// MeanSquaredErrorLossOperation.cs:71-78: grad = (2/(R*C)) * (o - t)
template <typename T>
__global__ void __launch_bounds__(256)
mse_backward_kernel(const T* __restrict__ o, const T* __restrict__ t, T* __restrict__ g, int64_t n,
                    T scale) {
  chain_begin();
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
    g[i] = mul_rn(scale, sub_rn(o[i], t[i]));
}
// CategoricalCrossEntropyLossOperation.cs:72-83: grad = -scale*y / (yHat + eps)
template <typename T>
__global__ void __launch_bounds__(256)
cce_backward_kernel(const T* __restrict__ o, const T* __restrict__ t, T* __restrict__ g, int64_t n,
                    T scale) {
  chain_begin();
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
    g[i] = div_rn(mul_rn(-scale, t[i]), add_rn(o[i], Eps15<T>::v()));
}

template <typename T>
static prad_status loss_forward_t(prad_ctx* ctx, const void* o, const void* t, void* loss,
                                  int64_t rows, int cols, int kind) {
  int64_t n = rows * cols;
  const T divisor = kind == 0 ? (T)(rows * cols) : (T)rows;
  if (n <= LOSS_SMALL) {
    launch_chained(loss_small_kernel<T>, 1, LOSS_SMALL_THREADS, 0, ctx->stream, (const T*)o, (const T*)t, (T*)loss, (int)n, kind, divisor);
    PRAD_LAUNCHED(ctx);
    return PRAD_OK;
  }
  int grid = stream_grid(ctx, n, LOSS_THREADS * 4, 4);
  prad_status s = ensure_workspace(ctx, (size_t)grid * sizeof(double));
  if (s) return s;
  loss_partial_kernel<T><<<grid, LOSS_THREADS, 0, ctx->stream>>>((const T*)o, (const T*)t,
                                                                  (double*)ctx->ws, n, kind);
  PRAD_LAUNCHED(ctx);
  loss_final_kernel<T><<<1, 32, 0, ctx->stream>>>((const double*)ctx->ws, grid, (T*)loss, divisor);
  PRAD_LAUNCHED(ctx);
  return PRAD_OK;
}

// ---------------------------------------------------------------- Swish
// SwishOperation.cs:41-107: y = x * sigmoid(beta x) with beta a [1 x 1] weight; the managed code
// computes in double whatever the storage type and stores back.  The backward is the one written
// there: dx = dy * sigmoid * ((1 + beta x) * (1 - sigmoid)); dBeta = sum dy * (x s (1 - s) - x^2 s^2).
template <typename T>
__global__ void __launch_bounds__(LOSS_THREADS)
swish_forward_kernel(const T* __restrict__ x, const T* __restrict__ beta, T* __restrict__ y, int64_t n) {
  const double b = (double)beta[0];
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    const double xv = (double)x[i];
    const double sig = __ddiv_rn(1.0, __dadd_rn(1.0, exp(__dmul_rn(-b, xv))));
    y[i] = (T)__dmul_rn(xv, sig);
  }
}
template <typename T>
__global__ void __launch_bounds__(LOSS_THREADS)
swish_backward_kernel(const T* __restrict__ x, const T* __restrict__ beta, const T* __restrict__ dy,
                      T* __restrict__ dx, double* __restrict__ partial, int64_t n) {
  const double b = (double)beta[0];
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  double acc = 0.0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    const double xv = (double)x[i], d = (double)dy[i];
    const double sig = __ddiv_rn(1.0, __dadd_rn(1.0, exp(__dmul_rn(-b, xv))));
    const double om = __dsub_rn(1.0, sig);
    dx[i] = (T)__dmul_rn(d, __dmul_rn(sig, __dmul_rn(__dadd_rn(1.0, __dmul_rn(b, xv)), om)));
    const double wrt = __dsub_rn(__dmul_rn(xv, __dmul_rn(sig, om)), __dmul_rn(__dmul_rn(xv, xv), __dmul_rn(sig, sig)));
    acc += (double)(T)__dmul_rn(d, wrt);      // each term is rounded to T before it is added, as there
  }
  double s = block_sum_d<LOSS_THREADS>(acc);
  if (threadIdx.x == 0) partial[blockIdx.x] = s;
}
template <typename T>
__global__ void swish_final_kernel(const double* __restrict__ partial, int nblocks, T* dbeta, int accumulate) {
  if (threadIdx.x == 0 && blockIdx.x == 0) {
    double s = 0.0;
    for (int b = 0; b < nblocks; ++b) s += partial[b];
    dbeta[0] = accumulate ? add_rn(dbeta[0], (T)s) : (T)s;
  }
}

template <typename T>
static prad_status swish_backward_t(prad_ctx* ctx, const void* x, const void* beta, const void* dy, void* dx,
                                    void* dbeta, int64_t n, int accumulate) {
  int grid = stream_grid(ctx, n, LOSS_THREADS * 4, 4);
  prad_status s = ensure_workspace(ctx, (size_t)grid * sizeof(double));
  if (s) return s;
  swish_backward_kernel<T><<<grid, LOSS_THREADS, 0, ctx->stream>>>((const T*)x, (const T*)beta, (const T*)dy,
                                                                    (T*)dx, (double*)ctx->ws, n);
  PRAD_LAUNCHED(ctx);
  swish_final_kernel<T><<<1, 32, 0, ctx->stream>>>((const double*)ctx->ws, grid, (T*)dbeta, accumulate);
  PRAD_LAUNCHED(ctx);
  return PRAD_OK;
}

// ---------------------------------------------------------------- SwigLU
// SwigLUOperation.cs:59-145: y = swish(x w_j + b_j) * (x v_j + c_j) with per-column w, v, b, c and
// the constructor's scalar beta; double arithmetic throughout, as there.  Backward as written:
// der = swish + beta * sigmoid * (1 - swish); the four per-column sums run over the rows.
// One thread per column and band of rows (consecutive threads = consecutive columns, so a row
// segment is read contiguously); bands are added in band order by the second kernel.
struct SwigLUParams { const void *w, *v, *b, *c; double beta; };

template <typename T>
__global__ void __launch_bounds__(128)
swiglu_forward_kernel(const T* __restrict__ x, SwigLUParams p, T* __restrict__ y, int64_t rows, int cols,
                      int64_t rows_per_band) {
  const int j = blockIdx.x * 128 + threadIdx.x;
  if (j >= cols) return;
  const double w = (double)((const T*)p.w)[j], v = (double)((const T*)p.v)[j];
  const double b = (double)((const T*)p.b)[j], c = (double)((const T*)p.c)[j];
  const int64_t r1 = min(rows, (int64_t)(blockIdx.y + 1) * rows_per_band);
  for (int64_t i = (int64_t)blockIdx.y * rows_per_band; i < r1; ++i) {
    const double xv = (double)x[i * cols + j];
    const double f = __dadd_rn(__dmul_rn(xv, w), b);
    const double swish = __dmul_rn(f, __ddiv_rn(1.0, __dadd_rn(1.0, exp(__dmul_rn(-p.beta, f)))));
    y[i * cols + j] = (T)__dmul_rn(swish, __dadd_rn(__dmul_rn(xv, v), c));
  }
}
template <typename T>
__global__ void __launch_bounds__(128)
swiglu_backward_kernel(const T* __restrict__ x, SwigLUParams p, const T* __restrict__ dy, T* __restrict__ dx,
                       double* __restrict__ partial, int64_t rows, int cols, int64_t rows_per_band) {
  const int j = blockIdx.x * 128 + threadIdx.x;
  if (j >= cols) return;
  const double w = (double)((const T*)p.w)[j], v = (double)((const T*)p.v)[j];
  const double b = (double)((const T*)p.b)[j], c = (double)((const T*)p.c)[j];
  const int64_t r1 = min(rows, (int64_t)(blockIdx.y + 1) * rows_per_band);
  double s_w = 0.0, s_v = 0.0, s_b = 0.0, s_c = 0.0;
  for (int64_t i = (int64_t)blockIdx.y * rows_per_band; i < r1; ++i) {
    const double xv = (double)x[i * cols + j], d = (double)dy[i * cols + j];
    const double f = __dadd_rn(__dmul_rn(xv, w), b);
    const double sig = __ddiv_rn(1.0, __dadd_rn(1.0, exp(__dmul_rn(-p.beta, f))));
    const double swish = __dmul_rn(f, sig);
    const double der = __dadd_rn(swish, __dmul_rn(__dmul_rn(p.beta, sig), __dsub_rn(1.0, swish)));
    const double lin = __dadd_rn(__dmul_rn(xv, v), c);
    dx[i * cols + j] = (T)__dmul_rn(d, __dmul_rn(v, der));
    s_w = __dadd_rn(s_w, __dmul_rn(d, __dmul_rn(__dmul_rn(xv, der), lin)));
    s_v = __dadd_rn(s_v, __dmul_rn(d, __dmul_rn(swish, xv)));
    s_b = __dadd_rn(s_b, __dmul_rn(d, __dmul_rn(der, lin)));
    s_c = __dadd_rn(s_c, __dmul_rn(d, swish));
  }
  double* out = partial + ((int64_t)blockIdx.y * 4) * cols + j;
  out[0] = s_w; out[cols] = s_v; out[2 * (int64_t)cols] = s_b; out[3 * (int64_t)cols] = s_c;
}
template <typename T>
__global__ void __launch_bounds__(128)
swiglu_final_kernel(const double* __restrict__ partial, int bands, int cols, T* dw, T* dv, T* db, T* dc) {
  const int j = blockIdx.x * 128 + threadIdx.x;
  if (j >= cols) return;
  double s[4] = {0.0, 0.0, 0.0, 0.0};
  for (int band = 0; band < bands; ++band)
#pragma unroll
    for (int q = 0; q < 4; ++q) s[q] = __dadd_rn(s[q], partial[((int64_t)band * 4 + q) * cols + j]);
  dw[j] = (T)s[0]; dv[j] = (T)s[1]; db[j] = (T)s[2]; dc[j] = (T)s[3];
}

static int swiglu_bands(const prad_ctx* ctx, int64_t rows, int cols) {
  const int64_t col_blocks = ceil_div(cols, 128);
  int64_t bands = ceil_div((int64_t)ctx->sm_count * 8, col_blocks);
  if (bands > ceil_div(rows, 16)) bands = ceil_div(rows, 16);   // at least 16 rows per band
  return (int)(bands < 1 ? 1 : bands);
}

// ---------------------------------------------------------------- BatchNormalization
// BatchNormalizationOperation.cs:52-158, as written: one population over the whole matrix; the
// variance loop and the normalisation use the SUM S of the elements and the sum V of squared
// deviations from S (the local variables at that point), while the fields read by the backward
// are S / n and V / n.  Everything in double.  stats (device, 4 doubles) = { S/n, V/n, S, V }.
template <typename T>
__global__ void __launch_bounds__(LOSS_THREADS)
bn_partial_kernel(const T* __restrict__ x, const double* __restrict__ stats, double* __restrict__ partial,
                  int64_t n, int second) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  const double S = second ? stats[2] : 0.0;
  double acc = 0.0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    const double v = (double)x[i];
    if (second) { const double d = __dsub_rn(v, S); acc += __dmul_rn(d, d); }
    else acc += v;
  }
  double s = block_sum_d<LOSS_THREADS>(acc);
  if (threadIdx.x == 0) partial[blockIdx.x] = s;
}
__global__ void bn_final_kernel(const double* __restrict__ partial, int nblocks, double* stats, double n, int second) {
  if (threadIdx.x == 0 && blockIdx.x == 0) {
    double s = 0.0;
    for (int b = 0; b < nblocks; ++b) s += partial[b];
    stats[second ? 3 : 2] = s;
    stats[second ? 1 : 0] = s / n;
  }
}
template <typename T>
__global__ void __launch_bounds__(LOSS_THREADS)
bn_forward_kernel(const T* __restrict__ x, const double* __restrict__ stats, T* __restrict__ y, int64_t n) {
  const double S = stats[2], den = sqrt(__dadd_rn(stats[3], 1E-6));
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
    y[i] = (T)__ddiv_rn(__dsub_rn((double)x[i], S), den);
}
template <typename T>
__global__ void __launch_bounds__(LOSS_THREADS)
bn_backward_kernel(const T* __restrict__ x, const double* __restrict__ stats, const T* __restrict__ dy,
                   T* __restrict__ dx, int64_t n) {
  const double mean = stats[0], nn = (double)n;
  const double inv = __ddiv_rn(1.0, sqrt(__dadd_rn(stats[1], 1E-6)));
  const double inv3 = __dmul_rn(__dmul_rn(inv, inv), inv);
  const double dy_dmean = __ddiv_rn(-inv, nn);
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    const double xm = __dsub_rn((double)x[i], mean);
    const double dy_dvar = __dmul_rn(__dmul_rn(-0.5, xm), inv3);
    const double dvar_dx = __ddiv_rn(__dmul_rn(2.0, xm), nn);
    dx[i] = (T)__dmul_rn(__dadd_rn(__dadd_rn(inv, __dmul_rn(dy_dvar, dvar_dx)), dy_dmean), (double)dy[i]);
  }
}

}  // namespace prad

using namespace prad;

extern "C" {

prad_status prad_mse_forward(prad_ctx* ctx, prad_dtype dt, const void* out, const void* target,
                             void* loss_out, int64_t rows, int cols) {
  PRAD_CHECK_CTX(ctx);
  PRAD_REQUIRE(dtype_ok(dt) && rows > 0 && cols > 0 && out && target && loss_out, PRAD_ERR_INVALID,
               "prad_mse_forward: bad argument");
  return dt == PRAD_F32 ? loss_forward_t<float>(ctx, out, target, loss_out, rows, cols, 0)
                        : loss_forward_t<double>(ctx, out, target, loss_out, rows, cols, 0);
}

prad_status prad_cce_forward(prad_ctx* ctx, prad_dtype dt, const void* out, const void* target,
                             void* loss_out, int64_t rows, int cols) {
  PRAD_CHECK_CTX(ctx);
  PRAD_REQUIRE(dtype_ok(dt) && rows > 0 && cols > 0 && out && target && loss_out, PRAD_ERR_INVALID,
               "prad_cce_forward: bad argument");
  return dt == PRAD_F32 ? loss_forward_t<float>(ctx, out, target, loss_out, rows, cols, 1)
                        : loss_forward_t<double>(ctx, out, target, loss_out, rows, cols, 1);
}

prad_status prad_mse_backward(prad_ctx* ctx, prad_dtype dt, const void* out, const void* target,
                              void* grad, int64_t rows, int cols, int64_t rows_total) {
  PRAD_CHECK_CTX(ctx);
  PRAD_REQUIRE(dtype_ok(dt) && rows >= 0 && cols >= 0 && rows_total >= 1, PRAD_ERR_INVALID,
               "prad_mse_backward: bad argument");
  int64_t n = rows * cols;
  if (n == 0) return PRAD_OK;
  PRAD_REQUIRE(out && target && grad, PRAD_ERR_INVALID, "prad_mse_backward: null pointer");
  int grid = stream_grid(ctx, n, 256 * 4, 8);
  if (dt == PRAD_F32)
    launch_chained(mse_backward_kernel<float>, grid, 256, 0, ctx->stream, (const float*)out, (const float*)target, (float*)grad, n, 2.0f / (float)(rows_total * cols));
  else
    launch_chained(mse_backward_kernel<double>, grid, 256, 0, ctx->stream, (const double*)out, (const double*)target, (double*)grad, n, 2.0 / (double)(rows_total * cols));
  PRAD_LAUNCHED(ctx);
  return PRAD_OK;
}

prad_status prad_cce_backward(prad_ctx* ctx, prad_dtype dt, const void* out, const void* target,
                              void* grad, int64_t rows, int cols, int64_t rows_total) {
  PRAD_CHECK_CTX(ctx);
  PRAD_REQUIRE(dtype_ok(dt) && rows >= 0 && cols >= 0 && rows_total >= 1, PRAD_ERR_INVALID,
               "prad_cce_backward: bad argument");
  int64_t n = rows * cols;
  if (n == 0) return PRAD_OK;
  PRAD_REQUIRE(out && target && grad, PRAD_ERR_INVALID, "prad_cce_backward: null pointer");
  int grid = stream_grid(ctx, n, 256 * 4, 8);
  if (dt == PRAD_F32)
    launch_chained(cce_backward_kernel<float>, grid, 256, 0, ctx->stream, (const float*)out, (const float*)target, (float*)grad, n, 1.0f / (float)rows_total);
  else
    launch_chained(cce_backward_kernel<double>, grid, 256, 0, ctx->stream, (const double*)out, (const double*)target, (double*)grad, n, 1.0 / (double)rows_total);
  PRAD_LAUNCHED(ctx);
  return PRAD_OK;
}

prad_status prad_swish_forward(prad_ctx* ctx, prad_dtype dt, const void* x, const void* beta, void* y, int64_t n) {
  PRAD_CHECK_CTX(ctx);
  PRAD_REQUIRE(dtype_ok(dt) && n >= 0 && (n == 0 || (x && beta && y)), PRAD_ERR_INVALID,
               "prad_swish_forward: bad dtype, null pointer or negative size");
  if (n == 0) return PRAD_OK;
  const int grid = stream_grid(ctx, n, LOSS_THREADS * 4, 4);
  if (dt == PRAD_F32) swish_forward_kernel<float><<<grid, LOSS_THREADS, 0, ctx->stream>>>((const float*)x, (const float*)beta, (float*)y, n);
  else swish_forward_kernel<double><<<grid, LOSS_THREADS, 0, ctx->stream>>>((const double*)x, (const double*)beta, (double*)y, n);
  PRAD_LAUNCHED(ctx);
  return PRAD_OK;
}

prad_status prad_swish_backward(prad_ctx* ctx, prad_dtype dt, const void* x, const void* beta, const void* dy,
                                void* dx, void* dbeta, int64_t n, int accumulate) {
  PRAD_CHECK_CTX(ctx);
  PRAD_REQUIRE(dtype_ok(dt) && n >= 0 && beta && dbeta && (n == 0 || (x && dy && dx)), PRAD_ERR_INVALID,
               "prad_swish_backward: bad dtype, null pointer or negative size");
  return dt == PRAD_F32 ? swish_backward_t<float>(ctx, x, beta, dy, dx, dbeta, n, accumulate)
                        : swish_backward_t<double>(ctx, x, beta, dy, dx, dbeta, n, accumulate);
}

prad_status prad_swiglu_forward(prad_ctx* ctx, prad_dtype dt, const void* x, const void* w, const void* v,
                                const void* b, const void* c, double beta, void* y, int64_t rows, int cols) {
  PRAD_CHECK_CTX(ctx);
  PRAD_REQUIRE(dtype_ok(dt) && rows >= 0 && cols >= 0, PRAD_ERR_INVALID, "prad_swiglu_forward: bad argument");
  if (rows == 0 || cols == 0) return PRAD_OK;
  PRAD_REQUIRE(x && w && v && b && c && y, PRAD_ERR_INVALID, "prad_swiglu_forward: null pointer");
  int bands = swiglu_bands(ctx, rows, cols);
  const int64_t rpb = ceil_div(rows, bands);
  bands = (int)ceil_div(rows, rpb);
  const dim3 grid((unsigned)ceil_div(cols, 128), (unsigned)bands);
  SwigLUParams p{w, v, b, c, beta};
  if (dt == PRAD_F32) swiglu_forward_kernel<float><<<grid, 128, 0, ctx->stream>>>((const float*)x, p, (float*)y, rows, cols, rpb);
  else swiglu_forward_kernel<double><<<grid, 128, 0, ctx->stream>>>((const double*)x, p, (double*)y, rows, cols, rpb);
  PRAD_LAUNCHED(ctx);
  return PRAD_OK;
}

prad_status prad_swiglu_backward(prad_ctx* ctx, prad_dtype dt, const void* x, const void* w, const void* v,
                                 const void* b, const void* c, double beta, const void* dy, void* dx, void* dw,
                                 void* dv, void* db, void* dc, int64_t rows, int cols) {
  PRAD_CHECK_CTX(ctx);
  PRAD_REQUIRE(dtype_ok(dt) && rows >= 0 && cols >= 0, PRAD_ERR_INVALID, "prad_swiglu_backward: bad argument");
  if (cols == 0) return PRAD_OK;
  PRAD_REQUIRE(w && v && b && c && dw && dv && db && dc && (rows == 0 || (x && dy && dx)), PRAD_ERR_INVALID,
               "prad_swiglu_backward: null pointer");
  int bands = rows == 0 ? 0 : swiglu_bands(ctx, rows, cols);
  const int64_t rpb = bands ? ceil_div(rows, bands) : 1;
  bands = (int)ceil_div(rows, rpb);
  prad_status st = ensure_workspace(ctx, (size_t)(bands ? bands : 1) * 4 * cols * sizeof(double));
  if (st) return st;
  SwigLUParams p{w, v, b, c, beta};
  const unsigned cb = (unsigned)ceil_div(cols, 128);
  if (bands) {
    const dim3 grid(cb, (unsigned)bands);
    if (dt == PRAD_F32) swiglu_backward_kernel<float><<<grid, 128, 0, ctx->stream>>>((const float*)x, p, (const float*)dy, (float*)dx, (double*)ctx->ws, rows, cols, rpb);
    else swiglu_backward_kernel<double><<<grid, 128, 0, ctx->stream>>>((const double*)x, p, (const double*)dy, (double*)dx, (double*)ctx->ws, rows, cols, rpb);
    PRAD_LAUNCHED(ctx);
  }
  if (dt == PRAD_F32) swiglu_final_kernel<float><<<cb, 128, 0, ctx->stream>>>((const double*)ctx->ws, bands, cols, (float*)dw, (float*)dv, (float*)db, (float*)dc);
  else swiglu_final_kernel<double><<<cb, 128, 0, ctx->stream>>>((const double*)ctx->ws, bands, cols, (double*)dw, (double*)dv, (double*)db, (double*)dc);
  PRAD_LAUNCHED(ctx);
  return PRAD_OK;
}

prad_status prad_batchnorm_forward(prad_ctx* ctx, prad_dtype dt, const void* x, void* y, void* stats, int64_t rows,
                                   int cols) {
  PRAD_CHECK_CTX(ctx);
  PRAD_REQUIRE(dtype_ok(dt) && rows >= 0 && cols >= 0, PRAD_ERR_INVALID, "prad_batchnorm_forward: bad argument");
  const int64_t n = rows * cols;
  if (n == 0) return PRAD_OK;
  PRAD_REQUIRE(x && y && stats, PRAD_ERR_INVALID, "prad_batchnorm_forward: null pointer");
  const int grid = stream_grid(ctx, n, LOSS_THREADS * 4, 4);
  prad_status st = ensure_workspace(ctx, (size_t)grid * sizeof(double));
  if (st) return st;
  double* part = (double*)ctx->ws;
  double* sd = (double*)stats;
  for (int second = 0; second < 2; ++second) {
    if (dt == PRAD_F32) bn_partial_kernel<float><<<grid, LOSS_THREADS, 0, ctx->stream>>>((const float*)x, sd, part, n, second);
    else bn_partial_kernel<double><<<grid, LOSS_THREADS, 0, ctx->stream>>>((const double*)x, sd, part, n, second);
    PRAD_LAUNCHED(ctx);
    bn_final_kernel<<<1, 32, 0, ctx->stream>>>(part, grid, sd, (double)n, second);
    PRAD_LAUNCHED(ctx);
  }
  if (dt == PRAD_F32) bn_forward_kernel<float><<<grid, LOSS_THREADS, 0, ctx->stream>>>((const float*)x, sd, (float*)y, n);
  else bn_forward_kernel<double><<<grid, LOSS_THREADS, 0, ctx->stream>>>((const double*)x, sd, (double*)y, n);
  PRAD_LAUNCHED(ctx);
  return PRAD_OK;
}

prad_status prad_batchnorm_backward(prad_ctx* ctx, prad_dtype dt, const void* x, const void* stats, const void* dy,
                                    void* dx, int64_t rows, int cols) {
  PRAD_CHECK_CTX(ctx);
  PRAD_REQUIRE(dtype_ok(dt) && rows >= 0 && cols >= 0, PRAD_ERR_INVALID, "prad_batchnorm_backward: bad argument");
  const int64_t n = rows * cols;
  if (n == 0) return PRAD_OK;
  PRAD_REQUIRE(x && stats && dy && dx, PRAD_ERR_INVALID, "prad_batchnorm_backward: null pointer");
  const int grid = stream_grid(ctx, n, LOSS_THREADS * 4, 4);
  if (dt == PRAD_F32) bn_backward_kernel<float><<<grid, LOSS_THREADS, 0, ctx->stream>>>((const float*)x, (const double*)stats, (const float*)dy, (float*)dx, n);
  else bn_backward_kernel<double><<<grid, LOSS_THREADS, 0, ctx->stream>>>((const double*)x, (const double*)stats, (const double*)dy, (double*)dx, n);
  PRAD_LAUNCHED(ctx);
  return PRAD_OK;
}

}  // extern "C"

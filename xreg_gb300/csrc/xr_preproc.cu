// xr_preproc.cu -- data preparation either side of the hot path, on the device:
//
// * HU -> linear attenuation (the kernel is in xr_volume.cu).
// * Fixed-image downsampling for a coarser registration level (DownsampleProjData
//   -> DownsampleImage, lib/image/xregProjData.cpp:40-53,
//   lib/itk/xregITKResampleUtils.h:51-131,183-187): for factor < 1, a discrete
//   Gaussian (ITK DiscreteGaussianImageFilter, variance (0.5/factor)^2 in pixels,
//   maximum error 0.01, kernel width at most 32, edge pixels replicated) along x
//   then y in double, rounded to the float image type; then resampling onto
//   floor(n * factor + 0.5) pixels with the same origin and spacing / factor, so
//   output pixel i reads the smoothed image at continuous index i / factor.  The
//   interpolator is DownsampleImage's default, the cubic B-spline (ITK
//   BSplineInterpolateImageFunction, order 3): coefficients by Unser's recursive
//   prefilter (pole sqrt(3) - 2, gain 6, mirror boundaries, causal start summed
//   to a 1e-10 horizon), along x then y in double; evaluation with the 4 x 4
//   cubic B-spline weights around floor(x) - 1, indices mirrored at 0 and n - 1;
//   points outside [-0.5, n - 0.5) get 0.
// * Projection pre-processing (ProjPreProc, lib/image/xregProjPreProc.cpp:31-139):
//   boundary crop (CropImage2DBoundary, lib/itk/xregITKCropPadUtils.h:89-114) and
//   the log remap (ImageIntensLogTransFilter::GenerateData,
//   lib/image/xregImageIntensLogTrans.cpp:52-146 with UseMaxIntensityAsI0):
//   I0 = max of the image smoothed by a discrete Gaussian of variance 2;
//   out = -log(x / I0) for x > 1e-6, else -log(min_pos / I0) with min_pos the
//   smallest value above 1e-6, all in float.
//
// The discrete Gaussian kernel is Lindeberg's discrete analogue
// T(k, t) = exp(-t) I_k(t) (t = variance, I_k the modified Bessel function),
// taken out from the centre until its two-sided sum reaches 1 - max_error and
// normalised to sum 1 — the construction ITK's GaussianOperator follows.  Here
// I_k is summed from its power series in double.
//
// The smoothing and the spline run in float-float (about 48 bits) instead of
// double: this GPU issues one double instruction per 64 cycles and scheduler, and
// its results are rounded to float.  Values that float-float cannot carry
// (infinities, NaN, magnitudes near the end of float's range) take the double
// operations.
#include "xr_gradtile.cuh"
#include "xr_internal.h"

#include <cmath>
#include <vector>

namespace xr {
namespace {

constexpr int kMaxTaps = 32;
using gt::FF;

struct GaussKernel {
  int radius;
  double c[kMaxTaps + 1];
  float hi[kMaxTaps + 1], lo[kMaxTaps + 1];  // c = hi + lo
};

__device__ __forceinline__ FF two_sum(float a, float b) {
  const float s = __fadd_rn(a, b), t = __fsub_rn(s, a);
  return FF{s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, t)), __fsub_rn(b, t))};
}
__device__ __forceinline__ FF renorm(float hi, float lo) {
  const float s = __fadd_rn(hi, lo);
  return FF{s, __fsub_rn(lo, __fsub_rn(s, hi))};
}
__device__ __forceinline__ FF ff_mul(FF a, FF b) {
  const float p = __fmul_rn(a.hi, b.hi);
  return renorm(p, __fmaf_rn(a.lo, b.hi, __fmaf_rn(a.hi, b.lo, __fmaf_rn(a.hi, b.hi, -p))));
}
__device__ __forceinline__ FF ff_sum(FF a, FF b) {
  const FF s = two_sum(a.hi, b.hi);
  return renorm(s.hi, __fadd_rn(s.lo, __fadd_rn(a.lo, b.lo)));
}
__device__ __forceinline__ FF ff_of(double v) {
  const float hi = (float)v;
  return FF{hi, (float)(v - (double)hi)};
}
__device__ __forceinline__ FF ff_of(float v) { return FF{v, 0.0f}; }
__device__ __forceinline__ FF ff_of(float2 v) { return FF{v.x, v.y}; }
__device__ __forceinline__ double value(float v) { return (double)v; }
__device__ __forceinline__ double value(float2 v) { return (double)v.x + (isfinite(v.x) ? (double)v.y : 0.0); }
constexpr float kHuge = 1.0e37f;  // magnitudes above it are left to double

// One pixel of the separable pass along x (dir 0) or y (dir 1), edges replicated,
// in double.
template <typename TIn>
__device__ __noinline__ double gauss_at_double(const TIn* __restrict__ in, int rows, int cols, int r, int c, int dir,
                                               const GaussKernel& k) {
  double s = __dmul_rn(k.c[0], value(in[(int64_t)r * cols + c]));
  for (int t = 1; t <= k.radius; ++t) {
    const int64_t a = dir == 0 ? (int64_t)r * cols + max(c - t, 0) : (int64_t)max(r - t, 0) * cols + c;
    const int64_t b = dir == 0 ? (int64_t)r * cols + min(c + t, cols - 1) : (int64_t)min(r + t, rows - 1) * cols + c;
    s = __dadd_rn(s, __dmul_rn(k.c[t], __dadd_rn(value(in[a]), value(in[b]))));
  }
  return s;
}

// The same in float-float: c_t (a + b) with the sum and the product exact to about
// 2^-47; a result that is not finite or not below kHuge is taken in double.
template <typename TIn, int DIR>
__device__ __forceinline__ FF gauss_at(const TIn* __restrict__ in, int rows, int cols, int r, int c,
                                       const GaussKernel& k) {
  const FF m = ff_of(in[(int64_t)r * cols + c]);
  FF acc = ff_mul(m, FF{k.hi[0], k.lo[0]});
#pragma unroll 4
  for (int t = 1; t <= k.radius; ++t) {
    const int64_t ia = DIR == 0 ? (int64_t)r * cols + max(c - t, 0) : (int64_t)max(r - t, 0) * cols + c;
    const int64_t ib = DIR == 0 ? (int64_t)r * cols + min(c + t, cols - 1) : (int64_t)min(r + t, rows - 1) * cols + c;
    const FF a = ff_of(in[ia]), b = ff_of(in[ib]);
    const FF s = two_sum(a.hi, b.hi);
    const float e = __fadd_rn(s.lo, __fadd_rn(a.lo, b.lo));
    const float p = __fmul_rn(s.hi, k.hi[t]);
    const float pe = __fmaf_rn(e, k.hi[t], __fmaf_rn(s.hi, k.lo[t], __fmaf_rn(s.hi, k.hi[t], -p)));
    const FF q = two_sum(acc.hi, p);
    acc = FF{q.hi, __fadd_rn(acc.lo, __fadd_rn(q.lo, pe))};
  }
  acc = renorm(acc.hi, acc.lo);
  if (fabsf(acc.hi) < kHuge && acc.lo == acc.lo) return acc;
  return ff_of(gauss_at_double(in, rows, cols, r, c, DIR, k));
}

// Separable pass along x: float in, float-float out.
__global__ void gauss_x_kernel(const float* __restrict__ in, int rows, int cols, const GaussKernel k,
                               float2* __restrict__ out) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= cols) return;
  for (int r = blockIdx.y; r < rows; r += gridDim.y) {
    const FF v = gauss_at<float, 0>(in, rows, cols, r, c, k);
    out[(int64_t)r * cols + c] = make_float2(v.hi, isfinite(v.hi) ? v.lo : 0.0f);
  }
}

// Pass along y, rounded to the float image type; *beyond is set when a value is not
// finite or not below kHuge.
__global__ void gauss_y_kernel(const float2* __restrict__ in, int rows, int cols, const GaussKernel k,
                               float* __restrict__ out, int* __restrict__ beyond) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= cols) return;
  for (int r = blockIdx.y; r < rows; r += gridDim.y) {
    const float v = gauss_at<float2, 1>(in, rows, cols, r, c, k).hi;
    out[(int64_t)r * cols + c] = v;
    if (!(fabsf(v) < kHuge)) *beyond = 1;
  }
}

// The passes in double, for images that spline_kernel does not take.
template <typename TIn>
__global__ void gauss_pass_kernel(const TIn* __restrict__ in, int rows, int cols, int dir, GaussKernel k,
                                  double* __restrict__ out) {
  const int64_t n = (int64_t)rows * cols;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int r = (int)(i / cols), c = (int)(i - (int64_t)r * cols);
    // explicitly rounded (no fused multiply-add): the same operations as the oracle
    double s = __dmul_rn(k.c[0], (double)in[i]);
    for (int t = 1; t <= k.radius; ++t) {
      int a, b;
      if (dir == 0) {
        a = max(c - t, 0); b = min(c + t, cols - 1);
        s = __dadd_rn(s, __dmul_rn(k.c[t], __dadd_rn((double)in[(int64_t)r * cols + a], (double)in[(int64_t)r * cols + b])));
      } else {
        a = max(r - t, 0); b = min(r + t, rows - 1);
        s = __dadd_rn(s, __dmul_rn(k.c[t], __dadd_rn((double)in[(int64_t)a * cols + c], (double)in[(int64_t)b * cols + c])));
      }
    }
    out[i] = s;
  }
}

// Second smoothing pass result rounded to the float image type, widened back
// to double as the B-spline prefilter's input.
__global__ void round_to_float_kernel(double* __restrict__ v, int64_t n) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    v[i] = (double)(float)v[i];
}

__global__ void widen_kernel(const float* __restrict__ in, int64_t n, double* __restrict__ out) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    out[i] = (double)in[i];
}

// Cubic B-spline prefilter of a line of `len` samples, `stride` apart, into v (from
// src, where given, else in place).  z = the pole, gain = (1 - z)(1 - 1/z), horizon =
// terms of the causal start.
__device__ void bspline_prefilter_line(double* __restrict__ v, int len, int64_t stride, double z, double gain,
                                       int horizon, const float* __restrict__ src = nullptr) {
  if (src) {
#pragma unroll 8
    for (int n = 0; n < len; ++n) v[n * stride] = __dmul_rn((double)__ldg(src + n * stride), gain);
  } else {
    for (int n = 0; n < len; ++n) v[n * stride] = __dmul_rn(v[n * stride], gain);
  }
  // causal initialisation (mirror boundaries)
  {
    double zn = z, sum;
    if (horizon < len) {
      sum = v[0];
      for (int n = 1; n < horizon; ++n) {
        sum = __dadd_rn(sum, __dmul_rn(zn, v[n * stride]));
        zn = __dmul_rn(zn, z);
      }
      v[0] = sum;
    } else {
      const double iz = __ddiv_rn(1.0, z);
      double z2n = pow(z, (double)(len - 1));
      sum = __dadd_rn(v[0], __dmul_rn(z2n, v[(int64_t)(len - 1) * stride]));
      z2n = __dmul_rn(z2n, __dmul_rn(z2n, iz));
      for (int n = 1; n <= len - 2; ++n) {
        sum = __dadd_rn(sum, __dmul_rn(__dadd_rn(zn, z2n), v[n * stride]));
        zn = __dmul_rn(zn, z);
        z2n = __dmul_rn(z2n, iz);
      }
      v[0] = __ddiv_rn(sum, __dsub_rn(1.0, __dmul_rn(zn, zn)));
    }
  }
  for (int n = 1; n < len; ++n) v[n * stride] = __dadd_rn(v[n * stride], __dmul_rn(z, v[(n - 1) * stride]));
  // anti-causal initialisation and recursion
  {
    const int64_t a = (int64_t)(len - 1) * stride, b = (int64_t)(len - 2) * stride;
    v[a] = __dmul_rn(__ddiv_rn(z, __dsub_rn(__dmul_rn(z, z), 1.0)), __dadd_rn(__dmul_rn(z, v[b]), v[a]));
  }
  for (int n = len - 2; n >= 0; --n) v[n * stride] = __dmul_rn(z, __dsub_rn(v[(n + 1) * stride], v[n * stride]));
}

// `count` lines, line l at c + l * line_stride; one thread per line.
__global__ void bspline_prefilter_kernel(double* __restrict__ c, int count, int len, int64_t line_stride,
                                         int64_t stride, double z, double gain, int horizon) {
  const int l = blockIdx.x * blockDim.x + threadIdx.x;
  if (l < count && len >= 2) bspline_prefilter_line(c + (int64_t)l * line_stride, len, stride, z, gain, horizon);
}

__device__ __forceinline__ int mirror_index(int k, int n) {
  if (n == 1) return 0;
  if (k < 0) k = -k;
  if (k > n - 1) k = (n - 1) - (k - (n - 1));
  return k;
}

__device__ __forceinline__ void cubic_weights(double x, int i1, double w[4]) {
  const double t = __dsub_rn(x, (double)i1);
  w[3] = __dmul_rn(__dmul_rn(__dmul_rn(1.0 / 6.0, t), t), t);
  w[0] = __dsub_rn(__dadd_rn(1.0 / 6.0, __dmul_rn(__dmul_rn(0.5, t), __dsub_rn(t, 1.0))), w[3]);
  w[2] = __dsub_rn(__dadd_rn(t, w[0]), __dmul_rn(2.0, w[3]));
  w[1] = __dsub_rn(__dsub_rn(__dsub_rn(1.0, w[0]), w[2]), w[3]);
}

// Output pixels i0, i0 + step, ...: pixel (r, c) = cubic B-spline of the coefficients
// at (c / factor, r / factor).
__device__ void bspline_resample(const double* __restrict__ coef, int rows, int cols, double factor, int orows,
                                 int ocols, int64_t i0, int64_t step, float* __restrict__ out) {
  const int64_t n = (int64_t)orows * ocols;
  for (int64_t i = i0; i < n; i += step) {
    const int r = (int)(i / ocols), c = (int)(i - (int64_t)r * ocols);
    const double x = __ddiv_rn((double)c, factor), y = __ddiv_rn((double)r, factor);
    if (!(x >= -0.5 && x < cols - 0.5 && y >= -0.5 && y < rows - 0.5)) { out[i] = 0.0f; continue; }
    const int x1 = (int)floorf((float)x), y1 = (int)floorf((float)y);  // index of weight 1
    double wx[4], wy[4];
    cubic_weights(x, x1, wx);
    cubic_weights(y, y1, wy);
    int ix[4], iy[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      ix[k] = mirror_index(x1 - 1 + k, cols);
      iy[k] = mirror_index(y1 - 1 + k, rows);
    }
    double acc = 0.0;
#pragma unroll
    for (int b = 0; b < 4; ++b)
#pragma unroll
      for (int a = 0; a < 4; ++a)
        acc = __dadd_rn(acc, __dmul_rn(__dmul_rn(wx[a], wy[b]), coef[(int64_t)iy[b] * cols + ix[a]]));
    out[i] = (float)acc;
  }
}

__global__ void bspline_resample_kernel(const double* __restrict__ coef, int rows, int cols, double factor,
                                        int orows, int ocols, float* __restrict__ out) {
  bspline_resample(coef, rows, cols, factor, orows, ocols, (int64_t)blockIdx.x * blockDim.x + threadIdx.x,
                   (int64_t)gridDim.x * blockDim.x, out);
}

// What spline_kernel does in double for an image with values that float-float does
// not carry (*beyond): its first pass widens and prefilters the rows, its second the
// columns, one thread a line over all blocks, and spline_double_kernel interpolates.
struct SplineDouble {
  const float* img;
  int rows, cols;
  double* coef;
};

template <bool COLUMNS>
__device__ __noinline__ void spline_lines_double(const float* __restrict__ img, int rows, int cols,
                                                 double* __restrict__ coef, double z, double gain, int horizon) {
  const int threads = gridDim.x * gridDim.y * blockDim.x;
  const int first = (blockIdx.y * gridDim.x + blockIdx.x) * blockDim.x + threadIdx.x;
  for (int l = first; l < (COLUMNS ? cols : rows); l += threads) {
    if constexpr (COLUMNS) bspline_prefilter_line(coef + l, rows, cols, z, gain, horizon);
    else bspline_prefilter_line(coef + (int64_t)l * cols, cols, 1, z, gain, horizon, img + (int64_t)l * cols);
  }
}

__global__ void spline_double_kernel(const double* __restrict__ coef, int rows, int cols, double factor, int orows,
                                     int ocols, const int* __restrict__ beyond, float* __restrict__ out) {
  if (!*beyond) return;
  bspline_resample(coef, rows, cols, factor, orows, ocols, (int64_t)blockIdx.x * blockDim.x + threadIdx.x,
                   (int64_t)gridDim.x * blockDim.x, out);
}

// The spline along one axis, prefilter and interpolation together, in float-float:
// `lines` lines of `len` contiguous samples in, out[j][line] (transposed, so that
// the same kernel takes the other axis next) = the spline at j / factor.
// The recursions decay by |z| = 0.27 a sample, so a line is cut into chunks that
// start kWarm samples early from zero (0.27^28 = 1e-16): a warp takes 32 lines by
// one chunk, its samples and coefficients in shared memory (33-word pitch: lanes
// along samples or along lines meet no bank conflicts).  One thread per line in
// double took 864 us along the rows of a 1436 x 1436 image and 1406 along its
// columns, one chain of dependent double operations each; the two passes of this
// kernel take 27 and 15 (quarter-size output).
constexpr int kChunk = 64, kWarm = 28;
constexpr int kSpan = kChunk + 3 + 2 * kWarm;  // coefficients -1 .. kChunk + 1 and both warm-ups
constexpr int kOuts = kChunk + 8;              // candidate outputs of a chunk (factor < 1), with room for rounding

template <typename TIn, typename TOut>
__global__ void __launch_bounds__(32) spline_kernel(const TIn* __restrict__ in, int lines, int len, double factor,
                                                    int outs, double z_d, double gain_d, int horizon,
                                                    const int* __restrict__ beyond, const SplineDouble dbl,
                                                    TOut* __restrict__ out) {
  __shared__ float hi[kSpan][33], lo[kSpan][33];
  __shared__ FF w[kOuts][4];
  __shared__ int first[kOuts];  // index of an output's second coefficient, -1: outside the image
  if (*beyond) {
    spline_lines_double<sizeof(TOut) == sizeof(float)>(dbl.img, dbl.rows, dbl.cols, dbl.coef, z_d, gain_d, horizon);
    return;
  }
  const int lane = threadIdx.x, l0 = blockIdx.y * 32;
  if (l0 >= lines) return;  // a block for the double columns alone
  const int start = blockIdx.x * kChunk;  // this chunk's outputs have floor(position) in [start, start + kChunk)
  const int k0 = max(start - 1 - kWarm, 0), k1 = min(start + kChunk + 2 + kWarm, len);
  for (int k = k0 + lane; k < k1; k += 32) {
#pragma unroll
    for (int r = 0; r < 32; r += 16) {  // 16 loads in flight
      TIn v[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) v[i] = in[(int64_t)min(l0 + r + i, lines - 1) * len + k];
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const FF f = ff_of(v[i]);
        hi[k - k0][r + i] = f.hi;
        lo[k - k0][r + i] = f.lo;
      }
    }
  }
  // outputs of this chunk and their weights, one output per lane at a time
  const bool tail = start + kChunk >= len;  // positions past the last sample belong to the last chunk
  const int jb = max((int)((float)start * (float)factor) - 2, 0);
  const int je = tail ? outs : min(outs, (int)((float)(start + kChunk) * (float)factor) + 3);
  int j0 = outs, j1 = 0;
  for (int j = jb + lane; j < je; j += 32) {
    const double x = __ddiv_rn((double)j, factor);
    const int x1 = (int)floorf((float)x);
    if (x1 < start || (x1 >= start + kChunk && !tail)) continue;
    j0 = min(j0, j);
    j1 = max(j1, j + 1);
    double wd[4];
    cubic_weights(x, x1, wd);
    for (int a = 0; a < 4; ++a) w[j - jb][a] = ff_of(wd[a]);
    first[j - jb] = x < len - 0.5 ? x1 : -1;
  }
  for (int o = 16; o > 0; o >>= 1) {
    j0 = min(j0, __shfl_xor_sync(0xffffffffu, j0, o));
    j1 = max(j1, __shfl_xor_sync(0xffffffffu, j1, o));
  }
  __syncwarp();
  // causal, then anti-causal recursion of this lane's line
  const FF z = ff_of(z_d), gain = ff_of(gain_d);
  const int n = k1 - k0;
  FF c{0.0f, 0.0f};
  int k = 0;
  if (k0 == 0) {  // the line's own start (mirror boundary), summed to the horizon
    FF zn = z;
    c = ff_mul(FF{hi[0][lane], lo[0][lane]}, gain);
    for (int i = 1; i < horizon; ++i) {
      c = ff_sum(c, ff_mul(zn, ff_mul(FF{hi[i][lane], lo[i][lane]}, gain)));
      zn = ff_mul(zn, z);
    }
    hi[0][lane] = c.hi;
    lo[0][lane] = c.lo;
    k = 1;
  }
  // c = gain s[k] + z c: hi + lo without renormalising (lo stays below an ulp or
  // two of hi, the recursion contracts), so that a step's dependent chain is one
  // product and one sum; the next sample is read before this one is stored
  FF v = ff_mul(FF{hi[k][lane], lo[k][lane]}, gain);
  for (; k < n; ++k) {
    const FF nx{hi[min(k + 1, n - 1)][lane], lo[min(k + 1, n - 1)][lane]};
    const float q = __fmul_rn(z.hi, c.hi);
    const float qe = __fmaf_rn(z.hi, c.lo, __fmaf_rn(z.lo, c.hi, __fmaf_rn(z.hi, c.hi, -q)));
    c = two_sum(v.hi, q);
    c.lo = __fadd_rn(c.lo, __fadd_rn(qe, v.lo));
    hi[k][lane] = c.hi;
    lo[k][lane] = c.lo;
    v = ff_mul(nx, gain);
  }
  k = n - 1;
  if (k1 == len) {  // the line's own end
    const FF b{hi[n - 2][lane], lo[n - 2][lane]};
    c = ff_mul(ff_of(__ddiv_rn(z_d, __dsub_rn(__dmul_rn(z_d, z_d), 1.0))), ff_sum(ff_mul(z, b), c));
    hi[k][lane] = c.hi;
    lo[k][lane] = c.lo;
    --k;
  } else {
    c = FF{0.0f, 0.0f};
  }
  const int kl = max(start - 2, 0) - k0;  // a mirrored index reaches start - 2
  v = FF{hi[k][lane], lo[k][lane]};
  for (; k >= kl; --k) {  // c = z (c - c+[k])
    const FF nx{hi[max(k - 1, 0)][lane], lo[max(k - 1, 0)][lane]};
    FF d = two_sum(c.hi, -v.hi);
    d.lo = __fadd_rn(d.lo, __fsub_rn(c.lo, v.lo));
    c.hi = __fmul_rn(z.hi, d.hi);
    c.lo = __fmaf_rn(z.hi, d.lo, __fmaf_rn(z.lo, d.hi, __fmaf_rn(z.hi, d.hi, -c.hi)));
    hi[k][lane] = c.hi;
    lo[k][lane] = c.lo;
    v = nx;
  }
  if (l0 + lane >= lines) return;
  for (int j = j0; j < j1; ++j) {
    v = FF{0.0f, 0.0f};
    const int x1 = first[j - jb];
    if (x1 >= 0) {
#pragma unroll
      for (int a = 0; a < 4; ++a) {
        const int i = mirror_index(x1 - 1 + a, len) - k0;
        v = ff_sum(v, ff_mul(w[j - jb][a], FF{hi[i][lane], lo[i][lane]}));
      }
    }
    if constexpr (sizeof(TOut) == sizeof(float2)) out[(int64_t)j * lines + l0 + lane] = make_float2(v.hi, v.lo);
    else out[(int64_t)j * lines + l0 + lane] = v.hi;
  }
}

// exp(-t) I_k(t) from the power series of I_k.
double scaled_bessel_i(int k, double t) {
  double term = 1.0;
  for (int j = 1; j <= k; ++j) term *= (0.5 * t) / j;  // (t/2)^k / k!
  double sum = term;
  const double q = 0.25 * t * t;
  for (int m = 1; m < 500; ++m) {
    term *= q / ((double)m * (double)(m + k));
    sum += term;
    if (term < 1e-18 * sum) break;
  }
  return std::exp(-t) * sum;
}

}  // namespace

// Discrete Gaussian taps c[0..radius] (normalised so c0 + 2 sum c_k = 1):
// e^{-t} I_0(t), e^{-t} I_1(t), then the Bessel recurrence
// c_k = c_{k-2} - 2 (k - 1) c_{k-1} / t until the two-sided sum reaches
// 1 - max_error or max_width one-sided taps.
int discrete_gaussian_taps(double variance, double max_error, int max_width, double* out) {
  std::vector<double> c;
  const double cap = 1.0 - max_error;
  c.push_back(scaled_bessel_i(0, variance));
  double sum = c[0];
  c.push_back(scaled_bessel_i(1, variance));
  sum += 2.0 * c[1];
  for (int k = 2; sum < cap && (int)c.size() < kMaxTaps + 1; ++k) {
    c.push_back(c[k - 2] - 2.0 * (k - 1) * c[k - 1] / variance);
    sum += 2.0 * c.back();
    if ((int)c.size() > max_width) break;  // one-sided length limit
  }
  for (double& v : c) v /= sum;
  for (size_t i = 0; i < c.size(); ++i) out[i] = c[i];
  return (int)c.size() - 1;
}

}  // namespace xr

using namespace xr;

extern "C" XR_API xr_status xr_hu_to_lin_att(const float* d_hu, int64_t n, float* d_mu, void* stream) {
  if (!d_hu || !d_mu || n < 0) return fail(XR_ERR_INVALID_ARG, "xr_hu_to_lin_att: bad argument");
  if (n == 0) return XR_OK;
  XR_CUDA_TRY(launch_hu_to_mu(d_hu, n, d_mu, static_cast<cudaStream_t>(stream)));
  return XR_OK;
}

extern "C" XR_API xr_status xr_downsample_image_size(int64_t rows, int64_t cols, double factor, int64_t* out_rows,
                                                    int64_t* out_cols) {
  if (!out_rows || !out_cols || rows < 1 || cols < 1 || !(factor > 0.0) || factor > 1.0)
    return fail(XR_ERR_INVALID_ARG, "xr_downsample_image_size: need rows, cols >= 1 and 0 < factor <= 1");
  *out_rows = (int64_t)((double)rows * factor + 0.5);
  *out_cols = (int64_t)((double)cols * factor + 0.5);
  if (*out_rows < 1 || *out_cols < 1) return fail(XR_ERR_INVALID_ARG, "xr_downsample_image_size: empty result");
  return XR_OK;
}

static GaussKernel gauss_kernel(double variance) {
  GaussKernel k{};
  k.radius = discrete_gaussian_taps(variance, 0.01, 32, k.c);
  for (int t = 0; t <= k.radius; ++t) {
    k.hi[t] = (float)k.c[t];
    k.lo[t] = (float)(k.c[t] - (double)k.hi[t]);
  }
  return k;
}

static dim3 image_grid(int64_t rows, int64_t cols) {
  return dim3((unsigned)((cols + 127) / 128), (unsigned)std::min<int64_t>(rows, 65535));
}

static unsigned grid_for(int64_t n) { return (unsigned)std::min<int64_t>((n + 255) / 256, 8192); }

struct Spline {
  double z = std::sqrt(3.0) - 2.0;
  double gain = (1.0 - z) * (1.0 - 1.0 / z);
  int horizon = (int)std::ceil(std::log(1.0e-10) / std::log(std::fabs(z)));
};

// Cubic B-spline coefficients of a rows x cols double image in place: along x
// (one thread per row), then along y (one thread per column).
static cudaError_t bspline_coefficients(double* c, int64_t rows, int64_t cols, cudaStream_t s) {
  const Spline p;
  bspline_prefilter_kernel<<<(unsigned)((rows + 127) / 128), 128, 0, s>>>(c, (int)rows, (int)cols, cols, 1, p.z, p.gain,
                                                                          p.horizon);
  bspline_prefilter_kernel<<<(unsigned)((cols + 127) / 128), 128, 0, s>>>(c, (int)cols, (int)rows, 1, cols, p.z, p.gain,
                                                                          p.horizon);
  return cudaGetLastError();
}

extern "C" XR_API xr_status xr_downsample_image(const float* d_src, int64_t rows, int64_t cols, double factor,
                                               double* d_scratch, float* d_dst, void* stream) {
  int64_t orows = 0, ocols = 0;
  xr_status st = xr_downsample_image_size(rows, cols, factor, &orows, &ocols);
  if (st != XR_OK) return st;
  if (!d_src || !d_dst || !d_scratch) return fail(XR_ERR_INVALID_ARG, "xr_downsample_image: NULL pointer");
  if (rows > (1 << 20) || cols > (1 << 20)) return fail(XR_ERR_INVALID_ARG, "xr_downsample_image: image too large");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int64_t n = rows * cols;
  double* a = d_scratch;
  double* b = d_scratch + n;
  const double sigma = 0.5 / factor;
  // Chunked float-float passes where a line has a chunk's samples and the output is
  // smaller on both axes (their buffers share the scratch: smoothed floats, then a
  // flag, in the second half; the row pass's output over the first).  Otherwise,
  // small or hardly reduced images, the double kernels.
  if (factor < 1.0 && rows >= kChunk && cols >= kChunk && orows < rows && ocols < cols) {
    const GaussKernel k = gauss_kernel(sigma * sigma);
    const Spline p;
    float2* x_out = reinterpret_cast<float2*>(a);  // smoothed along x, then the spline along x [ocols][rows]
    float* smooth = reinterpret_cast<float*>(b);
    int* beyond = reinterpret_cast<int*>(smooth + n);
    XR_CUDA_TRY(cudaMemsetAsync(beyond, 0, sizeof(int), s));
    gauss_x_kernel<<<image_grid(rows, cols), 128, 0, s>>>(d_src, (int)rows, (int)cols, k, x_out);
    gauss_y_kernel<<<image_grid(rows, cols), 128, 0, s>>>(x_out, (int)rows, (int)cols, k, smooth, beyond);
    auto grid = [](int64_t len, int64_t lines) {
      return dim3((unsigned)((len + kChunk - 1) / kChunk), (unsigned)((lines + 31) / 32));
    };
    // an image with values beyond float-float: the coefficients lie where x_out does
    const SplineDouble dbl{smooth, (int)rows, (int)cols, a};
    spline_kernel<float, float2><<<grid(cols, rows), 32, 0, s>>>(smooth, (int)rows, (int)cols, factor, (int)ocols, p.z,
                                                                 p.gain, p.horizon, beyond, dbl, x_out);
    dim3 columns = grid(rows, ocols);  // a thread for each column in the double case
    columns.y = std::max(columns.y, (unsigned)((cols + 32 * columns.x - 1) / (32 * columns.x)));
    spline_kernel<float2, float><<<columns, 32, 0, s>>>(x_out, (int)ocols, (int)rows, factor, (int)orows, p.z, p.gain,
                                                        p.horizon, beyond, dbl, d_dst);
    spline_double_kernel<<<std::min<unsigned>(grid_for(orows * ocols), 256), 256, 0, s>>>(
        a, (int)rows, (int)cols, factor, (int)orows, (int)ocols, beyond, d_dst);
    XR_CUDA_TRY(cudaGetLastError());
    return XR_OK;
  }
  if (factor < 1.0) {
    const GaussKernel k = gauss_kernel(sigma * sigma);
    gauss_pass_kernel<float><<<grid_for(n), 256, 0, s>>>(d_src, (int)rows, (int)cols, 0, k, a);
    gauss_pass_kernel<double><<<grid_for(n), 256, 0, s>>>(a, (int)rows, (int)cols, 1, k, b);
    round_to_float_kernel<<<grid_for(n), 256, 0, s>>>(b, n);
  } else {
    widen_kernel<<<grid_for(n), 256, 0, s>>>(d_src, n, b);
  }
  XR_CUDA_TRY(bspline_coefficients(b, rows, cols, s));
  bspline_resample_kernel<<<grid_for(orows * ocols), 256, 0, s>>>(b, (int)rows, (int)cols, factor, (int)orows,
                                                                  (int)ocols, d_dst);
  XR_CUDA_TRY(cudaGetLastError());
  return XR_OK;
}

extern "C" XR_API xr_status xr_camera_crop_boundary(const xr_camera_desc* src, int64_t width, xr_camera_desc* out) {
  if (!src || !out) return fail(XR_ERR_INVALID_ARG, "xr_camera_crop_boundary: NULL argument");
  if (width < 0 || src->num_det_rows - 2 * width < 2 || src->num_det_cols - 2 * width < 2)
    return fail(XR_ERR_INVALID_ARG, "xr_camera_crop_boundary: the crop leaves fewer than 2 rows or columns");
  // UpdateCameraModelFor2DROI in float: the principal point moves by the crop,
  // and CameraModel::setup(K, E, ...) derives the focal length again from K
  // (FocalLenFromIntrins, xregPerspectiveXform.cpp:186-190)
  xr_camera_desc d = *src;
  float K[9];
  for (int i = 0; i < 9; ++i) K[i] = (float)src->intrins[i];
  K[2] -= (float)width;
  K[5] -= (float)width;
  for (int i = 0; i < 9; ++i) d.intrins[i] = K[i];
  for (int i = 0; i < 16; ++i) d.extrins[i] = (float)src->extrins[i];
  const float rs = (float)src->det_row_spacing, cs = (float)src->det_col_spacing;
  d.det_row_spacing = rs;
  d.det_col_spacing = cs;
  d.focal_len = (std::fabs(K[0] * cs) + std::fabs(K[4] * ((rs < 0) ? cs : rs))) / 2.0f;
  d.num_det_rows = src->num_det_rows - 2 * width;
  d.num_det_cols = src->num_det_cols - 2 * width;
  *out = d;
  return XR_OK;
}

namespace xr {
namespace {

__global__ void crop_kernel(const float* __restrict__ in, int cols, int width, int orows, int ocols,
                            float* __restrict__ out) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= ocols) return;
  for (int r = blockIdx.y; r < orows; r += gridDim.y)
    out[(int64_t)r * ocols + c] = in[(int64_t)(r + width) * cols + (c + width)];
}

constexpr int kRedBlocks = 1024;  // partials of the statistics (the scratch holds as many)
constexpr float kLogEps = 1.0e-6f;

// Second Gaussian pass (along y) rounded to float, reduced to its maximum, and
// the smallest source value above 1e-6; per-block partials.
__global__ void log_remap_stats_kernel(const float2* __restrict__ a, const float* __restrict__ src, int rows,
                                       int cols, const GaussKernel k, float* __restrict__ part_max,
                                       float* __restrict__ part_min) {
  float mx = -INFINITY, mn = INFINITY;
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < cols; c += gridDim.x * blockDim.x)
    for (int r = blockIdx.y; r < rows; r += gridDim.y) {
      mx = fmaxf(mx, gauss_at<float2, 1>(a, rows, cols, r, c, k).hi);
      const float x = src[(int64_t)r * cols + c];
      if (x > kLogEps) mn = fminf(mn, x);
    }
  __shared__ float smx[32], smn[32];
  for (int o = 16; o > 0; o >>= 1) {
    mx = fmaxf(mx, __shfl_down_sync(0xffffffffu, mx, o));
    mn = fminf(mn, __shfl_down_sync(0xffffffffu, mn, o));
  }
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (lane == 0) { smx[w] = mx; smn[w] = mn; }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int j = 1; j < (int)(blockDim.x >> 5); ++j) { mx = fmaxf(mx, smx[j]); mn = fminf(mn, smn[j]); }
    part_max[blockIdx.y * gridDim.x + blockIdx.x] = mx;
    part_min[blockIdx.y * gridDim.x + blockIdx.x] = mn;
  }
}

// scal[0] = I0, scal[1] = -log(min_pos / I0) (min_pos 0 when no value exceeds 1e-6).
__global__ void log_remap_finalize_kernel(const float* __restrict__ part_max, const float* __restrict__ part_min,
                                          int nblk, int use_max, float i0, float* __restrict__ scal) {
  float mx = -INFINITY, mn = INFINITY;
  for (int j = threadIdx.x; j < nblk; j += 32) { mx = fmaxf(mx, part_max[j]); mn = fminf(mn, part_min[j]); }
  for (int o = 16; o > 0; o >>= 1) {
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
  }
  if (threadIdx.x != 0) return;
  const float I0 = use_max ? mx : i0;
  const float min_pos = (mn == INFINITY) ? 0.0f : mn;
  scal[0] = I0;
  scal[1] = -logf(__fdiv_rn(min_pos, I0));
}

__global__ void log_remap_kernel(const float* __restrict__ src, int64_t n, const float* __restrict__ scal,
                                 float* __restrict__ out) {
  const float I0 = scal[0], out_max = scal[1];
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const float x = src[i];
    out[i] = (x > kLogEps) ? -logf(__fdiv_rn(x, I0)) : out_max;
  }
}

}  // namespace
}  // namespace xr

extern "C" XR_API xr_status xr_crop_image_boundary(const float* d_src, int64_t rows, int64_t cols, int64_t width,
                                                  float* d_dst, void* stream) {
  if (!d_src || !d_dst) return fail(XR_ERR_INVALID_ARG, "xr_crop_image_boundary: NULL pointer");
  if (width < 0 || rows - 2 * width < 1 || cols - 2 * width < 1 || rows > (1 << 30) || cols > (1 << 30))
    return fail(XR_ERR_INVALID_ARG, "xr_crop_image_boundary: the crop leaves no pixels");
  const int64_t orows = rows - 2 * width, ocols = cols - 2 * width;
  crop_kernel<<<image_grid(orows, ocols), 128, 0, static_cast<cudaStream_t>(stream)>>>(
      d_src, (int)cols, (int)width, (int)orows, (int)ocols, d_dst);
  XR_CUDA_TRY(cudaGetLastError());
  return XR_OK;
}

extern "C" XR_API xr_status xr_log_remap(const float* d_src, int64_t rows, int64_t cols, int32_t use_max_as_i0,
                                        float i0, double* d_scratch, float* d_dst, void* stream) {
  if (!d_src || !d_dst || !d_scratch) return fail(XR_ERR_INVALID_ARG, "xr_log_remap: NULL pointer");
  if (rows < 1 || cols < 1 || rows > (1 << 20) || cols > (1 << 20))
    return fail(XR_ERR_INVALID_ARG, "xr_log_remap: bad image size");
  if (!use_max_as_i0 && !(i0 > 0.0f)) return fail(XR_ERR_INVALID_ARG, "xr_log_remap: I0 must be positive");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int64_t n = rows * cols;
  float2* a = reinterpret_cast<float2*>(d_scratch);
  float* part_max = reinterpret_cast<float*>(d_scratch + n);
  float* part_min = part_max + kRedBlocks;
  float* scal = part_min + kRedBlocks;
  const GaussKernel k = gauss_kernel(2.0);
  gauss_x_kernel<<<image_grid(rows, cols), 128, 0, s>>>(d_src, (int)rows, (int)cols, k, a);
  const unsigned bx = (unsigned)std::min<int64_t>((cols + 255) / 256, 64);
  const dim3 grid(bx, (unsigned)std::min<int64_t>(rows, kRedBlocks / bx));
  const int nblk = (int)(grid.x * grid.y);
  log_remap_stats_kernel<<<grid, 256, 0, s>>>(a, d_src, (int)rows, (int)cols, k, part_max, part_min);
  log_remap_finalize_kernel<<<1, 32, 0, s>>>(part_max, part_min, nblk, use_max_as_i0, i0, scal);
  log_remap_kernel<<<grid_for(n), 256, 0, s>>>(d_src, n, scal, d_dst);
  XR_CUDA_TRY(cudaGetLastError());
  return XR_OK;
}

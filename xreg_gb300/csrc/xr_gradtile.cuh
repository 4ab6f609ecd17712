// xr_gradtile.cuh -- device code shared by the split grad-NCC metric kernels
// (xr_metrics.cu) and the fused evaluation kernel (xr_raycast.cu): compensated
// reductions, the moments of one tile of a moving image's gradients, and the
// per-image FP64 combine.  Both paths run exactly this code
// on the same tiles, so their similarity values are identical bit for bit.
//
// Gradients (xregImgSimMetric2DGradImgCPU.cpp:48-65,86-101): OpenCV's sigma-0
// Gaussian [1 4 6 4 1]/16 (or [1 2 1]/4), then the 3x3 Sobel in x and y, with
// BORDER_REFLECT_101; NCC of each direction (xregImgSimMetric2DNCCCPU.cpp:
// 53-63,164-209), sim = 0.5 (s_x + s_y) (xregImgSimMetric2DGradNCCCPU.cpp:51-65).
#pragma once

#include "xr_internal.h"

namespace xr {
namespace gt {

constexpr int kThreads = 256;                     // block size of the NCC and patch kernels
// A tile is 2 x 2 strips, one per warp: a strip is kStripRows rows of the columns
// whose blur and Sobel stencils a warp's 32 columns hold.
constexpr int kStripRows = 32;
constexpr int kGH = 2 * kStripRows;               // tile rows
template <int KR>
constexpr int kTileCols = 2 * (32 - 2 * (KR + 1));
constexpr int kGW = kTileCols<2>;                 // tile columns of the 5x5 blur (52)
static_assert(kGH == kMetricTileRows && kGW == kMetricTileCols, "the host's tile counts");
constexpr int kTileThreads = 128;                 // the four warps
constexpr int kFinalizeThreads = 128;             // threads of the per-image combine

__device__ __forceinline__ int reflect101(int i, int n) {
  if (i < 0) i = -i;
  if (i >= n) i = 2 * (n - 1) - i;
  return i;
}

// A float-float value hi + lo (about 48 significant bits).
struct FF {
  float hi, lo;
};

// Knuth's two-sum on the FP32 pipe for float-float values: this GPU's FP64 pipe
// is slow enough that block reductions in double kept it 82 % busy and bounded
// the grad-NCC moment kernel.  Explicit _rn intrinsics keep every step unfused.
__device__ __forceinline__ FF ff_add(FF a, FF b) {
  const float s = __fadd_rn(a.hi, b.hi);
  const float bb = __fsub_rn(s, a.hi);
  float e = __fadd_rn(__fsub_rn(a.hi, __fsub_rn(s, bb)), __fsub_rn(b.hi, bb));  // s + e = a.hi + b.hi exactly
  e = __fadd_rn(e, __fadd_rn(a.lo, b.lo));
  const float hi = __fadd_rn(s, e);
  return FF{hi, __fsub_rn(e, __fsub_rn(hi, s))};
}

// a b exactly as a float-float (the rounding error of the product from one fma).
__device__ __forceinline__ FF ff_prod(float a, float b) {
  const float p = __fmul_rn(a, b);
  return FF{p, fmaf(a, b, -p)};
}

__device__ __forceinline__ FF ff_shfl_down(FF v, int o) {
  return FF{__shfl_down_sync(0xffffffffu, v.hi, o), __shfl_down_sync(0xffffffffu, v.lo, o)};
}

// Blur and Sobel arithmetic with every rounding explicit (no contraction), so
// every kernel that forms gradients gives the same bits.
__device__ __forceinline__ float blur5(float a, float b, float c, float d, float e) {
  return __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(0.0625f, a), __fmul_rn(0.25f, b)), __fmul_rn(0.375f, c)),
                             __fmul_rn(0.25f, d)),
                   __fmul_rn(0.0625f, e));
}
__device__ __forceinline__ float blur3(float a, float b, float c) {
  return __fadd_rn(__fadd_rn(__fmul_rn(0.25f, a), __fmul_rn(0.5f, b)), __fmul_rn(0.25f, c));
}
// Sobel at the centre of the blurred 3x3 neighbourhood a0 b0 c0 / a1 . c1 / a2 b2 c2
__device__ __forceinline__ void sobel3(float a0, float b0, float c0, float a1, float c1, float a2, float b2, float c2,
                                       float& gx, float& gy) {
  gx = __fadd_rn(__fadd_rn(__fsub_rn(c0, a0), __fmul_rn(2.0f, __fsub_rn(c1, a1))), __fsub_rn(c2, a2));
  gy = __fadd_rn(__fadd_rn(__fsub_rn(a2, a0), __fmul_rn(2.0f, __fsub_rn(b2, b0))), __fsub_rn(c2, c0));
}
// One pixel's contribution to the six moments.
__device__ __forceinline__ void moments_add(float (&m)[6], float gx, float gy, float fx, float fy) {
  m[0] = __fadd_rn(m[0], gx);
  m[1] = __fmaf_rn(gx, gx, m[1]);
  m[2] = __fmaf_rn(gx, fx, m[2]);
  m[3] = __fadd_rn(m[3], gy);
  m[4] = __fmaf_rn(gy, gy, m[4]);
  m[5] = __fmaf_rn(gy, fy, m[5]);
}

__device__ __forceinline__ double warp_sum_d(double v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

// Block-wide sum of K doubles per thread over the first nw warps (the others
// must hold zeros); result valid in thread 0.
template <int K>
__device__ __forceinline__ void block_sum_d(double (&v)[K], double* red /* [K][32] */, int nw) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const double w = warp_sum_d(v[k]);
    if (lane == 0 && warp < nw) red[k * 32 + warp] = w;
  }
  __syncthreads();
  if (warp == 0) {
#pragma unroll
    for (int k = 0; k < K; ++k) {
      double w = (lane < nw) ? red[k * 32 + lane] : 0.0;
      w = warp_sum_d(w);
      v[k] = w;
    }
  }
}

__device__ __forceinline__ double ncc_sim_from_moments(double sm, double smm, double smf, double n,
                                                       const FixedNCC& fx) {
  const double mean = sm / n;
  double var = (smm - n * mean * mean) / (n - 1.0);
  if (var < 0.0) var = 0.0;
  double sd = sqrt(var);
  if (sd < 1.0e-6) sd = 1.0e-6;
  const double cov = smf - mean * fx.sum_fhat;
  const double ncc = cov / (n * fx.sd * sd);
  return (1.0 - ncc) * 0.5;
}

// A pixel of a tile's input; CG reads through L2 only (pixels written earlier in
// the same kernel by other blocks).
template <bool CG>
__device__ __forceinline__ float tile_px(const float* __restrict__ p) {
  return CG ? __ldcg(p) : __ldg(p);
}

// Moments of the moving gradients over the kGH x kTileCols<KR> tile at (y0, x0), by
// the block's first four warps (all of its threads call it): each lane owns a
// column and goes down its strip's rows; the horizontal neighbours come by
// shuffles, the vertical ones stay in registers, so a pixel is read once from
// global memory and nothing goes through shared memory.  Sums are plain float over
// 8 rows of a column, float-float over the column, the lanes and the warps.  The
// value of moment k (S_gx, S_gx^2, S_gx fx, S_gy, S_gy^2, S_gy fy) is returned in
// thread k < 6.  red: [6][4].
// Bound by instruction issue: about 50 per pixel and lane, of which 26 of 32 lanes
// and 32 of 38 rows count.  100 images of 384^2 with their combines: 61 us, 150 with
// the tile's rows blurred in shared memory (5 loads and an index division per
// blurred value); one image 16 us.
template <int KR, bool CG>
__device__ double grad_tile_moments(const float* __restrict__ src, int rows, int cols, int y0, int x0,
                                    const float* __restrict__ fhx, const float* __restrict__ fhy,
                                    const uint8_t* __restrict__ mask, FF* red) {
  constexpr int H = KR + 1, kWin = 2 * KR + 1, kGroup = 8;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (warp < 4) {
    const int xs = x0 + (warp & 1) * (32 - 2 * H), ys = y0 + (warp >> 1) * kStripRows;  // the strip's first pixel
    const int x = xs - H + lane;
    // Rows / cols past the image's last pixel plus the halo only feed pixels that are
    // skipped; clamping before the reflection keeps every read inside the image.
    const float* pc = src + reflect101(min(x, cols - 1 + H), cols);
    const int xf = min(max(x, 0), cols - 1);  // lanes without a pixel of their own read some fixed value
    const bool owner = lane >= H && lane < 32 - H && x < cols;
    float hb[kWin];           // horizontally blurred rows
    float bl[3], lf[3], rt[3];  // blurred rows and their left and right neighbours
    FF acc[6];
#pragma unroll
    for (int q = 0; q < 6; ++q) acc[q] = FF{0.0f, 0.0f};
    auto row_of = [&](int r) -> const float* {  // input row r of the strip, from its first halo row
      const int y = min(ys - H + r, rows - 1 + H);
      return pc + (int64_t)reflect101(y, rows) * cols;
    };
    // takes one input row: the newest blurred row follows (garbage until the window is full)
    auto push = [&](float p) {
      float h = p;
      if constexpr (KR == 2)
        h = blur5(__shfl_up_sync(0xffffffffu, p, 2), __shfl_up_sync(0xffffffffu, p, 1), p,
                  __shfl_down_sync(0xffffffffu, p, 1), __shfl_down_sync(0xffffffffu, p, 2));
      else if constexpr (KR == 1)
        h = blur3(__shfl_up_sync(0xffffffffu, p, 1), p, __shfl_down_sync(0xffffffffu, p, 1));
#pragma unroll
      for (int i = 0; i + 1 < kWin; ++i) hb[i] = hb[i + 1];
      hb[kWin - 1] = h;
      bl[0] = bl[1]; bl[1] = bl[2];
      lf[0] = lf[1]; lf[1] = lf[2];
      rt[0] = rt[1]; rt[1] = rt[2];
      if constexpr (KR == 2) bl[2] = blur5(hb[0], hb[1], hb[2], hb[3], hb[4]);
      else if constexpr (KR == 1) bl[2] = blur3(hb[0], hb[1], hb[2]);
      else bl[2] = hb[0];
      lf[2] = __shfl_up_sync(0xffffffffu, bl[2], 1);
      rt[2] = __shfl_down_sync(0xffffffffu, bl[2], 1);
    };
#pragma unroll
    for (int i = 0; i < kWin; ++i) hb[i] = 0.0f;
#pragma unroll
    for (int i = 0; i < 3; ++i) bl[i] = lf[i] = rt[i] = 0.0f;
    {
      float p[2 * H];
#pragma unroll
      for (int i = 0; i < 2 * H; ++i) p[i] = tile_px<CG>(row_of(i));
#pragma unroll
      for (int i = 0; i < 2 * H; ++i) push(p[i]);
    }
#pragma unroll 1
    for (int g = 0; g < kStripRows && ys + g < rows; g += kGroup) {
      float p[kGroup], fx[kGroup], fy[kGroup], m[6] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
      const int64_t first = (int64_t)(ys + g) * cols + xf;
      auto sums = [&](int i) {
        float gx, gy;
        sobel3(lf[0], bl[0], rt[0], lf[1], rt[1], lf[2], bl[2], rt[2], gx, gy);
        moments_add(m, gx, gy, fx[i], fy[i]);
      };
      if (!mask && ys + g + H >= 0 && ys + g + kGroup + H <= rows) {  // no row to reflect, none to skip
        const float* q = pc + (int64_t)(ys + g + H) * cols;
#pragma unroll
        for (int i = 0; i < kGroup; ++i) {
          p[i] = tile_px<CG>(q + (int64_t)i * cols);
          fx[i] = __ldg(fhx + first + (int64_t)i * cols);
          fy[i] = __ldg(fhy + first + (int64_t)i * cols);
        }
#pragma unroll
        for (int i = 0; i < kGroup; ++i) {
          push(p[i]);
          sums(i);
        }
      } else {
        bool use[kGroup];
#pragma unroll
        for (int i = 0; i < kGroup; ++i) p[i] = tile_px<CG>(row_of(2 * H + g + i));
#pragma unroll
        for (int i = 0; i < kGroup; ++i) {
          const int64_t pix = first + (int64_t)i * cols;
          use[i] = owner && ys + g + i < rows && (!mask || mask[pix]);
          fx[i] = use[i] ? __ldg(fhx + pix) : 0.0f;
          fy[i] = use[i] ? __ldg(fhy + pix) : 0.0f;
        }
#pragma unroll
        for (int i = 0; i < kGroup; ++i) {
          push(p[i]);
          if (use[i]) sums(i);
        }
      }
#pragma unroll
      for (int q = 0; q < 6; ++q) {
        const float t = __fadd_rn(acc[q].hi, m[q]), d = __fsub_rn(t, acc[q].hi);
        acc[q].lo = __fadd_rn(acc[q].lo, __fadd_rn(__fsub_rn(acc[q].hi, __fsub_rn(t, d)), __fsub_rn(m[q], d)));
        acc[q].hi = t;
      }
    }
#pragma unroll
    for (int q = 0; q < 6; ++q) {
      acc[q].hi = owner ? acc[q].hi : 0.0f;
      acc[q].lo = owner ? acc[q].lo : 0.0f;
    }
    // over the lanes: the halves of the warp take three moments each, then 16 lanes each
    const bool upper = lane >= 16;
    FF v[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      const FF mine = upper ? acc[q + 3] : acc[q], theirs = upper ? acc[q] : acc[q + 3];
      const FF got{__shfl_xor_sync(0xffffffffu, theirs.hi, 16), __shfl_xor_sync(0xffffffffu, theirs.lo, 16)};
      v[q] = ff_add(mine, got);
    }
#pragma unroll
    for (int q = 0; q < 3; ++q) {
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) v[q] = ff_add(v[q], ff_shfl_down(v[q], o));
      if ((lane & 15) == 0) red[(q + (upper ? 3 : 0)) * 4 + warp] = v[q];
    }
  }
  __syncthreads();
  double out = 0.0;
  if (threadIdx.x < 6) {
    FF t = red[threadIdx.x * 4];
#pragma unroll
    for (int w = 1; w < 4; ++w) t = ff_add(t, red[threadIdx.x * 4 + w]);
    out = (double)t.hi + (double)t.lo;
  }
  __syncthreads();  // red is reused by the caller's next tile
  return out;
}

// Per-image combine: the tile partials (nblk x 6 doubles, read through L2 when
// CG) summed by the first kFinalizeThreads threads with that stride, then
// across their warps; the similarity value (valid in thread 0).
template <bool CG>
__device__ float grad_finalize_image(const double* __restrict__ p, int nblk, double n, const FixedNCC& fx,
                                     const FixedNCC& fy, double* red /* [6][4] */) {
  constexpr int kW = kFinalizeThreads / 32;
  double a[6] = {0, 0, 0, 0, 0, 0};
  if (threadIdx.x < kFinalizeThreads)
    for (int k = threadIdx.x; k < nblk; k += kFinalizeThreads)
      for (int j = 0; j < 6; ++j) a[j] = __dadd_rn(a[j], CG ? __ldcg(p + 6 * k + j) : p[6 * k + j]);
  {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      const double w = warp_sum_d(a[k]);
      if (lane == 0 && warp < kW) red[k * kW + warp] = w;
    }
    __syncthreads();
    if (warp == 0) {
#pragma unroll
      for (int k = 0; k < 6; ++k) a[k] = warp_sum_d((lane < kW) ? red[k * kW + lane] : 0.0);
    }
  }
  float out = 0.0f;
  if (threadIdx.x == 0) {
    const double sx = ncc_sim_from_moments(a[0], a[1], a[2], n, fx);
    const double sy = ncc_sim_from_moments(a[3], a[4], a[5], n, fy);
    // 0.5 * (float(s_x) + float(s_y)) as in ImgSimMetric2DGradNCCCPU::compute
    out = 0.5f * ((float)sx + (float)sy);
  }
  __syncthreads();  // red is reused
  return out;
}

// Mean over views of one candidate's values (ImgSimMetric2DCombineMean,
// xregImgSimMetric2DCombine.cpp:79-96).
__device__ __forceinline__ float combine_mean(const float* const* view_sims, int nviews, int64_t i, bool cg) {
  float s = 0.0f;
  for (int v = 0; v < nviews; ++v) s += cg ? __ldcg(view_sims[v] + i) : view_sims[v][i];
  return s / (float)nviews;
}

}  // namespace gt
}  // namespace xr

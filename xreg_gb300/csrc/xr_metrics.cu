// xr_metrics.cu -- 2D similarity metric kernels.
//
// NCC (xregImgSimMetric2DNCCCPU.cpp:53-63,164-209): per moving image the sums
// S_m, S_mm, S_mf (f = zero-mean fixed image) are accumulated per thread in
// compensated (Kahan) float, reduced per block in double, and combined per image
// in double:  mean_m = S_m/n, var_m = (S_mm - n mean_m^2)/(n-1), sd = max(1e-6, sqrt),
// cov = S_mf - mean_m * sum(f), ncc = cov / (n sd_f sd_m), sim = (1 - ncc)/2.
//
// Gradient images (xregImgSimMetric2DGradImgCPU.cpp:48-65,86-101): 5x5 Gaussian
// with OpenCV's fixed sigma-0 kernel [1 4 6 4 1]/16 (3x3: [1 2 1]/4), then 3x3
// Sobel in x and y, BORDER_REFLECT_101 everywhere.  A block stages a 32x32 tile
// plus halo in shared memory; the blurred tile is computed over the
// reflect-extended input, which equals the reflect-extended blurred image because
// the kernels are symmetric.
//
// Patch NCC (xregImgSimMetric2DPatchNCCCPU.cpp:205-287,558-619): a thread scores
// one or four patches of a column, two-pass mean / sample std dev over the (2r+1)^2
// window from a shared-memory tile, score 1 - sum((m - mu_m)/sd_m * fhat), mean over
// patches, weighted where asked.  The fixed side (per-patch mean and 1/(sd n)) is
// pre-computed once.
#include "xr_cmaes_core.h"
#include "xr_gradtile.cuh"

#include <cfloat>

namespace xr {
namespace {

constexpr int kT = 32;          // output tile edge for gradient kernels
using gt::kThreads;

using gt::FF;
using gt::ff_add;
using gt::ff_prod;
using gt::ff_shfl_down;
using gt::reflect101;
using gt::warp_sum_d;
using gt::ncc_sim_from_moments;

struct Kahan {
  float s = 0.0f, c = 0.0f;
  __device__ __forceinline__ void add(float x) {
    const float y = x - c;
    const float t = s + y;
    c = (t - s) - y;
    s = t;
  }
  __device__ __forceinline__ double value() const { return (double)s - (double)c; }
  __device__ __forceinline__ FF ff() const { return FF{s, -c}; }
};

// Block-wide sum of K float-float values per thread, returned in double by
// thread 0 (the other threads get undefined values).
template <int K>
__device__ __forceinline__ void block_sum_ff(FF (&v)[K], double (&out)[K], FF* red /* [K][32] */) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    FF w = v[k];
    for (int o = 16; o > 0; o >>= 1) w = ff_add(w, ff_shfl_down(w, o));
    if (lane == 0) red[k * 32 + warp] = w;
  }
  __syncthreads();
  if (warp == 0) {
#pragma unroll
    for (int k = 0; k < K; ++k) {
      FF w = (lane < nw) ? red[k * 32 + lane] : FF{0.0f, 0.0f};
      for (int o = 16; o > 0; o >>= 1) w = ff_add(w, ff_shfl_down(w, o));
      out[k] = (double)w.hi + (double)w.lo;
    }
  }
}

// Block-wide sum of K doubles per thread over all warps; result valid in thread 0.
template <int K>
__device__ __forceinline__ void block_sum_d(double (&v)[K], double* red /* [K][32] */) {
  gt::block_sum_d<K>(v, red, (int)(blockDim.x >> 5));
}

// ------------------------------------------------------------------ setup --
__global__ void image_sum_kernel(const float* __restrict__ img, int64_t n, const uint8_t* __restrict__ mask,
                                 double* __restrict__ out) {
  __shared__ double red[2 * 32];
  double v[2] = {0.0, 0.0};
  for (int64_t i = threadIdx.x; i < n; i += blockDim.x)
    if (!mask || mask[i]) { v[0] += (double)img[i]; v[1] += 1.0; }
  block_sum_d<2>(v, red);
  if (threadIdx.x == 0) { out[0] = v[0]; out[2] = v[1]; }
}

__global__ void image_var_kernel(const float* __restrict__ img, int64_t n, const uint8_t* __restrict__ mask,
                                 double* __restrict__ out) {
  __shared__ double red[1 * 32];
  const double mean = out[0] / out[2];
  double v[1] = {0.0};
  for (int64_t i = threadIdx.x; i < n; i += blockDim.x)
    if (!mask || mask[i]) { const double d = (double)img[i] - mean; v[0] += d * d; }
  block_sum_d<1>(v, red);
  if (threadIdx.x == 0) out[1] = v[0];
}

__global__ void sub_scalar_kernel(const float* __restrict__ in, int64_t n, float value, float* __restrict__ out) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    out[i] = in[i] - value;
}

// ---------------------------------------------------------------- NCC -----
__global__ void __launch_bounds__(kThreads) ncc_moments_kernel(const float* __restrict__ mov, int64_t npix,
                                                               const float* __restrict__ fhat,
                                                               const uint8_t* __restrict__ mask,
                                                               double* __restrict__ partials) {
  __shared__ FF red[3 * 32];
  const int64_t img = blockIdx.y;
  const float* m = mov + img * npix;
  Kahan s0, s1, s2;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < npix; i += (int64_t)gridDim.x * blockDim.x) {
    if (mask && !mask[i]) continue;
    const float x = m[i];
    s0.add(x);
    s1.add(x * x);
    s2.add(x * fhat[i]);
  }
  FF f[3] = {s0.ff(), s1.ff(), s2.ff()};
  double v[3];
  block_sum_ff<3>(f, v, red);
  if (threadIdx.x == 0) {
    double* o = partials + (img * gridDim.x + blockIdx.x) * 3;
    o[0] = v[0]; o[1] = v[1]; o[2] = v[2];
  }
}

// One block per image (as grad_finalize_kernel).
__global__ void ncc_finalize_kernel(const double* __restrict__ partials, int nblk, int64_t nimgs, double n,
                                    FixedNCC fx, float* __restrict__ sims) {
  __shared__ double red[3 * 32];
  const int64_t img = blockIdx.x;
  double a[3] = {0, 0, 0};
  const double* p = partials + img * nblk * 3;
  for (int k = threadIdx.x; k < nblk; k += blockDim.x) {
    a[0] += p[3 * k];
    a[1] += p[3 * k + 1];
    a[2] += p[3 * k + 2];
  }
  block_sum_d<3>(a, red);
  if (threadIdx.x == 0) sims[img] = (float)ncc_sim_from_moments(a[0], a[1], a[2], n, fx);
}

// ------------------------------------------------------ gradient images ---
// Stages rows [y0-H, y0+kT+H) x cols [x0-H, x0+kT+H) of an image (reflected at
// the borders), blurs with radius KR and applies Sobel on the kT x kT tile.
template <int KR>
struct GradTile {
  static constexpr int H = KR + 1;            // total halo
  static constexpr int WI = kT + 2 * H;       // staged input edge
  static constexpr int WB = kT + 2;           // blurred region edge
  float in[WI][WI + 1];
  float hb[WI][WB + 1];
  float bl[WB][WB + 1];

  __device__ void load(const float* __restrict__ img, int rows, int cols, int y0, int x0) {
    for (int i = threadIdx.x; i < WI * WI; i += blockDim.x) {
      const int r = i / WI, c = i - r * WI;
      // Rows/cols past the last tile pixel only feed pixels that are skipped;
      // clamping before the reflection keeps every read inside the image.
      const int gr = reflect101(min(y0 - H + r, rows - 1 + H), rows);
      const int gc = reflect101(min(x0 - H + c, cols - 1 + H), cols);
      in[r][c] = img[(int64_t)gr * cols + gc];
    }
    __syncthreads();
  }

  __device__ void blur() {
    if constexpr (KR == 0) {
      for (int i = threadIdx.x; i < WB * WB; i += blockDim.x) {
        const int r = i / WB, c = i - r * WB;
        bl[r][c] = in[r][c];
      }
      __syncthreads();
    } else {
    // horizontal pass over all staged rows, blurred columns [x0-1, x0+kT+1)
    for (int i = threadIdx.x; i < WI * WB; i += blockDim.x) {
      const int r = i / WB, c = i - r * WB;
      float s;
      if (KR == 2) {
        s = 0.0625f * in[r][c] + 0.25f * in[r][c + 1] + 0.375f * in[r][c + 2] + 0.25f * in[r][c + 3] +
            0.0625f * in[r][c + 4];
      } else {
        s = 0.25f * in[r][c] + 0.5f * in[r][c + 1] + 0.25f * in[r][c + 2];
      }
      hb[r][c] = s;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < WB * WB; i += blockDim.x) {
      const int r = i / WB, c = i - r * WB;
      float s;
      if (KR == 2) {
        s = 0.0625f * hb[r][c] + 0.25f * hb[r + 1][c] + 0.375f * hb[r + 2][c] + 0.25f * hb[r + 3][c] +
            0.0625f * hb[r + 4][c];
      } else {
        s = 0.25f * hb[r][c] + 0.5f * hb[r + 1][c] + 0.25f * hb[r + 2][c];
      }
      bl[r][c] = s;
    }
    __syncthreads();
    }
  }

  // Sobel at tile pixel (ty, tx) in [0, kT).
  __device__ __forceinline__ void sobel(int ty, int tx, float& gx, float& gy) const {
    const int r = ty + 1, c = tx + 1;
    const float a = bl[r - 1][c - 1], b = bl[r - 1][c], cc = bl[r - 1][c + 1];
    const float d = bl[r][c - 1], f = bl[r][c + 1];
    const float g = bl[r + 1][c - 1], h = bl[r + 1][c], ii = bl[r + 1][c + 1];
    gx = ((cc - a) + 2.0f * (f - d)) + (ii - g);
    gy = ((g - a) + 2.0f * (h - b)) + (ii - cc);
  }
};

template <int KR>
__global__ void __launch_bounds__(kThreads) grad_images_kernel(const float* __restrict__ imgs, int rows, int cols,
                                                               float* __restrict__ gx, float* __restrict__ gy) {
  __shared__ GradTile<KR> t;
  const int tiles_x = (cols + kT - 1) / kT;
  const int y0 = (blockIdx.x / tiles_x) * kT, x0 = (blockIdx.x % tiles_x) * kT;
  const int64_t npix = (int64_t)rows * cols;
  const int64_t img = blockIdx.y;
  t.load(imgs + img * npix, rows, cols, y0, x0);
  t.blur();
  for (int i = threadIdx.x; i < kT * kT; i += blockDim.x) {
    const int ty = i / kT, tx = i - ty * kT;
    if (y0 + ty >= rows || x0 + tx >= cols) continue;
    float a, b;
    t.sobel(ty, tx, a, b);
    const int64_t o = img * npix + (int64_t)(y0 + ty) * cols + x0 + tx;
    gx[o] = a;
    gy[o] = b;
  }
}

// Moments of the moving gradients, one tile per block (gt::grad_tile_moments,
// shared with the fused evaluation kernel).
using gt::kGH;
using gt::kGW;

template <int KR>
__global__ void __launch_bounds__(gt::kTileThreads, 5) grad_moments_kernel(const float* __restrict__ imgs, int rows,
                                                                        int cols, const float* __restrict__ fhx,
                                                                        const float* __restrict__ fhy,
                                                                        const uint8_t* __restrict__ mask,
                                                                        double* __restrict__ partials) {
  __shared__ FF red[6 * 4];
  const int tiles_x = (cols + gt::kTileCols<KR> - 1) / gt::kTileCols<KR>;
  const int y0 = (blockIdx.x / tiles_x) * kGH, x0 = (blockIdx.x % tiles_x) * gt::kTileCols<KR>;
  const int64_t img = blockIdx.y;
  const double v = gt::grad_tile_moments<KR, false>(imgs + img * (int64_t)rows * cols, rows, cols, y0, x0, fhx, fhy, mask,
                                                    red);
  if (threadIdx.x < 6) partials[(img * gridDim.x + blockIdx.x) * 6 + threadIdx.x] = v;
}

// One block of 128 threads per image: the tile partials combined in double
// (gt::grad_finalize_image, shared with the fused evaluation kernel).
__global__ void grad_finalize_kernel(const double* __restrict__ partials, int nblk, int64_t nimgs, double n,
                                     FixedNCC fx, FixedNCC fy, float* __restrict__ sims) {
  __shared__ double red[6 * (gt::kFinalizeThreads / 32)];
  const int64_t img = blockIdx.x;
  const float v = gt::grad_finalize_image<false>(partials + img * nblk * 6, nblk, n, fx, fy, red);
  if (threadIdx.x == 0) sims[img] = v;
}

// Batched grad-NCC over many jobs' images (launch_grad_multi): one block per
// tile, grid-stride; the counters of FusedJob::cnt (images, then poses)
// chain the per-image combine and the mean over views behind the tiles.
// A device CMA-ES job's update from its lambda values (the float means over
// views, widened to double as the host step does) by a whole block: the stages
// of cma::update (cmaes_UpdateDistribution, then cmaes_TestForTermination),
// the ranks, recombination sums and covariance entries one per thread.
__device__ __noinline__ void cma_update_block(void* state, const float* vals, CmaReport* report) {
  __shared__ double scal[3];
  const cma::View s = cma::view(state);
  const int n = s.h->n, lam = s.h->lam, mu = s.h->mu, nt = blockDim.x, tid = threadIdx.x;
  for (int k = tid; k < lam; k += nt) s.fv[k] = (double)__ldcg(vals + k);
  __syncthreads();
  for (int k = tid; k < lam; k += nt) cma::rank(s, k);
  __syncthreads();
  if (tid == 0) cma::keep_best(s);
  __syncthreads();
  for (int t = tid; t < 2 * n; t += nt) cma::recombine(s, t);
  __syncthreads();
  if (tid == 0) cma::paths(s, scal);
  __syncthreads();
  for (int t = tid; t < mu * n; t += nt) cma::steps(s, t);
  __syncthreads();
  for (int e = tid; e < n * (n + 1) / 2; e += nt) cma::covariance(s, e, scal);
  __syncthreads();
  if (tid == 0) cma::step_size(s, scal);
  for (int e = tid; e < n * n; e += nt) cma::eig_cb(s, e);
  __syncthreads();
  for (int e = tid; e < n * (n + 1) / 2; e += nt) cma::eig_btcb(s, e);
  __syncthreads();
  const int pairs = cma::rr_pairs(n), rounds = cma::rr_rounds(n);
  for (int sweep = 0; sweep < cma::kMaxSweeps; ++sweep) {
    if (tid == 0) s.h->rotated = 0;
    __syncthreads();
    for (int r = 0; r < rounds; ++r) {
      for (int i = tid; i < pairs; i += nt) cma::rot_params(n, s.A, r, i, s.rot, &s.h->rotated);
      __syncthreads();
      for (int e = tid; e < pairs * n; e += nt) cma::rot_cols(n, s.A, s.V, r, e / n, s.rot, e % n);
      __syncthreads();
      for (int e = tid; e < pairs * n; e += nt) cma::rot_rows(n, s.A, r, e / n, s.rot, e % n);
      __syncthreads();
    }
    const int rotated = *(volatile int32_t*)&s.h->rotated;
    __syncthreads();  // every thread has read the flag before the next sweep clears it
    if (!rotated) break;
  }
  for (int e = tid; e < n * n; e += nt) cma::eig_bv(s, e);
  __syncthreads();
  for (int e = tid; e < n * n; e += nt) s.B[e] = s.T[e];
  __syncthreads();
  if (tid == 0) {
    cma::finish(s);
    if (report) {
      report->reason = s.h->reason;
      double r = 0.0, t = 0.0;
      for (int i = 0; i < n; ++i) {
        const double sd = s.h->sigma * sqrt(s.C[i * n + i]);
        if (i < 3) r = fmax(r, sd);
        else t = fmax(t, sd);
      }
      report->sd_rot = r;
      report->sd_trans = t;
    }
  }
  __syncthreads();
}

__global__ void cma_update_kernel(const CmaUpdateJob* __restrict__ jobs) {
  cma_update_block(jobs[blockIdx.x].cma, jobs[blockIdx.x].vals, jobs[blockIdx.x].report);
}

// The last tile of an image combines its moments (FP64); the last view of a
// pose, the mean over views; the last pose of a job with a device optimizer,
// the optimizer's update (the whole block).  Out of line so the tile loop keeps
// the register budget of the per-view moments kernel (40 registers, 6 blocks
// per SM, where the inlined FP64 combine took 80 and 3).
__device__ __noinline__ void grad_multi_finish(const FusedJob& J, const FusedView& V, int64_t k, int mt, int64_t nimg,
                                               double* dred, int* job_done) {
  __threadfence();
  const float sim = gt::grad_finalize_image<true>(V.partials + k * mt * 6, mt, V.n_used, V.fx, V.fy, dred);
  if (threadIdx.x == 0) {
    int done = 0;
    V.sims[k] = sim;
    __threadfence();
    unsigned int* cp = J.cnt + nimg * mt + nimg + k;
    if (atomicAdd(cp, 1u) + 1u == (unsigned int)J.nviews) {  // every view of this pose
      *cp = 0u;
      __threadfence();
      float sum = 0.0f;
      for (int w = 0; w < J.nviews; ++w) sum += __ldcg(J.views[w].sims + k);
      J.out[k] = sum / (float)J.nviews;  // ImgSimMetric2DCombineMean (as gt::combine_mean)
      if (J.cma) {  // the job's last pose: its optimizer's update by this block
        __threadfence();
        unsigned int* cj = J.cnt + nimg * mt + nimg + J.pop;
        if (atomicAdd(cj, 1u) + 1u == (unsigned int)J.pop) {
          *cj = 0u;
          done = 1;
        }
      }
    }
    *job_done = done;
  }
  __syncthreads();
  if (*job_done) {
    __threadfence();
    cma_update_block(J.cma, J.out, J.report);
  }
}

__global__ void __launch_bounds__(gt::kTileThreads, 5) grad_multi_kernel(const FusedJob* __restrict__ jobs, int njobs,
                                                                      long long total) {
  __shared__ FF red[6 * 4];
  __shared__ double dred[6 * (gt::kFinalizeThreads / 32)];
  __shared__ int s_last, s_job_done;
  for (long long t = blockIdx.x; t < total; t += gridDim.x) {
    int j = 0;
    while (j + 1 < njobs && jobs[j + 1].tile_begin <= t) ++j;
    const FusedJob& J = jobs[j];
    const int rows = J.d.p.rows, cols = J.d.p.cols, mt = J.mt_x * J.mt_y;
    const long long local = t - J.tile_begin;
    const int64_t img = local / mt;  // projection: view-major (view * pop + pose)
    const int M = (int)(local - img * mt);
    const int64_t nimg = (int64_t)J.nviews * J.pop, v = img / J.pop, k = img - v * J.pop;
    const FusedView& V = J.views[v];
    const double val = gt::grad_tile_moments<2, false>(J.d.p.out + img * (int64_t)rows * cols, rows, cols,
                                                       (M / J.mt_x) * kGH, (M % J.mt_x) * kGW, V.fhx, V.fhy, V.mask, red);
    if (threadIdx.x < 6) {
      V.partials[(k * mt + M) * 6 + threadIdx.x] = val;
      __threadfence();
      __syncwarp(0x3f);
    }
    if (threadIdx.x == 0) {
      unsigned int* ci = J.cnt + nimg * mt + img;
      s_last = atomicAdd(ci, 1u) + 1u == (unsigned int)mt;
      if (s_last) *ci = 0u;
    }
    __syncthreads();
    if (s_last) grad_multi_finish(J, V, k, mt, nimg, dred, &s_job_done);  // every tile of this image is in
    __syncthreads();
  }
}

// ------------------------------------------------------------ patch NCC ---
constexpr int kPC = 16;  // patch centres per tile edge

// Per-patch statistics of a fixed image (ComputePatchMeanStdDev,
// xregImgSimMetric2DPatchNCCCPU.cpp:558-619, in double): pixels that count are
// all of them, or the masked-in ones when use_mask_stats; the mean is divided
// and the variance formed only when more than one pixel counts; sd >= 1e-6.
// mean / scale = 1 / (sd n) give the scaled fixed patch (f - mean) scale.
// wvar (optional): the squared sd used as a patch weight (with the mask when
// there is one, xregImgSimMetric2DPatchNCCCPU.cpp:402-411); ucount (optional):
// masked-in pixels of the patch.
__device__ void patch_stats_d(const float* __restrict__ img, int cols, int r0, int c0, int d,
                              const uint8_t* __restrict__ mask, int use_mask, double* mu_out, double* sd_out,
                              int* n_out) {
  int n = 0;
  double s = 0;
  for (int r = 0; r < d; ++r)
    for (int c = 0; c < d; ++c) {
      const int64_t i = (int64_t)(r0 + r) * cols + c0 + c;
      if (!use_mask || !mask || mask[i]) { s += img[i]; ++n; }
    }
  double var = 0;
  if (n > 1) {
    s /= (double)n;
    for (int r = 0; r < d; ++r)
      for (int c = 0; c < d; ++c) {
        const int64_t i = (int64_t)(r0 + r) * cols + c0 + c;
        if (!use_mask || !mask || mask[i]) { const double t = img[i] - s; var += t * t; }
      }
    var /= (double)(n - 1);
  }
  double sd = sqrt(var);
  if (sd < 1.0e-6) sd = 1.0e-6;
  *mu_out = s;
  *sd_out = sd;
  *n_out = n;
}

__global__ void patch_fixed_stats_kernel(const float* __restrict__ img, int cols, int radius, int stride, int ncr,
                                         int ncc, const uint8_t* __restrict__ mask, int use_mask_stats,
                                         float* __restrict__ mean, float* __restrict__ scale,
                                         float* __restrict__ wvar, int* __restrict__ ucount) {
  const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= (int64_t)ncr * ncc) return;
  const int pr = (int)(p / ncc), pc = (int)(p - (int64_t)pr * ncc);
  const int r0 = pr * stride, c0 = pc * stride, d = 2 * radius + 1;
  double mu, sd;
  int n;
  patch_stats_d(img, cols, r0, c0, d, mask, use_mask_stats, &mu, &sd, &n);
  if (mean) {
    mean[p] = (float)mu;
    scale[p] = (float)(1.0 / (sd * (double)n));
  }
  if (wvar) {
    if (mask && !use_mask_stats) patch_stats_d(img, cols, r0, c0, d, mask, 1, &mu, &sd, &n);
    wvar[p] = (float)(sd * sd);
  }
  if (ucount) {
    int k = 0;
    for (int r = 0; r < d; ++r)
      for (int c = 0; c < d; ++c) k += (!mask || mask[(int64_t)(r0 + r) * cols + c0 + c]) ? 1 : 0;
    ucount[p] = k;
  }
}

// Shared-memory layout of patch_ncc_kernel for one tile of kPC x kPC patch centres.
struct PatchLayout {
  int Wr, Wc;    // patch-window region (moving gradient / fixed tiles)
  int WIr, WIc;  // staged input
  int WBr, WBc;  // blurred
  size_t fbytes;  // float part
  size_t bytes;   // plus the Wr x Wc mask tile
  __host__ __device__ static PatchLayout make(int radius, int stride, int grad, int kr) {
    PatchLayout L;
    L.Wc = (kPC - 1) * stride + 2 * radius + 1;
    L.Wr = L.Wc;
    L.WBc = grad ? L.Wc + 2 : L.Wc;
    L.WBr = grad ? L.Wr + 2 : L.Wr;
    L.WIc = grad ? L.WBc + 2 * kr : L.Wc;
    L.WIr = grad ? L.WBr + 2 * kr : L.Wr;
    const size_t w = (size_t)L.Wr * L.Wc;
    const size_t fl = grad ? ((size_t)L.WIr * L.WIc + (size_t)L.WIr * L.WBc + (size_t)L.WBr * L.WBc + 4 * w)
                           : ((size_t)L.WIr * L.WIc + w);
    L.fbytes = fl * sizeof(float);
    L.bytes = L.fbytes + ((w + 15) & ~(size_t)15);
    return L;
  }
};

// Score 1 - sum over masked-in pixels of (m - mu_m) / sd_m * (f - fmean) fscale,
// moving statistics over all pixels (masked-in ones when use_mask_stats); the
// unmasked case is the plain patch NCC.  *var = sd_m^2.
__device__ __forceinline__ float patch_score(const float* __restrict__ m, const float* __restrict__ f,
                                             const uint8_t* __restrict__ mk, int W, int r0, int c0, int d,
                                             float fmean, float fscale, int use_mask_stats, int mask_in_sums) {
  float s = 0.0f;
  int n = 0;
  for (int r = 0; r < d; ++r)
    for (int c = 0; c < d; ++c)
      if (!use_mask_stats || !mk || mk[(r0 + r) * W + c0 + c]) { s += m[(r0 + r) * W + c0 + c]; ++n; }
  const float mu = n > 1 ? s / (float)n : s;
  float v = 0.0f, cov = 0.0f;
  for (int r = 0; r < d; ++r)
    for (int c = 0; c < d; ++c) {
      const int i = (r0 + r) * W + c0 + c;
      const float dm = m[i] - mu;
      if (!use_mask_stats || !mk || mk[i]) v = fmaf(dm, dm, v);
      if (!mk || !mask_in_sums || mk[i]) cov = fmaf(dm, f[i] - fmean, cov);
    }
  float sd = n > 1 ? sqrtf(v / (float)(n - 1)) : 0.0f;
  sd = fmaxf(sd, 1.0e-6f);
  return 1.0f - (cov / sd) * fscale;
}

// Sample variance (sd clamped at 1e-6, squared) of a d x d window with row pitch P.
__device__ __forceinline__ float patch_var(const float* __restrict__ m, int P, int r0, int c0, int d) {
  float s = 0.0f;
  for (int r = 0; r < d; ++r)
    for (int c = 0; c < d; ++c) s += m[(r0 + r) * P + c0 + c];
  const float n = (float)(d * d);
  const float mu = s / n;
  float v = 0.0f;
  for (int r = 0; r < d; ++r)
    for (int c = 0; c < d; ++c) {
      const float dm = m[(r0 + r) * P + c0 + c] - mu;
      v = fmaf(dm, dm, v);
    }
  const float sd = fmaxf(sqrtf(v / (n - 1.0f)), 1.0e-6f);
  return sd * sd;
}

// PASS 0: per image and direction, the sum over used patches with an unmasked
// centre of count x moving-patch variance (the normaliser of variance weights).
// PASS 1: per image and direction, the sum over used patches of
// count x weight x score (weight 1 when not weighting in the combine).
// The general kernel, one patch per thread: moving-variance weights, masked
// statistics, and tiles too large for patch_rows_kernel.
template <int GRAD, int KR, int PASS>
__global__ void __launch_bounds__(kThreads) patch_ncc_kernel(const float* __restrict__ imgs, int rows, int cols,
                                                             int radius, int stride, int ncr, int ncc,
                                                             PatchFixed px, PatchFixed py, PatchRun run,
                                                             double* __restrict__ partials) {
  extern __shared__ float sm[];
  __shared__ FF red[2 * 32];
  const PatchLayout L = PatchLayout::make(radius, stride, GRAD, KR);
  const int Wr = L.Wr, Wc = L.Wc, WIr = L.WIr, WIc = L.WIc, WBr = L.WBr, WBc = L.WBc;
  const int WW = Wr * Wc;
  float* s_in = sm;                              // WIr x WIc
  float* s_hb = s_in + WIr * WIc;                // WIr x WBc (GRAD)
  float* s_bl = s_hb + WIr * WBc;                // WBr x WBc (GRAD)
  float* s_mx = GRAD ? s_bl + WBr * WBc : s_in;  // Wr x Wc moving (gx or raw)
  float* s_my = s_mx + WW;                       // Wr x Wc moving gy
  float* s_fx = GRAD ? s_my + WW : s_in + WIr * WIc;  // Wr x Wc fixed (gx or raw)
  float* s_fy = s_fx + WW;
  uint8_t* s_mk = reinterpret_cast<uint8_t*>(reinterpret_cast<char*>(sm) + L.fbytes);  // Wr x Wc mask

  const int tiles_x = (ncc + kPC - 1) / kPC;
  const int tpr = blockIdx.x / tiles_x, tpc = blockIdx.x - tpr * tiles_x;
  const int pr0 = tpr * kPC, pc0 = tpc * kPC;
  const int y0 = pr0 * stride, x0 = pc0 * stride;  // top-left pixel of the window region
  const int64_t npix = (int64_t)rows * cols;
  const int64_t img = blockIdx.y;
  const float* src = imgs + img * npix;
  const int H = GRAD ? (KR + 1) : 0;
  const uint8_t* mk = run.mask ? s_mk : nullptr;

  for (int i = threadIdx.x; i < WIr * WIc; i += blockDim.x) {
    const int r = i / WIc, c = i - r * WIc;
    const int gr = reflect101(min(y0 - H + r, rows - 1 + H), rows);
    const int gc = reflect101(min(x0 - H + c, cols - 1 + H), cols);
    s_in[i] = src[(int64_t)gr * cols + gc];
  }
  for (int i = threadIdx.x; i < WW; i += blockDim.x) {
    const int r = i / Wc, c = i - r * Wc;
    const int gr = min(y0 + r, rows - 1), gc = min(x0 + c, cols - 1);
    if (PASS == 1) {
      s_fx[i] = px.img[(int64_t)gr * cols + gc];
      if (GRAD) s_fy[i] = py.img[(int64_t)gr * cols + gc];
    }
    if (run.mask) s_mk[i] = run.mask[(int64_t)gr * cols + gc];
  }
  __syncthreads();
  const bool need_grads = GRAD && (PASS == 1 || run.mvar == 2);
  if (need_grads) {
    if (KR == 0) {
      for (int i = threadIdx.x; i < WBr * WBc; i += blockDim.x) {
        const int r = i / WBc, c = i - r * WBc;
        s_bl[i] = s_in[r * WIc + c];
      }
    } else {
      for (int i = threadIdx.x; i < WIr * WBc; i += blockDim.x) {
        const int r = i / WBc, c = i - r * WBc;
        const float* q = s_in + r * WIc + c;
        s_hb[i] = (KR == 2) ? (0.0625f * q[0] + 0.25f * q[1] + 0.375f * q[2] + 0.25f * q[3] + 0.0625f * q[4])
                            : (0.25f * q[0] + 0.5f * q[1] + 0.25f * q[2]);
      }
      __syncthreads();
      for (int i = threadIdx.x; i < WBr * WBc; i += blockDim.x) {
        const int r = i / WBc, c = i - r * WBc;
        const float* q = s_hb + r * WBc + c;
        s_bl[i] = (KR == 2) ? (0.0625f * q[0] + 0.25f * q[WBc] + 0.375f * q[2 * WBc] + 0.25f * q[3 * WBc] +
                               0.0625f * q[4 * WBc])
                            : (0.25f * q[0] + 0.5f * q[WBc] + 0.25f * q[2 * WBc]);
      }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < WW; i += blockDim.x) {
      const int r = i / Wc + 1, c = i % Wc + 1;
      const float* q = s_bl;
      const float a = q[(r - 1) * WBc + c - 1], b = q[(r - 1) * WBc + c], cc = q[(r - 1) * WBc + c + 1];
      const float d = q[r * WBc + c - 1], f = q[r * WBc + c + 1];
      const float g = q[(r + 1) * WBc + c - 1], h = q[(r + 1) * WBc + c], ii = q[(r + 1) * WBc + c + 1];
      s_mx[i] = ((cc - a) + 2.0f * (f - d)) + (ii - g);
      s_my[i] = ((g - a) + 2.0f * (h - b)) + (ii - cc);
    }
  }
  __syncthreads();

  FF v[2] = {FF{0.0f, 0.0f}, FF{0.0f, 0.0f}};
  const int lr = threadIdx.x / kPC, lc = threadIdx.x % kPC;
  const int pc = pc0 + lc;
  const int d = 2 * radius + 1;
  const int c0 = lc * stride;
  {
    const int pr = pr0 + lr;
    if (pr < ncr && pc < ncc) {
      const int64_t pidx = (int64_t)pr * ncc + pc;
      const int cnt = run.cnt ? run.cnt[pidx] : 1;
      const int r0 = lr * stride;
      const bool centre = !mk || mk[(r0 + radius) * Wc + c0 + radius];
      if (cnt > 0) {
        // moving-patch variances used as weights: of the moving image itself
        // (mvar 1, shared by both directions) or of each gradient image (mvar 2)
        float var0 = 0.0f, var1 = 0.0f;
        if (run.mvar && centre) {
          if (run.mvar == 1) {
            var0 = GRAD ? patch_var(s_in + H * WIc + H, WIc, r0, c0, d) : patch_var(s_mx, Wc, r0, c0, d);
            var1 = var0;
          } else {
            var0 = patch_var(s_mx, Wc, r0, c0, d);
            if (GRAD) var1 = patch_var(s_my, Wc, r0, c0, d);
          }
        }
        if (PASS == 0) {
          v[0] = ff_prod((float)cnt, var0);
          v[1] = ff_prod((float)cnt, var1);
        } else {
          float w[2];
          for (int k = 0; k < 2; ++k) {
            const PatchFixed& P = k == 0 ? px : py;
            if (run.mvar) {
              float vk = k == 0 ? var0 : var1;
              if (run.normalize) {
                const float S = (float)run.mvar_sum[img * 2 + k];
                vk = S > 1.0e-6f ? vk / S : 0.0f;
              }
              w[k] = vk;
            } else {
              w[k] = P.w ? P.w[pidx] : 1.0f;
            }
          }
          float kept = 0.0f;  // per-patch score as xReg keeps it (0.5 (s_x + s_y) for GRAD)
          if (!run.weighted || fabsf(w[0]) > 1.0e-6f) {
            const float sc = patch_score(s_mx, s_fx, mk, Wc, r0, c0, d, px.mean[pidx], px.scale[pidx],
                                         run.use_mask_stats, run.mask_in_sums);
            v[0] = ff_prod((float)cnt, (run.weighted ? w[0] : 1.0f) * sc);
            kept += GRAD ? 0.5f * sc : sc;
          }
          if (GRAD && (!run.weighted || fabsf(w[1]) > 1.0e-6f)) {
            const float sc = patch_score(s_my, s_fy, mk, Wc, r0, c0, d, py.mean[pidx], py.scale[pidx],
                                         run.use_mask_stats, run.mask_in_sums);
            v[1] = ff_prod((float)cnt, (run.weighted ? w[1] : 1.0f) * sc);
            kept += 0.5f * sc;
          }
          if (run.scores) run.scores[img * (int64_t)ncr * ncc + pidx] = kept;
        }
      }
    }
  }
  double t[2];
  block_sum_ff<2>(v, t, red);
  if (threadIdx.x == 0) {
    double* o = partials + (img * gridDim.x + blockIdx.x) * 2;
    o[0] = t[0];
    o[1] = t[1];
  }
}

// ---- patches stacked in a column (the common case) ----
// A tile is 32 columns of patches by RB rows of them per warp; a thread scores RB patches
// of one column, so a pixel is read once for all of them and their row sums give
// every patch's mean.  Two channels run side by side as packed pairs (one
// instruction for two, each lane rounded as the scalar one): the two gradients of an
// image, or two images of the plain patch metric.  Per patch two passes as in
// patch_score: the mean, then the deviations.  Bound by the FP32 pipe (4 operations a
// pixel, patch and channel) at 24 warps an SM, for which the columns of a row are taken
// in two parts and a mask is kept in bytes (at 16 warps eight patches a thread were
// needed: masked calls and strides of 2 were 5 to 12 % slower).  20 images of 768^2, 11
// x 11, both gradients: 1175 us one channel at a time, now 632; 24 plain images of 384^2:
// 180 us, now 98; 8 images of 187 x 118 at stride 3, a whole call: 55 us, now 47.
// Every RB takes the same operations in the same order, patch by patch and up to the
// partial sums (one for 8 rows of patches), so an image's value does not depend on
// how many others share the launch.
// Pixel x of a row lies at (x mod stride) Wp + x / stride, so that the lanes of a
// read (one patch column each) are neighbours for every stride.
constexpr int kPartRows = 8;

struct PatchRows {
  int Wr, Wc, Wp, P;  // the tile's pixels, columns of a residue, pitch (stride Wp)
  int edge;           // of a patch, as offsets of its columns (four at a time; first in memory)
  size_t bytes;
  __host__ __device__ static PatchRows make(int radius, int stride, int grad, bool mask, int rb) {
    PatchRows L;
    L.Wc = 31 * stride + 2 * radius + 1;
    L.Wr = (8 * rb - 1) * stride + 2 * radius + 1;
    L.Wp = (L.Wc + stride - 1) / stride;
    L.P = stride * L.Wp;
    L.edge = (2 * radius + 4) & ~3;
    const int words = grad ? 4 : (rb > 1 ? 3 : 2);  // the moving side, in pairs but for rb 1, and the fixed one
    L.bytes = (size_t)L.edge * 4 + (size_t)L.Wr * L.P * (4 * words + (mask ? 1 : 0));
    return L;
  }
};

typedef unsigned long long u64;

// the same for one channel: the first value
template <typename V>
__device__ __forceinline__ V pack2(float a, float b) {
  if constexpr (sizeof(V) == 4) return a;
  else {
    u64 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
  }
}
__device__ __forceinline__ float2 unpack2(float v) { return make_float2(v, v); }
__device__ __forceinline__ float add2(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float fma2(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ float2 unpack2(u64 r) {
  float2 v;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(v.x), "=f"(v.y) : "l"(r));
  return v;
}
__device__ __forceinline__ u64 add2(u64 a, u64 b) {
  u64 d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ u64 fma2(u64 a, u64 b, u64 c) {
  u64 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}

// body(std::integral_constant<int, N>, offsets) for the columns of a patch row, in
// order, N at a time: all at once (HALVES: in two parts) where edge and stride (1 or 2)
// are known, else in fours
template <int DC, int SC, bool HALVES, typename Body>
__device__ __forceinline__ void patch_columns(int d, int Wp, const int4* __restrict__ offs, Body body) {
  if constexpr (DC > 0) {
    int o[DC];
#pragma unroll
    for (int c = 0; c < DC; ++c) o[c] = (c % SC) * Wp + c / SC;
    if constexpr (HALVES) {
      body(std::integral_constant<int, DC - DC / 2>(), o);
      int o2[DC / 2];
#pragma unroll
      for (int c = 0; c < DC / 2; ++c) o2[c] = o[DC - DC / 2 + c];
      body(std::integral_constant<int, DC / 2>(), o2);
    } else {
      body(std::integral_constant<int, DC>(), o);
    }
  } else {
    int c = 0;
#pragma unroll 1
    for (; c + 4 <= d; c += 4) {
      const int4 q = offs[c >> 2];
      const int o[4] = {q.x, q.y, q.z, q.w};
      body(std::integral_constant<int, 4>(), o);
    }
    const int4 q = offs[c >> 2];  // d is odd
    if (d & 2) {
      const int o[3] = {q.x, q.y, q.z};
      body(std::integral_constant<int, 3>(), o);
    } else {
      const int o[1] = {q.x};
      body(std::integral_constant<int, 1>(), o);
    }
  }
}

// a mask byte (-1 or 0) as 1 or 0 in every channel
template <typename V>
__device__ __forceinline__ V patch_mask(int m) {
  const float k = __uint_as_float((unsigned int)m & 0x3f800000u);
  return pack2<V>(k, k);
}

// Scores of RB stacked patches in both channels; their first window starts at m[0]
// (V: a pair of channels, or one), f[0] (as m, or FS: one value for both), mk[0] (MASK: -1 or 0 per
// pixel, f zero where it is 0), row pitch P.  DC and SC: the patch edge and stride when
// known.  scale(j): the patch's 1 / sd of the fixed side, per channel.
template <typename V, int RB, int DC, int SC, bool MASK, bool FS, typename Scale>
__device__ __forceinline__ void patch_column_scores(const V* __restrict__ m, const void* __restrict__ f,
                                                    const int8_t* __restrict__ mk, int P, int Wp, const int4* __restrict__ offs,
                                                    int d_rt, int stride_rt, const V (&fmean)[RB], Scale scale,
                                                    float2 (&score)[RB]) {
  const int d = DC > 0 ? DC : d_rt, stride = DC > 0 ? SC : stride_rt;
  const int span = (RB - 1) * stride + d;
  auto fixed = [&](int i) -> V {
    if constexpr (FS) {
      const float v = static_cast<const float*>(f)[i];
      return pack2<V>(v, v);
    } else {
      return static_cast<const V*>(f)[i];
    }
  };
  V mu[RB], v[RB], cov[RB];
#pragma unroll
  for (int j = 0; j < RB; ++j) mu[j] = v[j] = cov[j] = V(0);
#pragma unroll 1
  for (int r = 0; r < span; ++r) {
    const V* row = m + r * P;
    V h = V(0);
    patch_columns<DC, SC, RB == 4>(d, Wp, offs, [&](auto count, auto& o) {
      V x[count.value];
#pragma unroll
      for (int c = 0; c < count.value; ++c) x[c] = row[o[c]];
#pragma unroll
      for (int c = 0; c < count.value; ++c) h = add2(h, x[c]);
    });
#pragma unroll
    for (int j = 0; j < RB; ++j)
      if (r >= j * stride && r < j * stride + d) mu[j] = add2(mu[j], h);
  }
  const float n = (float)(d * d);
#pragma unroll
  for (int j = 0; j < RB; ++j) {  // negated
    const float2 t = unpack2(mu[j]);
    mu[j] = d > 1 ? pack2<V>(-(t.x / n), -(t.y / n)) : pack2<V>(-t.x, -t.y);
  }
#pragma unroll 1
  for (int r = 0; r < span; ++r) {
    const int row = r * P;
    patch_columns<DC, SC, RB == 4>(d, Wp, offs, [&](auto count, auto& o) {
      constexpr int N = count.value;
      V x[N], y[N], k[N];  // k: the mask twice
#pragma unroll
      for (int c = 0; c < N; ++c) {
        x[c] = m[row + o[c]];
        y[c] = fixed(row + o[c]);
        k[c] = MASK ? patch_mask<V>(mk[row + o[c]]) : V(0);
      }
#pragma unroll
      for (int j = 0; j < RB; ++j)
        if (r >= j * stride && r < j * stride + d) {
#pragma unroll
          for (int c = 0; c < N; ++c) {
            const V dm = add2(x[c], mu[j]), e = MASK ? fma2(k[c], fmean[j], y[c]) : add2(y[c], fmean[j]);
            v[j] = fma2(dm, dm, v[j]);
            cov[j] = fma2(dm, e, cov[j]);
          }
        }
    });
  }
  if constexpr (MASK) {
    // a masked-out pixel must not count, also where its product with 0 is not 0
#pragma unroll
    for (int j = 0; j < RB; ++j) {
      const float2 vv = unpack2(v[j]), fm = unpack2(fmean[j]), mj = unpack2(mu[j]);
      if (isfinite(vv.x) && isfinite(vv.y) && isfinite(fm.x) && isfinite(fm.y)) continue;
      float2 c2 = make_float2(0.0f, 0.0f);
#pragma unroll 1
      for (int r = j * stride; r < j * stride + d; ++r)
#pragma unroll 1
        for (int c = 0; c < d; ++c) {
          const int i = r * P + reinterpret_cast<const int*>(offs)[c];
          if (mk[i] == 0) continue;
          const float2 x = unpack2(m[i]), y = unpack2(fixed(i));
          c2.x = fmaf(x.x + mj.x, y.x + fm.x, c2.x);
          c2.y = fmaf(x.y + mj.y, y.y + fm.y, c2.y);
        }
      cov[j] = pack2<V>(c2.x, c2.y);
    }
  }
  auto value = [&](float vv, float cc, float sc) -> float {
    float sd = d > 1 ? sqrtf(vv / (n - 1.0f)) : 0.0f;
    sd = fmaxf(sd, 1.0e-6f);
    return 1.0f - (cc / sd) * sc;
  };
#pragma unroll
  for (int j = 0; j < RB; ++j) {
    const float2 vv = unpack2(v[j]), cc = unpack2(cov[j]), fs = scale(j);
    score[j] = make_float2(value(vv.x, cc.x, fs.x), value(vv.y, cc.y, fs.y));
  }
}

// Gradients of the moving image over the tile (top-left pixel x0, y0): a warp goes
// down 32 columns of a quarter of the rows, horizontal neighbours by shuffles, vertical
// ones in registers (as gt::grad_tile_moments).
template <int KR, typename At>
__device__ __forceinline__ void patch_tile_gradients(const float* __restrict__ src, int rows, int cols, int y0, int x0,
                                                     const PatchRows& L, At at, float2* __restrict__ s_m) {
  constexpr int H = KR + 1, kWin = 2 * KR + 1, kOut = 32 - 2 * H;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int strips = (L.Wc + kOut - 1) / kOut, chunk = (L.Wr + 3) / 4;
  for (int u = warp; u < strips * 4; u += kThreads / 32) {
    const int c0 = (u % strips) * kOut, r0 = (u / strips) * chunk, r1 = min(r0 + chunk, L.Wr);
    const int c = c0 - H + lane;
    const float* pc = src + reflect101(min(x0 + c, cols - 1 + H), cols);
    const bool owner = lane >= H && lane < 32 - H && c < L.Wc;
    const int ic = owner ? at(c) : 0;
    float hb[kWin], bl[3], lf[3], rt[3];
#pragma unroll
    for (int i = 0; i < kWin; ++i) hb[i] = 0.0f;
#pragma unroll
    for (int i = 0; i < 3; ++i) bl[i] = lf[i] = rt[i] = 0.0f;
    constexpr int kGroup = 6;  // rows in flight; 11 or 17 rows a warp at the default radius (8: 645 us for 632)
    for (int rb = r0 - 2 * H; rb < r1; rb += kGroup) {  // output rows rb .., from input rows rb + H ..
      float p[kGroup];
      if (y0 + rb + H >= 0 && y0 + rb + H + kGroup <= rows) {  // no row to reflect
        const float* q = pc + (int64_t)(y0 + rb + H) * cols;
#pragma unroll
        for (int i = 0; i < kGroup; ++i) p[i] = __ldg(q + (int64_t)i * cols);
      } else {
#pragma unroll
        for (int i = 0; i < kGroup; ++i)
          p[i] = __ldg(pc + (int64_t)reflect101(min(y0 + rb + i + H, rows - 1 + H), rows) * cols);
      }
#pragma unroll
      for (int i = 0; i < kGroup; ++i) {
        float h = p[i];
        if constexpr (KR == 2)
          h = gt::blur5(__shfl_up_sync(0xffffffffu, p[i], 2), __shfl_up_sync(0xffffffffu, p[i], 1), p[i],
                        __shfl_down_sync(0xffffffffu, p[i], 1), __shfl_down_sync(0xffffffffu, p[i], 2));
        else if constexpr (KR == 1)
          h = gt::blur3(__shfl_up_sync(0xffffffffu, p[i], 1), p[i], __shfl_down_sync(0xffffffffu, p[i], 1));
#pragma unroll
        for (int k = 0; k + 1 < kWin; ++k) hb[k] = hb[k + 1];
        hb[kWin - 1] = h;
        bl[0] = bl[1]; bl[1] = bl[2];
        lf[0] = lf[1]; lf[1] = lf[2];
        rt[0] = rt[1]; rt[1] = rt[2];
        if constexpr (KR == 2) bl[2] = gt::blur5(hb[0], hb[1], hb[2], hb[3], hb[4]);
        else if constexpr (KR == 1) bl[2] = gt::blur3(hb[0], hb[1], hb[2]);
        else bl[2] = hb[0];
        lf[2] = __shfl_up_sync(0xffffffffu, bl[2], 1);
        rt[2] = __shfl_down_sync(0xffffffffu, bl[2], 1);
        const int r = rb + i;
        if (owner && r >= r0 && r < r1) {
          float gx, gy;
          gt::sobel3(lf[0], bl[0], rt[0], lf[1], rt[1], lf[2], bl[2], rt[2], gx, gy);
          s_m[r * L.P + ic] = make_float2(gx, gy);
        }
      }
    }
  }
}

// Grid: tiles, then images (GRAD, RB 1) or pairs of images; kr: the blur's radius (GRAD).
// Partials: per image, sums over kPartRows rows by 32 columns of patches, nblk of them.
template <int GRAD, int RB, int DC, int SC, bool MASK>
__global__ void __launch_bounds__(kThreads, 3)
patch_rows_kernel(const float* __restrict__ imgs, int rows, int cols, int64_t nimgs, int kr, int radius, int stride_rt,
                  int ncr, int ncc, PatchFixed px, PatchFixed py, PatchRun run,
                  double* __restrict__ partials, int nblk) {
  constexpr int kWarps = kThreads / 32;
  constexpr bool kPairs = !GRAD && RB > 1;
  using V = std::conditional_t<GRAD || kPairs, u64, float>;
  extern __shared__ int4 smp[];
  __shared__ FF red[2][kThreads];
  const int stride = DC > 0 ? SC : stride_rt;
  const PatchRows L = PatchRows::make(radius, stride, GRAD, MASK, RB);
  const int size = L.Wr * L.P;
  int* s_off = reinterpret_cast<int*>(smp);
  V* s_m = reinterpret_cast<V*>(s_off + L.edge);
  float2* s_f = reinterpret_cast<float2*>(s_m + size);   // GRAD
  float* s_f1 = reinterpret_cast<float*>(s_f);           // plain
  int8_t* s_mk = reinterpret_cast<int8_t*>(GRAD ? reinterpret_cast<float*>(s_f + size) : s_f1 + size);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int tiles_x = (ncc + 31) / 32;
  const int tpr = blockIdx.x / tiles_x, tpc = blockIdx.x - tpr * tiles_x;
  const int pr0 = tpr * kWarps * RB, pc0 = tpc * 32;
  const int y0 = pr0 * stride, x0 = pc0 * stride;  // top-left pixel of the tile
  const int64_t npix = (int64_t)rows * cols;
  const int64_t img = kPairs ? 2 * (int64_t)blockIdx.y : (int64_t)blockIdx.y;
  const bool pair = kPairs && img + 1 < nimgs;  // a last image alone fills both channels
  const float* src = imgs + img * npix;
  auto at = [&](int x) -> int {
    const int q = x / stride;
    return (x - q * stride) * L.Wp + q;
  };
  if (threadIdx.x < L.edge) s_off[threadIdx.x] = at(threadIdx.x);

  // the fixed side, the mask and (plain patches) the images: a lane goes down a column,
  // four of its rows in flight; past the image the last pixel, which only patches outside
  // the grid read
  for (int c = lane; c < L.Wc; c += 32) {
    const int to = at(c);
    const int64_t gc = min(x0 + c, cols - 1);
    for (int r0 = warp; r0 < L.Wr; r0 += 4 * kWarps) {
      float a[4], b[4], b1[4];
      bool in[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int64_t g = (int64_t)min(y0 + r0 + k * kWarps, rows - 1) * cols + gc;
        in[k] = !MASK || run.mask[g];
        a[k] = __ldg(px.img + g);
        b[k] = GRAD ? __ldg(py.img + g) : __ldg(src + g);
        b1[k] = pair ? __ldg(src + npix + g) : b[k];
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int r = r0 + k * kWarps, i = r * L.P + to;
        if (r >= L.Wr) break;
        if constexpr (GRAD != 0) {
          s_f[i] = in[k] ? make_float2(a[k], b[k]) : make_float2(0.0f, 0.0f);
        } else {
          s_m[i] = pack2<V>(b[k], b1[k]);
          s_f1[i] = in[k] ? a[k] : 0.0f;
        }
        if constexpr (MASK) s_mk[i] = in[k] ? -1 : 0;
      }
    }
  }
  if constexpr (GRAD != 0) {
    if (kr == 2) patch_tile_gradients<2>(src, rows, cols, y0, x0, L, at, reinterpret_cast<float2*>(s_m));
    else if (kr == 1) patch_tile_gradients<1>(src, rows, cols, y0, x0, L, at, reinterpret_cast<float2*>(s_m));
    else patch_tile_gradients<0>(src, rows, cols, y0, x0, L, at, reinterpret_cast<float2*>(s_m));
  }
  __syncthreads();

  FF v[RB][2];
#pragma unroll
  for (int j = 0; j < RB; ++j) v[j][0] = v[j][1] = FF{0.0f, 0.0f};
  const int pc = pc0 + lane, prw = pr0 + warp * RB;
  if (pc < ncc && prw < ncr) {
    int cnt[RB];
    bool any = false;
    const int64_t pidx = (int64_t)prw * ncc + pc;
#pragma unroll
    for (int j = 0; j < RB; ++j) {
      cnt[j] = prw + j < ncr ? (run.cnt ? run.cnt[pidx + (int64_t)j * ncc] : 1) : 0;
      any = any || cnt[j] > 0;
    }
    if (any) {
      const int o = warp * RB * stride * L.P + lane;
      V fm[RB];
      float2 sc[RB];
      const PatchFixed& p1 = GRAD ? py : px;  // the second channel's fixed side
#pragma unroll
      for (int j = 0; j < RB; ++j) {
        const int64_t i = pidx + (int64_t)j * ncc;
        fm[j] = cnt[j] > 0 ? pack2<V>(-px.mean[i], -p1.mean[i]) : V(0);
      }
      const void* f0 = GRAD ? static_cast<const void*>(s_f + o) : static_cast<const void*>(s_f1 + o);
      patch_column_scores<V, RB, DC, SC, MASK, GRAD == 0>(
          s_m + o, f0, s_mk + o, L.P, L.Wp, smp, 2 * radius + 1, stride, fm,
          [&](int j) -> float2 {
            const int64_t i = pidx + (int64_t)j * ncc;
            return prw + j < ncr ? make_float2(px.scale[i], p1.scale[i]) : make_float2(0.0f, 0.0f);
          },
          sc);
#pragma unroll
      for (int j = 0; j < RB; ++j) {
        if (prw + j >= ncr) continue;
        const int64_t i = pidx + (int64_t)j * ncc;
        const int count = RB > 2 ? (run.cnt ? run.cnt[i] : 1) : cnt[j];
        if (count <= 0) continue;
        const float w[2] = {px.w ? px.w[i] : 1.0f, p1.w ? p1.w[i] : 1.0f};
        const float s2[2] = {sc[j].x, sc[j].y};
        float kept[2] = {0.0f, 0.0f};  // per-patch score as xReg keeps it (0.5 (s_x + s_y) for GRAD)
#pragma unroll
        for (int k = 0; k < 2; ++k)
          if (!run.weighted || fabsf(w[k]) > 1.0e-6f) {
            v[j][k] = ff_prod((float)count, (run.weighted ? w[k] : 1.0f) * s2[k]);
            kept[GRAD ? 0 : k] += GRAD ? 0.5f * s2[k] : s2[k];
          }
        if (run.scores) {
          const int64_t np = (int64_t)ncr * ncc;
          run.scores[img * np + i] = kept[0];
          if (pair) run.scores[(img + 1) * np + i] = kept[1];
        }
      }
    }
  }
  // sums by halves: a thread's rows, the warps of a part, the lanes
#pragma unroll
  for (int k = 0; k < 2; ++k) {
#pragma unroll
    for (int h = 1; h < RB; h *= 2)
#pragma unroll
      for (int j = 0; j < RB; j += 2 * h) v[j][k] = ff_add(v[j][k], v[j + h][k]);
    red[k][threadIdx.x] = v[0][k];
  }
  __syncthreads();
  constexpr int kPart = kPartRows / RB;  // warps of a part
  const int part_row = tpr * (kWarps / kPart) + warp;
  if (warp < kWarps / kPart && part_row * kPartRows < ncr) {
    double t[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      FF w[kPart];
#pragma unroll
      for (int i = 0; i < kPart; ++i) w[i] = red[k][(warp * kPart + i) * 32 + lane];
#pragma unroll
      for (int h = 1; h < kPart; h *= 2)
#pragma unroll
        for (int i = 0; i < kPart; i += 2 * h) w[i] = ff_add(w[i], w[i + h]);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) w[0] = ff_add(w[0], ff_shfl_down(w[0], o));
      t[k] = (double)w[0].hi + (double)w[0].lo;
    }
    if (lane == 0) {
      double* o = partials + (img * nblk + part_row * tiles_x + tpc) * 2;
      o[0] = t[0];
      o[1] = GRAD ? t[1] : 0.0;
      if (pair) {
        o += 2 * (int64_t)nblk;
        o[0] = t[1];
        o[1] = 0.0;
      }
    }
  }
}

// Per image (one block each): the two sums over the blocks' partials.
__device__ __forceinline__ void patch_partials_sum(const double* __restrict__ p, int nblk, double (&v)[2],
                                                   double* red) {
  v[0] = 0.0;
  v[1] = 0.0;
  for (int k = threadIdx.x; k < nblk; k += blockDim.x) {
    v[0] += p[2 * k];
    v[1] += p[2 * k + 1];
  }
  block_sum_d<2>(v, red);
}

__global__ void patch_sum_partials_kernel(const double* __restrict__ partials, int nblk, double* __restrict__ out) {
  __shared__ double red[2 * 32];
  const int64_t img = blockIdx.x;
  double v[2];
  patch_partials_sum(partials + img * nblk * 2, nblk, v, red);
  if (threadIdx.x == 0) {
    out[img * 2] = v[0];
    out[img * 2 + 1] = v[1];
  }
}

// Value per image: sum / denominator per direction; FLT_MAX where normalised
// moving variances sum to at most 1e-6; patch grad-NCC 0.5 (s_x + s_y) in float.
__global__ void patch_finalize_kernel(const double* __restrict__ partials, int nblk, double den_x, double den_y,
                                      int grad, int mvar, int normalize, const double* __restrict__ mvar_sum,
                                      float* __restrict__ sims) {
  __shared__ double red[2 * 32];
  const int64_t img = blockIdx.x;
  double v[2];
  patch_partials_sum(partials + img * nblk * 2, nblk, v, red);
  if (threadIdx.x != 0) return;
  const bool chk = mvar && normalize;
  if (chk && mvar == 1 && !((float)mvar_sum[img * 2] > 1.0e-6f)) {
    sims[img] = FLT_MAX;
    return;
  }
  const float sx = (chk && !((float)mvar_sum[img * 2] > 1.0e-6f)) ? FLT_MAX : (float)(v[0] / den_x);
  if (grad) {
    const float sy = (chk && !((float)mvar_sum[img * 2 + 1] > 1.0e-6f)) ? FLT_MAX : (float)(v[1] / den_y);
    sims[img] = 0.5f * (sx + sy);
  } else {
    sims[img] = sx;
  }
}

// cnt[idx[k]] += 1 for k < n (patch multiplicities of a drawn subset).
__global__ void patch_scatter_counts_kernel(const int32_t* __restrict__ idx, int64_t n, int32_t* __restrict__ cnt) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k < n) atomicAdd(cnt + idx[k], 1);
}

struct ViewPtrs {
  const float* p[16];
};

__global__ void combine_mean_kernel(ViewPtrs vp, int nviews, int64_t pop, float* __restrict__ out) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= pop) return;
  out[i] = gt::combine_mean(vp.p, nviews, i, false);
}

template <typename K>
cudaError_t set_smem(K kern, size_t bytes) {
  // above the default 48 KB the kernel must opt in; the kernels' own static
  // shared memory counts against the same 48 KB, so opt in with room to spare
  if (bytes > 40 * 1024) return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  return cudaSuccess;
}

}  // namespace

cudaError_t launch_image_stats(const float* img, int64_t npix, const uint8_t* mask, double* d_out, cudaStream_t s) {
  image_sum_kernel<<<1, 1024, 0, s>>>(img, npix, mask, d_out);
  image_var_kernel<<<1, 1024, 0, s>>>(img, npix, mask, d_out);
  return cudaGetLastError();
}

cudaError_t launch_sum_f(const float* in, int64_t n, const uint8_t* mask, double* d_out, cudaStream_t s) {
  image_sum_kernel<<<1, 1024, 0, s>>>(in, n, mask, d_out);
  return cudaGetLastError();
}

cudaError_t launch_sub_scalar(const float* in, int64_t n, double value, float* out, cudaStream_t s) {
  const int blocks = (int)((n + 255) / 256 < 4096 ? (n + 255) / 256 : 4096);
  sub_scalar_kernel<<<blocks > 0 ? blocks : 1, 256, 0, s>>>(in, n, (float)value, out);
  return cudaGetLastError();
}

cudaError_t launch_ncc_moments(const float* mov, int64_t npix, int64_t nimgs, const float* fhat,
                               const uint8_t* mask, double* partials, int nblk, cudaStream_t s) {
  if (nimgs <= 0) return cudaSuccess;
  const dim3 grid(nblk, (unsigned)nimgs);
  ncc_moments_kernel<<<grid, kThreads, 0, s>>>(mov, npix, fhat, mask, partials);
  return cudaGetLastError();
}

cudaError_t launch_ncc_finalize(const double* partials, int nblk, int64_t nimgs, int64_t n_used, FixedNCC fx,
                                float* sims, cudaStream_t s) {
  if (nimgs <= 0) return cudaSuccess;
  ncc_finalize_kernel<<<(unsigned)nimgs, 128, 0, s>>>(partials, nblk, nimgs, (double)n_used, fx, sims);
  return cudaGetLastError();
}

cudaError_t launch_grad_images(const float* img, int rows, int cols, int64_t nimgs, int smooth_ksize, float* gx,
                               float* gy, cudaStream_t s) {
  const int tiles = ((rows + kT - 1) / kT) * ((cols + kT - 1) / kT);
  const dim3 grid(tiles, (unsigned)nimgs);
  switch (smooth_ksize) {
    case 0: grad_images_kernel<0><<<grid, kThreads, 0, s>>>(img, rows, cols, gx, gy); break;
    case 3: grad_images_kernel<1><<<grid, kThreads, 0, s>>>(img, rows, cols, gx, gy); break;
    case 5: grad_images_kernel<2><<<grid, kThreads, 0, s>>>(img, rows, cols, gx, gy); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

cudaError_t launch_grad_moments(const float* mov, int rows, int cols, int64_t nimgs, int smooth_ksize,
                                const float* fhat_x, const float* fhat_y, const uint8_t* mask, double* partials,
                                cudaStream_t s, int* nblk_out) {
  int tw = 0;
  switch (smooth_ksize) {
    case 0: tw = gt::kTileCols<0>; break;
    case 3: tw = gt::kTileCols<1>; break;
    case 5: tw = gt::kTileCols<2>; break;
    default: return cudaErrorInvalidValue;
  }
  const int tiles = ((rows + kGH - 1) / kGH) * ((cols + tw - 1) / tw);
  if (nblk_out) *nblk_out = tiles;
  if (nimgs <= 0 || !partials) return cudaSuccess;
  const dim3 grid(tiles, (unsigned)nimgs);
  constexpr int nt = gt::kTileThreads;
  switch (smooth_ksize) {
    case 0: grad_moments_kernel<0><<<grid, nt, 0, s>>>(mov, rows, cols, fhat_x, fhat_y, mask, partials); break;
    case 3: grad_moments_kernel<1><<<grid, nt, 0, s>>>(mov, rows, cols, fhat_x, fhat_y, mask, partials); break;
    default: grad_moments_kernel<2><<<grid, nt, 0, s>>>(mov, rows, cols, fhat_x, fhat_y, mask, partials); break;
  }
  return cudaGetLastError();
}

cudaError_t launch_grad_multi(const FusedJob* d_jobs, int njobs, long long total, cudaStream_t s) {
  if (total <= 0) return cudaSuccess;
  int dev = 0, sms = 0, per_sm = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e == cudaSuccess)
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, grad_multi_kernel, gt::kTileThreads, 0);
  if (e != cudaSuccess) return e;
  const long long cap = (long long)sms * (per_sm > 0 ? per_sm : 1);
  grad_multi_kernel<<<(unsigned)(total < cap ? total : cap), gt::kTileThreads, 0, s>>>(d_jobs, njobs, total);
  return cudaGetLastError();
}

cudaError_t launch_cma_updates(const CmaUpdateJob* d_jobs, int njobs, cudaStream_t s) {
  if (njobs <= 0) return cudaSuccess;
  cma_update_kernel<<<(unsigned)njobs, 128, 0, s>>>(d_jobs);
  return cudaGetLastError();
}

cudaError_t launch_grad_finalize(const double* partials, int nblk, int64_t nimgs, int64_t n_used, FixedNCC fx,
                                 FixedNCC fy, float* sims, cudaStream_t s) {
  if (nimgs <= 0) return cudaSuccess;
  grad_finalize_kernel<<<(unsigned)nimgs, 128, 0, s>>>(partials, nblk, nimgs, (double)n_used, fx, fy, sims);
  return cudaGetLastError();
}

cudaError_t launch_patch_fixed_stats(const float* img, int rows, int cols, int radius, int stride, int ncr, int ncc,
                                     const uint8_t* mask, int use_mask_stats, float* mean, float* scale, float* wvar,
                                     int* ucount, cudaStream_t s) {
  (void)rows;
  const int64_t n = (int64_t)ncr * ncc;
  if (n <= 0) return cudaSuccess;
  patch_fixed_stats_kernel<<<(unsigned)((n + 127) / 128), 128, 0, s>>>(img, cols, radius, stride, ncr, ncc, mask,
                                                                       use_mask_stats, mean, scale, wvar, ucount);
  return cudaGetLastError();
}

// Patches a thread scores in a column (patch_rows_kernel).  One while a patch a thread
// does not fill the GPU (1024 threads an SM): four would leave SMs idle (6 images of
// 311 x 476, 15 x 15 at stride 3, a whole call: 56 us against 81 with four; 16 of 215 x
// 493, 11 x 11 at stride 2, above the line: 79 against 60).  Four while two blocks' tiles
// fit an SM (228 KB, 4 KB of static and 1 KB of reserved memory a block): one block of 8
// warps cannot hide its own staging (24 images of 384^2 at stride 3, 7 x 7, 11 x 11 and
// 15 x 15, masked: 88, 104, 125 us with four, 62, 79, 104 with one; at stride 2, 15 x 15,
// both gradients, 96 KB: 179 with four, 234 with one).  The general kernel with masked
// statistics, moving-variance weights or tiles too large.
constexpr size_t kPatchSmem = 200 * 1024;
constexpr size_t kPatchSmemFour = 109 * 1024;

static size_t patch_rows_bytes(int radius, int stride, int grad, const PatchRun& run, int rb) {
  return PatchRows::make(radius, stride, grad, run.mask != nullptr, rb).bytes;
}

static bool patch_general(int radius, int stride, int grad, const PatchRun& run) {
  return run.mvar || (run.mask && (run.use_mask_stats || !run.mask_in_sums)) ||
         patch_rows_bytes(radius, stride, grad, run, 1) > kPatchSmem;
}

// tiles of `rows` by 32 patches
static int patch_tiles(int ncr, int ncc, int rows) { return ((ncr + rows - 1) / rows) * ((ncc + 31) / 32); }

static int patch_general_tiles(int ncr, int ncc) { return ((ncr + kPC - 1) / kPC) * ((ncc + kPC - 1) / kPC); }

static cudaError_t patch_rb(int radius, int stride, int grad, const PatchRun& run, int ncr, int ncc, int64_t nimgs,
                            int* rb) {
  int dev = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return e;
  const bool many = (int64_t)ncr * ncc * nimgs > (int64_t)sms * 1024;
  *rb = many && patch_rows_bytes(radius, stride, grad, run, 4) <= kPatchSmemFour ? 4 : 1;
  return e;
}

int patch_ncc_max_blocks(int ncr, int ncc) {
  return max(patch_general_tiles(ncr, ncc), patch_tiles(ncr, ncc, kPartRows));
}

template <int GRAD, int RB, int DC, int SC, bool MASK>
static cudaError_t launch_rows(const float* mov, int rows, int cols, int kr, int radius, int stride, int ncr, int ncc,
                               int64_t nimgs, const PatchFixed& px, const PatchFixed& py, const PatchRun& run,
                               double* partials, int nblk, cudaStream_t s) {
  const size_t bytes = patch_rows_bytes(radius, stride, GRAD, run, RB);
  const cudaError_t e = set_smem(patch_rows_kernel<GRAD, RB, DC, SC, MASK>, bytes);
  if (e != cudaSuccess) return e;
  const dim3 grid(patch_tiles(ncr, ncc, 8 * RB), (unsigned)(!GRAD && RB > 1 ? (nimgs + 1) / 2 : nimgs));
  patch_rows_kernel<GRAD, RB, DC, SC, MASK><<<grid, kThreads, bytes, s>>>(mov, rows, cols, nimgs, kr, radius, stride, ncr,
                                                                     ncc, px, py, run, partials, nblk);
  return cudaGetLastError();
}

cudaError_t launch_patch_ncc(const float* mov, int rows, int cols, int64_t nimgs, int grad, int smooth_ksize,
                             int radius, int stride, int ncr, int ncc, PatchFixed px, PatchFixed py, PatchRun run,
                             int pass, double* partials, cudaStream_t s, int* nblk_out) {
  const int kr = smooth_ksize == 5 ? 2 : (smooth_ksize == 3 ? 1 : 0);
  if (smooth_ksize != 0 && smooth_ksize != 3 && smooth_ksize != 5) return cudaErrorInvalidValue;
  const bool general = patch_general(radius, stride, grad, run);
  const int nblk = general ? patch_general_tiles(ncr, ncc) : patch_tiles(ncr, ncc, kPartRows);
  if (nblk_out) *nblk_out = nblk;
  if (nimgs <= 0 || !partials) return cudaSuccess;
  // One limit of radius and stride for every form, the general kernel's: options and the
  // number of images do not decide what is refused.
  const PatchLayout L = PatchLayout::make(radius, stride, grad, kr);
  if (L.bytes > kPatchSmem) return cudaErrorInvalidValue;
  if (!general) {
    if (pass != 1) return cudaErrorInvalidValue;
    int rb = 1;
    const cudaError_t e = patch_rb(radius, stride, grad, run, ncr, ncc, nimgs, &rb);
    if (e != cudaSuccess) return e;
    // the columns of xReg's default patches (11 x 11) unroll at strides 1 and 2 (24 masked
    // images of 384^2 at stride 2, a whole call: 63 us against 95 by fours)
#define XR_ROWS(G, R, D, S, M) \
  return launch_rows<G, R, D, S, M>(mov, rows, cols, kr, radius, stride, ncr, ncc, nimgs, px, py, run, partials, nblk, s)
#define XR_ROWS_R(G, R, M)                                 \
  if (radius == 5 && stride == 1) XR_ROWS(G, R, 11, 1, M); \
  if (radius == 5 && stride == 2) XR_ROWS(G, R, 11, 2, M); \
  XR_ROWS(G, R, 0, 0, M)
#define XR_ROWS_G(G)                                 \
  if (run.mask && rb == 1) { XR_ROWS_R(G, 1, true); } \
  if (run.mask) { XR_ROWS_R(G, 4, true); }            \
  if (rb == 1) { XR_ROWS_R(G, 1, false); }            \
  XR_ROWS_R(G, 4, false)
    if (grad) { XR_ROWS_G(1); }
    XR_ROWS_G(0);
#undef XR_ROWS_G
#undef XR_ROWS_R
#undef XR_ROWS
  }
  const dim3 grid(nblk, (unsigned)nimgs);
  cudaError_t e = cudaSuccess;
#define XR_PATCH_LAUNCH(G, K, P)                                                                                       \
  e = set_smem(patch_ncc_kernel<G, K, P>, L.bytes);                                                                    \
  if (e != cudaSuccess) return e;                                                                                      \
  patch_ncc_kernel<G, K, P><<<grid, kThreads, L.bytes, s>>>(mov, rows, cols, radius, stride, ncr, ncc, px, py, run,    \
                                                            partials);
#define XR_PATCH_PASS(G, K)    \
  if (pass == 0) {             \
    XR_PATCH_LAUNCH(G, K, 0)   \
  } else {                     \
    XR_PATCH_LAUNCH(G, K, 1)   \
  }
  if (!grad) {
    XR_PATCH_PASS(0, 0)
  } else if (kr == 0) {
    XR_PATCH_PASS(1, 0)
  } else if (kr == 1) {
    XR_PATCH_PASS(1, 1)
  } else {
    XR_PATCH_PASS(1, 2)
  }
#undef XR_PATCH_PASS
#undef XR_PATCH_LAUNCH
  return cudaGetLastError();
}

cudaError_t launch_patch_sum_partials(const double* partials, int nblk, int64_t nimgs, double* out, cudaStream_t s) {
  if (nimgs <= 0) return cudaSuccess;
  patch_sum_partials_kernel<<<(unsigned)nimgs, 256, 0, s>>>(partials, nblk, out);
  return cudaGetLastError();
}

cudaError_t launch_patch_finalize(const double* partials, int nblk, int64_t nimgs, double den_x, double den_y,
                                  int grad, int mvar, int normalize, const double* mvar_sum, float* sims,
                                  cudaStream_t s) {
  if (nimgs <= 0) return cudaSuccess;
  patch_finalize_kernel<<<(unsigned)nimgs, 256, 0, s>>>(partials, nblk, den_x, den_y, grad, mvar, normalize,
                                                       mvar_sum, sims);
  return cudaGetLastError();
}

cudaError_t launch_patch_scatter_counts(const int32_t* idx, int64_t n, int32_t* cnt, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  patch_scatter_counts_kernel<<<(unsigned)((n + 127) / 128), 128, 0, s>>>(idx, n, cnt);
  return cudaGetLastError();
}

cudaError_t launch_combine_mean(const float* const* view_sims, int nviews, int64_t pop, float* out, cudaStream_t s) {
  if (nviews < 1 || nviews > 16) return cudaErrorInvalidValue;
  ViewPtrs vp;
  for (int v = 0; v < 16; ++v) vp.p[v] = v < nviews ? view_sims[v] : nullptr;
  combine_mean_kernel<<<(unsigned)((pop + 127) / 128), 128, 0, s>>>(vp, nviews, pop, out);
  return cudaGetLastError();
}

}  // namespace xr

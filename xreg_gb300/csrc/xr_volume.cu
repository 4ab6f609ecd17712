// xr_volume.cu -- volume set-up: HU to attenuation, the statistics of a volume
// (largest magnitude, support box, macro-cell occupancy) in one pass, and its
// cell copy and 16-bit voxels in another.  All bound by HBM.
#include "xr_cells.h"
#include "xr_internal.h"

#include <algorithm>

namespace xr {
namespace {

constexpr int kThreads = 256;

// ------------------------------------------------------ HU to attenuation --
// HUToLinAttFilter::GenerateData (lib/image/xregHUToLinAtt.cpp:45-69):
// mu = max(hu scale + mu_w - mu_lower, 0) in double, stored as float.  Three
// double operations per voxel bound the pass (722 us for 512 x 512 x 300, 0.63 GB
// of traffic), so the sum is formed in float-float, whose error is far below the
// spacing of the float result, and the double operations run only where that
// error could decide the rounding (105 us).  The result is the double one for every
// input.
constexpr double kMuW = 0.02683 * 1.0, kMuA = 0.02485 * 0.0001, kHuLower = -1000.0;
constexpr double kHuScale = (kMuW - kMuA) * 1.0e-3;
constexpr double kMuLower = (kHuLower * kHuScale) + kMuW;

// out of line: its double instructions would otherwise be issued for every voxel
__device__ __noinline__ float hu_to_mu_double(float hu) {
  const double v = ((double)hu * kHuScale) + kMuW - kMuLower;
  return (float)(v > 0.0 ? v : 0.0);
}

__device__ __forceinline__ float hu_to_mu(float hu) {
  // At hu_lower the double result is 0, and it grows with hu: 0 below it too (and for NaN).
  if (!(hu > (float)kHuLower)) return 0.0f;
  constexpr float s_hi = (float)kHuScale, s_lo = (float)(kHuScale - (double)s_hi);
  constexpr double c = kMuW - kMuLower;
  constexpr float c_hi = (float)c, c_lo = (float)(c - (double)c_hi);
  const float p = __fmul_rn(hu, s_hi);
  const float pe = __fmaf_rn(hu, s_lo, __fmaf_rn(hu, s_hi, -p));  // hu scale = p + pe
  const float t = __fadd_rn(p, c_hi), b = __fsub_rn(t, p);
  float e = __fadd_rn(__fsub_rn(p, __fsub_rn(t, b)), __fsub_rn(c_hi, b));  // t + e = p + c_hi exactly
  e = __fadd_rn(e, __fadd_rn(pe, c_lo));
  const float hi = __fadd_rn(t, e), lo = __fsub_rn(e, __fsub_rn(hi, t));
  // The float-float value and the double one both lie within 2^-45 (|p| + c) of
  // the exact one (a few roundings at 2^-47 of the terms, and at 2^-53).
  const float tol = __fmul_rn(__fadd_rn(fabsf(p), c_hi), 0x1p-44f);
  if (__fadd_rn(hi, __fadd_rn(lo, tol)) == hi && __fadd_rn(hi, __fsub_rn(lo, tol)) == hi && hi > 0.0f) return hi;
  return hu_to_mu_double(hu);
}

__global__ void hu_to_mu_kernel(const float* __restrict__ hu, int64_t n, float* __restrict__ mu) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  for (; i + 3 * stride < n; i += 4 * stride) {  // four loads in flight
    float v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = hu[i + k * stride];
#pragma unroll
    for (int k = 0; k < 4; ++k) mu[i + k * stride] = hu_to_mu(v[k]);
  }
  for (; i < n; i += stride) mu[i] = hu_to_mu(hu[i]);
}

// ------------------------------------------------------------- statistics --
constexpr int kSegX = 1024;                   // voxels of a row per block
constexpr int kSegBits = kSegX / 8 + 2;       // macro cells they reach along x, one more on each side
constexpr int kSegWords = (kSegBits + 31) / 32;

// A block takes 8 x 8 rows (one macro cell in y and z) of kSegX voxels, a warp a
// row at a time and a lane four neighbours of every 128: ballots of the lanes with a
// non-zero voxel (any, the last, one of the first two) give the macro cells along x,
// the row's place in its macro cell those along y and z.  A macro cell m is occupied
// when a voxel in [8m - 1, 8m + 9] on every axis is not zero (VolView::occ).  One
// read of the volume where the largest magnitude, the box and the occupancy took
// one each (58 + 268 + 372 us for 512 x 512 x 300).  Its reads would take 46 us; with
// a ballot per 32 voxels it was bound by instructions at 97, with the box's atomics
// per warp (they all meet in one L2 sector) at 91, now 63.  VEC: rows start on 16 bytes.
template <bool VEC>
__global__ void __launch_bounds__(kThreads) volume_stats_kernel(const float* __restrict__ vox, int nx, int ny, int nz,
                                                                int nxs, int nyb, uint32_t* __restrict__ occ, int nmx,
                                                                int nmy, int nmz, VolStats* __restrict__ stats) {
  __shared__ uint32_t bits[3][3][kSegWords];  // macro cells (z, y) - 1 .. + 1 around the block's, x from 128 xs - 1
  __shared__ unsigned int found[7];  // as VolStats: largest magnitude, box
  for (int i = threadIdx.x; i < 9 * kSegWords; i += kThreads) (&bits[0][0][0])[i] = 0u;
  if (threadIdx.x < 7) found[threadIdx.x] = 0u;
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int xs = (int)(blockIdx.x % nxs), yb = (int)(blockIdx.x / nxs % nyb), zb = (int)(blockIdx.x / nxs / nyb);
  const int x0 = xs * kSegX, xe = min(nx, x0 + kSegX);
  float mx = 0.0f;
  int lo[3] = {0x7fffffff, 0x7fffffff, 0x7fffffff}, hi[3] = {-1, -1, -1};
  for (int r = warp; r < 64; r += kThreads / 32) {
    const int ry = r & 7, rz = r >> 3, y = yb * 8 + ry, z = zb * 8 + rz;
    if (y >= ny || z >= nz) continue;
    const float* row = vox + ((int64_t)z * ny + y) * nx;
    for (int xc = x0; xc < xe; xc += 512) {
      float v[4][4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int x = xc + 128 * k + 4 * lane;
        if constexpr (VEC) {
          const float4 q = x < xe ? __ldg(reinterpret_cast<const float4*>(row + x)) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
          v[k][0] = q.x; v[k][1] = q.y; v[k][2] = q.z; v[k][3] = q.w;
        } else {
#pragma unroll
          for (int i = 0; i < 4; ++i) v[k][i] = x + i < xe ? __ldg(row + x + i) : 0.0f;
        }
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        uint32_t w[4];  // not zero: but for the sign a bit is set (a NaN too)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          mx = fmaxf(mx, fabsf(v[k][i]));  // passes over NaN
          w[i] = __float_as_uint(v[k][i]);
        }
        const bool some = ((w[0] | w[1] | w[2] | w[3]) << 1) != 0u;
        const uint32_t any = __ballot_sync(0xffffffffu, some);
        if (!any) continue;
        const uint32_t last = __ballot_sync(0xffffffffu, (w[3] << 1) != 0u);
        const uint32_t first2 = __ballot_sync(0xffffffffu, ((w[0] | w[1]) << 1) != 0u);
        const int xk = xc + 128 * k, x = xk + 4 * lane;
        if (some && (x < lo[0] || x + 3 > hi[0]))
#pragma unroll
          for (int i = 0; i < 4; ++i)
            if ((w[i] << 1) != 0u) {
              lo[0] = min(lo[0], x + i);
              hi[0] = max(hi[0], x + i);
            }
        lo[1] = min(lo[1], y); hi[1] = max(hi[1], y);
        lo[2] = min(lo[2], z); hi[2] = max(hi[2], z);
        // lane j reports the chunk's macro cell j - 1: its lanes 2j - 2 and 2j - 1, the last voxel of
        // lane 2j - 3 and the first two of lane 2j
        const int s = 2 * lane - 3;
        const bool set = lane < 18 && ((((s >= 0 ? any >> s : any << -s) & 6u) | ((s >= 0 ? last >> s : last << -s) & 1u)) != 0u ||
                                       (lane < 16 && ((first2 >> (2 * lane)) & 1u)));
        const uint32_t m18 = __ballot_sync(0xffffffffu, set);
        if (lane < 2) {
          const int b0 = (xk - x0) / 8;  // bit 0: macro cell 128 xs - 1
          const uint32_t word = lane == 0 ? m18 << (b0 & 31) : (b0 & 31) ? m18 >> (32 - (b0 & 31)) : 0u;
          if (word)
            for (int dz = rz < 2 ? 0 : 1; dz <= (rz == 7 ? 2 : 1); ++dz)
              for (int dy = ry < 2 ? 0 : 1; dy <= (ry == 7 ? 2 : 1); ++dy)
                if (word & ~bits[dz][dy][(b0 >> 5) + lane]) atomicOr(&bits[dz][dy][(b0 >> 5) + lane], word);
        }
      }
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    lo[0] = min(lo[0], __shfl_xor_sync(0xffffffffu, lo[0], o));
    hi[0] = max(hi[0], __shfl_xor_sync(0xffffffffu, hi[0], o));
  }
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if (lane == 0) {  // one atomic per block and value: they all meet in one L2 sector
    atomicMax(&found[0], __float_as_uint(mx));
    if (hi[0] >= 0)
      for (int k = 0; k < 3; ++k) {
        atomicMax(&found[1 + k], 0x7fffffffu - (unsigned int)lo[k]);
        atomicMax(&found[4 + k], (unsigned int)hi[k] + 1u);
      }
  }
  __syncthreads();
  if (threadIdx.x < 7 && found[threadIdx.x]) {
    unsigned int* g = threadIdx.x == 0 ? &stats->max_bits : threadIdx.x < 4 ? &stats->lo[threadIdx.x - 1] : &stats->hi[threadIdx.x - 4];
    atomicMax(g, found[threadIdx.x]);
  }
  for (int i = threadIdx.x; i < 9 * kSegBits; i += kThreads) {
    const int d = i / kSegBits, b = i - d * kSegBits;
    if (!((bits[d / 3][d % 3][b >> 5] >> (b & 31)) & 1u)) continue;
    const int mxi = xs * (kSegX / 8) + b - 1, myi = yb + d % 3 - 1, mzi = zb + d / 3 - 1;
    if (mxi < 0 || mxi >= nmx || myi < 0 || myi >= nmy || mzi < 0 || mzi >= nmz) continue;
    const int m = (mzi * nmy + myi) * nmx + mxi;
    const uint32_t bit = 1u << (m & 31);
    if (!(occ[m >> 5] & bit)) atomicOr(&occ[m >> 5], bit);
  }
}

// ------------------------------------------------------------------ cells --
template <int VT>
__device__ __forceinline__ uint32_t half_pair(float a, float b) {
  if constexpr (VT == XR_VOXEL_F16) {
    const __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
  } else {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
  }
}

// The cell copy (see xr_raycast.cu) and, when out_vox is set, the voxels in the
// volume's own type.  Voxels are x fastest and cells z fastest, so a block takes
// 32 x 32 cells in x and z through shared memory and walks kBuildY of them in y:
// one new plane of 33 x 33 voxels per step (read along x), its cells written by
// lanes along z, 512 bytes or 1 KB together.  One thread per cell reading along x
// wrote 16 bytes at a time, half sectors (2251 us for 512 x 512 x 300 FP16 and
// another 79 for the voxels, now 320 for both, 5.3 TB/s).
constexpr int kBuildY = 16, kTile = 32, kPlane = kTile + 1;

template <int VT>
__global__ void __launch_bounds__(kThreads) build_cells_kernel(const float* __restrict__ vox, int nx, int ny, int nz,
                                                               float scale, bool weighted, int32_t csx, int32_t csy,
                                                               int tx, int tz, void* __restrict__ out,
                                                               void* __restrict__ out_vox) {
  __shared__ float plane[2][kPlane * kPlane];  // [y parity][z][x], odd pitch: columns are free of bank conflicts
  const int bx = (int)(blockIdx.x % tx), bz = (int)(blockIdx.x / tx % tz), by = (int)(blockIdx.x / tx / tz);
  const int cx0 = bx * kTile, cz0 = bz * kTile, cy0 = by * kBuildY;  // first cell (index + 1)
  const int cy1 = min(cy0 + kBuildY, ny + 1);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int kPer = (kPlane * kPlane + kThreads - 1) / kThreads;
  float v[kPer];
  // plane of voxels with index y (clamped), x from cx0 - 1, z from cz0 - 1 (clamped)
  auto fetch = [&](int y) {
    y = min(max(y, 0), ny - 1);
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
      const int i = threadIdx.x + k * kThreads, zi = i / kPlane, xi = i - zi * kPlane;
      const int x = min(max(cx0 - 1 + xi, 0), nx - 1), z = min(max(cz0 - 1 + zi, 0), nz - 1);
      if (i < kPlane * kPlane) v[k] = __ldg(vox + ((int64_t)z * ny + y) * nx + x);
    }
  };
  auto stage = [&](float* p) {
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
      const int i = threadIdx.x + k * kThreads;
      if (i < kPlane * kPlane) p[i] = VT == XR_VOXEL_F32 ? v[k] : v[k] * scale;
    }
  };
  fetch(cy0 - 1);
  stage(plane[0]);
  fetch(cy0);
  stage(plane[1]);
  __syncthreads();
  for (int cy = cy0; cy < cy1; ++cy) {
    const float* p0 = plane[(cy - cy0) & 1];
    const float* p1 = plane[(cy - cy0 + 1) & 1];
    const bool more = cy + 1 < cy1;
    if (more) fetch(cy + 1);
    if (cz0 + lane <= nz) {
#pragma unroll
      for (int k = 0; k < kTile / (kThreads / 32); ++k) {
        const int xi = warp + k * (kThreads / 32);
        if (cx0 + xi > nx) continue;
        const int o = lane * kPlane + xi;
        // z-pairs: v000 v001 v100 v101 v010 v011 v110 v111 (vxyz)
        const float c[8] = {p0[o], p0[o + kPlane], p0[o + 1], p0[o + kPlane + 1],
                            p1[o], p1[o + kPlane], p1[o + 1], p1[o + kPlane + 1]};
        const int64_t cell = (int64_t)(cx0 + xi) * csx + (int64_t)cy * csy + cz0 + lane;
        if constexpr (VT == XR_VOXEL_F32) {
          float* q = static_cast<float*>(out) + 8 * cell;
          float d[4];  // the x + 1 corners, as cells hold them
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int k0 = (i & 1) + 4 * (i >> 1);
            d[i] = weighted ? c[k0 + 2] : __fsub_rn(c[k0 + 2], c[k0]);
          }
          asm volatile("st.global.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(q), "f"(c[0]), "f"(c[1]), "f"(d[0]),
                       "f"(d[1]), "f"(c[4]), "f"(c[5]), "f"(d[2]), "f"(d[3])
                       : "memory");
        } else {
          static_cast<uint4*>(out)[cell] = make_uint4(half_pair<VT>(c[0], c[1]), half_pair<VT>(c[2], c[3]),
                                                      half_pair<VT>(c[4], c[5]), half_pair<VT>(c[6], c[7]));
        }
      }
    }
    if (out_vox && cy < ny) {  // voxels (cx0 + lane, cy, cz0 + ..): plane p1, one in from its corner
      for (int zi = warp; zi < kTile; zi += kThreads / 32) {
        const int x = cx0 + lane, z = cz0 + zi;
        if (x >= nx || z >= nz) continue;
        const float a = p1[(zi + 1) * kPlane + lane + 1];
        const int64_t i = ((int64_t)z * ny + cy) * nx + x;
        if constexpr (VT == XR_VOXEL_F32) static_cast<float*>(out_vox)[i] = a;
        else if constexpr (VT == XR_VOXEL_F16) static_cast<__half*>(out_vox)[i] = __float2half_rn(a);
        else static_cast<__nv_bfloat16*>(out_vox)[i] = __float2bfloat16_rn(a);
      }
    }
    __syncthreads();
    if (more) {
      stage(plane[(cy - cy0) & 1]);
      __syncthreads();
    }
  }
}

// Voxels in the volume's own 16-bit type, for volumes without a cell copy.
template <int VT>
__global__ void convert_voxels_kernel(const float* __restrict__ in, int64_t n, float scale, void* out) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const float v = in[i] * scale;
    if constexpr (VT == XR_VOXEL_F16) static_cast<__half*>(out)[i] = __float2half_rn(v);
    else static_cast<__nv_bfloat16*>(out)[i] = __float2bfloat16_rn(v);
  }
}

}  // namespace

cudaError_t launch_hu_to_mu(const float* hu, int64_t n, float* mu, cudaStream_t s) {
  hu_to_mu_kernel<<<(unsigned)std::min<int64_t>((n + 1023) / 1024, 8192), kThreads, 0, s>>>(hu, n, mu);
  return cudaGetLastError();
}

cudaError_t launch_volume_stats(const float* vox, int nx, int ny, int nz, uint32_t* d_occ, int nmx, int nmy, int nmz,
                                VolStats* d_stats, cudaStream_t s) {
  const size_t words = ((size_t)nmx * nmy * nmz + 31) / 32;
  cudaError_t e = cudaMemsetAsync(d_occ, 0, words * sizeof(uint32_t), s);
  if (e == cudaSuccess) e = cudaMemsetAsync(d_stats, 0, sizeof(VolStats), s);
  if (e != cudaSuccess) return e;
  const int64_t nxs = ((int64_t)nx + kSegX - 1) / kSegX, nyb = ((int64_t)ny + 7) / 8, nzb = ((int64_t)nz + 7) / 8;
  const bool vec = nx % 4 == 0 && reinterpret_cast<uintptr_t>(vox) % 16 == 0;
  const auto kernel = vec ? volume_stats_kernel<true> : volume_stats_kernel<false>;
  kernel<<<(unsigned)(nxs * nyb * nzb), kThreads, 0, s>>>(vox, nx, ny, nz, (int)nxs, (int)nyb, d_occ, nmx, nmy, nmz,
                                                          d_stats);
  return cudaGetLastError();
}

cudaError_t launch_build_cells(const float* vox_f32, int nx, int ny, int nz, int32_t voxel_type, float scale,
                               bool weighted, void* out, void* out_vox, cudaStream_t s) {
  int32_t cs[2];
  cell_strides(nx, ny, nz, cs);
  const int64_t tx = (nx + (int64_t)kTile) / kTile, tz = (nz + (int64_t)kTile) / kTile,
                ty = (ny + (int64_t)kBuildY) / kBuildY;
  const unsigned blocks = (unsigned)(tx * ty * tz);
  switch (voxel_type) {
    case XR_VOXEL_F32:
      build_cells_kernel<XR_VOXEL_F32><<<blocks, kThreads, 0, s>>>(vox_f32, nx, ny, nz, 1.0f, weighted, cs[0], cs[1], (int)tx,
                                                                   (int)tz, out, out_vox);
      break;
    case XR_VOXEL_F16:
      build_cells_kernel<XR_VOXEL_F16><<<blocks, kThreads, 0, s>>>(vox_f32, nx, ny, nz, scale, weighted, cs[0], cs[1], (int)tx,
                                                                   (int)tz, out, out_vox);
      break;
    case XR_VOXEL_BF16:
      build_cells_kernel<XR_VOXEL_BF16><<<blocks, kThreads, 0, s>>>(vox_f32, nx, ny, nz, scale, weighted, cs[0], cs[1], (int)tx,
                                                                    (int)tz, out, out_vox);
      break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

cudaError_t launch_convert_voxels(const float* vox_f32, int64_t n, int32_t voxel_type, float scale, void* out,
                                  cudaStream_t s) {
  if (voxel_type == XR_VOXEL_F16) convert_voxels_kernel<XR_VOXEL_F16><<<2048, kThreads, 0, s>>>(vox_f32, n, scale, out);
  else if (voxel_type == XR_VOXEL_BF16)
    convert_voxels_kernel<XR_VOXEL_BF16><<<2048, kThreads, 0, s>>>(vox_f32, n, scale, out);
  else return cudaErrorInvalidValue;
  return cudaGetLastError();
}

}  // namespace xr

// xr_raycast.cu -- line-integral DRR kernels (one thread per detector ray).
//
// Semantics follow RayCasterLineIntCPU (xregRayCastLineIntCPU.cpp:106-290):
//   * ray from the pinhole to the detector pixel, clipped against the index
//     box [0, n-1]^3 with the segment-limited slab test
//     (xregSpatialPrimitives.cpp:176-221);
//   * if the clipped parameter interval is longer than 2e-3, both ends move
//     1e-3 inward (segment-parameter units, xregRayCastLineIntCPU.cpp:233-236);
//   * floor(len_mm / step) + 1 samples, positions advanced by repeated addition
//     of the step vector (:253-277);
//   * software trilinear interpolation with ITK's boundary rule (a neighbour
//     past the last index keeps no weight), never texture filtering;
//   * ray sum (or max) times the step in mm (:279); replace / accumulate /
//     background images as in RayCasterCPU::pre_compute (xregRayCastBaseCPU.cpp:128-158).
//
// The per-ray geometry (detector point, slab test, nudge, step count, start
// point, step vector) is xReg's own float arithmetic in Eigen's evaluation order
// (xf::ray_setup, xr_xfloat.h), so sample counts and sample positions are the
// reference's, bit for bit.  The interpolation and the sum use ordinary float
// arithmetic.
//
// Volume layouts (same values, same arithmetic, bit-identical results):
//   LINEAR  voxels x-fastest; a sample issues 8 scalar loads.
//   CELL8   for every trilinear cell (ix, iy, iz) in [-1, n-1]^3 the 8 corner
//           values (voxel indices clamped to [0, n-1]) are stored contiguously as
//           z-pairs (v000 v001 v100 v101 v010 v011 v110 v111, vxyz), so each pair
//           the packed FP32 blend needs is one 64-bit register: one 16-byte load per sample for FP16/BF16, two
//           for FP32, or one 32-byte load for FP32 (the 256-bit read, layout 2).
//           It spends 8x the voxel bytes of HBM to cut L1 requests per sample
//           from 8 to 1-2; the linear kernel is bound by exactly those requests.
//           Float32 cells hold, in place of the x + 1 corners, their differences
//           to the x corners (v1yz - v0yz), the first blend's slope (but for
//           VolView::weighted volumes, which hold the corners).
//           Cells are numbered z fastest, then x, then y (VolView::cs).  The
//           border cells (index -1 and n-1) are constant along their axis: a
//           position that rounding carries past a face of the volume reads the
//           face's values with no clamp in the sample loop.
#include "xr_cells.h"
#include "xr_gradtile.cuh"
#include "xr_internal.h"

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cfloat>

namespace xr {
namespace {

template <int VT>
struct Vox;
template <>
struct Vox<XR_VOXEL_F32> {
  __device__ __forceinline__ static float ld(const void* b, int i) {
    return __ldg(static_cast<const float*>(b) + i);
  }
  // 8 corners of cell c (CELL8 layout)
  __device__ __forceinline__ static void cell(const void* b, unsigned int c, float v[8]) {
    const float4* p = static_cast<const float4*>(b) + 2 * (size_t)c;
    const float4 lo = __ldg(p), hi = __ldg(p + 1);
    v[0] = lo.x; v[1] = lo.y; v[2] = lo.z; v[3] = lo.w;
    v[4] = hi.x; v[5] = hi.y; v[6] = hi.z; v[7] = hi.w;
  }
  // The same 32-byte cell with one 256-bit load (sm_100+ .v8 form); cells are
  // 32-byte aligned because the buffer is and every cell is 32 bytes.
  __device__ __forceinline__ static void cell_wide(const void* b, unsigned int c, float v[8]) {
    const float* p = static_cast<const float*>(b) + 8 * (size_t)c;
    asm("ld.global.nc.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
        : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
        : "l"(p));
  }
};
// FP16 volumes are blended on their half2 words (interp8_h16 below), so their
// corners are read as raw 16-bit values and never widened.
template <>
struct Vox<XR_VOXEL_F16> {
  __device__ __forceinline__ static unsigned int ld16(const void* b, int i) {
    return __ldg(static_cast<const unsigned short*>(b) + i);
  }
  // the 4 z-pair words of cell c (CELL8 layout)
  __device__ __forceinline__ static void cell_words(const void* b, unsigned int c, unsigned int w[4]) {
    const uint4 q = __ldg(static_cast<const uint4*>(b) + c);
    w[0] = q.x; w[1] = q.y; w[2] = q.z; w[3] = q.w;
  }
};
template <>
struct Vox<XR_VOXEL_BF16> {
  __device__ __forceinline__ static float ld(const void* b, int i) {
    return __bfloat162float(__ldg(static_cast<const __nv_bfloat16*>(b) + i));
  }
  __device__ __forceinline__ static void cell_words(const void* b, unsigned int c, unsigned int w[4]) {
    const uint4 q = __ldg(static_cast<const uint4*>(b) + c);
    w[0] = q.x; w[1] = q.y; w[2] = q.z; w[3] = q.w;
  }
};

constexpr int kThreads = 256;
// Resident blocks per SM the DRR kernels are compiled for: 48 registers, which
// hold four cells in flight per thread; measured faster than 40 or 64.
constexpr int kMinBlocksPerSM = 5;
// Warps per block of drr_kernel and drr_jobs_kernel.  Rays differ in length, and a
// block keeps its place until its longest is done: 4 warps measured 1.5 to 4 %
// faster than 8 (population 4867 -> 4785 us, FP16 coarse 2837 -> 2718, BF16 1570 ->
// 1521), 2 or 1 mixed (4749 / 2728 / 1545, 5178 / 2710 / 1497).
constexpr int kWarps = kDrrWarps;
constexpr int kMaxWarps = 8;  // of a drr_kernel block: 8 warps across where the caller asks for them
constexpr int kDeepBlocksPerSM = 4;  // of the deep march (launch_t): 128 registers
// CELL8 data read with one 256-bit load per sample (float32 volumes only).
constexpr int kLayoutCell8Wide = 2;
__device__ __forceinline__ int clampi(int v, int lo, int hi) { return max(min(v, hi), lo); }

// Trilinear of the 8 corners in cell order (z-pairs: v000 v001 v100 v101 v010
// v011 v110 v111, vxyz) as three levels of a + f (b - a), each difference
// rounded once and each blend one fma.  DIFF: v[2], v[3], v[6], v[7] already
// hold the x differences (float32 cells).  10 operations (14 without DIFF)
// where the weighted form (1 - f) a + f b takes 17.  A term whose far corners
// are zero stays exact to an ulp (b - a = -a exactly), so rays that graze the
// body keep their relative error; elsewhere the error is that of the weighted
// form, an ulp of the largest corner.
template <bool DIFF>
__device__ __forceinline__ float interp8(const float v[8], float fx, float fy, float fz) {
  const float d00 = DIFF ? v[2] : __fsub_rn(v[2], v[0]), d01 = DIFF ? v[3] : __fsub_rn(v[3], v[1]);
  const float d10 = DIFF ? v[6] : __fsub_rn(v[6], v[4]), d11 = DIFF ? v[7] : __fsub_rn(v[7], v[5]);
  const float a00 = __fmaf_rn(d00, fx, v[0]), a01 = __fmaf_rn(d01, fx, v[1]);
  const float a10 = __fmaf_rn(d10, fx, v[4]), a11 = __fmaf_rn(d11, fx, v[5]);
  const float b0 = __fmaf_rn(__fsub_rn(a10, a00), fy, a00);
  const float b1 = __fmaf_rn(__fsub_rn(a11, a01), fy, a01);
  return __fmaf_rn(__fsub_rn(b1, b0), fz, b0);
}

// The weighted form, for volumes whose differences could overflow or be
// undefined (VolView::weighted: an infinite voxel, or one above 2^126).
__device__ __forceinline__ float interp8_weighted(const float v[8], float fx, float fy, float fz) {
  const float gx = 1.0f - fx, gy = 1.0f - fy, gz = 1.0f - fz;
  const float a00 = fmaf(v[2], fx, v[0] * gx);
  const float a01 = fmaf(v[3], fx, v[1] * gx);
  const float a10 = fmaf(v[6], fx, v[4] * gx);
  const float a11 = fmaf(v[7], fx, v[5] * gx);
  const float b0 = fmaf(a10, fy, a00 * gy);
  const float b1 = fmaf(a11, fy, a01 * gy);
  return fmaf(b1, fz, b0 * gz);
}

// ---- packed FP32 pairs (sm_100+ f32x2): each lane rounds exactly as the
// scalar instruction with the same rounding mode, so results are bit-identical
// to the scalar code and only the instruction count changes.
__device__ __forceinline__ unsigned long long pk2(float a, float b) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void upk2(unsigned long long r, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(r));
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
  unsigned long long d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ unsigned long long add2_rm(unsigned long long a, unsigned long long b) {
  unsigned long long d;
  asm("add.rm.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ unsigned long long sub2(unsigned long long a, unsigned long long b) {
  unsigned long long d;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
// The two bf16 values of w less the floats of q, each difference rounded once as
// after widening (sub.f32.bf16, sm_100+).
__device__ __forceinline__ unsigned long long sub_bf16(unsigned int w, unsigned long long q) {
  float a, b, c, d;
  upk2(q, a, b);
  asm("{\n\t.reg .b16 l, h;\n\tmov.b32 {l, h}, %2;\n\t"
      "sub.rn.f32.bf16 %0, l, %3;\n\tsub.rn.f32.bf16 %1, h, %4;\n\t}"
      : "=f"(c), "=f"(d)
      : "r"(w), "f"(a), "f"(b));
  return pk2(c, d);
}
// interp8 on the z-pairs of a bf16 cell, w: (v000, v001) (v100, v101) (v010, v011)
// (v110, v111); the x and y blends run on pairs, the z blend in scalar.  The upper x
// corners are never widened: their differences come from the stored words (48 images
// of 300 x 260, 1522 us with eight corners widened, now 1441).
__device__ __forceinline__ float interp8_pairs(const unsigned int w[4], unsigned long long fxy, float fz) {
  float fx, fy;
  upk2(fxy, fx, fy);
  const unsigned long long q0 = pk2(__uint_as_float(w[0] << 16), __uint_as_float(w[0] & 0xffff0000u));
  const unsigned long long q2 = pk2(__uint_as_float(w[2] << 16), __uint_as_float(w[2] & 0xffff0000u));
  const unsigned long long FX = pk2(fx, fx), FY = pk2(fy, fy);
  const unsigned long long ay0 = fma2(sub_bf16(w[1], q0), FX, q0);  // (a00, a01)
  const unsigned long long ay1 = fma2(sub_bf16(w[3], q2), FX, q2);  // (a10, a11)
  const unsigned long long B = fma2(sub2(ay1, ay0), FY, ay0);       // (b0, b1)
  float b0, b1;
  upk2(B, b0, b1);
  return __fmaf_rn(__fsub_rn(b1, b0), fz, b0);
}

// ---- FP16 cells: the trilinear on the stored half2 words, with no
// conversion of the corners.  The x blend runs on the (z0, z1) pairs in half
// arithmetic (fma.rn.f16x2); the y blend is four mixed-precision fmas
// (fma.rn.f32.f16: exact products of halves added in float); the z blend is
// float.  The x and y weights are scaled by 2^15 before they are rounded to
// half, so a fraction as small as one float ulp of a position (>= 2^-24) is
// still a normal half; the stored values are below 1 (the volume's maximum is
// stored in [0.5, 1)), so the half blend cannot overflow; the volume's
// inv_scale removes the scales exactly.  Error: the half rounding of the four weights
// and of the x blend, about 1e-3 of a sample at worst, within the 2e-3 bound
// for half-precision volumes.  Every FP16 path (layouts, loops, the fused
// kernel) uses this one function, so they agree bit for bit.
__device__ __forceinline__ unsigned int h2_mul(unsigned int a, unsigned int b) {
  unsigned int d;
  asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
__device__ __forceinline__ unsigned int h2_fma(unsigned int a, unsigned int b, unsigned int c) {
  unsigned int d;
  asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}
// y blend of the half pairs a0 = (a00, a01), a1 = (a10, a11) with the half
// weights (low gy, high fy) of wy: b0 = a00 gy + a10 fy, b1 = a01 gy + a11 fy
__device__ __forceinline__ void h2_yblend(unsigned int a0, unsigned int a1, unsigned int wy, float& b0, float& b1) {
  asm("{\n\t.reg .b16 p0, p1, q0, q1, g, f;\n\t.reg .f32 t, u;\n\t"
      "mov.b32 {p0, p1}, %2;\n\tmov.b32 {q0, q1}, %3;\n\tmov.b32 {g, f}, %4;\n\t"
      "fma.rn.f32.f16 t, p0, g, %5;\n\tfma.rn.f32.f16 %0, q0, f, t;\n\t"
      "fma.rn.f32.f16 u, p1, g, %5;\n\tfma.rn.f32.f16 %1, q1, f, u;\n\t}"
      : "=f"(b0), "=f"(b1)
      : "r"(a0), "r"(a1), "r"(wy), "f"(0.0f));
}
// halves g (low) and f (high)
__device__ __forceinline__ unsigned int h2_pack(float g, float f) {
  unsigned int d;
  asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(f), "f"(g));
  return d;
}
// w: (v000, v001) (v100, v101) (v010, v011) (v110, v111), low half z = 0; fx, fy:
// the fractions times kH16 (the cell walk's positions carry that scale, so the
// four weights take two subtractions and two conversions; with the x weights
// converted one by one 20 images of 768^2 took 6555 us, now 6318, a pose of two views
// of 384^2 149, now 139); returns the sample times 2^30.
__device__ __forceinline__ float interp8_h16(const unsigned int w[4], float fx, float fy, float fz) {
  const float gx = __fsub_rn(kH16, fx);
  unsigned int GX, FX;  // each weight twice, from one conversion of both
  asm("{\n\t.reg .b16 g, f;\n\tmov.b32 {g, f}, %2;\n\tmov.b32 %0, {g, g};\n\tmov.b32 %1, {f, f};\n\t}"
      : "=r"(GX), "=r"(FX)
      : "r"(h2_pack(gx, fx)));
  const unsigned int wy = h2_pack(__fsub_rn(kH16, fy), fy);
  const unsigned int A0 = h2_fma(w[1], FX, h2_mul(w[0], GX));  // (a00, a01)
  const unsigned int A1 = h2_fma(w[3], FX, h2_mul(w[2], GX));  // (a10, a11)
  float b0, b1;
  h2_yblend(A0, A1, wy, b0, b1);
  return __fmaf_rn(__fsub_rn(b1, b0), fz, b0);
}

template <int KERNEL>
__device__ __forceinline__ float fold(float sum, float v) {
  if (KERNEL == XR_LINE_INT_MAX) return (sum < v) ? v : sum;
  return __fadd_rn(sum, v);
}

// A sample's fractions within its cell.
struct Frac3 {
  float x, y, z;
};
struct Frac21 {
  unsigned long long xy;
  float z;
};

// One cell's corners, as loaded (a bf16 value is the upper half of the float with
// the same value, so a word widens with one shift and one mask, exactly).
template <int VT, int LAYOUT>
struct CellData {
  static constexpr int kWords = VT == XR_VOXEL_F32 ? 8 : 4;
  unsigned int w[kWords];
  // cell number c, or (BYTES) the cell at byte offset c
  template <bool BYTES = false>
  __device__ __forceinline__ void load(const void* data, unsigned int c) {
    if constexpr (BYTES) {
      data = static_cast<const char*>(data) + c;
      c = 0;
    }
    if constexpr (VT != XR_VOXEL_F32) Vox<VT>::cell_words(data, c, w);
    else {
      float v[8];
      if constexpr (LAYOUT == kLayoutCell8Wide) Vox<VT>::cell_wide(data, c, v);
      else Vox<VT>::cell(data, c, v);
#pragma unroll
      for (int k = 0; k < 8; ++k) w[k] = __float_as_uint(v[k]);
    }
  }
  __device__ __forceinline__ float value(const Frac3& f) const {
    if constexpr (VT == XR_VOXEL_F16) return interp8_h16(w, f.x, f.y, f.z);  // x and y scaled by kH16
    else {
      float v[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        if constexpr (VT == XR_VOXEL_BF16) v[k] = __uint_as_float((k & 1) ? (w[k >> 1] & 0xffff0000u) : (w[k >> 1] << 16));
        else v[k] = __uint_as_float(w[k]);
      }
      return interp8<VT == XR_VOXEL_F32>(v, f.x, f.y, f.z);
    }
  }
  __device__ __forceinline__ float value(const Frac21& f) const {
    static_assert(VT == XR_VOXEL_BF16, "");
    return interp8_pairs(w, f.xy, f.z);
  }
  // of a volume with VolView::weighted, whose float32 cells hold their corners
  __device__ __forceinline__ float weighted_value(const Frac21& f) const {
    Frac3 g;
    upk2(f.xy, g.x, g.y);
    g.z = f.z;
    return weighted_value(g);
  }
  __device__ __forceinline__ float weighted_value(const Frac3& f) const {
    float v[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      if constexpr (VT == XR_VOXEL_F32) v[k] = __uint_as_float(w[k]);
      else v[k] = __uint_as_float((k & 1) ? (w[k >> 1] & 0xffff0000u) : (w[k >> 1] << 16));
    }
    return interp8_weighted(v, f.x, f.y, f.z);
  }
};

// How a kernel blends a volume's corners: the cells' kernels know it (their volumes are
// weighted or not), those of the LINEAR layout ask the volume.
enum class Blend { kDifferences, kWeights, kVolume };
template <int VT, Blend BLEND>
__device__ __forceinline__ bool by_weights(const VolView& vol) {
  return VT != XR_VOXEL_F16 && (BLEND == Blend::kWeights || (BLEND == Blend::kVolume && vol.weighted));
}

// Trilinear sample at index position (px, py, pz) with ITK's boundary rule:
// positions past a face take the face's values.  The cell is floor(position)
// clamped to [-1, n-1], the fraction saturated to [0, 1] (a NaN position reads
// cell 0 with fraction 0).  INSIDE (LINEAR only): the caller has shown that the
// position lies in [0, n-1) on every axis, where no clamp changes anything.  A
// weighted volume's cells end at n-2 (fraction 1 on the last voxel), without the
// border's: there a corner of weight 0 decides whether an infinity makes a NaN.
template <int VT, int LAYOUT, bool INSIDE, Blend BLEND>
__device__ __forceinline__ float sample(const VolView& vol, const void* data, float px, float py, float pz) {
  const bool weighted = by_weights<VT, BLEND>(vol);
  int ix = __float2int_rd(px), iy = __float2int_rd(py), iz = __float2int_rd(pz);
  if (!INSIDE) {
    const int b = weighted ? 1 : 0;
    ix = clampi(ix, b - 1, vol.nx - 1 - b);
    iy = clampi(iy, b - 1, vol.ny - 1 - b);
    iz = clampi(iz, b - 1, vol.nz - 1 - b);
  }
  float fx = px - (float)ix, fy = py - (float)iy, fz = pz - (float)iz;
  if (!INSIDE) {
    fx = __saturatef(fx);
    fy = __saturatef(fy);
    fz = __saturatef(fz);
  }
  if constexpr (LAYOUT == XR_LAYOUT_LINEAR) {
    int sx = 1, sy = vol.nx, sz = vol.nx * vol.ny;
    if (!INSIDE) {  // border cells: both corners are the face's voxel
      sx = (ix >= 0 && ix < vol.nx - 1) ? sx : 0;
      sy = (iy >= 0 && iy < vol.ny - 1) ? sy : 0;
      sz = (iz >= 0 && iz < vol.nz - 1) ? sz : 0;
      ix = max(ix, 0);
      iy = max(iy, 0);
      iz = max(iz, 0);
    }
    const int b = (iz * vol.ny + iy) * vol.nx + ix;
    if constexpr (VT == XR_VOXEL_F16) {  // the CELL8 words, packed from 8 scalar reads
      unsigned int w[4];
      w[0] = Vox<VT>::ld16(data, b) | (Vox<VT>::ld16(data, b + sz) << 16);
      w[1] = Vox<VT>::ld16(data, b + sx) | (Vox<VT>::ld16(data, b + sz + sx) << 16);
      w[2] = Vox<VT>::ld16(data, b + sy) | (Vox<VT>::ld16(data, b + sz + sy) << 16);
      w[3] = Vox<VT>::ld16(data, b + sy + sx) | (Vox<VT>::ld16(data, b + sz + sy + sx) << 16);
      return interp8_h16(w, fx * kH16, fy * kH16, fz);
    } else {
      float v[8];
      v[0] = Vox<VT>::ld(data, b);
      v[1] = Vox<VT>::ld(data, b + sz);
      v[2] = Vox<VT>::ld(data, b + sx);
      v[3] = Vox<VT>::ld(data, b + sz + sx);
      v[4] = Vox<VT>::ld(data, b + sy);
      v[5] = Vox<VT>::ld(data, b + sz + sy);
      v[6] = Vox<VT>::ld(data, b + sy + sx);
      v[7] = Vox<VT>::ld(data, b + sz + sy + sx);
      return weighted ? interp8_weighted(v, fx, fy, fz) : interp8<false>(v, fx, fy, fz);
    }
  } else {
    const unsigned int c = (unsigned int)(ix + 1) * (unsigned int)vol.cs[0] +
                           (unsigned int)(iy + 1) * (unsigned int)vol.cs[1] + (unsigned int)(iz + 1);
    CellData<VT, LAYOUT> q;
    q.load(data, c);
    constexpr float kS = VT == XR_VOXEL_F16 ? kH16 : 1.0f;
    if constexpr (BLEND == Blend::kWeights) return q.weighted_value(Frac3{fx, fy, fz});
    else return q.value(Frac3{fx * kS, fy * kS, fz});
  }
}

// Walks the macro cells of the ray p0 + k st from k = kstart towards kend
// (dir +1 forward, -1 backward) and returns the ray parameter at which it
// enters the first macro cell whose (dilated) occupancy bit is set, or +inf
// (-inf backward) when none is met before kend.  Macro cell m spans continuous
// index [8m, 8m + 8) on each axis; the first and the last on an axis run on past
// the volume.  The walk advances the parameter of each axis' next boundary by its
// spacing: with inv = 1 / st within a few ulps and at most a few hundred steps
// the parameters stay well inside the one-sample margin the caller leaves on each
// side.  A step takes about 15 instructions; forming each boundary's parameter
// from the cell index took three times that, a quarter of a ray's instructions.
__device__ __forceinline__ float macro_march(const VolView& v, const float p0[3], const float st[3],
                                             const float inv[3], float kstart, float kend, int dir) {
  const int nm[3] = {v.nmx, v.nmy, v.nmz};
  const int stride[3] = {1, v.nmx, v.nmx * v.nmy};
  const float fdir = (float)dir;
  float t[3], dt[3];  // parameter along the walk (fdir k) of the axis' next boundary, its spacing
  int step[3], left[3], idx = 0;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const float q = p0[a] + kstart * st[a], d = fdir * st[a];
    const int m = clampi(__float2int_rd(q) >> kMacroShift, 0, nm[a] - 1);
    idx += m * stride[a];
    const bool up = d > 1.0e-20f, down = d < -1.0e-20f;
    step[a] = up ? stride[a] : -stride[a];
    left[a] = up ? nm[a] - 1 - m : down ? m : 0;  // boundaries ahead
    const float bound = (float)((up ? m + 1 : m) << kMacroShift);
    dt[a] = fabsf(inv[a]) * (float)(1 << kMacroShift);
    t[a] = left[a] > 0 ? fdir * ((bound - p0[a]) * inv[a]) : INFINITY;
  }
  float k = fdir * kstart;
  const float tend = fdir * kend;
  for (;;) {  // at most the boundaries ahead: each step uses one up
    if ((__ldg(v.occ + (idx >> 5)) >> (idx & 31)) & 1u) return fdir * k;
    const float tn = fminf(t[0], fminf(t[1], t[2]));
    if (!(tn <= tend)) return fdir * INFINITY;  // past the end, or no boundary ahead
    k = fmaxf(k, tn);
    const int a = t[0] == tn ? 0 : t[1] == tn ? 1 : 2;
#pragma unroll
    for (int b = 0; b < 3; ++b)
      if (a == b) {
        idx += step[b];
        t[b] = --left[b] > 0 ? t[b] + dt[b] : INFINITY;
      }
  }
}

// Position of a ray's next sample in the cell layouts, for rays whose positions
// stay in [-1, n) on every axis (trace_pixel).  next() returns the cell of the
// current position (its byte offset when the copy is below 4 GB, BYTES, which
// spares the 64-bit multiply of an index: FP16 loop 7443 -> 7175 us on 20 images
// of 768^2; its number otherwise) and the fractions, then advances by one step.
// floor(p) comes from one round-down addition of the axis' constant K = 2^23 + m
// (VolView::kfl, m a whole number): for -1 <= p < 2^24 - K the sum rounded down
// is exactly K + floor(p), whose bit pattern is 0x4B000000 + m + floor(p).  The
// constants are chosen so that the biases of the three axes cancel in the cell
// (wrapping 32-bit arithmetic): no conversion and no correction remain.  FP16
// walks x and y in units of 2^-15 voxel (a power of two: every operation rounds
// as unscaled), which makes the fractions the scaled weights interp8_h16 takes.
template <int VT, bool BYTES>
struct CellWalk {
  using Frac = Frac3;
  static constexpr unsigned int kUnit = BYTES ? (VT == XR_VOXEL_F32 ? 32u : 16u) : 1u;
  static constexpr float kScale = VT == XR_VOXEL_F16 ? kH16 : 1.0f;
  float px, py, pz, sx, sy, sz, kx, ky, kz;
  unsigned int csx, csy;
  __device__ __forceinline__ CellWalk(const VolView& v, float x, float y, float z, float dx, float dy, float dz)
      : px(x * kScale), py(y * kScale), pz(z), sx(dx * kScale), sy(dy * kScale), sz(dz), kx(v.kfl[0]), ky(v.kfl[1]),
        kz(v.kfl[2]), csx((unsigned int)v.cs[0] * kUnit), csy((unsigned int)v.cs[1] * kUnit) {}
  __device__ __forceinline__ unsigned int next(Frac& f) {
    const float tx = __fadd_rd(px, kx), ty = __fadd_rd(py, ky), tz = __fadd_rd(pz, kz);
    f.x = __fsub_rn(px, __fsub_rn(tx, kx));
    f.y = __fsub_rn(py, __fsub_rn(ty, ky));
    f.z = __fsub_rn(pz, __fsub_rn(tz, kz));
    px = __fadd_rn(px, sx);
    py = __fadd_rn(py, sy);
    pz = __fadd_rn(pz, sz);
    return __float_as_uint(ty) * csy + (__float_as_uint(tx) * csx + __float_as_uint(tz) * kUnit);
  }
};
// BF16: x and y as one packed pair (each lane rounds as the scalar instruction,
// so positions, cells and fractions are the same).
template <bool BYTES>
struct CellWalk<XR_VOXEL_BF16, BYTES> {
  using Frac = Frac21;
  static constexpr unsigned int kUnit = BYTES ? 16u : 1u;
  unsigned long long P, S, K;
  float pz, sz, kz;
  unsigned int csx, csy;
  __device__ __forceinline__ CellWalk(const VolView& v, float x, float y, float z, float dx, float dy, float dz)
      : P(pk2(x, y)), S(pk2(dx, dy)), K(pk2(v.kfl[0], v.kfl[1])), pz(z), sz(dz), kz(v.kfl[2]),
        csx((unsigned int)v.cs[0] * kUnit), csy((unsigned int)v.cs[1] * kUnit) {}
  __device__ __forceinline__ unsigned int next(Frac& f) {
    const unsigned long long T = add2_rm(P, K);
    const float tz = __fadd_rd(pz, kz);
    f.xy = sub2(P, sub2(T, K));
    f.z = __fsub_rn(pz, __fsub_rn(tz, kz));
    float tx, ty;
    upk2(T, tx, ty);
    P = add2(P, S);
    pz = __fadd_rn(pz, sz);
    return __float_as_uint(ty) * csy + (__float_as_uint(tx) * csx + __float_as_uint(tz) * kUnit);
  }
};

// n samples of one ray from the current position on, in order, from the cells
// (positions within [-1, n) on every axis).  Four cells are in flight per thread.
// Float32 and FP16 load four, then blend four, in scalar arithmetic; BF16, whose
// widening makes it the most instruction-bound, runs on packed pairs and reloads
// each cell's registers as soon as it is blended.  Measured on sum launches of
// the 256^3 / 384^2 population (float32, 100 poses), a 320 x 320 x 256 / 192^2 one
// (FP16, 171 images) and a 256 x 256 x 200 / 300 x 260 one (BF16, 48 images), in us:
// scalar batches of four 5144 / 2873 / 1726, packed batches - / 3025 / 1690,
// packed reload 7029 / 3464 / 1613 (the reload form spills at float32's and
// FP16's register need), scalar reload of three 5317 / - / -.
// WEIGHTED: of a VolView::weighted volume, by weights (no DEEP).
template <int VT, int KERNEL, int LAYOUT, bool BYTES, bool DEEP, bool WEIGHTED>
__device__ __forceinline__ float march_cells(const VolView& vol, float px, float py, float pz, float sx, float sy,
                                             float sz, unsigned int n, float sum) {
  using Cell = CellData<VT, LAYOUT>;
  using Walk = CellWalk<VT, BYTES>;
  using Frac = typename Walk::Frac;
  const void* data = vol.cells;
  Walk walk(vol, px, py, pz, sx, sy, sz);
  auto value = [](const Cell& q, const Frac& f) {
    if constexpr (WEIGHTED) return q.weighted_value(f);
    else return q.value(f);
  };
  if constexpr (DEEP) {  // batches of eight, the last one masked
    constexpr unsigned int kDeep = 8;
    unsigned int c = 0;
    while (n > 0) {
      const unsigned int m = min(n, kDeep);
      Frac f[kDeep];
      Cell q[kDeep];
#pragma unroll
      for (unsigned int k = 0; k < kDeep; ++k) {
        const unsigned int ck = walk.next(f[k]);
        c = k < m ? ck : c;  // past the last sample: the last cell again
        q[k].template load<BYTES>(data, c);
      }
#pragma unroll
      for (unsigned int k = 0; k < kDeep; ++k) {
        const float v = fold<KERNEL>(sum, value(q[k], f[k]));
        sum = k < m ? v : sum;
      }
      n -= m;
    }
    return sum;
  }
  if constexpr (VT == XR_VOXEL_BF16 && !WEIGHTED) {
    if (n >= 4) {
      Frac f[4];
      Cell q[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) q[k].template load<BYTES>(data, walk.next(f[k]));
      for (n -= 4; n >= 4; n -= 4) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          sum = fold<KERNEL>(sum, value(q[k], f[k]));
          q[k].template load<BYTES>(data, walk.next(f[k]));
        }
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) sum = fold<KERNEL>(sum, value(q[k], f[k]));
    }
  } else {
    for (; n >= 4; n -= 4) {
      Frac f[4];
      Cell q[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) q[k].template load<BYTES>(data, walk.next(f[k]));
#pragma unroll
      for (int k = 0; k < 4; ++k) sum = fold<KERNEL>(sum, value(q[k], f[k]));
    }
  }
  for (; n > 0; --n) {
    Frac f;
    Cell q;
    q.template load<BYTES>(data, walk.next(f));
    sum = fold<KERNEL>(sum, value(q, f));
  }
  return sum;
}

// The same through sample(): the LINEAR layout, and rays that march_cells does
// not take.
template <int VT, int KERNEL, int LAYOUT, bool INSIDE, Blend BLEND>
__device__ __forceinline__ float march_samples(const VolView& vol, const void* data, float px, float py, float pz,
                                               float sx, float sy, float sz, unsigned int n, float sum) {
  if (LAYOUT == XR_LAYOUT_LINEAR || BLEND != Blend::kDifferences) {
    for (; n >= 2; n -= 2) {
      const float v0 = sample<VT, LAYOUT, INSIDE, BLEND>(vol, data, px, py, pz);
      px = __fadd_rn(px, sx); py = __fadd_rn(py, sy); pz = __fadd_rn(pz, sz);
      const float v1 = sample<VT, LAYOUT, INSIDE, BLEND>(vol, data, px, py, pz);
      px = __fadd_rn(px, sx); py = __fadd_rn(py, sy); pz = __fadd_rn(pz, sz);
      sum = fold<KERNEL>(fold<KERNEL>(sum, v0), v1);
    }
  }
  for (; n > 0; --n) {
    const float v0 = sample<VT, LAYOUT, INSIDE, BLEND>(vol, data, px, py, pz);
    px = __fadd_rn(px, sx); py = __fadd_rn(py, sy); pz = __fadd_rn(pz, sz);
    sum = fold<KERNEL>(sum, v0);
  }
  return sum;
}

// Traces the ray of pixel (row, col) of projection proj and stores the result
// (the caller checks that the pixel exists).  Returns the number of samples of
// the reference step rule; *loaded receives how many of them were loaded (the
// others were proven zero and skipped).
template <int VT, int KERNEL, int LAYOUT, bool DEEP, Blend BLEND>
__device__ __forceinline__ unsigned long long trace_pixel(const DrrParams& p, const int64_t proj, const int row,
                                                          const int col, unsigned int* loaded) {
  float sum = (KERNEL == XR_LINE_INT_MAX) ? -FLT_MAX : 0.0f;
  unsigned long long ns = 0;
  *loaded = 0;
  {
    // xReg's per-ray float set-up (xf::ray_setup): clipped, nudged segment,
    // start point, step vector and the step-count quotient
    const float maxb[3] = {(float)(p.vol.nx - 1), (float)(p.vol.ny - 1), (float)(p.vol.nz - 1)};
    float st0[3], stv[3], quot;
    bool hit = xf::ray_setup(p.geo[proj], (float)col, (float)row, maxb, p.step, st0, stv, quot);
    if (hit) {
      float px = st0[0], py = st0[1], pz = st0[2];
      // num_steps = size_t(quotient) through a saturating 32-bit conversion (a
      // 64-bit one runs on the slow FP64 pipe): above 2^32 - 1 it saturates and
      // NaN gives 0, so the max_steps test (max_steps < 2^31) decides as with 64 bits
      unsigned long long nsteps = __float2uint_rz(quot);
      if (!(nsteps <= p.max_steps)) {
        // A ray longer than the volume diagonal allows can only come from a
        // non-finite or degenerate pose: count it and leave the pixel unsampled
        // rather than loop for an unbounded time.
        atomicAdd(p.err_counter, 1u);
        nsteps = 0;
        hit = false;
      }
      const float sx = stv[0], sy = stv[1], sz = stv[2];
      // reciprocal steps for the skipping bounds (never for sample positions), to an
      // ulp or two: the bounds leave a sample on each side
      const float inv_st[3] = {__fdividef(1.0f, sx), __fdividef(1.0f, sy), __fdividef(1.0f, sz)};
      const void* data = (LAYOUT != XR_LAYOUT_LINEAR) ? p.vol.cells : p.vol.voxels;
      // Samples [first, last] may touch non-zero voxels; the others interpolate
      // only zeros, so for the sum they add exactly +0 and need no load.  The
      // samples before `first` still advance the position by the same float
      // additions, so every sampled position is the one the reference uses.
      unsigned int first = 0, last = (unsigned int)nsteps;
      if (KERNEL == XR_LINE_INT_SUM && p.vol.has_support && hit) {
        float lo = 0.0f, hi = (float)nsteps;
        if (p.vol.sup_lo[0] > p.vol.sup_hi[0]) hi = -1.0f;  // all-zero volume
        const float st[3] = {sx, sy, sz}, p0[3] = {px, py, pz};
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          if (fabsf(st[k]) > 1.0e-20f) {
            // reciprocal steps: a few ulps of error, inside the one-sample margins below
            float a = (p.vol.sup_lo[k] - p0[k]) * inv_st[k], b = (p.vol.sup_hi[k] - p0[k]) * inv_st[k];
            if (a > b) { const float t = a; a = b; b = t; }
            lo = fmaxf(lo, a);
            hi = fminf(hi, b);
          } else if (!(p0[k] > p.vol.sup_lo[k] && p0[k] < p.vol.sup_hi[k])) {
            hi = -1.0f;
          }
        }
        if (!(lo <= hi)) {
          last = 0;
          first = 1;  // no sample can be non-zero
        } else {
          const float f0 = floorf(lo) - 1.0f, f1 = ceilf(hi) + 1.0f;
          first = f0 > 0.0f ? (unsigned int)f0 : 0u;
          last = f1 < (float)nsteps ? (unsigned int)f1 : (unsigned int)nsteps;
        }
      }
      // Repeated addition drifts by at most a half-ulp of a coordinate below 2^e
      // per sample: with fewer than 2^(22-e) samples positions stay within an
      // eighth of a voxel of the exact ray.
      const int ebits = 32 - __clz(max(p.vol.nx, max(p.vol.ny, p.vol.nz)));
      const bool drift_ok = hit && ebits <= 22 && last < (1u << (22 - ebits));
      if (KERNEL == XR_LINE_INT_SUM && p.vol.occ && drift_ok && first <= last) {
        // Macro-cell trim: walk the macro grid from each end of [first, last]
        // to the first occupied macro cell; the samples before (after) it lie in
        // empty macro cells and add exactly 0.  The occupancy is dilated by one
        // trilinear cell, so a sample whose float position strays less than a
        // voxel from the exact ray still reads only zero corners.
        {
          const float p0[3] = {px, py, pz}, st[3] = {sx, sy, sz};
          const float kf = macro_march(p.vol, p0, st, inv_st, (float)first, (float)last, 1);
          if (kf == INFINITY) {
            first = 1u;
            last = 0u;  // every sample is zero
          } else {
            const float f = floorf(kf) - 1.0f;
            if (f > (float)first) first = (unsigned int)f;
            const float kl = macro_march(p.vol, p0, st, inv_st, (float)last, (float)first, -1);
            if (kl == -INFINITY) {
              first = 1u;
              last = 0u;
            } else {
              const float l = ceilf(kl) + 1.0f;
              if (l < (float)last) last = (unsigned int)l;
            }
          }
        }
      }
      // With both ends within three quarters of a voxel of [0, n-1] (the segment is
      // straight) and a drift below an eighth, every position stays in [-1, n):
      // march_cells, whose loads no clamp bounds.  Rays of ordinary frames all lie
      // there; a NaN or infinite start or step does not, nor one that a focal point
      // millions of voxels away rounds off the volume: those take the clamped
      // sampler.  On the LINEAR layout, and of weighted volumes, rays a quarter voxel
      // inside run without clamps.
      constexpr bool kWeights = BLEND == Blend::kWeights, kInside = LAYOUT == XR_LAYOUT_LINEAR || kWeights;
      bool unclamped = drift_ok && (LAYOUT == XR_LAYOUT_LINEAR || p.vol.kfl[0] > 0.0f);
      if (unclamped) unclamped = xf::samples_within(st0, stv, first, last, maxb, kInside ? -0.25f : 0.75f);
      if (hit) {
        // advance to sample `first` (four additions per trip: the skipped samples
        // are a large part of a trimmed ray); x and y as one packed pair, whose
        // lanes round as the scalar additions do
        unsigned int skip = first <= last ? first : last + 1u;
        {
          unsigned long long P = pk2(px, py);
          const unsigned long long S = pk2(sx, sy);
          for (; skip >= 4; skip -= 4) {
            P = add2(P, S); pz = __fadd_rn(pz, sz);
            P = add2(P, S); pz = __fadd_rn(pz, sz);
            P = add2(P, S); pz = __fadd_rn(pz, sz);
            P = add2(P, S); pz = __fadd_rn(pz, sz);
          }
          for (; skip > 0; --skip) {
            P = add2(P, S); pz = __fadd_rn(pz, sz);
          }
          upk2(P, px, py);
        }
        // samples first..last in order
        const unsigned int n = first <= last ? last - first + 1u : 0u;
        *loaded = n;
        if (unclamped) {
          if constexpr (LAYOUT == XR_LAYOUT_LINEAR)
            sum = march_samples<VT, KERNEL, LAYOUT, true, BLEND>(p.vol, data, px, py, pz, sx, sy, sz, n, sum);
          else
            sum = p.vol.cell_bytes
                      ? march_cells<VT, KERNEL, LAYOUT, true, DEEP, kWeights>(p.vol, px, py, pz, sx, sy, sz, n, sum)
                      : march_cells<VT, KERNEL, LAYOUT, false, DEEP, kWeights>(p.vol, px, py, pz, sx, sy, sz, n, sum);
        } else {
          sum = march_samples<VT, KERNEL, LAYOUT, false, BLEND>(p.vol, data, px, py, pz, sx, sy, sz, n, sum);
        }
        sum = __fmul_rn(sum, p.step);
        if (VT != XR_VOXEL_F32) sum = __fmul_rn(sum, p.vol.inv_scale);
        ns = nsteps + 1;
      }
    }
    // aa_sum = 0 + sum (xregRayCastLineIntCPU.cpp:189,282), then the store rule.
    const float aa = __fadd_rn(0.0f, sum);
    const int64_t npix = (int64_t)p.rows * p.cols;
    const int64_t pix = (int64_t)row * p.cols + col;
    const int64_t oidx = proj * npix + pix;
    float prev;
    if (p.bg_projs) prev = p.bg_projs[(int64_t)p.cam_idx[proj] * npix + pix];
    else if (p.store == XR_PROJ_STORE_REPLACE) prev = p.default_bg;
    else prev = p.out[oidx];
    p.out[oidx] = (KERNEL == XR_LINE_INT_MAX) ? ((prev < aa) ? aa : prev) : __fadd_rn(prev, aa);
  }
  return ns;
}

// The pixel of a lane in its warp's 8 x 4 (wl 3) or 4 x 8 (wl 2) patch: four
// consecutive lanes are a 2 x 2 block, eight a 4 x 2 block.
__device__ __forceinline__ void lane_pixel(int lane, int wl, int& col, int& row) {
  col = (lane & 1) + ((lane >> 1) & ((1 << wl) - 2));  // lane bits 0, 2 (and 3 when wide)
  row = ((lane >> 1) & 1) + ((lane >> (wl + 1)) << 1);
}

template <int VT, int KERNEL, int LAYOUT, bool DEEP, Blend BLEND>
__global__ void __launch_bounds__(32 * kMaxWarps, (DEEP ? kDeepBlocksPerSM : kMinBlocksPerSM * 8 / kWarps) * kWarps / kMaxWarps)
drr_kernel(const DrrParams p, const int64_t proj_base) {
  // Each warp covers an 8 x 4 (or, tall, 4 x 8) patch of pixels so its 32 rays
  // stay close inside the volume; a block is bw x bh warps, kWarps or bw of them.  The
  // projection is the fastest grid index: blocks resident at the same time trace
  // the same detector tile for many nearby poses, whose footprints overlap in L2.
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int bw = p.block_warps_x;
  const int wl = p.warp_tall ? 2 : 3;  // log2 of the warp's width in pixels
  const int wc = 1 << wl, wr = 32 >> wl;
  int lc, lr;
  lane_pixel(lane, wl, lc, lr);
  const int col = blockIdx.y * (wc * bw) + (warp % bw) * wc + lc;
  const int row = blockIdx.z * (p.block_warps_y * wr) + (warp / bw) * wr + lr;
  const int64_t proj = proj_base + blockIdx.x;
  unsigned long long ns = 0;
  unsigned int nl = 0;
  if (col < p.cols && row < p.rows) ns = trace_pixel<VT, KERNEL, LAYOUT, DEEP, BLEND>(p, proj, row, col, &nl);
  if (p.sample_counter) {
    unsigned long long nlw = nl;
    for (int o = 16; o > 0; o >>= 1) {
      ns += __shfl_down_sync(0xffffffffu, ns, o);
      nlw += __shfl_down_sync(0xffffffffu, nlw, o);
    }
    if (lane == 0 && ns) atomicAdd(p.sample_counter, ns);
    if (lane == 0 && nlw && p.loaded_counter) atomicAdd(p.loaded_counter, nlw);
  }
}

// ---- brick-staged variant (layout 3: float32 CELL8 cells, sum kernel) ----
// One block traces 16x16 rays of one projection.  Their samples are taken in
// slabs of cells along the rays' dominant axis: for each slab the block copies
// the cells its rays reach there (a box from every ray's cell at the slab entry
// and an estimate of its exit, widened by one cell) into shared memory, then
// each ray takes its samples in that slab from the copy; a sample whose cell
// falls outside the box reads global memory.  Positions, cells, fractions and
// the order of the sum are those of drr_kernel (support-box skipping included,
// no macro-cell trim), so every value is identical.  The staged alternative to
// gathering through L1, measured against it; never chosen by the autotuner.
constexpr int kLayoutBrick = 3;
constexpr int kBrickCells = 1400;  // 43.75 KB of 32-byte cells
constexpr int kBrickDepth = 16;    // cells per slab along the dominant axis

// Cell (numbered from 0: floor + 1) and fractions of a position, clamped as sample() does.
template <Blend BLEND>
__device__ __forceinline__ void cell3(const VolView& vol, const float pos[3], int c[3], float f[3]) {
  const int n[3] = {vol.nx, vol.ny, vol.nz};
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const int b = BLEND == Blend::kWeights ? 1 : 0;
    const int i = clampi(__float2int_rd(pos[a]), b - 1, n[a] - 1 - b);
    f[a] = __saturatef(pos[a] - (float)i);
    c[a] = i + 1;
  }
}

template <Blend BLEND>
__device__ __forceinline__ float brick_value(const float v[8], const float f[3]) {
  return BLEND == Blend::kWeights ? interp8_weighted(v, f[0], f[1], f[2]) : interp8<true>(v, f[0], f[1], f[2]);
}

// The ray's remaining samples k..last from global memory, in order.
template <Blend BLEND>
__device__ __forceinline__ float brick_march_global(const VolView& vol, float pos[3], const float st[3],
                                                    unsigned int& k, unsigned int last, float sum) {
  for (; k <= last; ++k) {
    int c[3];
    float f[3], v[8];
    cell3<BLEND>(vol, pos, c, f);
    Vox<XR_VOXEL_F32>::cell_wide(vol.cells, (unsigned int)c[0] * vol.cs[0] + (unsigned int)c[1] * vol.cs[1] + (unsigned int)c[2], v);
    sum = __fadd_rn(sum, brick_value<BLEND>(v, f));
    pos[0] = __fadd_rn(pos[0], st[0]);
    pos[1] = __fadd_rn(pos[1], st[1]);
    pos[2] = __fadd_rn(pos[2], st[2]);
  }
  return sum;
}

template <Blend BLEND>
__global__ void __launch_bounds__(kThreads, 4) drr_brick_kernel(const DrrParams p, const int64_t proj_base) {
  __shared__ float4 s_cells[2 * kBrickCells];
  __shared__ int s_code, s_amin, s_amax, s_lo[3], s_hi[3];
  const int tid = threadIdx.x;
  const int col = blockIdx.y * 16 + (tid & 15), row = blockIdx.z * 16 + (tid >> 4);
  const int64_t proj = proj_base + blockIdx.x;
  const VolView& vol = p.vol;
  const int ncell[3] = {vol.nx + 1, vol.ny + 1, vol.nz + 1};
  const float4* cells = static_cast<const float4*>(vol.cells);
  if (tid == 0) {
    s_code = -1;
    s_amin = 0x7fffffff;
    s_amax = -1;
  }
  const bool pixel = col < p.cols && row < p.rows;
  float sum = 0.0f, pos[3] = {0.0f, 0.0f, 0.0f}, st[3] = {0.0f, 0.0f, 0.0f};
  unsigned long long ns = 0;
  unsigned int nl = 0, k = 1, last = 0;  // samples k..last remain
  if (pixel) {
    // xReg's per-ray float set-up and drr_kernel's support-box bounds
    const float maxb[3] = {(float)(vol.nx - 1), (float)(vol.ny - 1), (float)(vol.nz - 1)};
    float st0[3], quot;
    bool hit = xf::ray_setup(p.geo[proj], (float)col, (float)row, maxb, p.step, st0, st, quot);
    unsigned long long nsteps = hit ? __float2uint_rz(quot) : 0ull;
    if (hit && !(nsteps <= p.max_steps)) {
      atomicAdd(p.err_counter, 1u);
      nsteps = 0;
      hit = false;
    }
    if (hit) {
      unsigned int first = 0, lst = (unsigned int)nsteps;
      if (vol.has_support) {
        float lo = 0.0f, hi = (float)nsteps;
        if (vol.sup_lo[0] > vol.sup_hi[0]) hi = -1.0f;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          if (fabsf(st[a]) > 1.0e-20f) {
            const float inv = 1.0f / st[a];
            float u = (vol.sup_lo[a] - st0[a]) * inv, w = (vol.sup_hi[a] - st0[a]) * inv;
            if (u > w) { const float t = u; u = w; w = t; }
            lo = fmaxf(lo, u);
            hi = fminf(hi, w);
          } else if (!(st0[a] > vol.sup_lo[a] && st0[a] < vol.sup_hi[a])) {
            hi = -1.0f;
          }
        }
        if (!(lo <= hi)) {
          lst = 0;
          first = 1;
        } else {
          const float f0 = floorf(lo) - 1.0f, f1 = ceilf(hi) + 1.0f;
          first = f0 > 0.0f ? (unsigned int)f0 : 0u;
          lst = f1 < (float)nsteps ? (unsigned int)f1 : (unsigned int)nsteps;
        }
      }
      pos[0] = st0[0]; pos[1] = st0[1]; pos[2] = st0[2];
      for (unsigned int i = 0, skip = first <= lst ? first : lst + 1u; i < skip; ++i) {
        pos[0] = __fadd_rn(pos[0], st[0]);
        pos[1] = __fadd_rn(pos[1], st[1]);
        pos[2] = __fadd_rn(pos[2], st[2]);
      }
      k = first;
      last = lst;
      nl = first <= lst ? lst - first + 1u : 0u;
      ns = nsteps + 1;
    }
  }
  __syncthreads();
  // the block's axis and direction: claimed by the first ray that has samples
  int code = -1;
  if (k <= last) {
    int a = 0;
    float m = fabsf(st[0]);
    if (fabsf(st[1]) > m) { a = 1; m = fabsf(st[1]); }
    if (fabsf(st[2]) > m) { a = 2; m = fabsf(st[2]); }
    code = m > 0.0f ? 2 * a + (st[a] > 0.0f ? 1 : 0) : -1;
    if (code >= 0) atomicCAS(&s_code, -1, code);
  }
  __syncthreads();
  const int bcode = s_code, ax = bcode >> 1, dir = (bcode & 1) ? 1 : -1;
  const bool staged = k <= last && bcode >= 0 && code == bcode;
  if (k <= last && !staged) sum = brick_march_global<BLEND>(vol, pos, st, k, last, sum);  // another axis: global reads
  if (staged) {  // the cells of this ray's first and (about) last samples along the axis
    int c0[3], c1[3];
    float f[3];
    cell3<BLEND>(vol, pos, c0, f);
    const float e = (float)(last - k);
    const float pe[3] = {pos[0] + e * st[0], pos[1] + e * st[1], pos[2] + e * st[2]};
    cell3<BLEND>(vol, pe, c1, f);
    atomicMin(&s_amin, min(c0[ax], c1[ax]) - 1);
    atomicMax(&s_amax, max(c0[ax], c1[ax]) + 1);
  }
  __syncthreads();
  if (bcode >= 0) {
    const int amin = max(s_amin, 0), amax = min(s_amax, ncell[ax] - 1);
    int z = dir > 0 ? amin : amax;  // first cell of the slab along the axis
    for (int guard = 0; guard < 8192 && (dir > 0 ? z <= amax : z >= amin); ++guard) {
      if (tid < 3) {
        s_lo[tid] = 0x7fffffff;
        s_hi[tid] = -1;
      }
      __syncthreads();
      const int zfar = (dir > 0 ? z + kBrickDepth : z - kBrickDepth) - 1;  // index of the first cell past a full slab
      if (staged && k <= last) {
        int ce[3], cx[3];
        float f[3];
        cell3<BLEND>(vol, pos, ce, f);
        float m = ((float)zfar - pos[ax]) / st[ax];  // samples to the slab's far side, about
        m = fminf(fmaxf(m, 0.0f), (float)(last - k));
        const float pe[3] = {pos[0] + m * st[0], pos[1] + m * st[1], pos[2] + m * st[2]};
        cell3<BLEND>(vol, pe, cx, f);
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          if (a == ax) continue;
          atomicMin(&s_lo[a], min(ce[a], cx[a]) - 1);
          atomicMax(&s_hi[a], max(ce[a], cx[a]) + 1);
        }
      }
      __syncthreads();
      int lo[3], hi[3], lat = 1;
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        if (a == ax) continue;
        lo[a] = max(s_lo[a], 0);
        hi[a] = min(s_hi[a], ncell[a] - 1);
        lat *= hi[a] >= lo[a] ? hi[a] - lo[a] + 1 : 0;
      }
      // slab depth: the full one, thinner when the box would not fit
      int d = kBrickDepth;
      bool use = lat > 0;
      if (use && lat * d > kBrickCells) {
        d = kBrickCells / lat;
        if (d < 1) {
          d = kBrickDepth;
          use = false;  // too wide a box: this slab reads global memory
        }
      }
      lo[ax] = dir > 0 ? z : max(z - d + 1, 0);
      hi[ax] = dir > 0 ? min(z + d - 1, ncell[ax] - 1) : z;
      const int W = hi[0] - lo[0] + 1, H = hi[1] - lo[1] + 1, Dz = hi[2] - lo[2] + 1;
      if (use) {
        const int total = W * H * Dz;
        for (int i = tid; i < total; i += kThreads) {
          const int zz = lo[2] + i % Dz, x = lo[0] + (i / Dz) % W, y = lo[1] + i / (Dz * W);  // as cells lie
          const int64_t c = (int64_t)x * vol.cs[0] + (int64_t)y * vol.cs[1] + zz;
          s_cells[2 * i] = __ldg(cells + 2 * c);
          s_cells[2 * i + 1] = __ldg(cells + 2 * c + 1);
        }
      }
      __syncthreads();
      const int zend = dir > 0 ? z + d : z - d;  // first cell past this slab
      if (staged) {
        for (; k <= last; ++k) {
          int c[3];
          float f[3], v[8];
          cell3<BLEND>(vol, pos, c, f);
          if (dir > 0 ? c[ax] >= zend : c[ax] <= zend) break;
          const bool in = use && c[0] >= lo[0] && c[0] <= hi[0] && c[1] >= lo[1] && c[1] <= hi[1] && c[2] >= lo[2] &&
                          c[2] <= hi[2];
          if (in) {
            const int i = (c[2] - lo[2]) + Dz * ((c[0] - lo[0]) + W * (c[1] - lo[1]));
            const float4 q0 = s_cells[2 * i], q1 = s_cells[2 * i + 1];
            v[0] = q0.x; v[1] = q0.y; v[2] = q0.z; v[3] = q0.w;
            v[4] = q1.x; v[5] = q1.y; v[6] = q1.z; v[7] = q1.w;
          } else {
            Vox<XR_VOXEL_F32>::cell_wide(vol.cells, (unsigned int)c[0] * vol.cs[0] + (unsigned int)c[1] * vol.cs[1] + (unsigned int)c[2], v);
          }
          sum = __fadd_rn(sum, brick_value<BLEND>(v, f));
          pos[0] = __fadd_rn(pos[0], st[0]);
          pos[1] = __fadd_rn(pos[1], st[1]);
          pos[2] = __fadd_rn(pos[2], st[2]);
        }
      }
      __syncthreads();  // the copy is read by every ray before the next slab overwrites it
      z = zend;
    }
  }
  if (k <= last) sum = brick_march_global<BLEND>(vol, pos, st, k, last, sum);  // past the estimated range
  if (pixel) {
    sum = __fmul_rn(sum, p.step);
    const float aa = __fadd_rn(0.0f, sum);
    const int64_t npix = (int64_t)p.rows * p.cols;
    const int64_t pix = (int64_t)row * p.cols + col;
    const int64_t oidx = proj * npix + pix;
    float prev;
    if (p.bg_projs) prev = p.bg_projs[(int64_t)p.cam_idx[proj] * npix + pix];
    else if (p.store == XR_PROJ_STORE_REPLACE) prev = p.default_bg;
    else prev = p.out[oidx];
    p.out[oidx] = __fadd_rn(prev, aa);
  }
  if (p.sample_counter) {
    const int lane = tid & 31;
    unsigned long long nlw = nl;
    for (int o = 16; o > 0; o >>= 1) {
      ns += __shfl_down_sync(0xffffffffu, ns, o);
      nlw += __shfl_down_sync(0xffffffffu, nlw, o);
    }
    if (lane == 0 && ns) atomicAdd(p.sample_counter, ns);
    if (lane == 0 && nlw && p.loaded_counter) atomicAdd(p.loaded_counter, nlw);
  }
}

// Fused evaluation: a persistent multi-job DRR loop (every block takes the
// next (job, tile, projection) item from a global counter; projections are
// the fastest index within a job), with each job's grad-NCC (5x5 smoothing) computed inside the same launch.
// No block ever waits for another.  After a block writes a DRR tile it
// counts the tile towards every 64x52 metric tile whose input (the tile with
// its 3-pixel blur + Sobel halo, clipped to the image) the tile overlaps; the
// block whose count completes a metric tile computes that tile's moments at
// once, reading the DRR pixels back through L2 (gt::grad_tile_moments, the
// split path's own tile code); the block that completes an image's metric
// tiles combines its partials in FP64 (gt::grad_finalize_image), and the block
// that completes a pose's views writes the mean over views.  Counters are
// zero between launches: whoever completes one resets it.  Stores are made
// visible device-wide (fence) before each count; counted data is read through
// L2 (ld.global.cg), never through the incoherent L1.
constexpr int kFusedKR = 2;  // 5x5 smoothing, xReg's default

// Metric tiles the DRR tile [r0, r1) x [c0, c1) feeds, and how many DRR tiles
// (tw x th pixels) feed each; claims (into claim[]) those whose count this
// tile completes.
__device__ __forceinline__ int fused_count_tile(const FusedJob& J, unsigned int* cnt_tile, int r0, int r1, int c0,
                                                int c1, int tw, int th, int* claim) {
  constexpr int H = kFusedKR + 1;
  const int rows = J.d.p.rows, cols = J.d.p.cols;
  int n = 0;
  const int my0 = max(0, (r0 - H) / gt::kGH - 1), my1 = min(J.mt_y - 1, (r1 - 1 + H) / gt::kGH);
  const int mx0 = max(0, (c0 - H) / gt::kGW - 1), mx1 = min(J.mt_x - 1, (c1 - 1 + H) / gt::kGW);
  for (int my = my0; my <= my1; ++my) {
    const int er0 = max(0, my * gt::kGH - H), er1 = min(rows, my * gt::kGH + gt::kGH + H);
    if (!(er0 < r1 && r0 < er1)) continue;
    for (int mx = mx0; mx <= mx1; ++mx) {
      const int ec0 = max(0, mx * gt::kGW - H), ec1 = min(cols, mx * gt::kGW + gt::kGW + H);
      if (!(ec0 < c1 && c0 < ec1)) continue;
      const unsigned int target = (unsigned int)(((er1 - 1) / th - er0 / th + 1) * ((ec1 - 1) / tw - ec0 / tw + 1));
      unsigned int* c = cnt_tile + my * J.mt_x + mx;
      if (atomicAdd(c, 1u) + 1u == target) {
        *c = 0u;  // completed: zero for the next launch
        claim[n++] = my * J.mt_x + mx;
      }
    }
  }
  return n;
}

// The metric stage of a claimed tile, out of line: its registers do not
// constrain the DRR loop's (it runs a few times per image, the loop for every
// sample).  Returns, in thread 0, whether the image is complete.
__device__ __noinline__ bool fused_metric_tile(const FusedJob& J, int64_t proj, int M, gt::FF* red) {
  const DrrParams& P = J.d.p;
  const int rows = P.rows, cols = P.cols, mt = J.mt_x * J.mt_y;
  const int64_t nimg = (int64_t)J.nviews * J.pop;
  const int64_t v = proj / J.pop, k = proj - v * J.pop;
  const FusedView& V = J.views[v];
  const double val = gt::grad_tile_moments<2, true>(P.out + proj * (int64_t)rows * cols, rows, cols,
                                                    (M / J.mt_x) * gt::kGH, (M % J.mt_x) * gt::kGW, V.fhx, V.fhy, V.mask,
                                                    red);
  bool last = false;
  if (threadIdx.x < 6) {
    V.partials[(k * mt + M) * 6 + threadIdx.x] = val;
    __threadfence();
    __syncwarp(0x3f);
  }
  if (threadIdx.x == 0) {
    unsigned int* ci = J.cnt + nimg * mt + proj;
    last = atomicAdd(ci, 1u) + 1u == (unsigned int)mt;
    if (last) *ci = 0u;
  }
  return last;
}

// Every metric tile of image proj is in: its FP64 combine, then (by the block
// that completes the pose's views) the mean over views.
__device__ __noinline__ void fused_metric_image(const FusedJob& J, int64_t proj, double* red) {
  const int mt = J.mt_x * J.mt_y;
  const int64_t nimg = (int64_t)J.nviews * J.pop;
  const int64_t v = proj / J.pop, k = proj - v * J.pop;
  const FusedView& V = J.views[v];
  __threadfence();
  const float sim = gt::grad_finalize_image<true>(V.partials + k * mt * 6, mt, V.n_used, V.fx, V.fy, red);
  if (threadIdx.x == 0) {
    V.sims[k] = sim;
    __threadfence();
    unsigned int* cp = J.cnt + nimg * mt + nimg + k;
    if (atomicAdd(cp, 1u) + 1u == (unsigned int)J.nviews) {  // every view of this pose
      *cp = 0u;
      __threadfence();
      float sum = 0.0f;
      for (int w = 0; w < J.nviews; ++w) sum += __ldcg(J.views[w].sims + k);
      J.out[k] = sum / (float)J.nviews;  // ImgSimMetric2DCombineMean (as gt::combine_mean)
    }
  }
}

// Resident blocks per SM: 48 registers, but for BF16, whose reload form spills in this
// kernel at 48 (3 views of 250 x 240 under 57 poses 4158 us, at 64 registers 2804).
constexpr int fused_blocks(int vt) { return vt == XR_VOXEL_BF16 ? kMinBlocksPerSM - 1 : kMinBlocksPerSM; }

template <int VT, int LAYOUT, Blend BLEND>
__global__ void __launch_bounds__(kThreads, fused_blocks(VT))
eval_fused_kernel(const FusedJob* __restrict__ jobs, int njobs, long long total, unsigned long long* counter) {
  // under 1 KB of shared memory: the SM's unified L1 stays with the DRR gathers
  __shared__ long long s_item;
  __shared__ gt::FF s_red[6 * 4];
  __shared__ double s_dred[6 * (gt::kFinalizeThreads / 32)];
  __shared__ int s_claim[16];
  __shared__ int s_nclaim, s_last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (;;) {
    if (threadIdx.x == 0) s_item = (long long)atomicAdd(counter, 1ull);
    __syncthreads();
    const long long item = s_item;
    __syncthreads();
    if (item >= total) break;
    int j = 0;
    while (j + 1 < njobs && jobs[j + 1].d.item_begin <= item) ++j;
    const FusedJob& J = jobs[j];
    const DrrParams& P = J.d.p;
    const long long local = item - J.d.item_begin;
    const int64_t proj = (int64_t)(local % P.num_projs);
    const int tile = (int)(local / P.num_projs);
    const int ty = tile / J.d.tiles_x, tx = tile - ty * J.d.tiles_x;
    // the job's block shape (as drr_kernel): bw warps across, each warp 8x4
    // pixels (or 4x8 when tall)
    const int bw = P.block_warps_x, wl = P.warp_tall ? 2 : 3;
    const int wc = 1 << wl, wr = 32 >> wl, tw = wc * bw, th = (8 / bw) * wr;
    int lc, lr;
    lane_pixel(lane, wl, lc, lr);
    const int col = tx * tw + (warp % bw) * wc + lc;
    const int row = ty * th + (warp / bw) * wr + lr;
    unsigned int nl;
    if (col < P.cols && row < P.rows) trace_pixel<VT, XR_LINE_INT_SUM, LAYOUT, false, BLEND>(P, proj, row, col, &nl);
    if (!J.metric) continue;
    __threadfence();  // this block's DRR pixels, visible device-wide before they are counted
    __syncthreads();
    const int mt = J.mt_x * J.mt_y;
    if (threadIdx.x == 0)
      s_nclaim = fused_count_tile(J, J.cnt + proj * mt, ty * th, min(ty * th + th, P.rows), tx * tw,
                                  min(tx * tw + tw, P.cols), tw, th, s_claim);
    __syncthreads();
    const int nclaim = s_nclaim;
    for (int c = 0; c < nclaim; ++c) {
      __threadfence();
      const bool last = fused_metric_tile(J, proj, s_claim[c], s_red);
      if (threadIdx.x == 0) s_last = last;
      __syncthreads();
      if (s_last) fused_metric_image(J, proj, s_dred);  // every tile of this image is in
      __syncthreads();
    }
  }
}

// One launch over several jobs without a work counter: blockIdx.x numbers
// every job's (tile, projection) items in the multi-job kernel's order and
// the hardware block scheduler hands them out; each block is one tile in its
// job's block shape, as drr_kernel.  64 registers (4 blocks per SM): the job's
// parameters come from global memory instead of the constant bank; measured
// 3.4% faster than 48 on an uneven set of 8 jobs.
// GROUPED: every job's items are pose groups (MultiJobDrr::pose_group); a
// separate instantiation, so the per-projection kernels keep their registers.
constexpr int jobs_threads(bool grouped) { return grouped ? kThreads : 32 * kWarps; }
template <int VT, int LAYOUT, bool GROUPED, Blend BLEND>
__global__ void __launch_bounds__(jobs_threads(GROUPED), (kMinBlocksPerSM - 1) * kThreads / jobs_threads(GROUPED))
drr_jobs_kernel(const MultiJobDrr* __restrict__ jobs, int njobs, long long item0) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long item = item0 + blockIdx.x;
  int lo = 0, hi = njobs - 1;  // last job whose items start at or before this one
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (jobs[mid].item_begin <= item) lo = mid; else hi = mid - 1;
  }
  const MultiJobDrr& J = jobs[lo];
  const long long local = item - J.item_begin;
  const long long nproj = J.p.num_projs;
  int64_t proj;
  int col, row;
  if constexpr (GROUPED) {
    // 4 consecutive projections x an 8x8-pixel tile.  When the 4 share a camera
    // and the tile's central ray meets the volume at nearly the same cells under
    // all 4 poses (late CMA-ES generations), their rays through a pixel nearly
    // coincide: each warp takes a 2x4-pixel sub-tile under all 4 poses, so its
    // lanes share cells; otherwise each pair of warps takes one projection's
    // tile.  The rays and their values are the same either way.
    const long long ngrp = (nproj + 3) / 4;
    const int64_t p0 = (int64_t)(local % ngrp) * 4;
    const int tile = (int)(local / ngrp);
    const int ty = tile / J.tiles_x, tx = tile - ty * J.tiles_x;
    bool coherent = p0 + 3 < nproj;
    if (coherent) {
      // where the tile's central ray of the first pose enters and leaves the
      // volume, in that pose's camera coordinates; the other poses' camera ->
      // index affines must put those points within a voxel of it (the
      // deviation is affine, so the segment's ends bound it along the ray)
      const ProjGeom& g0 = J.p.geo[p0];
      const float maxb[3] = {(float)(J.p.vol.nx - 1), (float)(J.p.vol.ny - 1), (float)(J.p.vol.nz - 1)};
      float st0[3], stv[3], quot;
      const int cc = min(tx * 8 + 4, J.p.cols - 1), rc = min(ty * 8 + 4, J.p.rows - 1);
      coherent = xf::ray_setup(g0, (float)cc, (float)rc, maxb, J.p.step, st0, stv, quot) && quot < 1.0e6f;
      if (coherent) {
        xf::Affine M0, Mi;
        for (int k = 0; k < 9; ++k) M0.L[k] = g0.M[k];
        for (int k = 0; k < 3; ++k) M0.t[k] = g0.M[9 + k];
        xf::inverse(M0, Mi);
        float ends[2][3], cam[2][3];
        for (int k = 0; k < 3; ++k) {
          ends[0][k] = st0[k];
          ends[1][k] = st0[k] + quot * stv[k];
        }
        xf::apply(Mi, ends[0], cam[0]);
        xf::apply(Mi, ends[1], cam[1]);
        float dev = 0.0f;
        for (int q = 1; q < 4; ++q) {
          const ProjGeom& g = J.p.geo[p0 + q];
          coherent = coherent && J.p.cam_idx[p0 + q] == J.p.cam_idx[p0];
          for (int e = 0; e < 2; ++e)
            for (int i = 0; i < 3; ++i) {
              const float v = g.M[3 * i] * cam[e][0] + g.M[3 * i + 1] * cam[e][1] + g.M[3 * i + 2] * cam[e][2] +
                              g.M[9 + i];
              dev = fmaxf(dev, fabsf(v - ends[e][i]));
            }
        }
        coherent = coherent && dev < 1.0f;
      }
    }
    int q;
    if (coherent) {
      q = lane >> 3;
      col = tx * 8 + (warp & 3) * 2 + (lane & 1);
      row = ty * 8 + (warp >> 2) * 4 + ((lane & 7) >> 1);
    } else {
      q = warp >> 1;
      int lc, lr;
      lane_pixel(lane, 3, lc, lr);
      col = tx * 8 + lc;
      row = ty * 8 + (warp & 1) * 4 + lr;
    }
    proj = p0 + q;
    if (proj >= nproj) return;
  } else {
    proj = (int64_t)(local % nproj);
    const int tile = (int)(local / nproj);
    const int ty = tile / J.tiles_x, tx = tile - ty * J.tiles_x;
    const int bw = J.p.block_warps_x, wl = J.p.warp_tall ? 2 : 3;
    const int wc = 1 << wl, wr = 32 >> wl;
    int lc, lr;
    lane_pixel(lane, wl, lc, lr);
    col = tx * (wc * bw) + (warp % bw) * wc + lc;
    row = ty * ((kWarps / bw) * wr) + (warp / bw) * wr + lr;
  }
  if (col >= J.p.cols || row >= J.p.rows) return;
  unsigned int nl;
  trace_pixel<VT, XR_LINE_INT_SUM, LAYOUT, false, BLEND>(J.p, proj, row, col, &nl);
}

constexpr int kMaxDevices = 64;

template <int VT, int LAYOUT, Blend BLEND>
cudaError_t launch_fused_t(const FusedJob* d_jobs, int njobs, long long total, unsigned long long* d_counter,
                           int* blocks_out, cudaStream_t s) {
  static std::atomic<int> cached[kMaxDevices];  // blocks per device; zero = not known yet
  int dev = 0, sms = 0, per_sm = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
  int blocks = cached[dev].load(std::memory_order_relaxed);
  if (!blocks) {
    // the kernel's shared memory is small: the smallest carve-out that holds
    // every resident block leaves the rest of the SM's unified L1 to the gathers
    cudaFuncAttributes fa{};
    int smem_sm = 0;
    cudaError_t e = cudaFuncGetAttributes(&fa, eval_fused_kernel<VT, LAYOUT, BLEND>);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
    if (e != cudaSuccess) return e;
    const double need = (double)(fa.sharedSizeBytes + 1024) * fused_blocks(VT);
    const int pct = std::min(100, (int)std::ceil(100.0 * need / (double)std::max(smem_sm, 1)) + 1);
    e = cudaFuncSetAttribute(eval_fused_kernel<VT, LAYOUT, BLEND>, cudaFuncAttributePreferredSharedMemoryCarveout, pct);
    if (e != cudaSuccess) return e;
    e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, eval_fused_kernel<VT, LAYOUT, BLEND>, kThreads, 0);
    if (e != cudaSuccess) return e;
    blocks = sms * (per_sm > 0 ? per_sm : 1);
    cached[dev].store(blocks, std::memory_order_relaxed);
  }
  *blocks_out = blocks;
  cudaError_t e = cudaMemsetAsync(d_counter, 0, sizeof(unsigned long long), s);
  if (e != cudaSuccess) return e;
  eval_fused_kernel<VT, LAYOUT, BLEND><<<blocks, kThreads, 0, s>>>(d_jobs, njobs, total, d_counter);
  return cudaGetLastError();
}

template <int VT, int LAYOUT, bool GROUPED, Blend BLEND>
cudaError_t launch_jobs_g(const MultiJobDrr* d_jobs, int njobs, long long total, cudaStream_t s) {
  static std::atomic<bool> carveout_set[kMaxDevices];
  int dev = 0;
  if (cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < kMaxDevices &&
      !carveout_set[dev].load(std::memory_order_relaxed)) {
    cudaFuncSetAttribute(drr_jobs_kernel<VT, LAYOUT, GROUPED, BLEND>, cudaFuncAttributePreferredSharedMemoryCarveout,
                         (int)cudaSharedmemCarveoutMaxL1);
    carveout_set[dev].store(true, std::memory_order_relaxed);
  }
  const long long max_x = 0x7fffffff;
  for (long long base = 0; base < total; base += max_x) {
    const long long n = (total - base) < max_x ? (total - base) : max_x;
    drr_jobs_kernel<VT, LAYOUT, GROUPED, BLEND><<<(unsigned)n, jobs_threads(GROUPED), 0, s>>>(d_jobs, njobs, base);
  }
  return cudaGetLastError();
}

template <int VT, int LAYOUT, Blend BLEND>
cudaError_t launch_jobs_t(const MultiJobDrr* d_jobs, int njobs, long long total, bool grouped, cudaStream_t s) {
  return grouped ? launch_jobs_g<VT, LAYOUT, true, BLEND>(d_jobs, njobs, total, s)
                 : launch_jobs_g<VT, LAYOUT, false, BLEND>(d_jobs, njobs, total, s);
}

template <int VT, int KERNEL, int LAYOUT, bool DEEP, Blend BLEND>
cudaError_t launch_depth(const DrrParams& p, cudaStream_t s) {
  // The kernel uses no shared memory: ask for the largest L1 (the gathers hit
  // it), once per device (a preference; setting it twice is harmless).
  static std::atomic<bool> carveout_set[kMaxDevices];
  int dev = 0;
  if (cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < kMaxDevices &&
      !carveout_set[dev].load(std::memory_order_relaxed)) {
    cudaFuncSetAttribute(drr_kernel<VT, KERNEL, LAYOUT, DEEP, BLEND>, cudaFuncAttributePreferredSharedMemoryCarveout,
                         (int)cudaSharedmemCarveoutMaxL1);
    carveout_set[dev].store(true, std::memory_order_relaxed);
  }
  const int bw = p.block_warps_x;
  const int wc = p.warp_tall ? 4 : 8;
  const int tx = wc * bw, ty = p.block_warps_y * (32 / wc);
  const int64_t max_x = 0x7fffffff;
  for (int64_t base = 0; base < p.num_projs; base += max_x) {
    const int64_t n = (p.num_projs - base) < max_x ? (p.num_projs - base) : max_x;
    const dim3 grid((unsigned)n, (p.cols + tx - 1) / tx, (p.rows + ty - 1) / ty);
    drr_kernel<VT, KERNEL, LAYOUT, DEEP, BLEND><<<grid, 32 * bw * p.block_warps_y, 0, s>>>(p, base);
  }
  return cudaGetLastError();
}

// A launch of few rays is bound by the latency of a ray's loads one after another
// (a quarter of the warps the SMs hold, data that no earlier pose brought into L2),
// so it takes eight cells in flight per thread at 128 registers where a large one
// takes four at 48.  Up to twice the rays that are resident at 128 registers;
// measured, four against eight, in us with the geometry launch: 256^3 float32, one
// pose of 256^2 116 / 64, 330^2 114 / 87, 384^2 113 / 94; 320 x 320 x 256 FP16,
// three views of 192^2 127 / 98; BF16, two views of 240^2 84 / 83, of 300 x 260
// (156,000 rays) 97 / 98; FP16, two views of 384^2 (294,912 rays) 148 / 150.
template <int VT, int KERNEL, int LAYOUT>
cudaError_t launch_t(const DrrParams& p, cudaStream_t s) {
  if constexpr (LAYOUT == XR_LAYOUT_LINEAR) {
    return launch_depth<VT, KERNEL, LAYOUT, false, Blend::kVolume>(p, s);
  } else {
    // Volumes with an infinity have a march of their own, four by weights (20 images
    // of 256^2 of a 256 x 256 x 200 float32 volume: 616 us through the clamped sampler).
    if constexpr (VT != XR_VOXEL_F16)
      if (p.vol.weighted) return launch_depth<VT, KERNEL, LAYOUT, false, Blend::kWeights>(p, s);
    static std::atomic<int> cached[kMaxDevices];  // SMs per device; zero = not known yet
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < kMaxDevices) {
      sms = cached[dev].load(std::memory_order_relaxed);
      if (!sms && cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess)
        cached[dev].store(sms, std::memory_order_relaxed);
    }
    if (p.num_projs * p.rows * p.cols <= 2 * (int64_t)sms * kDeepBlocksPerSM * 32 * kWarps)
      return launch_depth<VT, KERNEL, LAYOUT, true, Blend::kDifferences>(p, s);
    return launch_depth<VT, KERNEL, LAYOUT, false, Blend::kDifferences>(p, s);
  }
}

template <int VT, int KERNEL>
cudaError_t launch_layout(const DrrParams& p, cudaStream_t s) {
  if (p.vol.layout == kLayoutCell8Wide) {
    if constexpr (VT == XR_VOXEL_F32) return launch_t<VT, KERNEL, kLayoutCell8Wide>(p, s);
    return cudaErrorInvalidValue;
  }
  if (p.vol.layout == XR_LAYOUT_CELL8) return launch_t<VT, KERNEL, XR_LAYOUT_CELL8>(p, s);
  return launch_t<VT, KERNEL, XR_LAYOUT_LINEAR>(p, s);
}

template <int VT>
cudaError_t launch_kernel_id(const DrrParams& p, cudaStream_t s) {
  return p.kernel_id == XR_LINE_INT_MAX ? launch_layout<VT, XR_LINE_INT_MAX>(p, s)
                                        : launch_layout<VT, XR_LINE_INT_SUM>(p, s);
}

}  // namespace

template <Blend BLEND>
cudaError_t launch_brick_t(const DrrParams& p, cudaStream_t s) {
  static std::atomic<bool> carveout_set[kMaxDevices];
  int dev = 0;
  if (cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < kMaxDevices &&
      !carveout_set[dev].load(std::memory_order_relaxed)) {
    // four resident blocks of 44 KB each, the rest of the SM's unified L1 for the global reads
    cudaFuncSetAttribute(drr_brick_kernel<BLEND>, cudaFuncAttributePreferredSharedMemoryCarveout, 80);
    carveout_set[dev].store(true, std::memory_order_relaxed);
  }
  const int64_t max_x = 0x7fffffff;
  for (int64_t base = 0; base < p.num_projs; base += max_x) {
    const int64_t n = (p.num_projs - base) < max_x ? (p.num_projs - base) : max_x;
    const dim3 grid((unsigned)n, (p.cols + 15) / 16, (p.rows + 15) / 16);
    drr_brick_kernel<BLEND><<<grid, kThreads, 0, s>>>(p, base);
  }
  return cudaGetLastError();
}

cudaError_t launch_brick(const DrrParams& p, cudaStream_t s) {
  if (p.vol.voxel_type != XR_VOXEL_F32 || !p.vol.cells || p.kernel_id != XR_LINE_INT_SUM) return cudaErrorInvalidValue;
  return p.vol.weighted ? launch_brick_t<Blend::kWeights>(p, s) : launch_brick_t<Blend::kDifferences>(p, s);
}

cudaError_t launch_drr(const DrrParams& params, cudaStream_t s) {
  DrrParams p = params;
  if (p.num_projs <= 0) return cudaSuccess;
  if (p.vol.layout == kLayoutBrick) return launch_brick(p, s);
  if (!(p.block_warps_x == 1 || p.block_warps_x == 2 || p.block_warps_x == 4 || p.block_warps_x == 8))
    return cudaErrorInvalidValue;
  p.block_warps_y = std::max(kWarps / p.block_warps_x, 1);
  if (p.warp_tall != 0 && p.warp_tall != 1) return cudaErrorInvalidValue;
  if (p.vol.layout != XR_LAYOUT_LINEAR && !p.vol.cells) return cudaErrorInvalidValue;
  if (p.vol.layout == kLayoutCell8Wide && p.vol.voxel_type != XR_VOXEL_F32) return cudaErrorInvalidValue;
  switch (p.vol.voxel_type) {
    case XR_VOXEL_F32: return launch_kernel_id<XR_VOXEL_F32>(p, s);
    case XR_VOXEL_F16: return launch_kernel_id<XR_VOXEL_F16>(p, s);
    case XR_VOXEL_BF16: return launch_kernel_id<XR_VOXEL_BF16>(p, s);
    default: return cudaErrorInvalidValue;
  }
}

// CALL(voxel type, layout, blend) for the jobs' voxel type and layout: the cell layouts
// by their blend, LINEAR by each volume's own.
#define XR_BY_VOLUME(CALL)                                                                                        \
  switch (voxel_type * 4 + layout) {                                                                              \
    case XR_VOXEL_F32 * 4 + XR_LAYOUT_LINEAR: return CALL(XR_VOXEL_F32, XR_LAYOUT_LINEAR, Blend::kVolume);        \
    case XR_VOXEL_F32 * 4 + kLayoutCell8Wide:                                                                     \
      return weighted ? CALL(XR_VOXEL_F32, kLayoutCell8Wide, Blend::kWeights)                                     \
                      : CALL(XR_VOXEL_F32, kLayoutCell8Wide, Blend::kDifferences);                                \
    case XR_VOXEL_F16 * 4 + XR_LAYOUT_LINEAR: return CALL(XR_VOXEL_F16, XR_LAYOUT_LINEAR, Blend::kVolume);        \
    case XR_VOXEL_F16 * 4 + XR_LAYOUT_CELL8: return CALL(XR_VOXEL_F16, XR_LAYOUT_CELL8, Blend::kDifferences);     \
    case XR_VOXEL_BF16 * 4 + XR_LAYOUT_LINEAR: return CALL(XR_VOXEL_BF16, XR_LAYOUT_LINEAR, Blend::kVolume);      \
    case XR_VOXEL_BF16 * 4 + XR_LAYOUT_CELL8:                                                                     \
      return weighted ? CALL(XR_VOXEL_BF16, XR_LAYOUT_CELL8, Blend::kWeights)                                     \
                      : CALL(XR_VOXEL_BF16, XR_LAYOUT_CELL8, Blend::kDifferences);                                \
    default: return cudaErrorInvalidValue;                                                                        \
  }

cudaError_t launch_eval_fused(const FusedJob* d_jobs, int njobs, long long total, int32_t voxel_type, int32_t layout,
                              bool weighted, unsigned long long* d_counter, int* blocks_out, cudaStream_t s) {
  *blocks_out = 0;
  if (total <= 0) return cudaSuccess;
#define XR_FUSED(V, L, B) launch_fused_t<V, L, B>(d_jobs, njobs, total, d_counter, blocks_out, s)
  XR_BY_VOLUME(XR_FUSED)
#undef XR_FUSED
}

cudaError_t launch_drr_jobs(const MultiJobDrr* d_jobs, int njobs, long long total, int32_t voxel_type, int32_t layout,
                            bool weighted, bool grouped, cudaStream_t s) {
  if (total <= 0) return cudaSuccess;
#define XR_JOBS(V, L, B) launch_jobs_t<V, L, B>(d_jobs, njobs, total, grouped, s)
  XR_BY_VOLUME(XR_JOBS)
#undef XR_JOBS
}
#undef XR_BY_VOLUME

}  // namespace xr

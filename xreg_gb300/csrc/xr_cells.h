// xr_cells.h -- numbering of the cell copy of a volume (CELL8 layout, see
// xr_raycast.cu) and the constants of the sample loop's round-down floor.  Host
// code: the kernels get its results in VolView.
#pragma once

#include <cstddef>
#include <cstdint>

#include "xreg_gb300.h"

namespace xr {

constexpr float kH16 = 32768.0f;  // scale of the FP16 x and y positions and weights

// The x and y strides of the cell copy, cells.  Long ones are padded to 2 modulo 8:
// the L1 serves a cell load in passes of 4 lanes (32-byte cells) or 8 lanes (16-byte
// cells), one wavefront per pass unless two of its cells share a bank group, i.e. a
// cell number modulo 4 or 8; with these strides the cells of a pass's 2 x 2 or 4 x 2
// pixel block (lane_pixel) mostly differ there.  Measured against unpadded strides,
// and 4 x 1 and 4 x 2 blocks, on the launches of march_cells: float32 5409 -> 5130 us
// (9.8 -> 8.9 wavefronts per load, 8 is the least), FP16 2994 -> 2871 (12.4 -> 11.5),
// BF16 unchanged.  Short ones are not: on a stack of 4 slices the padding would
// double the copy.
inline void cell_strides_wide(int64_t nx, int64_t nz, int64_t cs[2]) {
  auto pad = [](int64_t n) { return n < 56 ? n : n + ((2 - n) & 7); };  // at most an eighth more
  cs[0] = pad(nz + 1);
  cs[1] = pad(cs[0] * (nx + 1));
}

// Whether a volume has a cell copy: the kernels number cells in 32 bits.  Only
// volumes of 2^31 voxels with two very short axes have more cells, and are read as
// they lie.
inline bool cells_numbered(int64_t nx, int64_t ny, int64_t nz) {
  int64_t cs[2];
  cell_strides_wide(nx, nz, cs);
  return cs[1] <= 0x7fffffff && cs[1] * (ny + 1) < (int64_t(1) << 32);
}

// VolView::cs (zeros where cells are not numbered).
inline void cell_strides(int64_t nx, int64_t ny, int64_t nz, int32_t cs[2]) {
  int64_t w[2];
  cell_strides_wide(nx, nz, w);
  const bool ok = cells_numbered(nx, ny, nz);
  cs[0] = ok ? (int32_t)w[0] : 0;
  cs[1] = ok ? (int32_t)w[1] : 0;
}

// Bytes of the cell copy (cells numbered z fastest, then x, then y).
inline size_t cell_layout_bytes(int64_t nx, int64_t ny, int64_t nz, int32_t voxel_type) {
  int32_t cs[2];
  cell_strides(nx, ny, nz, cs);
  const size_t ncell = (size_t)cs[1] * (size_t)(ny + 1);
  return ncell * (voxel_type == XR_VOXEL_F32 ? 32 : 16);
}

// VolView::kfl and cell_bytes; zeros in kfl where there are none.  Whole numbers
// 1 <= m <= 2^22 that turn bias + m + floor(p) per axis into the cell (floor(p) + 1
// per axis, in strides of cs[0] u, cs[1] u and u bytes or, with u 1, cells) modulo
// 2^32: the sum of the biases, negated, in the mixed base of the strides, plus one
// each.  m_y <= 2^32 / (cs[1] u), m_x and m_z stay within a slab's cells; none where
// 2^23 + m + floor(p) could reach 2^24: slabs below 2^10 (bytes or cells), or axes
// above 2^22.
inline void cell_floor_constants(int64_t nx, int64_t ny, int64_t nz, int32_t voxel_type, float kfl[3], int32_t* bytes) {
  int32_t cs[2];
  cell_strides(nx, ny, nz, cs);
  *bytes = cell_layout_bytes(nx, ny, nz, voxel_type) < (uint64_t(1) << 32) ? 1 : 0;
  const uint32_t u = !*bytes ? 1u : (voxel_type == XR_VOXEL_F32 ? 32u : 16u);
  const uint32_t sx = (uint32_t)cs[0] * u, sy = (uint32_t)cs[1] * u;
  for (int k = 0; k < 3; ++k) kfl[k] = 0.0f;
  if (sy <= 1024) return;  // also where cells are not numbered
  const float scale = voxel_type == XR_VOXEL_F16 ? kH16 : 1.0f;  // of the x and y positions
  const uint32_t bias_xy = voxel_type == XR_VOXEL_F16 ? 0x52800000u : 0x4B000000u;  // bits of 2^23 scale
  const uint32_t t = 0u - bias_xy * (sx + sy) - 0x4B000000u * u;
  const uint32_t my = t / sy, mx = (t % sy) / sx, mz = (t % sy) % sx / u;
  if (mx + nx >= (1 << 23) - 2 || my + ny >= (1 << 23) - 2 || mz + nz >= (1 << 23) - 2) return;
  kfl[0] = (8388609.0f + (float)mx) * scale;
  kfl[1] = (8388609.0f + (float)my) * scale;
  kfl[2] = 8388609.0f + (float)mz;
}

}  // namespace xr

// Restates on the host how the DRR kernel reads the cell copy: every ray of an
// image is set up (xf::ray_setup), its samples are chosen, and where the kernel
// would take the unclamped march the cell addresses of all samples are formed as
// the march forms them (round-down addition of the floor constants, wrapping
// 32-bit products) and compared with the copy's size and with floor(position).
// Reads cases of doubles from a file, writes six counts for each (checked by
// tests/test_ray_cells_cpu.py).
#include <cfenv>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "xr_cells.h"
#include "xr_xfloat.h"

namespace {

float add_down(float a, float b) {
  volatile float x = a, y = b;
  std::fesetround(FE_DOWNWARD);
  volatile float r = x + y;
  std::fesetround(FE_TONEAREST);
  return r;
}

uint32_t bits(float v) {
  if (v != v) return 0x7fffffffu;  // the GPU's NaN
  uint32_t u;
  std::memcpy(&u, &v, 4);
  return u;
}

struct Counts {
  double hits = 0, unclamped = 0, samples = 0, outside = 0, wrong = 0, guarded = 0;
};

// The kernel's rule but for the guard: samples drift by less than an eighth of a voxel.
bool drift_ok(const int32_t n[3], uint32_t last) {
  const int32_t m = std::fmax(n[0], std::fmax(n[1], n[2]));
  int e = 0;
  while ((m >> e) != 0) ++e;
  return e <= 22 && last < (1u << (22 - e));
}

Counts run(const int32_t n[3], int vt, float step, int rows, int cols, const xr::xf::RayFrame& g, bool guard) {
  Counts c;
  int32_t cs[2], bytes;
  float kfl[3];
  xr::cell_strides(n[0], n[1], n[2], cs);
  xr::cell_floor_constants(n[0], n[1], n[2], vt, kfl, &bytes);
  const uint64_t copy = xr::cell_layout_bytes(n[0], n[1], n[2], vt);
  const uint32_t cell = vt == XR_VOXEL_F32 ? 32 : 16, unit = bytes ? cell : 1;
  const float scale = vt == XR_VOXEL_F16 ? xr::kH16 : 1.0f;
  const float maxb[3] = {(float)(n[0] - 1), (float)(n[1] - 1), (float)(n[2] - 1)};
  for (int row = 0; row < rows; ++row)
    for (int col = 0; col < cols; ++col) {
      float p[3], st[3], quot;
      if (!xr::xf::ray_setup(g, (float)col, (float)row, maxb, step, p, st, quot)) continue;
      // float to unsigned as the GPU converts: NaN and negatives 0, saturating
      const uint32_t nsteps = !(quot >= 1.0f) ? 0u : quot >= 4294967296.0f ? 0xffffffffu : (uint32_t)quot;
      if (nsteps > 100000u) continue;  // the kernel's limit on a ray's samples
      ++c.hits;
      if (!drift_ok(n, nsteps) || !(kfl[0] > 0.0f)) continue;
      const bool in = xr::xf::samples_within(p, st, 0u, nsteps, maxb, 0.75f);
      if (!in) ++c.guarded;
      if (guard && !in) continue;
      ++c.unclamped;
      for (int k = 0; k < 3; ++k)
        if (k < 2) p[k] *= scale, st[k] *= scale;
      for (uint32_t i = 0; i <= nsteps; ++i) {
        uint32_t t[3];
        for (int k = 0; k < 3; ++k) t[k] = bits(add_down(p[k], kfl[k]));
        const uint32_t a = t[1] * ((uint32_t)cs[1] * unit) + (t[0] * ((uint32_t)cs[0] * unit) + t[2] * unit);
        const uint64_t at = bytes ? a : (uint64_t)a * cell;
        ++c.samples;
        if (at + cell > copy) ++c.outside;
        else {
          const int64_t x = (int64_t)std::floor(p[0] / scale) + 1, y = (int64_t)std::floor(p[1] / scale) + 1,
                        z = (int64_t)std::floor(p[2]) + 1;
          if ((uint64_t)(x * cs[0] + y * (int64_t)cs[1] + z) * cell != at) ++c.wrong;
        }
        for (int k = 0; k < 3; ++k) p[k] = xr::xf::add(p[k], st[k]);
      }
    }
  return c;
}

}  // namespace

int main(int argc, char** argv) {
  if (argc == 6) {  // nx ny nz voxel type, "numbering": strides, bytes, constants
    const int64_t n[3] = {std::atoll(argv[1]), std::atoll(argv[2]), std::atoll(argv[3])};
    const int vt = std::atoi(argv[4]);
    int32_t cs[2], bytes;
    float kfl[3];
    xr::cell_strides(n[0], n[1], n[2], cs);
    xr::cell_floor_constants(n[0], n[1], n[2], vt, kfl, &bytes);
    std::printf("%d %d %d %llu %d %.1f %.1f %.1f\n", xr::cells_numbered(n[0], n[1], n[2]) ? 1 : 0, cs[0], cs[1],
                (unsigned long long)xr::cell_layout_bytes(n[0], n[1], n[2], vt), bytes, kfl[0], kfl[1], kfl[2]);
    return 0;
  }
  if (argc != 3) return 2;
  std::FILE* f = std::fopen(argv[1], "rb");
  std::FILE* o = std::fopen(argv[2], "wb");
  if (!f || !o) return 2;
  // n[3], voxel type, step, rows, cols, guard, K[9], E[16], focal length, frame, phys -> idx [12], pose [12]
  double h[8 + 9 + 16 + 2 + 24];
  while (std::fread(h, sizeof(double), sizeof(h) / sizeof(double), f) == sizeof(h) / sizeof(double)) {
    const int32_t n[3] = {(int32_t)h[0], (int32_t)h[1], (int32_t)h[2]};
    xr::xf::Camera cam;
    for (int k = 0; k < 9; ++k) cam.K[k] = (float)h[8 + k];
    for (int k = 0; k < 16; ++k) cam.E[k] = (float)h[17 + k];
    cam.focal_len = (float)h[33];
    cam.frame = (int32_t)h[34];
    xr::xf::Affine p2i, pose;
    for (int k = 0; k < 9; ++k) p2i.L[k] = (float)h[35 + k], pose.L[k] = (float)h[47 + k];
    for (int k = 0; k < 3; ++k) p2i.t[k] = (float)h[44 + k], pose.t[k] = (float)h[56 + k];
    xr::xf::RayFrame g;
    xr::xf::ray_frame(cam, p2i, pose, g);
    const Counts c = run(n, (int)h[3], (float)h[4], (int)h[5], (int)h[6], g, h[7] != 0.0);
    const double out[6] = {c.hits, c.unclamped, c.samples, c.outside, c.wrong, c.guarded};
    std::fwrite(out, sizeof(double), 6, o);
  }
  std::fclose(f);
  std::fclose(o);
  return 0;
}

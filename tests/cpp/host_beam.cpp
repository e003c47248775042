// The beams of the ray caster (asc_rays.cuh) compiled as host C++, a warp at a
// time (host_warp.h): an image as k_raycast casts it.
#include "host_warp.h"
#include "../../include/autoscoper_gb300.h"
#include "../../autoscoper_gb300/csrc/asc_rays.cuh"

using namespace asc;

// The clearance grid by its definition: the maximum over the axes of the
// distance from the cell's span to a voxel above the threshold, least over
// those voxels; an axis after the other, since the norm is separable.
static std::vector<uint8_t> clearance(const uint16_t* vol, int nx, int ny, int nz, float threshold)
{
  int n[3] = {nx, ny, nz};
  std::vector<uint8_t> d((size_t)nx * ny * nz);
  for (size_t i = 0; i < d.size(); ++i) d[i] = (float)vol[i] > threshold ? 0 : CLEAR_MAX;
  for (int axis = 0; axis < 3; ++axis) {
    int g[3] = {n[0], n[1], n[2]};
    g[axis] = clear_dim(n[axis]);
    std::vector<uint8_t> e((size_t)g[0] * g[1] * g[2]);
    const size_t step = axis == 0 ? 1 : (axis == 1 ? n[0] : (size_t)n[0] * n[1]);
    for (int z = 0; z < g[2]; ++z)
      for (int y = 0; y < g[1]; ++y)
        for (int x = 0; x < g[0]; ++x) {
          int at[3] = {x, y, z}, best = CLEAR_MAX;
          const int c = at[axis];
          at[axis] = 0;
          const uint8_t* line = d.data() + ((size_t)at[2] * n[1] + at[1]) * n[0] + at[0];
          for (int v = std::max(0, 2 * c - CLEAR_MAX); v < std::min(n[axis], 2 * c + 3 + CLEAR_MAX); ++v)
            best = std::min(best, std::max((int)line[v * step], std::max(std::max(2 * c - v, v - 2 * c - 2), 0)));
          e[((size_t)z * g[1] + y) * g[0] + x] = (uint8_t)best;
        }
    d.swap(e);
    n[axis] = g[axis];
  }
  return d;
}

// counts: samples of the whole rays, marched ones, lane slots, beams without
// an occupied interval.
extern "C" void hr_cast(const uint16_t* vol, int nx, int ny, int nz, int skip, const float* m, const float* vp,
                        float step, float cutoff, int w, int h, float* out, long long* counts)
{
  std::vector<uint32_t> pairs(padded_words(nx, ny, nz, ASC_STORE_U16));
  const auto at = [&](int x, int y, int z) { return (uint32_t)vol[((size_t)z * ny + y) * nx + x]; };
  pack_pairs(nx, ny, nz, ASC_STORE_U16, at, pairs.data());
  const int px = nx + 2 * PAD, pxy = px * (ny + 2 * PAD);
  DevVolume V{pairs.data(), nx, ny, nz, px, pxy, ASC_STORE_U16, 1.0f / 65535.0f, 0.f};
  V.gmax = volume_gmax(nx, ny, nz, [&](int x, int y, int z) { return (float)at(x, y, z); });
  const Cutoff cut = make_cutoff(cutoff, V.norm, V.gmax);
  std::vector<uint8_t> clr;
  if (skip) clr = clearance(vol, nx, ny, nz, occupancy_threshold(cut));
  df sx, sy;
  df_split((double)vp[2] / w, sx.h, sx.l);
  df_split((double)vp[3] / h, sy.h, sy.l);
  const RayScene s{m, vp, sx, sy, step, skip ? clr.data() : nullptr, w, h};
  static RaySlots<32> S;
  static float exact[EXACT_FLOATS];
  for (int i = 0; i < 4; ++i) counts[i] = 0;
  for (int y = 0; y < h; ++y)
    for (int x = 0; x < w; ++x) {
      RaySetup r;
      if (ray_setup(m, vp, x, y, sx, sy, step, nx, ny, nz, r)) counts[0] += r.K;
    }
  for (int y0 = 0; y0 < h; y0 += 4)
    for (int x0 = 0; x0 < w; x0 += 8)
      host_warp::run([&] {
        const int lane = threadIdx.x, x = x0 + (lane & 7), y = y0 + (lane >> 3);
        const bool valid = x < w && y < h;
        const Beam b = beam_mask(V, s, std::min(x, w - 1), std::min(y, h - 1));
        float d = 0.f;
        unsigned marched = 0, slots = 0;
        if (b.mask) {
          d = ray_beam<1>(V, s, cut, make_float4(cut.raw - cut.t0, cut.hi0 + cut.t0, cut.t1, 0.f), S, x, y, valid, b,
                          marched, slots);
          for (unsigned f = __ballot_sync(FULL_WARP, valid && d != d); f; f &= f - 1) {
            const int q = __ffs(f) - 1;
            const int rx = __shfl_sync(FULL_WARP, x, q), ry = __shfl_sync(FULL_WARP, y, q);
            const float e = march_exact(V, s, cut, rx, ry, exact);
            if (lane == q) d = e;
          }
        } else if (lane == 0) {
          ++counts[3];
        }
        if (valid) out[(size_t)y * w + x] = d;
        counts[1] += marched;
        if (lane == 0) counts[2] += slots;
      });
}

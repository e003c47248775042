// One march block (asc_march.cuh) compiled as host C++: the pairs of a ray
// inside the padded grid against the clamped samples one at a time.
#include <cstring>
#include <vector>

#include "host_march_shim.h"
#include "../../include/autoscoper_gb300.h"
#include "../../autoscoper_gb300/csrc/asc_march.cuh"

using namespace asc;

// Segments [j0, j1] of every ray of a w x h image, marched both ways:
// counts[0] segments, [1] rays that are not inside, [2] differing sums.
template <int STORE, int PAIRS, bool EXACT>
static void run(const DevVolume& V, const Cutoff& cut, const float* m, const float* vp, float step, int w, int h,
                long long* counts)
{
  df sx, sy;
  df_split((double)vp[2] / w, sx.h, sx.l);
  df_split((double)vp[3] / h, sy.h, sy.l);
  for (int y = 0; y < h; ++y)
    for (int x = 0; x < w; ++x) {
      RaySetup r;
      if (!ray_setup(m, vp, x, y, sx, sy, step, V.nx, V.ny, V.nz, r) || r.K <= 0) continue;
      const bool in = ray_inside(V, r);
      counts[1] += !in;
      float lo, hi;
      cutoff_bounds(cut, r.dX.h, r.dY.h, r.dZ.h, lo, hi);
      for (int kb = 0; kb < r.K; kb += REBASE) {
        const int n = std::min(REBASE, r.K - kb), j0 = (x * 7 + y) % n;
        for (int j1 = j0; j1 < n; j1 += 1 + (j1 - j0)) {
          const float a = march_block<STORE, EXACT, PAIRS>(V, r, kb, j0, j1, lo, hi, cut, in);
          const float b = march_block<STORE, EXACT, PAIRS>(V, r, kb, j0, j1, lo, hi, cut, false);
          ++counts[0];
          counts[2] += std::memcmp(&a, &b, 4) != 0;
        }
      }
    }
}

template <int STORE>
static void run_all(const DevVolume& V, const Cutoff& cut, const float* m, const float* vp, float step, int w, int h,
                    long long* counts)
{
  run<STORE, 1, false>(V, cut, m, vp, step, w, h, counts);
  run<STORE, 2, false>(V, cut, m, vp, step, w, h, counts);
  run<STORE, 1, true>(V, cut, m, vp, step, w, h, counts);
}

extern "C" void hb_blocks(const uint32_t* stored, int nx, int ny, int nz, int storage, const float* m, const float* vp,
                          float step, float cutoff, int w, int h, long long* counts)
{
  std::vector<uint32_t> pairs(padded_words(nx, ny, nz, storage));
  pack_pairs(nx, ny, nz, storage, [&](int x, int y, int z) { return stored[((size_t)z * ny + y) * nx + x]; },
             pairs.data());
  const int px = nx + 2 * PAD, pxy = px * (ny + 2 * PAD);
  DevVolume V{pairs.data(), nx, ny, nz, px, pxy, storage, 1.0f / 65535.0f, 0.f};
  V.gmax = 65535.0f;
  const Cutoff cut = make_cutoff(cutoff, V.norm, V.gmax);
  counts[0] = counts[1] = counts[2] = 0;
  if (storage == ASC_STORE_U16) run_all<ASC_STORE_U16>(V, cut, m, vp, step, w, h, counts);
  if (storage == ASC_STORE_BF16) run_all<ASC_STORE_BF16>(V, cut, m, vp, step, w, h, counts);
  if (storage == ASC_STORE_F32) run_all<ASC_STORE_F32>(V, cut, m, vp, step, w, h, counts);
}

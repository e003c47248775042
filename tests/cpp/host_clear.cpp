// The clearance grid kernel's phases (asc_clear.cuh) compiled as host C++: a
// block's threads one after the other, its warps by host_warp.h.
#include "host_warp.h"
inline uint2 make_uint2(unsigned x, unsigned y) { return {x, y}; }
#include "../../include/autoscoper_gb300.h"
#include "../../autoscoper_gb300/csrc/asc_clear.cuh"

using namespace asc;

template <int STORE>
static void build(const DevVolume& V, float threshold, uint8_t* clr)
{
  static ClearWork w;
  for (int cz = 0; cz < clear_dim(V.nz); cz += CB)
    for (int cy = 0; cy < clear_dim(V.ny); cy += CB)
      for (int cx = 0; cx < clear_dim(V.nx); cx += CB) {
        std::memset(&w, 0xff, sizeof w);
        host_warp::run([&] {
          for (int i = 0; i < CLEAR_Z * CLEAR_Y / 2; ++i) clear_load<STORE>(V, threshold, w, i, cx, cy, cz);
        });
        std::vector<uint2> acc(CLEAR_THREADS, uint2{0u, 0u});
        std::vector<unsigned> n(3 * CLEAR_THREADS, 0u);
        for (int round = 0; CLEAR_ROUND * round <= CLEAR_REACH; ++round) {
          for (int t = 0; t < CLEAR_THREADS; ++t) clear_reach(w, t, round, acc[t]);
          for (int t = 0; t < CLEAR_THREADS; ++t) clear_count(w, t, round, reinterpret_cast<unsigned(&)[3]>(n[3 * t]));
        }
        for (int t = 0; t < CLEAR_THREADS; ++t) clear_bytes(w, t, reinterpret_cast<unsigned(&)[3]>(n[3 * t]));
        for (int t = 0; t < CLEAR_THREADS; ++t) clear_store(w, t, V, cx, cy, cz, clr);
      }
}

extern "C" void hc_grid(const uint32_t* stored, int nx, int ny, int nz, int storage, float threshold, uint8_t* clr)
{
  std::vector<uint32_t> pairs(padded_words(nx, ny, nz, storage));
  pack_pairs(nx, ny, nz, storage, [&](int x, int y, int z) { return stored[((size_t)z * ny + y) * nx + x]; },
             pairs.data());
  const int px = nx + 2 * PAD;
  const DevVolume V{pairs.data(), nx, ny, nz, px, px * (ny + 2 * PAD), storage, 1.0f / 65535.0f, 0.f};
  if (storage == ASC_STORE_U16) build<ASC_STORE_U16>(V, threshold, clr);
  if (storage == ASC_STORE_BF16) build<ASC_STORE_BF16>(V, threshold, clr);
  if (storage == ASC_STORE_F32) build<ASC_STORE_F32>(V, threshold, clr);
}

// The ray march of a beam (32 neighbouring rays) by one warp, shared by the
// batched engine (k_ray) and the plain ray caster (k_raycast), and the exact
// march of one ray by one warp.
//
// A beam's crossing of the volume is cut into 64 intervals, two per lane,
// and the clearance grid says which of them may hold a sample above the
// cutoff (beam_mask).  A beam without any is done: its pixels are 0.  In an
// occupied beam each lane sets its ray up in double-float, trims the runs of
// occupied intervals with its own clearances, cuts them into segments at the
// multiples of REBASE samples (next_segment) and marches these one after the
// other, the warp's lanes side by side; it adds the segments' sums in order
// (add_block).  Which samples are skipped changes no bit of the result: a
// sample at or below the cutoff leaves its segment's sum as it is, and the
// segments' bounds at multiples of REBASE do not depend on it.
//
// A clearance answers for 15 voxels at most, so pixels of more than about three
// voxels, or a crossing of more than 1700, leave intervals that no clearance
// clears.  The rays of such a beam find their own intervals (ray_mask); the same
// march follows.  k_ray over 64 candidates of a 320^3 bone in two views of 152^2
// (4 voxels a pixel): 545 us with a walk of each ray through 8-voxel cells, 1588
// with the beams' intervals alone (4 times the samples), 520 with the rays' own; of
// a 512^3 bone at 243^2 2360, 12600 and 2340.
//
// What bounds it is instruction issue: 74 % of the slots, and the packed FP32
// pairs of the sample loop take two.  A beam serves its 32 rays with one byte
// per interval and lane; rays that walked 8-voxel cells by themselves spent
// half of their instructions on the walk.  Neighbours' segments are of nearly
// equal length (a warp's lanes march 85 % of the samples that its slots have
// room for), so sorting a block's segments by length, with its barriers, costs
// more than the idle lanes do (12.6 ms against 12.2 on the batch below).
// k_ray over 300 candidates x 2 views of 1024^2 (three bones of up to 4.8 M
// voxels): 16.5 ms with the walk (15.7 G warp instructions), 12.2 with beams,
// 11.8 with the sample loop's unpacking split over two units and no clamp in it
// (march_block), 11.3 with the warp met again before each march (march_beam;
// 12.1 G); 100 candidates of a 128^3 bone at 512^2: 2.55, 1.44, 1.42 and 1.37
// ms.
#pragma once

#include "asc_march.cuh"

namespace asc {

constexpr int RTX = 16, RTY = 16;     // a ray tile, pixels
constexpr int BEAMS = RTX * RTY / 32;  // its beams
constexpr int NRAY = 256;             // threads per block of the marching kernels
constexpr unsigned FULL_WARP = 0xffffffffu;

// What an image's rays share.
struct RayScene {
  const float* m;
  const float* vp;
  df sx, sy;
  float step;
  const uint8_t* clr;  // the clearance grid; null: every sample is marched
  int w, h;
};

// The pixel of this lane in beam `sub` of the tile at (x0, y0): a beam is a
// (1 << shape) x (32 >> shape) block of pixels.
__device__ __forceinline__ void beam_pixel(int x0, int y0, int sub, int shape, int& x, int& y)
{
  const int lane = threadIdx.x & 31, across = 4 - shape;  // log2 of the beams per tile row
  x = x0 + ((sub & ((1 << across) - 1)) << shape) + (lane & ((1 << shape) - 1));
  y = y0 + ((sub >> across) << (5 - shape)) + (lane >> shape);
}

struct Beam {
  unsigned long long mask;  // bit i: interval [t0 + i len, t0 + (i + 1) len) may hold samples above the cutoff
  float t0, len;
  float err;
  bool wide;  // an interval reaches farther than a clearance answers for: each ray finds its own (ray_mask)
};

// The occupied intervals of this warp's 32 rays.  Every lane passes a pixel
// of the image (lanes past its edge the edge's).
__device__ __forceinline__ Beam beam_mask(const DevVolume& V, const RayScene& s, int x, int y)
{
  const float nx = (float)V.nx, ny = (float)V.ny, nz = (float)V.nz;
  const BeamRay r = beam_ray(s.m, s.vp, s.sx.h, s.sy.h, (float)x, (float)y, s.step, nx, ny, nz);
  Beam b;
  b.err = r.err;
  // t >= 0, so the order of the floats is the order of their bits
  const bool hit = r.far > r.near;
  const float t0 = __uint_as_float(__reduce_min_sync(FULL_WARP, __float_as_uint(hit ? r.near : 3.0e38f)));
  const float t1 = __uint_as_float(__reduce_max_sync(FULL_WARP, __float_as_uint(hit ? r.far : 0.f)));
  b.t0 = t0;
  b.len = (t1 - t0) * (1.0f / 64.0f);
  b.mask = 0ull;
  b.wide = false;
  if (!(t1 > t0)) return b;
  if (!s.clr) {
    b.mask = ~0ull;
    return b;
  }
  float D[3], w[3];
  for (int i = 0; i < 3; ++i) {
    D[i] = __shfl_sync(FULL_WARP, r.D[i], 12);  // a ray near the middle of the block
    w[i] = __uint_as_float(__reduce_max_sync(FULL_WARP, __float_as_uint(fabsf(r.D[i] - D[i]))));
  }
  const float half = 0.5f * b.len, c0 = fmaf((float)(threadIdx.x & 31) + 0.5f, b.len, t0);
  bool wide = false;
  const bool lo = beam_occupied(s.clr, V.nx, V.ny, V.nz, r.O, D, w, c0, half, r.err, wide);
  const bool hi = beam_occupied(s.clr, V.nx, V.ny, V.nz, r.O, D, w, fmaf(32.0f, b.len, c0), half, r.err, wide);
  b.wide = __any_sync(FULL_WARP, wide);
  b.mask = (unsigned long long)__ballot_sync(FULL_WARP, lo) | (unsigned long long)__ballot_sync(FULL_WARP, hi) << 32;
  return b;
}

// A ray's set-up, kept in the thread's own slots of shared memory: the march
// of a segment reads it once, and in registers it would spill.
template <int THREADS>
struct RaySlots {
  float4 q[3][THREADS];  // X, Y, Z, dX, dY, dZ as double-floats
};

// What the clearances along a ray need of it: sample k lies at X - k dX.
struct ClearRay {
  float X, Y, Z, dX, dY, dZ;
  float per;  // samples per voxel of the fastest axis
};
template <class Slots>
__device__ __forceinline__ ClearRay clear_ray(const Slots& S)
{
  const float4 q0 = S.q[0][threadIdx.x], q1 = S.q[1][threadIdx.x], q2 = S.q[2][threadIdx.x];
  const float dX = q1.z, dY = q2.x, dZ = q2.z;
  return ClearRay{q0.x, q0.z, q1.x, dX, dY, dZ,
                  0.99999f * approx_rcp(fmaxf(fabsf(dX), fmaxf(fabsf(dY), fabsf(dZ))))};
}

// Samples of clear space from sample k on, on either side; 0: sample k may count.
__device__ __forceinline__ int clear_samples(const DevVolume& V, const uint8_t* __restrict__ clr, const ClearRay& r,
                                             float err, int k)
{
  const float kf = (float)k;
  const float e = clearance_at(clr, V.nx, V.ny, V.nz, fmaf(-kf, r.dX, r.X), fmaf(-kf, r.dY, r.Y),
                               fmaf(-kf, r.dZ, r.Z)) - 1.0f - err;
  return e >= 0.f ? (int)fminf(e * r.per, 1.0e6f) + 1 : 0;
}

// The occupied intervals of this lane's ray (tf: RaySetup::tf) in a wide beam,
// from tests at equal distances along the beam's crossing: enough of them that
// a clearance of half its range clears the stretch of one, and at least a test
// per 8 samples up to one per interval.  Rays that cross few voxels are left to
// the trims of their ends, which reach as far (SHORT): 64 candidates in two views
// at 4 voxels a pixel, k_ray of a 160^3 bone 165 us without tests and 148 with
// them, of a 128^3 one 107 and 115.  The tests do not wait for one another, where
// hopping from clearance to clearance is a chain of loads: a cast of 32^2 pixels
// of a 320^3 bone 62 us with hops, 54 with tests.  FLIGHT: loads in flight, which
// shorten a single image (four; 58 us with two) but crowd L1 when every warp
// marches (64 candidates of a 512^3 bone: 2.48 ms with four, 2.33 with two).
constexpr float CLEAR_HALF = 0.5f * (CLEAR_MAX - 1);
constexpr int SHORT = 10;  // in units of 2 CLEAR_HALF voxels
template <int FLIGHT, class Slots>
__device__ __forceinline__ unsigned long long ray_mask(const DevVolume& V, const uint8_t* __restrict__ clr,
                                                       const Slots& S, int K, float tf, const Beam& b)
{
  const float4 q0 = S.q[0][threadIdx.x], q1 = S.q[1][threadIdx.x], q2 = S.q[2][threadIdx.x];
  const float dX = q1.z, dY = q2.x, dZ = q2.z;
  const float d = K > 0 ? fmaxf(fabsf(dX), fmaxf(fabsf(dY), fabsf(dZ))) : 0.f;  // voxels a sample
  const unsigned far = __reduce_max_sync(FULL_WARP, (unsigned)fminf(b.len * d * (32.0f / CLEAR_HALF), 4096.0f));
  if (far <= SHORT || 4.0f * (float)far > 64.0f * b.len) return ~0ull;  // a test for fewer than four samples gains nothing
  const unsigned tests = max(far, (unsigned)fminf(8.0f * b.len, 64.0f));
  int lt = 0;  // log2 of the tests made
  while ((1u << lt) < tests) ++lt;
  const float len = b.len * (lt <= 6 ? (float)(64 >> lt) : 1.0f / (float)(1 << (lt - 6)));
  const float need = fmaf(0.5f * len, d, 1.0f + b.err);
  const unsigned long long bits = lt <= 6 ? ~0ull >> (64 - (64 >> lt)) : 1ull;
  unsigned long long mask = 0ull;
#pragma unroll FLIGHT
  for (int j = 0; j < 1 << lt; ++j) {
    const float k = tf - fmaf((float)j + 0.5f, len, b.t0);
    const float e = clearance_at(clr, V.nx, V.ny, V.nz, fmaf(-k, dX, q0.x), fmaf(-k, dY, q0.z), fmaf(-k, dZ, q1.x));
    if (!(e >= need)) mask |= bits << (lt <= 6 ? j << (6 - lt) : j >> (lt - 6));
  }
  return mask;
}

// A ray's place in its beam's runs: the intervals left, the samples
// [k, ke] left of the current run, and the open segment (march block pb,
// extent [pf, pl]; pf < 0 when none is open).
struct RunState {
  unsigned long long mask;
  int k, ke;
  int pb, pf, pl;
};

// The ray's next segment: block start kb (a multiple of REBASE) and the
// occupied extent [kb + js, kb + je], in increasing k; false when the ray is
// done.  Runs are trimmed from both ends by the clearance at the end's
// sample, up to TRIMS times: four trims leave 2 % more samples than an exact
// box per 8-voxel cell did (39.1 against 38.2 a ray on the benchmark's bones,
// none 47.2, two 40.8).
constexpr int TRIMS = 4;
template <class Slots>
__device__ __forceinline__ bool next_segment(const DevVolume& V, const uint8_t* __restrict__ clr, const Slots& S,
                                             int K, float tf, const Beam& b, RunState& s, int& kb, int& js, int& je)
{
  for (;;) {
    while (s.k > s.ke && s.mask) {
      // the run of intervals farthest from the camera (samples count from the far side)
      const int i1 = 63 - __clzll((long long)s.mask);
      const unsigned long long above = ~(s.mask << (63 - i1));
      const int i0 = above ? i1 + 1 - __clzll((long long)above) : 0;
      s.mask &= (1ull << i0) - 1ull;
      const float tb = fmaf((float)(i1 + 1), b.len, b.t0), ta = fmaf((float)i0, b.len, b.t0);
      const float slack = fmaf(4.0e-6f, tb, 0.01f);  // the rounding of t
      if (i1 < 63) s.k = max(s.k, (int)ceilf(tf - tb - slack));
      s.ke = i0 > 0 ? min(K - 1, (int)floorf(tf - ta + slack)) : K - 1;
      if (clr) {
        const ClearRay r = clear_ray(S);
        for (int t = 0; t < TRIMS && s.k <= s.ke; ++t) {
          const int f = clear_samples(V, clr, r, b.err, s.k), l = clear_samples(V, clr, r, b.err, s.ke);
          s.k += f;
          s.ke -= l;
          if (f + l == 0) break;
        }
      }
    }
    if (s.k > s.ke) break;
    const int bb = (int)((unsigned)s.k / REBASE), hi = min(s.ke, bb * REBASE + REBASE - 1);
    if (s.pf >= 0 && s.pb != bb) break;
    if (s.pf < 0) {
      s.pb = bb;
      s.pf = s.k;
    }
    s.pl = hi;
    s.k = hi + 1;
  }
  if (s.pf < 0) return false;
  kb = s.pb * REBASE;
  js = s.pf - kb;
  je = s.pl - kb;
  s.pf = -1;
  return true;
}

// The segments of this lane's ray (K samples; 0: none), marched side by side
// with the warp's other lanes.  tf: RaySetup::tf, negative for a ray that is
// not ray_inside().  Returns their sum in raw units: NaN when a sample fell in
// the cutoff's band.  marched: this lane's samples; slots: what the warp's
// lanes had room for.
template <int STORE, int PAIRS, class Slots>
__device__ __forceinline__ float march_beam(const DevVolume& V, const uint8_t* __restrict__ clr, const Slots& S,
                                            int K, float tf, const Beam& b, float4 band, const Cutoff& cut,
                                            unsigned& marched, unsigned& slots)
{
  RunState run{b.mask, 0, -1, 0, -1, 0};
  if (b.wide) run.mask &= ray_mask<2 * PAIRS>(V, clr, S, K, fabsf(tf), b);
  if (K <= 0) run.mask = 0;
  df total{0.f, 0.f};  // NaN once a segment met the cutoff's band
  for (;;) {
    // A segment or an empty one in the same registers, and what depends on it
    // after the warp has met again: with the march under next_segment's own
    // result the compiler ran all that follows twice, for the lanes that had
    // a segment and for the others (k_ray 11.81 ms against 11.31 here).
    int kb = 0, js = 0, je = -1;
    {
      int a, f, l;
      if (next_segment(V, clr, S, K, fabsf(tf), b, run, a, f, l)) {
        kb = a;
        js = f;
        je = l;
      }
    }
    const int len = je - js + 1;
    float p = 0.f;
    if (len > 0) {
      RaySetup r;
      const float4 q0 = S.q[0][threadIdx.x], q1 = S.q[1][threadIdx.x], q2 = S.q[2][threadIdx.x];
      r.X = df{q0.x, q0.y};
      r.Y = df{q0.z, q0.w};
      r.Z = df{q1.x, q1.y};
      r.dX = df{q1.z, q1.w};
      r.dY = df{q2.x, q2.y};
      r.dZ = df{q2.z, q2.w};
      // this ray's band: raw - t0, hi0 + t0 and t1 (cutoff_bounds)
      const float D = fabsf(q1.z) + fabsf(q2.x) + fabsf(q2.z);
      p = march_block<STORE, false, PAIRS>(V, r, kb, js, je, fmaf(-band.z, D, band.x), fmaf(band.z, D, band.y), cut,
                                           tf > 0.f);
    }
    if (block_flagged(p))
      total.h = __int_as_float(0x7fffffff);  // NaN stays NaN through add_block
    else
      add_block(total, p);
    const unsigned most = __reduce_max_sync(FULL_WARP, (unsigned)len);
    if (most == 0) break;
    marched += (unsigned)len;
    slots += 32u * most;
  }
  return total.h + total.l;
}

// The DRR sum of the ray at pixel (x, y) (valid: inside the image) of this
// warp's beam.  band: the cutoff's raw - t0, hi0 + t0 and t1.
template <int PAIRS, class Slots>
__device__ __forceinline__ float ray_beam(const DevVolume& V, const RayScene& s, const Cutoff& cut, float4 band,
                                          Slots& S, int x, int y, bool valid, const Beam& b, unsigned& marched,
                                          unsigned& slots)
{
  int K = 0;
  float tf = 0.f;
  {
    RaySetup r;
    if (valid && ray_setup(s.m, s.vp, x, y, s.sx, s.sy, s.step, V.nx, V.ny, V.nz, r)) {
      S.q[0][threadIdx.x] = make_float4(r.X.h, r.X.l, r.Y.h, r.Y.l);
      S.q[1][threadIdx.x] = make_float4(r.Z.h, r.Z.l, r.dX.h, r.dX.l);
      S.q[2][threadIdx.x] = make_float4(r.dY.h, r.dY.l, r.dZ.h, r.dZ.l);
      K = r.K;
      tf = ray_inside(V, r) ? r.tf : -r.tf;
    }
  }
  if (V.storage == ASC_STORE_F32) return march_beam<ASC_STORE_F32, PAIRS>(V, s.clr, S, K, tf, b, band, cut, marched, slots);
  if (V.storage == ASC_STORE_BF16) return march_beam<ASC_STORE_BF16, PAIRS>(V, s.clr, S, K, tf, b, band, cut, marched, slots);
  if (V.storage == ASC_STORE_F16) return march_beam<ASC_STORE_F16, PAIRS>(V, s.clr, S, K, tf, b, band, cut, marched, slots);
  return march_beam<ASC_STORE_U16, PAIRS>(V, s.clr, S, K, tf, b, band, cut, marched, slots);
}

// The DRR sum of one ray (raw units) by one warp, every cutoff decision the
// exact one: the warp's lanes take the samples side by side (two of each
// march block), then the blocks' sums are taken in order, a lane per block,
// and added in order, so the bits are those of the serial march.  What bounds
// it is the loads' latency: with one marked ray per lane, marched serially,
// k_ray_fix took 184 us for the 7 800 marked rays of 300 candidates x 2 views
// and 44 us for a simplex step's few; here 58 and 16.
// v: EXACT_FLOATS shared words of the warp.
constexpr int EXACT_BLOCKS = 8;                                  // march blocks in flight
constexpr int EXACT_FLOATS = EXACT_BLOCKS * (REBASE + 1);
template <int STORE>
__device__ __forceinline__ float march_exact(const DevVolume& V, const RaySetup& r, const Cutoff& cut, float* v)
{
  const int lane = threadIdx.x & 31;
  float lo, hi;
  cutoff_bounds(cut, r.dX.h, r.dY.h, r.dZ.h, lo, hi);
  df total{0.f, 0.f};
  const int nb = (r.K + REBASE - 1) / REBASE;
  for (int b0 = 0; b0 < nb; b0 += EXACT_BLOCKS) {
    const int n = min(EXACT_BLOCKS, nb - b0);
    for (int i = lane; i < n * REBASE; i += 32) {
      const int b = i / REBASE, j = i % REBASE, kb = (b0 + b) * REBASE;
      v[b * (REBASE + 1) + j] = kb + j < r.K ? march_block<STORE, true>(V, r, kb, j, j, lo, hi, cut) : 0.f;
    }
    __syncwarp();
    float p = 0.f;
    if (lane < n)
      for (int j = 0; j < REBASE; ++j) p += v[lane * (REBASE + 1) + j];
    for (int b = 0; b < n; ++b) add_block(total, __shfl_sync(FULL_WARP, p, b));
    __syncwarp();
  }
  return total.h + total.l;
}

__device__ __forceinline__ float march_exact(const DevVolume& V, const RayScene& s, const Cutoff& cut, int x, int y,
                                             float* v)
{
  RaySetup r;
  if (!ray_setup(s.m, s.vp, x, y, s.sx, s.sy, s.step, V.nx, V.ny, V.nz, r) || r.K <= 0) return 0.f;
  if (V.storage == ASC_STORE_F32) return march_exact<ASC_STORE_F32>(V, r, cut, v);
  if (V.storage == ASC_STORE_BF16) return march_exact<ASC_STORE_BF16>(V, r, cut, v);
  if (V.storage == ASC_STORE_F16) return march_exact<ASC_STORE_F16>(V, r, cut, v);
  return march_exact<ASC_STORE_U16>(V, r, cut, v);
}

}  // namespace asc

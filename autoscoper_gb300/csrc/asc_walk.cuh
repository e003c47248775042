// The march of one ray by one thread over 8-voxel cells, host only: the
// kernels march beams over clearance grids (asc_rays.cuh); this form shares
// their ray set-up, march blocks and cutoff decisions, and the CPU tests hold
// those to the FP64 oracle through it.
#pragma once

#include "asc_march.cuh"

namespace asc {

// Occupancy of OCC^3-voxel cells for one cutoff (OCC = 8): cell (cx, cy, cz)
// is empty (byte 0) when every voxel of [8c-1, 8c+10) on each axis is <=
// cutoff.  That range holds the taps of nonzero weight of every sample at a
// texel coordinate in (8c-1, 8c+9), i.e. within one voxel of the cell's own
// [8c, 8c+8), so a walk may place a sample in a cell with an error of up to a
// voxel.  A trilinear sample is a convex combination of its taps (each FP32
// lerp stays between its ends), so a sample placed in an empty cell is <=
// cutoff and adds exactly nothing to the DRR (RayCaster_kernels.cu:189); the
// march skips it.
//
// An occupied cell also keeps the box of its voxels above the cutoff: a
// sample can touch such a voxel v only at texel coordinates in [v-1, v+1)
// per axis, and an eighth of a voxel of margin covers the walk's placement
// error (FP32 positions, ~1e-4 voxel).  The walk marches only the cell's
// samples that lie in the box, so a cell occupied by a few voxels costs a few
// samples.  Bounds are int16 eighths of a voxel, so trimming applies to
// volumes of at most OCC_TRIM_MAX voxels per axis.
constexpr int OCC = 8;
constexpr int OCC_LO = 1, OCC_HI = 2;  // apron voxels below and above a cell
// The grid holds OCC_PAD cells of margin on every side (cells -2 .. b + 1 of
// an axis of b cells), so that a walk, whose cells stay within one of the
// box's, indexes it without clamping.
constexpr int OCC_PAD = 2;
constexpr int OCC_TRIM_MAX = 4094;
__host__ __device__ __forceinline__ int occ_dim(int n) { return (n + OCC - 1) / OCC + 2 * OCC_PAD; }

// The grid of n cells: n occupancy bytes, then at the next 16-byte boundary
// n boxes, each an int4 of (lo | hi << 16) per axis x, y, z (int16 texel
// coordinates in eighths of a voxel) and a spare word.
__host__ __device__ __forceinline__ size_t occ_box_offset(size_t n) { return (n + 15) & ~(size_t)15; }
__host__ __device__ __forceinline__ size_t occ_grid_bytes(size_t n) { return occ_box_offset(n) + 16 * n; }

// Occupancy byte and box of cell (cx, cy, cz) (margin cells included) of an
// nx x ny x nz volume; val(x, y, z) is the voxel's raw value.
template <class Val>
__host__ __device__ inline uint8_t occ_cell(int cx, int cy, int cz, int nx, int ny, int nz, float cutoff, Val&& val,
                                            int* box)
{
  int lo[3] = {0x7fff, 0x7fff, 0x7fff}, hi[3] = {-0x7fff, -0x7fff, -0x7fff};
  bool any = false;
  const int a = -OCC_LO, e = OCC + OCC_HI;
  for (int z = max(cz * OCC + a, 0); z < min(cz * OCC + e, nz); ++z)
    for (int y = max(cy * OCC + a, 0); y < min(cy * OCC + e, ny); ++y)
      for (int x = max(cx * OCC + a, 0); x < min(cx * OCC + e, nx); ++x)
        if (val(x, y, z) > cutoff) {
          any = true;
          lo[0] = min(lo[0], 8 * (x - 1) - 1);
          hi[0] = max(hi[0], 8 * (x + 1) + 1);
          lo[1] = min(lo[1], 8 * (y - 1) - 1);
          hi[1] = max(hi[1], 8 * (y + 1) + 1);
          lo[2] = min(lo[2], 8 * (z - 1) - 1);
          hi[2] = max(hi[2], 8 * (z + 1) + 1);
        }
  for (int i = 0; i < 3; ++i) box[i] = (lo[i] & 0xffff) | (int)((unsigned)hi[i] << 16);
  box[3] = 0;
  // byte 2: the box covers the cell with a voxel to spare on every side, so
  // trimming keeps every sample the walk places in the cell
  const int c[3] = {cx, cy, cz};
  bool covers = true;
  for (int i = 0; i < 3; ++i) covers = covers && lo[i] <= 8 * (OCC * c[i] - 1) && hi[i] >= 8 * (OCC * c[i] + OCC + 1);
  return any ? (covers ? 2 : 1) : 0;
}


// A ray's walk through the occupancy grid (a 3-D DDA over cells, in units of
// samples): the sample index of each axis' next cell-plane crossing, the
// samples between crossings and the cell step per crossing.  FP32 throughout:
// a sample's cell comes out within ~1e-3 voxel of the exact one, far inside
// the one-voxel apron of the occupancy grid.
struct CellWalk {
  float tx, ty, tz;     // next crossing per axis (sample index; +inf if none)
  float dtx, dty, dtz;  // samples between crossings
  int cell;             // the current cell's index in the padded grid
  int ix, iy, iz;       // index change per crossing of each axis
  unsigned last;        // the grid's last index (a bound no walk reaches)
  int steps;            // crossings a ray can make through the grid
};

__device__ __forceinline__ void walk_axis(float C, float dC, float kf, float& t, float& dt, int& c, int& st)
{
  // coordinate at sample k: C - k dC
  const float X = fmaf(-kf, dC, C);
  c = __float2int_rd(X * (1.0f / OCC));
  if (dC > 0.f) {  // decreasing: next plane at OCC * c
    st = -1;
    const float ri = __frcp_rn(dC);
    dt = OCC * ri;
    t = fmaf(X - (float)(OCC * c), ri, kf);
  } else if (dC < 0.f) {  // increasing: next plane at OCC * (c + 1)
    st = 1;
    const float ri = __frcp_rn(dC);
    dt = -OCC * ri;
    t = fmaf(X - (float)(OCC * (c + 1)), ri, kf);
  } else {
    st = 0;
    dt = 3.0e38f;
    t = 3.0e38f;
  }
}

__device__ __forceinline__ CellWalk cell_walk(const DevVolume& V, const RaySetup& r, int k)
{
  CellWalk w;
  const float kf = (float)k;
  int cx, cy, cz, sx, sy, sz;
  walk_axis(r.X.h, r.dX.h, kf, w.tx, w.dtx, cx, sx);
  walk_axis(r.Y.h, r.dY.h, kf, w.ty, w.dty, cy, sy);
  walk_axis(r.Z.h, r.dZ.h, kf, w.tz, w.dtz, cz, sz);
  const int px = occ_dim(V.nx), py = occ_dim(V.ny), pz = occ_dim(V.nz);
  w.cell = ((cz + OCC_PAD) * py + (cy + OCC_PAD)) * px + (cx + OCC_PAD);
  w.ix = sx;
  w.iy = sy * px;
  w.iz = sz * px * py;
  w.last = (unsigned)(px * py * pz - 1);
  w.steps = 2 * (px + py + pz);
  return w;
}

// The walk's view of one ray for trimming a cell to its box: per axis
// ia = 1 / (8 dC) (box bounds are eighths of a voxel) and the start C
// (sample k sits at C - k dC); ia is NaN for an axis the ray runs parallel
// to and for every axis of a volume too large for the boxes (no bound).
struct RayTrim {
  float ia[3], c[3];
};

__device__ __forceinline__ RayTrim ray_trim(const DevVolume& V, const RaySetup& r)
{
  RayTrim t;
  const float C[3] = {r.X.h, r.Y.h, r.Z.h}, d[3] = {r.dX.h, r.dY.h, r.dZ.h};
  const bool big = V.nx > OCC_TRIM_MAX || V.ny > OCC_TRIM_MAX || V.nz > OCC_TRIM_MAX;
  for (int i = 0; i < 3; ++i) {
    t.ia[i] = big || d[i] == 0.f ? __int_as_float(0x7fffffff) : 0.125f * __frcp_rn(d[i]);
    t.c[i] = C[i];
  }
  return t;
}

// Walk state of one ray between calls of walk_segments: the next sample to
// place, and the open march block (index pb, occupied extent [pf, pl]; pf < 0
// when none is open).
struct WalkState {
  int k, kend;
  int pb, pf, pl;
};

// Walks samples s.k .. s.kend and hands each march block that holds occupied
// samples to emit(kb, js, je) -- block start kb (a multiple of REBASE) and the
// occupied extent [kb + js, kb + je] -- in increasing k.  emit returns false
// when it can take no more; the walk then stops, and a later call resumes
// where it stopped.  Returns true when the ray is done.  Without `occ` every
// sample counts as occupied.  The steps are bounded by the cells the ray
// crosses; past that bound the rest of the ray counts as occupied.
template <class Emit, class Trim>
__device__ __forceinline__ bool walk_segments(CellWalk& w, const uint8_t* __restrict__ occ, Trim&& trim, WalkState& s,
                                              Emit&& emit)
{
  const int4* __restrict__ boxes = occ ? (const int4*)(occ + occ_box_offset((size_t)w.last + 1)) : nullptr;
  int steps = w.steps;
  // tp: the cell's entry crossing; its first sample is floor(tp) + 1
  const float kendf = (float)s.kend;
  float tp = (float)s.k - 0.5f;
  while (tp < kendf) {
    bool full = true;
    unsigned cb = 0;  // the cell's occupancy byte; 1: trim to the box
    float tn = 3.0e38f;
    if (occ && steps > 0) {
      tn = fminf(w.tx, fminf(w.ty, w.tz));
      cb = __ldg(occ + min((unsigned)w.cell, w.last));
      full = cb != 0;
      --steps;
    }
    if (full) {
      // add the cell's samples [a, ke] that lie in its box to the open block(s)
      int ke = tn < kendf ? (int)floorf(tn) : s.kend;
      int a = (int)floorf(tp) + 1;
      if (cb == 1) {
        const int4 bx = __ldg(boxes + min((unsigned)w.cell, w.last));
        float klo = -1.0e9f, khi = 1.0e9f;
        const int pk[3] = {bx.x, bx.y, bx.z};
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          const float lo = (float)((pk[i] << 16) >> 16), hi = (float)(pk[i] >> 16);
          float ia, c;
          trim(i, ia, c);  // the ray's RayTrim entries of axis i
          const float ca = 8.0f * c * ia;  // C / dC
          const float k1 = fmaf(-hi, ia, ca), k2 = fmaf(-lo, ia, ca);
          klo = fmaxf(klo, fminf(k1, k2));  // a NaN bound (parallel axis) leaves klo and khi
          khi = fminf(khi, fmaxf(k1, k2));
        }
        a = max(a, (int)ceilf(klo));
        ke = min(ke, (int)floorf(khi));
      }
      for (; a <= ke;) {
        const int bb = (int)((unsigned)a / REBASE), hi = min(ke, bb * REBASE + REBASE - 1);
        if (s.pf >= 0 && s.pb != bb) {
          if (!emit(s.pb * REBASE, s.pf - s.pb * REBASE, s.pl - s.pb * REBASE)) {
            s.k = a;  // resume here; the walk state still describes this cell
            return false;
          }
          s.pf = -1;
        }
        if (s.pf < 0) {
          s.pb = bb;
          s.pf = a;
        }
        s.pl = hi;
        a = hi + 1;
      }
    }
    tp = tn;
    if (tn == w.tx) {
      w.cell += w.ix;
      w.tx += w.dtx;
    } else if (tn == w.ty) {
      w.cell += w.iy;
      w.ty += w.dty;
    } else {
      w.cell += w.iz;
      w.tz += w.dtz;
    }
  }
  s.k = s.kend + 1;
  if (s.pf >= 0) {
    if (!emit(s.pb * REBASE, s.pf - s.pb * REBASE, s.pl - s.pb * REBASE)) return false;
    s.pf = -1;
  }
  return true;
}

// One march pass over a whole ray: the march blocks that hold occupied
// samples, in order, each trimmed to its occupied extent, their sums combined
// in double-float.  EXACT false: *flagged is set when a sample fell in the
// cutoff's band (the pass's total then leaves the band's samples out).
template <int STORE, bool EXACT>
__device__ __forceinline__ float march_pass(const DevVolume& V, const uint8_t* __restrict__ occ, const RaySetup& r,
                                            const Cutoff& cut, bool* flagged)
{
  CellWalk w = cell_walk(V, r, 0);
  WalkState s{0, r.K - 1, 0, -1, 0};
  const RayTrim t = ray_trim(V, r);
  df total{0.f, 0.f};
  bool fl = false;
  float lo, hi;
  cutoff_bounds(cut, r.dX.h, r.dY.h, r.dZ.h, lo, hi);
  walk_segments(w, occ, [&](int i, float& ia, float& c) {
    ia = t.ia[i];
    c = t.c[i];
  }, s, [&](int kb, int js, int je) {
    const float p = march_block<STORE, EXACT>(V, r, kb, js, je, lo, hi, cut, ray_inside(V, r));
    if (!EXACT && block_flagged(p))
      fl = true;
    else
      add_block(total, p);
    return true;
  });
  if (flagged) *flagged = fl;
  return total.h + total.l;
}

// One whole ray, with every cutoff decision the exact one: the FP32 pass,
// and the exact pass when a sample fell in the band.  The result depends
// only on the samples above the cutoff, so it is the same with and without
// `occ`, and the same as the batched engine's.
template <int STORE>
__device__ __forceinline__ float march(const DevVolume& V, const uint8_t* __restrict__ occ, const RaySetup& r,
                                       const Cutoff& cut)
{
  if (r.K <= 0) return 0.f;
  bool flagged = false;
  const float d = march_pass<STORE, false>(V, occ, r, cut, &flagged);
  return flagged ? march_pass<STORE, true>(V, occ, r, cut, nullptr) : d;
}

}  // namespace asc

// The clearance grid (asc_march.cuh) of a volume, CB^3 cells per block.
//
// A cell's clearance is the number of distances d = 0, 1, .. CLEAR_MAX - 1
// within which (maximum norm) no voxel lies above the threshold.  Voxels are
// bits, so a distance is tested for a row of cells at once: the block's rows
// of voxels are ORed over the cell's reach along y (incrementally: two rows
// more per distance), then along z, and the reach along x is a windowed OR of
// the word's own bits.  Four distances a round, one per quarter of the block.
//
// What bounds it is reading the voxels, 7 times each from L2 (the block's
// cells and CLEAR_MAX - 1 voxels around them); a stored voxel holds its
// neighbours in x and y as well (DevVolume), so every other voxel of every
// other row is loaded, four loads in flight per warp.  By build, with the cast
// of 16 pixels after it taken off: 35 us for 128^3 voxels, 175 for 320^3 and 652
// for 512^3, where the same distances by a byte per voxel and axis, a voxel per
// load, took 122, 552 and 2182, and occupancy bits of 8^3 cells 88, 182 and 699.
#pragma once

#include "asc_march.cuh"

namespace asc {

constexpr int CB = 16;                           // cells of a block's edge
constexpr int CLEAR_REACH = CLEAR_MAX - 1;       // voxels around them
constexpr int CLEAR_Z = CLEAR_CELL * CB + 1 + 2 * CLEAR_REACH;  // slices read, from voxel CLEAR_CELL c - CLEAR_REACH on
constexpr int CLEAR_Y = CLEAR_Z + 1;             // rows, in pairs
constexpr int CLEAR_THREADS = 1024, CLEAR_ROUND = 4;
static_assert(CLEAR_CELL == 2 && CLEAR_REACH % 2 == 0 && CLEAR_Y <= 64, "rows of voxels in pairs, a 64-bit word each");
static_assert(CLEAR_Z * CB <= CLEAR_THREADS && CLEAR_ROUND * CB * CB == CLEAR_THREADS, "a thread per row and per cell row");

struct ClearWork {
  uint2 row[CLEAR_Z][CLEAR_Y];             // the voxels above the threshold: even ones, odd ones
  union {
    uint2 reach[CLEAR_ROUND][CLEAR_Z][CB];        // ORed over a cell's reach along y, per distance of the round
    uint32_t count[CLEAR_ROUND][CB][CB][CB / 4];  // at the end: a byte per cell, the quarter's clear distances
  };
};

// Row pair i of the block at cells (cx, cy, cz), by a warp: two voxels of two
// rows per lane.
template <int STORE>
__device__ __forceinline__ void clear_load(const DevVolume& V, float threshold, ClearWork& w, int i, int cx, int cy, int cz)
{
  const int iz = i / (CLEAR_Y / 2), iy = 2 * (i % (CLEAR_Y / 2));
  const int x = CLEAR_CELL * cx - CLEAR_REACH + 2 * (threadIdx.x & 31);
  const int y = CLEAR_CELL * cy - CLEAR_REACH + iy, z = CLEAR_CELL * cz - CLEAR_REACH + iz;
  bool a[4] = {false, false, false, false};
  if (x >= 0 && x < V.nx && y >= 0 && y < V.ny && z >= 0 && z < V.nz) {
    const Taps<STORE> t =
        fetch_taps<STORE>(V.pairs, (unsigned)(z + PAD) * (unsigned)V.pxy + (unsigned)(y + PAD) * (unsigned)V.px + (unsigned)(x + PAD),
                          (unsigned)V.px, (unsigned)V.pxy);
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      float lo, hi;
      if constexpr (STORE == ASC_STORE_F32) {
        lo = t.p[r].x;
        hi = t.p[r].y;
      } else {
        unpack<STORE>(t.w[r], lo, hi);
      }
      const bool in = y + r < V.ny;
      a[2 * r] = in && lo > threshold;
      a[2 * r + 1] = in && x + 1 < V.nx && hi > threshold;
    }
  }
  unsigned b[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) b[k] = __ballot_sync(0xffffffffu, a[k]);
  if ((threadIdx.x & 31) == 0) {
    w.row[iz][iy] = make_uint2(b[0], b[1]);
    w.row[iz][iy + 1] = make_uint2(b[2], b[3]);
  }
}

// Thread t's row (slice t / CB, cell row t % CB) of a round's distances: acc
// holds the OR of the round before.
__device__ __forceinline__ void clear_reach(ClearWork& w, int t, int round, uint2& acc)
{
  if (t >= CLEAR_Z * CB) return;
  const int z = t / CB, c = t % CB, y = CLEAR_CELL * c + CLEAR_REACH;  // the cell's first row
  const auto add = [&](int iy) {
    const uint2 r = w.row[z][iy];
    acc.x |= r.x;
    acc.y |= r.y;
  };
#pragma unroll
  for (int k = 0; k < CLEAR_ROUND; ++k) {
    const int d = CLEAR_ROUND * round + k;
    if (d > CLEAR_REACH) break;
    if (d == 0) {
      add(y);
      add(y + 1);
      add(y + 2);
    } else {
      add(y - d);
      add(y + 2 + d);
    }
    w.reach[k][z][c] = acc;
  }
}

// OR of `len` bits from each bit on.
__device__ __forceinline__ unsigned window_or(unsigned v, int len)
{
  int n = 1;
  for (; 2 * n <= len; n *= 2) v |= v >> n;
  return v | v >> (len - n);
}

// Bit c: cell c of the row (16 cells) holds no voxel within d of it along x.
__device__ __forceinline__ unsigned clear_cells(uint2 v, int d)
{
  // even voxels 2c - d .. 2c + 2 + d, odd ones alike; bit i of a word is voxel 2 i (+ 1) - CLEAR_REACH
  const int a = d / 2, b = (d + 1) / 2, first = CLEAR_REACH / 2;
  const unsigned any = window_or(v.x, 2 * a + 2) >> (first - a) | window_or(v.y, 2 * b + 1) >> (first - b);
  return ~any & 0xffffu;
}

// Thread t's cells (quarter t / CB^2: its distance of the round; cell row
// (y, z)): n counts, in bit planes, the distances at which each was clear.
__device__ __forceinline__ void clear_count(const ClearWork& w, int t, int round, unsigned (&n)[3])
{
  const int k = t / (CB * CB), cz = t / CB % CB, cy = t % CB, d = CLEAR_ROUND * round + k;
  if (d > CLEAR_REACH) return;
  uint2 v = make_uint2(0u, 0u);
  for (int z = CLEAR_CELL * cz + CLEAR_REACH - d; z <= CLEAR_CELL * cz + CLEAR_REACH + 2 + d; ++z) {
    const uint2 r = w.reach[k][z][cy];
    v.x |= r.x;
    v.y |= r.y;
  }
  const unsigned u = clear_cells(v, d), c0 = n[0] & u, c1 = n[1] & c0;
  n[0] ^= u;
  n[1] ^= c0;
  n[2] |= c1;
}

// The counts as bytes, after every thread's last clear_count.
__device__ __forceinline__ void clear_bytes(ClearWork& w, int t, const unsigned (&n)[3])
{
  const int k = t / (CB * CB), cz = t / CB % CB, cy = t % CB;
  for (int q = 0; q < CB / 4; ++q) {
    uint32_t v = 0;
#pragma unroll
    for (int p = 0; p < 3; ++p)
#pragma unroll
      for (int i = 0; i < 4; ++i) v |= (n[p] >> (4 * q + i) & 1u) << (8 * i + p);
    w.count[k][cz][cy][q] = v;
  }
}

// Thread t's four cells of the block at cells (cx, cy, cz): the quarters'
// counts added into the grid.
__device__ __forceinline__ void clear_store(const ClearWork& w, int t, const DevVolume& V, int cx, int cy, int cz,
                                            uint8_t* __restrict__ clr)
{
  const int gx = clear_dim(V.nx), gy = clear_dim(V.ny), gz = clear_dim(V.nz);
  const int q = t % (CB / 4), y = t / (CB / 4) % CB, z = t / (CB / 4 * CB), x = cx + 4 * q;
  if (x >= gx || cy + y >= gy || cz + z >= gz) return;
  uint32_t v = 0;
#pragma unroll
  for (int k = 0; k < CLEAR_ROUND; ++k) v += w.count[k][z][y][q];
  uint8_t* o = clr + ((size_t)(cz + z) * gy + (cy + y)) * gx + x;
  if (gx % 4 == 0) {  // o is aligned: clr is, as cudaMalloc's
    *reinterpret_cast<uint32_t*>(o) = v;
    return;
  }
  for (int i = 0; i < 4 && x + i < gx; ++i) o[i] = (uint8_t)(v >> (8 * i));
}

}  // namespace asc

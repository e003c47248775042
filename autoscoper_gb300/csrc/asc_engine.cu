// Batched registration engine: Tracker::minimizationFunc (Tracker.cpp:775-827)
// for many (bone, manipulator) candidates per pass, with the scene resident
// on the device.
//
// One evaluation is four launches on one stream (five with cf_model 1):
//   k_setup       a warp per item: FP64 pose composition, view matrices,
//                            viewports (Tracker.cpp:603-634) and crops; the
//                            last block: the tile layout of every crop, with
//                            prefix sums and each tile's (item, view);
//   k_ray         persistent: a warp per beam of 32 rays from an atomic
//                            queue, DRRs written to a packed buffer; rays
//                            with a sample within rounding of the cutoff are
//                            marked, their beams listed;
//   k_ray_fix     a warp per listed beam: its marked rays marched again with
//                            exact cutoff decisions;
//   k_view        persistent: 48x48 output tiles pulled from a queue; each
//                            stages DRR and radiograph regions with the chain's
//                            halo in shared memory, runs both filter chains,
//                            the masks and the NCC moments; the last tile of a
//                            view merges its tiles in FP64, the last view of an
//                            item sums the view costs.
// The PSO driver adds an update kernel before and a best-update kernel after,
// and captures one iteration as a CUDA graph.
#include <cuda_fp16.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <vector>

#include "asc_internal.cuh"
#include "asc_rays.cuh"

namespace asc {
const void* image_data(asc_image im, int* w, int* h, int* bps);
}

using namespace asc;

namespace {

constexpr int MAX_VIEWS = 16;  // views of an engine (a serving engine holds several jobs' views)
constexpr int MAX_SLOTS = 4;   // views one bone is scored in (the public bone desc's per-view settings)
constexpr int MAX_BONES = 64;
constexpr int MAX_FILTERS = 8;
#ifndef ASC_VT
#define ASC_VT 48
#endif
#ifndef ASC_VIEW_MINBLOCKS
#define ASC_VIEW_MINBLOCKS 3
#endif
constexpr int VT = ASC_VT;   // k_view output tile edge
constexpr int VNT = 256;     // k_view threads per block

struct FilterDev {
  int kind, K, R;
  float p0, p1, p2;
  float g[32];
};

struct ViewDev {
  double cam[12], cam_inv[12], ip[12], cvp[4];
  float ipf[4];
  int rw, rh;  // render size of this view's trial (Trial::render_width/height)
  const void* rad;
  int rad_w, rad_h, rad_bps;
  const float* bg;
  int bg_w, bg_h;
  float bg_thr;
  int n_drr, n_rad, h_drr, h_rad;
  FilterDev fdrr[MAX_FILTERS], frad[MAX_FILTERS];
};

struct BoneDev {
  DevVolume vol;
  float inv_scale[3], inv_trans[3];
  double pivot[12], pivot_inv[12], base[6];
  // per slot: the bone is scored in views view_of[0 .. n_slots), with that
  // view's RayCaster settings and its clearance grid
  float step[MAX_SLOTS], scale[MAX_SLOTS];
  Cutoff cut[MAX_SLOTS];
  const uint8_t* clr[MAX_SLOTS];
  int view_of[MAX_SLOTS];
  int n_slots;
  int visible;                    // RayCaster::setVisible: a hidden volume renders zeros
};

struct SceneDev {
  int n_views, n_bones, rw, rh, coverage, halo;  // rw, rh, halo: the largest of the views'
  int slots;     // (item, slot) entries per item: the most views a bone is scored in
  int cf_model;  // 0: 1 - NCC per view; 1: SAD ("hdist") per view
  ViewDev views[MAX_VIEWS];
  BoneDev bones[MAX_BONES];
};

struct IV {
  float m[12];
  float vp[4];
  float sx[2], sy[2];  // vp[2] / w and vp[3] / h as double-floats
  int w, h, ok, bone;
  int view, slot;  // the engine view and the bone's slot of this (item, view)
  int rtx, rty, ftx, fty;
  int err;        // the crop exceeded the render size (the reference throws)
  float band[3];  // the bone's cutoff here: raw - t0, hi0 + t0, t1 (k_ray's band)
  float step;     // the bone's sample distance here, and its volume's size (k_count_samples)
  int nx, ny, nz;
  long long pix;  // offset of this crop in the DRR buffer
};

struct Counters {
  int n_items, n_iv;
  int rtiles, ftiles;
  unsigned rnext;
  int fnext;
  int error;
  int nfix;   // rays whose march met the cutoff's band (k_ray_fix marches them again)
  int nfixb;  // beams holding such rays
  unsigned setup;  // blocks of k_setup done; 0 between evaluations
  unsigned long long samples, pixels;
  unsigned long long marched, slots;  // marched samples, 32 x warp-max span
};

struct Bufs {
  IV* iv;
  int* roff;       // n_iv + 1 prefix of ray tiles
  int* foff;       // n_iv + 1 prefix of view tiles
  float* drr;
  Moments* part;   // per view tile
  float2* fg;      // cf_model 1: masked DRR and radiograph per crop pixel
  double2* hmean;  // cf_model 1: per-iv means of f and g
  float* tsad;     // cf_model 1: per view tile SAD
  double* vcost;   // per iv
  unsigned* ivt;   // per-iv tile tickets
  unsigned* itt;   // per-item view tickets
  unsigned* fixb;  // beams (ray tile x BEAMS + its beam) holding rays to march again exactly (k_ray_fix)
  int* rtile_iv;   // per ray tile: its (item, view) (k_setup)
  int* ftile_iv;   // per view tile: its (item, view)
  Counters* C;
};

// The last view of an item is scored: its cost, and its views' costs.
__device__ void finish_item(const SceneDev* sc, const Bufs& b, int item, double* cost, double* view_cost_out)
{
  const int ns = sc->slots;
  double tot = 0;
  for (int j = 0; j < ns; ++j) {
    const double v = b.vcost[item * ns + j];
    tot += v;
    if (view_cost_out) view_cost_out[item * ns + j] = v;
  }
  cost[item] = tot < 0 ? 9999.0 : tot;  // Tracker.cpp:823-825
}

// ---------------------------------------------------------------- k_setup
// The FP64 set-up of an item (minimizationFunc's pose, then trackFrame's
// view matrix, viewport and crop for each of its views) by one warp, its
// intermediate frames in the warp's shared memory.  An FP64 operation takes
// a warp 16 issue cycles and its dependants ~40 whatever its active lanes, so
// what counts is the chain's length: the sines, the elements of a rotation
// or product, the volume's corners and the quotients are dealt to lanes, and
// the operands and the order of each stay those of frame_* (asc_internal.cuh).
constexpr int SETUP_THREADS = 256;
struct SetupWarp {
  double f[2][12];     // frames under construction (rotations, translation)
  double R[2][9];      // their next rotation
  double t[3][12];     // products
  double mv[4][12], imv[4][12];  // per view
  double film[4][4], corner[4][6];  // per view: the image's film-plane box, the volume's faces (setup_view)
};

// frame_rotate of f[side] about a by the angle of cosine c and sine s, by 16
// lanes per side; `on`: this side takes part.
__device__ __forceinline__ void warp_rotate(SetupWarp& w, int side, int e, bool on, double a0, double a1, double a2,
                                            double c, double s)
{
  const double mag = sqrt(a0 * a0 + a1 * a1 + a2 * a2);
  const double mine = (e % 3 == 0 ? a0 : (e % 3 == 1 ? a1 : a2)) / mag;
  const int first = (threadIdx.x & 16);
  a0 = __shfl_sync(FULL_WARP, mine, first);
  a1 = __shfl_sync(FULL_WARP, mine, first + 1);
  a2 = __shfl_sync(FULL_WARP, mine, first + 2);
  on = on && mag != 0 && e < 9;
  const int i = e / 3, j = e % 3;
  const double oc = 1.0 - c;
  if (on) {
    // row-vector rotation matrix: oc a_i a_j, plus c on the diagonal, plus or
    // minus s a_k off it
    const int lo = min(i, j), hi = max(i, j), k = 3 - lo - hi;
    const double al = lo == 0 ? a0 : (lo == 1 ? a1 : a2), ah = hi == 0 ? a0 : (hi == 1 ? a1 : a2);
    const double ak = k == 0 ? a0 : (k == 1 ? a1 : a2);
    const bool plus = (j - i + 3) % 3 == 1;  // (0,1), (1,2), (2,0)
    w.R[side][e] = i == j ? oc * al * al + c : oc * al * ah + (plus ? s : -s) * ak;
  }
  __syncwarp();
  double t = 0.0;
  if (on) {
    const double *f = w.f[side] + 3 * i, *R = w.R[side] + j;
    t = f[0] * R[0] + f[1] * R[3] + f[2] * R[6];
  }
  __syncwarp();
  if (on) w.f[side][e] = t;
  __syncwarp();
}

// out = a . b (frame_mul), an element per lane.
__device__ __forceinline__ void warp_mul(const double* a, const double* b, double* out, int lane)
{
  if (lane < 12) {
    const int c = lane / 3, i = lane % 3;
    const double r = a[i] * b[3 * c] + a[3 + i] * b[3 * c + 1] + a[6 + i] * b[3 * c + 2];
    out[lane] = c == 3 ? r + a[9 + i] : r;
  }
  __syncwarp();
}

__device__ __forceinline__ double shfl_min(double v, int o) { return fmin(v, __shfl_xor_sync(FULL_WARP, v, o)); }
__device__ __forceinline__ double shfl_max(double v, int o) { return fmax(v, __shfl_xor_sync(FULL_WARP, v, o)); }

// What an item's views need besides its pose, by a second warp meanwhile: 8
// lanes per view, the corners of its image in the film plane
// (calculate_viewport's rf) and the faces of the bone's box.
__device__ __forceinline__ void setup_view(const SceneDev* __restrict__ sc, int bi, SetupWarp& w)
{
  const BoneDev& B = sc->bones[bi];
  const int lane = threadIdx.x & 31, j = lane >> 3, l = lane & 7, first = lane & ~7;
  const ViewDev& V = sc->views[j < sc->slots && j < B.n_slots ? B.view_of[j] : 0];
  const int i = l % 3;
  const double *a = V.cam, *p = V.ip + (l < 3 ? 3 : 9);
  const double at = -(a[3 * i] * a[9] + a[3 * i + 1] * a[10] + a[3 * i + 2] * a[11]);
  const double q = a[3 * i] * p[0] + a[3 * i + 1] * p[1] + a[3 * i + 2] * p[2] + at;
  const double num = __shfl_sync(FULL_WARP, q, first + (l < 2 ? l : (l < 4 ? l + 1 : 0)));
  const double den = __shfl_sync(FULL_WARP, q, first + (l < 2 ? 2 : 5));
  if (l < 4) w.film[j][l] = -2 * num / den;
  if (l < 6) {
    const int k = l >> 1;
    const double face = k < 2 ? (double)(l & 1) : (double)(l & 1) - 1.0;
    w.corner[j][l] = (face - (double)B.inv_trans[k]) / (double)B.inv_scale[k];
  }
}

// The frame of yaw (cosine c, sine s) about z alone, what frame_rotate makes
// of the identity.
__device__ __forceinline__ void warp_yaw(double* f, int lane, double c, double s)
{
  if (lane < 12) {
    const double one = 1.0 - c + c;
    f[lane] = lane == 0 || lane == 4 ? c : (lane == 1 ? s : (lane == 3 ? -s : (lane == 8 ? one : 0.0)));
  }
  __syncwarp();
}

// The item's pose: its frame into w.f[0].
__device__ void setup_pose(const SceneDev* __restrict__ sc, int item, int bi, const double* __restrict__ manip,
                           SetupWarp& w)
{
  const double PI = 3.14159265358979323846;
  const int lane = threadIdx.x & 31, side = lane >> 4, e = lane & 15;
  const BoneDev& B = sc->bones[bi];
  const double* man = manip + 6 * item;
  // ---- minimizationFunc: pose . V^-1 . manip . V, then the xyzypr round trip.
  // side 0: the base pose's frame; side 1: the manipulator's
  const double v3 = man[3], v4 = man[4], v5 = man[5];
  const double ang = sqrt(v3 * v3 + v4 * v4 + v5 * v5);
  double c, s;
  sincos(PI * (lane < 3 ? B.base[3 + lane] : ang) / 180.0, &s, &c);
  warp_yaw(w.f[0], lane, __shfl_sync(FULL_WARP, c, 0), __shfl_sync(FULL_WARP, s, 0));
  if (side == 1 && e < 12) w.f[1][e] = e == 0 || e == 4 || e == 8 ? 1.0 : 0.0;
  __syncwarp();
  for (int k = 1; k < 3; ++k) {  // pitch about the new y, roll about the new x
    const double* ax = w.f[0] + 6 - 3 * k;
    const double a0 = side ? v3 : ax[0], a1 = side ? v4 : ax[1], a2 = side ? v5 : ax[2];
    const int from = side ? 3 : k;
    const double ck = __shfl_sync(FULL_WARP, c, from), sk = __shfl_sync(FULL_WARP, s, from);
    warp_rotate(w, side, e, side == 0 || (k == 1 && ang != 0), a0, a1, a2, ck, sk);
  }
  if (lane < 3) w.f[0][9 + lane] += B.base[lane];
  if (side == 1 && e < 3) w.f[1][9 + e] += man[e];
  __syncwarp();
  warp_mul(w.f[0], B.pivot_inv, w.t[0], lane);
  warp_mul(w.t[0], w.f[1], w.t[1], lane);
  warp_mul(w.t[1], B.pivot, w.t[2], lane);
  {
    const double* f = w.t[2];
    const double q = sqrt(f[5] * f[5] + f[8] * f[8]);
    const double y = lane == 0 ? f[1] : (lane == 1 ? -f[2] : f[5]), x = lane == 0 ? f[0] : (lane == 1 ? q : f[8]);
    const double ypr = 180.0 * atan2(y, x) / PI;
    sincos(PI * ypr / 180.0, &s, &c);
  }
  warp_yaw(w.f[0], lane, __shfl_sync(FULL_WARP, c, 0), __shfl_sync(FULL_WARP, s, 0));
  for (int k = 1; k < 3; ++k) {
    const double* ax = w.f[0] + 6 - 3 * k;
    const double a0 = ax[0], a1 = ax[1], a2 = ax[2];
    const double ck = __shfl_sync(FULL_WARP, c, k), sk = __shfl_sync(FULL_WARP, s, k);
    warp_rotate(w, side, e, side == 0, a0, a1, a2, ck, sk);
  }
  if (lane < 3) w.f[0][9 + lane] += w.t[2][9 + lane];
  __syncwarp();
}

// trackFrame (1a)-(1c) of the item's views, 8 lanes each.
__device__ void setup_views(const SceneDev* __restrict__ sc, int item, int bi, const Bufs& b, SetupWarp& w)
{
  const int lane = threadIdx.x & 31, ns = sc->slots, j = lane >> 3, l = lane & 7;
  const BoneDev& B = sc->bones[bi];
  const bool on = j < ns && j < B.n_slots;  // past the bone's views: a slot that adds nothing to the cost
  const int view = on ? B.view_of[j] : 0;
  const ViewDev& V = sc->views[view];
  double *mv = w.mv[j], *imv = w.imv[j];
  for (int q = l; q < 12; q += 8) {
    const int cc = q / 3, i = q % 3;
    const double *a = V.cam_inv, *t = w.f[0];
    const double r = a[i] * t[3 * cc] + a[3 + i] * t[3 * cc + 1] + a[6 + i] * t[3 * cc + 2];
    mv[q] = cc == 3 ? r + a[9 + i] : r;
  }
  __syncwarp();
  for (int q = l; q < 12; q += 8) {  // frame_inverse
    const int cc = q / 3, i = q % 3;
    imv[q] = cc < 3 ? mv[3 * i + cc] : -(mv[3 * i] * mv[9] + mv[3 * i + 1] * mv[10] + mv[3 * i + 2] * mv[11]);
  }
  const int first = lane & ~7;
  // calculate_viewport, the volume's corners a lane each
  const double rf0 = w.film[j][0], rf1 = w.film[j][1], rf2 = w.film[j][2], rf3 = w.film[j][3];
  double lo0, lo1, hi0, hi1;
  {
    const double p0 = w.corner[j][l >> 2], p1 = w.corner[j][2 + (l >> 1 & 1)], p2 = w.corner[j][4 + (l & 1)];
    double q[3];
    for (int i = 0; i < 3; ++i) q[i] = mv[i] * p0 + mv[3 + i] * p1 + mv[6 + i] * p2 + mv[9 + i];
    const double fx = -2 * q[0] / q[2], fy = -2 * q[1] / q[2];
    lo0 = fmin(1.0, fx);
    lo1 = fmin(1.0, fy);
    hi0 = fmax(-1.0, fx);
    hi1 = fmax(-1.0, fy);
  }
  for (int o = 1; o < 8; o <<= 1) {
    lo0 = shfl_min(lo0, o);
    lo1 = shfl_min(lo1, o);
    hi0 = shfl_max(hi0, o);
    hi1 = shfl_max(hi1, o);
  }
  __syncwarp();  // imv
  const bool seen = !((lo0 > rf2 && hi0 > rf2) || (lo1 > rf3 && hi1 > rf3) || (lo0 < rf0 && hi0 < rf0) ||
                      (lo1 < rf1 && hi1 < rf1) || (lo0 == 1.0 && lo1 == 1.0 && hi0 == -1.0 && hi1 == -1.0));
  if (lo0 < rf0) lo0 = rf0;
  if (lo1 < rf1) lo1 = rf1;
  if (hi0 > rf2) hi0 = rf2;
  if (hi1 > rf3) hi1 = rf3;
  const double vp2 = hi0 - lo0, vp3 = hi1 - lo1;
  // the crop's width (even lanes) and height (odd lanes), and its pixels' spacing
  const bool odd = l & 1;
  const double fs = (odd ? vp3 : vp2) * (odd ? V.rh : V.rw) / V.cvp[odd ? 3 : 2];
  unsigned n = fs > 0 ? (unsigned)fs : 0u;
  float sh = 0.f, sl = 0.f;
  const double spacing = (double)(float)(odd ? vp3 : vp2) / (double)n;
  if (n > 0) df_split(spacing, sh, sl);
  unsigned cw = __shfl_sync(FULL_WARP, n, first), ch = __shfl_sync(FULL_WARP, n, first + 1);
  const float syh = __shfl_sync(FULL_WARP, sh, first + 1), syl = __shfl_sync(FULL_WARP, sl, first + 1);
  if (j >= ns) return;
  const int k = item * ns + j;
  IV& r = b.iv[k];
  if (on)
    for (int q = l; q < 12; q += 8) {  // fold_matrix
      const int row = q / 4, cc = q % 4;
      const double last = cc < 3 ? 0.0 : 1.0;
      r.m[q] = (float)(imv[cc < 3 ? 3 * cc + row : 9 + row] * (double)B.inv_scale[row] + last * (double)B.inv_trans[row]);
    }
  if (l != 0) return;
  r.bone = bi;
  r.slot = j;
  r.view = on ? view : -1;
  r.w = r.h = r.ok = r.err = 0;
  r.rtx = r.rty = r.ftx = r.fty = 0;
  double vc = 0.0;
  if (on) {
    const Cutoff& cut = B.cut[j];
    r.band[0] = cut.raw - cut.t0;
    r.band[1] = cut.hi0 + cut.t0;
    r.band[2] = cut.t1;
    r.step = B.step[j];
    r.nx = B.vol.nx;
    r.ny = B.vol.ny;
    r.nz = B.vol.nz;
    if (!seen) {
      vc = 9999.0;  // Tracker.cpp:614-617
    } else {
      if (cw > (unsigned)V.rw || ch > (unsigned)V.rh) {
        r.err = 1;  // the reference throws (Tracker.cpp:625-629)
        cw = 0;
        ch = 0;
      }
      r.w = (int)cw;
      r.h = (int)ch;
      r.vp[0] = (float)lo0;
      r.vp[1] = (float)lo1;
      r.vp[2] = (float)vp2;
      r.vp[3] = (float)vp3;
      r.sx[0] = sh;
      r.sx[1] = sl;
      r.sy[0] = syh;
      r.sy[1] = syl;
      if (cw == 0 || ch == 0 || !B.visible) {
        // an empty crop, or the all-zero DRR of a hidden volume (RayCaster.cpp:131-134),
        // whose mask is empty: the degenerate NCC (1e5), or the SAD of no pixels
        vc = sc->cf_model ? 0.0 : 1.0 - 1e5;
      } else {
        r.ok = 1;
        r.rtx = (r.w + RTX - 1) / RTX;
        r.rty = (r.h + RTY - 1) / RTY;
        r.ftx = (r.w + VT - 1) / VT;
        r.fty = (r.h + VT - 1) / VT;
      }
    }
  }
  b.vcost[k] = vc;
  b.ivt[k] = 0;
}

// Exclusive sums over the block's threads of a, c and p, and their totals
// (s: 3 words of 8 bytes per warp).
__device__ __forceinline__ void block_scan3(int& a, int& c, long long& p, int& ta, int& tc, long long& tp,
                                            long long (*s)[SETUP_THREADS / 32])
{
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int ia = a, ic = c;
  long long ip = p;
  for (int o = 1; o < 32; o <<= 1) {
    const int ua = __shfl_up_sync(FULL_WARP, ia, o), uc = __shfl_up_sync(FULL_WARP, ic, o);
    const long long up = __shfl_up_sync(FULL_WARP, ip, o);
    if (lane >= o) {
      ia += ua;
      ic += uc;
      ip += up;
    }
  }
  __syncthreads();
  if (lane == 31) {
    s[0][warp] = ia;
    s[1][warp] = ic;
    s[2][warp] = ip;
  }
  __syncthreads();
  ta = tc = 0;
  tp = 0;
  int ba = 0, bc = 0;
  long long bp = 0;
  for (int q = 0; q < SETUP_THREADS / 32; ++q) {
    if (q == warp) {
      ba = ta;
      bc = tc;
      bp = tp;
    }
    ta += (int)s[0][q];
    tc += (int)s[1][q];
    tp += s[2][q];
  }
  a = ba + ia - a;
  c = bc + ic - c;
  p = bp + ip - p;
}

// p[from, to) = v by a warp, 16 bytes a lane between the ends.
__device__ __forceinline__ void warp_fill(int* __restrict__ p, int from, int to, int v, int lane)
{
  const int a = min((from + 3) & ~3, to), z = max(a, to & ~3);
  if (from + lane < a) p[from + lane] = v;
  for (int t = a + 4 * lane; t < z; t += 128) *(int4*)(p + t) = make_int4(v, v, v, v);
  if (z + lane < to) p[z + lane] = v;
}

// Every item's set-up, by one warp of its block (the SM's FP64 unit serves
// one at a time, a second warp the part that needs no pose); then the last block to finish lays the batch out: prefix sums of the tile counts and crop sizes (ray tiles, view
// tiles, DRR offsets), each tile's (item, view), so that the persistent
// kernels look a grabbed tile up with one load, the batch counters, and the
// items' view tickets (views finished here count as arrived).
// What bounds it is the latency of one FP64 chain (~70 cycles an operation).
// One thread per (item, view) took 78 us, with two launches after it for the
// layout and the tile map: 88 us for 4 candidates, 99 for 300; here 28 and 77.
__global__ void __launch_bounds__(SETUP_THREADS) k_setup(const SceneDev* __restrict__ sc, int n_items,
                                                         const int* __restrict__ bone_in,
                                                         const double* __restrict__ manip, Bufs b,
                                                         double* __restrict__ cost, double* __restrict__ view_cost_out,
                                                         int* __restrict__ error_out)
{
  __shared__ SetupWarp s_w;
  __shared__ long long s_scan[3][SETUP_THREADS / 32];
  __shared__ int s_ray[SETUP_THREADS + 1], s_view[SETUP_THREADS + 1];
  __shared__ int s_err;
  __shared__ bool s_last;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int bi = bone_in[blockIdx.x];
  if (bi < 0 || bi >= sc->n_bones) bi = 0;
  if (warp == 0) setup_pose(sc, blockIdx.x, bi, manip, s_w);
  if (warp == 1) setup_view(sc, bi, s_w);
  __syncthreads();
  if (warp == 0) {
    setup_views(sc, blockIdx.x, bi, b, s_w);
    __threadfence();
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    s_last = atomicAdd(&b.C->setup, 1u) == gridDim.x - 1;
    s_err = 0;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  const int nv = sc->slots, n_iv = n_items * nv;
  int ray = 0, view = 0;
  long long pix = 0;
  for (int k0 = 0; k0 < n_iv; k0 += SETUP_THREADS) {
    const int k = k0 + threadIdx.x;
    int a = 0, c = 0, ta, tc;
    long long p = 0, tp;
    if (k < n_iv) {
      const IV& r = b.iv[k];
      if (__ldcg(&r.err)) s_err = ASC_ERR_RANGE;
      a = __ldcg(&r.rtx) * __ldcg(&r.rty);
      c = __ldcg(&r.ftx) * __ldcg(&r.fty);
      p = (long long)__ldcg(&r.w) * __ldcg(&r.h);
    }
    block_scan3(a, c, p, ta, tc, tp, s_scan);
    s_ray[threadIdx.x] = ray + a;
    s_view[threadIdx.x] = view + c;
    if (k < n_iv) {
      b.iv[k].pix = pix + p;
      b.roff[k] = ray + a;
      b.foff[k] = view + c;
    }
    ray += ta;
    view += tc;
    pix += tp;
    if (threadIdx.x == 0) {
      s_ray[SETUP_THREADS] = ray;
      s_view[SETUP_THREADS] = view;
    }
    __syncthreads();
    for (int q = warp; q < SETUP_THREADS && k0 + q < n_iv; q += SETUP_THREADS / 32) {
      warp_fill(b.rtile_iv, s_ray[q], s_ray[q + 1], k0 + q, lane);
      warp_fill(b.ftile_iv, s_view[q], s_view[q + 1], k0 + q, lane);
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    b.roff[n_iv] = ray;
    b.foff[n_iv] = view;
    b.C->n_items = n_items;
    b.C->n_iv = n_iv;
    b.C->rtiles = ray;
    b.C->ftiles = view;
    b.C->rnext = 0;
    b.C->fnext = 0;
    b.C->error = s_err;
    if (error_out) *error_out = s_err;
    b.C->nfix = 0;
    b.C->nfixb = 0;
    b.C->samples = 0;
    b.C->marched = 0;
    b.C->slots = 0;
    b.C->pixels = (unsigned long long)pix;
    b.C->setup = 0;
  }
  // item tickets: views finished here count as arrived
  for (int item = threadIdx.x; item < n_items; item += blockDim.x) {
    unsigned pre = 0;
    for (int v = 0; v < nv; ++v) pre += __ldcg(&b.iv[item * nv + v].ok) ? 0u : 1u;
    b.itt[item] = pre;
    if (pre == (unsigned)nv) finish_item(sc, b, item, cost, view_cost_out);
  }
}

// ---------------------------------------------------------------- k_ray
#ifndef ASC_RAY_MINBLOCKS
#define ASC_RAY_MINBLOCKS 4  // 4 x 256 threads resident per SM (<= 64 registers)
#endif

// The scene of one (item, view) record's rays.
__device__ __forceinline__ RayScene ray_scene(const IV& r, const BoneDev& B, int skip)
{
  return RayScene{r.m, r.vp, df{r.sx[0], r.sx[1]}, df{r.sy[0], r.sy[1]}, B.step[r.slot],
                  skip ? B.clr[r.slot] : nullptr, r.w, r.h};
}

// The beams of the ray tiles, a warp each, from an atomic queue: a beam that
// meets nothing (beam_mask) writes zeros, the others are marched (ray_beam).
// shape: log2 of the width of a beam in its tile (2: 4 x 8 rays, 3: 8 x 4,
// 4: 16 x 2), the autotuner's choice.  A ray any of whose samples fell in
// the cutoff's band (march_block) leaves the mark -1 in its DRR pixel, and its
// beam goes on the fix list for k_ray_fix.
__global__ void __launch_bounds__(NRAY, ASC_RAY_MINBLOCKS) k_ray(const SceneDev* __restrict__ sc, Bufs b, int skip,
                                                                 int shape)
{
  __shared__ RaySlots<NRAY> S;
  const int lane = threadIdx.x & 31;
  const unsigned n = (unsigned)b.C->rtiles * BEAMS;
  unsigned long long marched = 0, slots = 0;
  unsigned next = 0;
  if (lane == 0) next = atomicAdd(&b.C->rnext, 1u);
  for (;;) {
    const unsigned id = __shfl_sync(FULL_WARP, next, 0);
    if (id >= n) break;
    if (lane == 0) next = atomicAdd(&b.C->rnext, 1u);  // taken while this beam is marched
    const int tile = (int)(id / BEAMS), k = b.rtile_iv[tile], t = tile - b.roff[k];
    const IV& r = b.iv[k];
    int x, y;
    beam_pixel((t % r.rtx) * RTX, (t / r.rtx) * RTY, (int)(id % BEAMS), shape, x, y);
    const bool valid = x < r.w && y < r.h;
    if (!__any_sync(FULL_WARP, valid)) continue;
    const BoneDev& B = sc->bones[r.bone];
    const RayScene s = ray_scene(r, B, skip);
    const Beam beam = beam_mask(B.vol, s, min(x, r.w - 1), min(y, r.h - 1));
    float* out = b.drr + r.pix + (long long)y * r.w + x;
    if (!beam.mask) {
      if (valid) *out = 0.f;
      continue;
    }
    unsigned done = 0, room = 0;
    const float d = ray_beam<1>(B.vol, s, B.cut[r.slot], make_float4(r.band[0], r.band[1], r.band[2], 0.f), S, x, y, valid,
                             beam, done, room);
    marched += done;
    slots += room;
    const bool flagged = valid && d != d;
    if (valid) *out = flagged ? -1.0f : fminf(fmaxf(d * B.scale[r.slot], 0.f), 1.f);
    if (__any_sync(FULL_WARP, flagged) && lane == 0) b.fixb[atomicAdd(&b.C->nfixb, 1)] = id;
  }
  for (int o = 16; o > 0; o >>= 1) marched += __shfl_xor_sync(FULL_WARP, marched, o);
  if (lane == 0 && slots) {
    atomicAdd(&b.C->marched, marched);
    atomicAdd(&b.C->slots, slots);
  }
}

// The marked rays of the beams on the fix list, marched again with every
// cutoff decision the exact one; each overwrites its mark.  Each takes a
// whole warp (march_exact), one after the other within a beam.
constexpr int FIX_THREADS = 128;
__global__ void __launch_bounds__(FIX_THREADS) k_ray_fix(const SceneDev* __restrict__ sc, Bufs b, int shape)
{
  __shared__ float s_v[FIX_THREADS / 32][EXACT_FLOATS];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5, n = b.C->nfixb;
  const int nw = gridDim.x * (FIX_THREADS / 32);
  for (int i = wib * gridDim.x + blockIdx.x; i < n; i += nw) {
    const unsigned id = b.fixb[i];
    const int tile = (int)(id / BEAMS), k = b.rtile_iv[tile], t = tile - b.roff[k];
    const IV& r = b.iv[k];
    int x, y;
    beam_pixel((t % r.rtx) * RTX, (t / r.rtx) * RTY, (int)(id % BEAMS), shape, x, y);
    const BoneDev& B = sc->bones[r.bone];
    const RayScene s = ray_scene(r, B, 0);
    unsigned m = __ballot_sync(FULL_WARP, x < r.w && y < r.h && b.drr[r.pix + (long long)y * r.w + x] < 0.f);
    if (lane == 0) atomicAdd(&b.C->nfix, __popc(m));
    for (; m; m &= m - 1) {
      const int rx = __shfl_sync(FULL_WARP, x, __ffs(m) - 1), ry = __shfl_sync(FULL_WARP, y, __ffs(m) - 1);
      const float d = march_exact(B.vol, s, B.cut[r.slot], rx, ry, s_v[wib]);
      if (lane == 0) b.drr[r.pix + (long long)ry * r.w + rx] = fminf(fmaxf(d * B.scale[r.slot], 0.f), 1.f);
    }
  }
}

// Trilinear samples of the reference's march over the last evaluation's
// crops, from their records (asc_engine_stats, asc_engine_counters): the
// evaluation itself sets up only the rays that meet an occupied interval.
__global__ void __launch_bounds__(NRAY) k_count_samples(Bufs b)
{
  unsigned long long n = 0;
  for (int tile = blockIdx.x; tile < b.C->rtiles; tile += gridDim.x) {
    const int k = b.rtile_iv[tile], t = tile - b.roff[k];
    const IV& r = b.iv[k];
    const int x = (t % r.rtx) * RTX + threadIdx.x % RTX, y = (t / r.rtx) * RTY + threadIdx.x / RTX;
    RaySetup rs;
    const bool hit = x < r.w && y < r.h && ray_setup(r.m, r.vp, x, y, df{r.sx[0], r.sx[1]}, df{r.sy[0], r.sy[1]},
                                                     r.step, r.nx, r.ny, r.nz, rs);
    n += __reduce_add_sync(FULL_WARP, hit ? (unsigned)rs.K : 0u);
  }
  if ((threadIdx.x & 31) == 0 && n) atomicAdd(&b.C->samples, n);
}

// ---------------------------------------------------------------- k_view
// A tile's region: region column rx, row ry <-> image (x0 + rx, y0 + ry),
// rows `P` floats apart.  The tile starts at column EX (a multiple of 4, so
// that four columns of the tile are 16 aligned bytes in every buffer) and row
// EY, the larger chain's halo.  `in`: the region that the chains read lies
// inside the image, and the stages skip every bounds test.
struct Region {
  int x0, y0, P, EX, EY, w, h;
  bool in;
};

__device__ __forceinline__ bool inside(const Region& g, int ry, int rx)
{
  int x = g.x0 + rx, y = g.y0 + ry;
  return x >= 0 && x < g.w && y >= 0 && y < g.h;
}

// A band of the region: the tile and `halo` pixels around it.
struct Band {
  int x0, x1, y0, y1;
};
__device__ __forceinline__ Band band(const Region& g, int halo)
{
  return Band{g.EX - halo, g.EX + VT + halo, g.EY - halo, g.EY + VT + halo};
}

// Calls f(ry, rx) for every position of a band, the positions dealt to the
// block's threads in row-major order (consecutive threads take consecutive
// columns, wrapping to the next row), so no lane idles on bands narrower or
// wider than a warp.
template <class F>
__device__ __forceinline__ void for_band(const Band& b, F&& f)
{
  const int bw = b.x1 - b.x0, n = bw * (b.y1 - b.y0);
  if (bw <= 0 || n <= 0) return;
  const int dq = VNT / bw, dr = VNT - dq * bw;
  int ry = (int)threadIdx.x / bw;
  int rx = (int)threadIdx.x - ry * bw;
  ry += b.y0;
  for (int i = threadIdx.x; i < n; i += VNT) {
    f(ry, b.x0 + rx);
    rx += dr;
    ry += dq;
    if (rx >= bw) {
      rx -= bw;
      ++ry;
    }
  }
}

// Calls f(ry, rx) for units of 4 columns of a row of a band (aligned, so up to
// 3 columns past the band on either side, whose results are not used), dealt
// to the threads in row-major order.  A unit is one row: taller ones load
// less, but their unrolled code runs once or twice a tile and waits for
// the instruction cache (units of 4 rows: 3.71 ms on 300 candidates x 2 views
// of 1024^2 with the four-filter chain, against 2.84).
template <class F>
__device__ __forceinline__ void for_units(const Band& b, F&& f)
{
  const int c0 = b.x0 >> 2;
  for_band(Band{c0, (b.x1 + 3) >> 2, b.y0, b.y1}, [&](int ry, int c) { f(ry, c << 2); });
}

__device__ __forceinline__ float4 lds4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float part(const float4& v, int i) { return i == 0 ? v.x : (i == 1 ? v.y : (i == 2 ? v.z : v.w)); }

// axy^e1 * v^e2 of ContrastFilter_kernels.cu (two powf there) as one exp2 of
// the summed logarithms; axy > 0.01 here.  v^0 is 1 for every v, as powf's.
__device__ __forceinline__ float contrast_pow(float axy, float v, float e1, float e2)
{
  float l = e1 * log2f(axy);
  if (e2 != 0.f) l = fmaf(e2, log2f(v), l);
  return exp2f(l);
}

__device__ __forceinline__ float contrast_px(float axy, float v, float e1, float e2)
{
  return axy > 0.01f ? contrast_pow(axy, v, e1, e2) : 0.0f;
}

__device__ __forceinline__ float clamp01(float v) { return fminf(fmaxf(v, 0.f), 1.f); }

// k_view's dynamic shared memory, in 4-byte words: 4 words that a unit's
// reads before a buffer's first row may touch, two stage buffers of P
// columns (run_chain), the VT x VT tile, then the region's per-column and per-row radiograph
// mapping (texel index and weight each).  halo: the larger chain's.
__host__ __device__ constexpr int view_ex(int halo) { return (halo + 3) & ~3; }
__host__ __device__ constexpr int view_pitch(int halo) { return VT + 2 * view_ex(halo); }
__host__ __device__ constexpr int view_rows(int halo) { return VT + 2 * halo; }
__host__ __device__ constexpr size_t view_tail_floats(int halo)
{
  return 4 + (size_t)2 * view_rows(halo) * view_pitch(halo) + (size_t)VT * VT;
}
__host__ __device__ constexpr size_t view_smem_floats(int halo)
{
  return view_tail_floats(halo) + (size_t)2 * (view_rows(halo) + view_pitch(halo));
}
// the widest chain an engine takes: three square stage buffers, the tile and
// ten words per row of the region in 224 KB (more than k_view needs)
__host__ __device__ constexpr bool view_fits(int halo)
{
  const size_t E = view_rows(halo);
  return (3 * E * E + (size_t)VT * VT + 10 * E) * 4 <= 224 * 1024;
}
static_assert(view_fits(42) && !view_fits(43) && view_smem_floats(42) * 4 + 2048 <= 227 * 1024,
              "the widest chain fits a block's shared memory");
constexpr int kNoTexel = -0x7fffffff;  // a column or row that maps outside the radiograph

// Gaussian (kind 3) or Sharpen (kind 4) with a K-tap kernel: the 1-D weights
// in registers, a horizontal pass into `tmp`, then a vertical pass, 4 columns
// at a time in 16-byte words.  Each output adds its taps in order.  Positions
// outside the image hold 0 in every stage buffer, which is the reference's
// skipping of out-of-image taps.
template <int K>
__device__ void blur_stage(const FilterDev& f, const float* in, float* out, float* tmp, const Region& g, int halo)
{
  constexpr int R = K / 2, Q = (R + 3) / 4, NV = 2 * Q + 1;  // words on either side, words of a unit's reads
  const int P = g.P;
  float w[K];
#pragma unroll
  for (int k = 0; k < K; ++k) w[k] = f.g[k];
  const Band b = band(g, halo);
  for_units(Band{b.x0, b.x1, b.y0 - R, b.y1 + R}, [&](int ry, int rx) {
    const float* p = in + ry * P + rx - 4 * Q;
    float v[4 * NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const float4 q = lds4(p + 4 * i);
      v[4 * i] = q.x;
      v[4 * i + 1] = q.y;
      v[4 * i + 2] = q.z;
      v[4 * i + 3] = q.w;
    }
    float s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int k = 0; k < K; ++k)
#pragma unroll
      for (int i = 0; i < 4; ++i) s[i] = fmaf(w[k], v[4 * Q - R + i + k], s[i]);
    *reinterpret_cast<float4*>(tmp + ry * P + rx) = make_float4(s[0], s[1], s[2], s[3]);
  });
  __syncthreads();
  const bool gauss = f.kind == 3;
  const float p1 = f.p1, p2 = f.p2;
  for_units(b, [&](int ry, int rx) {
    float s[4] = {0.f, 0.f, 0.f, 0.f};
    const float* p = tmp + (ry - R) * P + rx;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const float4 q = lds4(p + k * P);
      s[0] = fmaf(w[k], q.x, s[0]);
      s[1] = fmaf(w[k], q.y, s[1]);
      s[2] = fmaf(w[k], q.z, s[2]);
      s[3] = fmaf(w[k], q.w, s[3]);
    }
    if (gauss) {
#pragma unroll
      for (int i = 0; i < 4; ++i) s[i] = clamp01(s[i]);
    } else {
      const float4 q = lds4(in + ry * P + rx);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float v = part(q, i), blur = s[i];
        s[i] = fabsf(v - blur) > p2 ? clamp01(v + p1 * (v - blur)) : v;
      }
    }
    if (!g.in)
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (!inside(g, ry, rx + i)) s[i] = 0.f;
    *reinterpret_cast<float4*>(out + ry * P + rx) = make_float4(s[0], s[1], s[2], s[3]);
  });
}

// Any kernel size: per-element passes with the weights in shared memory.
__device__ void blur_stage_any(const FilterDev& f, const float* in, float* out, float* tmp, float* wsh,
                               const Region& g, int halo)
{
  const int P = g.P, K = f.K, R = f.R;
  const float p1 = f.p1, p2 = f.p2;
  if (threadIdx.x < K) wsh[threadIdx.x] = f.g[threadIdx.x];
  __syncthreads();
  const Band b = band(g, halo);
  for_band(Band{b.x0, b.x1, b.y0 - R, b.y1 + R}, [&](int ry, int rx) {
    const float* p = in + ry * P + rx - R;
    float sum = 0.f;
    for (int k = 0; k < K; ++k) sum = fmaf(wsh[k], p[k], sum);
    tmp[ry * P + rx] = sum;
  });
  __syncthreads();
  for_band(b, [&](int ry, int rx) {
    float r = 0.f;
    if (g.in || inside(g, ry, rx)) {
      const float* p = tmp + (ry - R) * P + rx;
      float blur = 0.f;
      for (int k = 0; k < K; ++k) blur = fmaf(wsh[k], p[k * P], blur);
      if (f.kind == 3) {
        r = clamp01(blur);
      } else {
        const float v = in[ry * P + rx];
        r = fabsf(v - blur) > p2 ? clamp01(v + p1 * (v - blur)) : v;
      }
    }
    out[ry * P + rx] = r;
  });
}

// SobelFilter_kernels.cu:63-113 at one pixel from its 3 x 3 neighbourhood.
__device__ __forceinline__ float sobel_px(float p00, float p01, float p02, float p10, float p11, float p12, float p20,
                                          float p21, float p22, float scale, float blend)
{
  const float horz = p02 + 2 * p12 + p22 - p00 - 2 * p10 - p20;
  const float vert = p00 + 2 * p01 + p02 - p20 - 2 * p21 - p22;
  const float grad = sqrtf(horz * horz + vert * vert);
  const float s = blend < 0.5f ? scale * grad + 2.0f * blend * p11 : 2.0f * (1.0f - blend) * scale * grad + p11;
  return clamp01(s);
}

// The six columns rx - 1 .. rx + 4 of row p (p: column rx).
__device__ __forceinline__ void six(const float* p, float* v)
{
  const float4 c = lds4(p);
  v[0] = p[-1];
  v[1] = c.x;
  v[2] = c.y;
  v[3] = c.z;
  v[4] = c.w;
  v[5] = p[4];
}

// Applies one filter from `in` to `out` (a blur: may be `in`) over the band of
// the tile and `halo` pixels around it; positions outside the image get 0.
// `tmp` holds the horizontal pass of a Gaussian/Sharpen blur, `wsh` the 1-D weights of a blur
// of uncommon size.
__device__ void apply_stage(const FilterDev& f, const float* in, float* out, float* tmp, float* wsh, const Region& g,
                            int halo)
{
  const int P = g.P;
  const int kind = f.kind, K = f.K;
  const float p0 = f.p0, p1 = f.p1;
  if (kind == 3 || kind == 4) {
    switch (K) {
      case 3: blur_stage<3>(f, in, out, tmp, g, halo); break;
      case 5: blur_stage<5>(f, in, out, tmp, g, halo); break;
      case 7: blur_stage<7>(f, in, out, tmp, g, halo); break;
      case 9: blur_stage<9>(f, in, out, tmp, g, halo); break;
      case 11: blur_stage<11>(f, in, out, tmp, g, halo); break;
      case 13: blur_stage<13>(f, in, out, tmp, g, halo); break;
      default: blur_stage_any(f, in, out, tmp, wsh, g, halo);
    }
  } else if (kind == 1) {
    for_units(band(g, halo), [&](int ry, int rx) {
      const float* p = in + ry * P + rx;
      float u[6], m[6], d[6], o[4];
      six(p - P, u);
      six(p, m);
      six(p + P, d);
#pragma unroll
      for (int i = 0; i < 4; ++i)
        o[i] = sobel_px(u[i], u[i + 1], u[i + 2], m[i], m[i + 1], m[i + 2], d[i], d[i + 1], d[i + 2], p0, p1);
      if (!g.in)
#pragma unroll 1
        for (int i = 0; i < 4; ++i) {
          const int y = g.y0 + ry, x = g.x0 + rx + i;
          if (x > 0 && x < g.w - 1 && y > 0 && y < g.h - 1) continue;
          float r = 0.f;
          if (x >= 0 && x < g.w && y >= 0 && y < g.h) {
            // image border: neighbours outside the image repeat the edge
            const int xm = x > 0 ? -1 : 0, xp = x < g.w - 1 ? 1 : 0, ym = y > 0 ? -P : 0, yp = y < g.h - 1 ? P : 0;
            const float* c = p + i;
            r = sobel_px(c[ym + xm], c[ym], c[ym + xp], c[xm], c[0], c[xp], c[yp + xm], c[yp], c[yp + xp], p0, p1);
          }
          if (i == 0) o[0] = r;
          if (i == 1) o[1] = r;
          if (i == 2) o[2] = r;
          if (i == 3) o[3] = r;
        }
      *reinterpret_cast<float4*>(out + ry * P + rx) = make_float4(o[0], o[1], o[2], o[3]);
    });
  } else if (kind == 0 && K == 3) {
    // ContrastFilter_kernels.cu:62-96 with a 3 x 3 box: the mean over the
    // window's in-image pixels (out-of-image positions hold 0, so the sum
    // runs over the whole window and only the count depends on the border)
    const float e1 = p0 - p1, e2 = p1;
    for_units(band(g, halo), [&](int ry, int rx) {
      const float* p = in + ry * P + rx;
      float u[6], m[6], d[6], o[4];
      six(p - P, u);
      six(p, m);
      six(p + P, d);
#pragma unroll
      for (int i = 0; i < 4; ++i)
        o[i] = (u[i] + u[i + 1] + u[i + 2]) + (m[i] + m[i + 1] + m[i + 2]) + (d[i] + d[i + 1] + d[i + 2]);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float axy = ninth(o[i]);
        if (!g.in) {
          const int y = g.y0 + ry, x = g.x0 + rx + i;
          if (!(x > 0 && x < g.w - 1 && y > 0 && y < g.h - 1)) {
            const bool at = x >= 0 && x < g.w && y >= 0 && y < g.h;
            const int cnt = (min(y + 2, g.h) - max(y - 1, 0)) * (min(x + 2, g.w) - max(x - 1, 0));
            axy = at ? o[i] / (float)cnt : 0.f;
          }
        }
        o[i] = contrast_px(axy, m[i + 1], e1, e2);
      }
      *reinterpret_cast<float4*>(out + ry * P + rx) = make_float4(o[0], o[1], o[2], o[3]);
    });
  } else if (kind == 0) {
    const int size = K, h0 = size / 2, h1 = (size + 1) / 2;
    const float e1 = p0 - p1, e2 = p1;
    for_band(band(g, halo), [&](int ry, int rx) {
      float r = 0.f;
      if (g.in || inside(g, ry, rx)) {
        const int x = g.x0 + rx, y = g.y0 + ry;
        const int i0 = max(y - h0, 0), i1 = min(y + h1, g.h);
        const int j0 = max(x - h0, 0), j1 = min(x + h1, g.w);
        float cnt = 0.f, sum = 0.f;
        for (int yy = i0; yy < i1; ++yy)
          for (int xx = j0; xx < j1; ++xx) {
            cnt += 1.0f;
            sum += in[(yy - g.y0) * P + (xx - g.x0)];
          }
        const float axy = sum / cnt, v = in[ry * P + rx];
        r = axy > 0.01f ? contrast_pow(axy, v, e1, e2) : 0.0f;
      }
      out[ry * P + rx] = r;
    });
  }
  __syncthreads();
}

// Runs a filter chain on the first of two stage buffers of `size` floats
// each (valid on the tile and its halo H); returns the one holding the result on the tile.
// Sobel and Contrast go from one buffer to the other; a blur's horizontal pass
// does, and its vertical pass, which reads the stage's input at the pixel
// itself alone, comes back into the input's.  (A third buffer would take a
// resident block from chains of halo 13 and more, and at 22 the last but one.)
// Not inlined: both chains of a tile run the same code, which with it fits the instruction cache.
__device__ __noinline__ float* run_chain(const FilterDev* fl, int nf, int H, float* buf, int size, float* wsh, Region g)
{
  int halo = H;
  float *in = buf, *other = buf + size;
  for (int s = 0; s < nf; ++s) {
    const bool blur = fl[s].kind == 3 || fl[s].kind == 4;
    halo -= fl[s].R;
    apply_stage(fl[s], in, blur ? in : other, other, wsh, g, halo);
    if (!blur) {
      float* t = in;
      in = other;
      other = t;
    }
  }
  return in;
}

// Calls f(i, ly, lx) for the tile's pixels, i = ly VT + lx, thread t taking t,
// t + VNT, ...
template <class F>
__device__ __forceinline__ void for_tile(F&& f)
{
  int ly = threadIdx.x / VT, lx = threadIdx.x % VT;
#pragma unroll 1
  for (int i = threadIdx.x; i < VT * VT; i += VNT) {
    f(i, ly, lx);
    lx += VNT % VT;
    ly += VNT / VT;
    if (lx >= VT) {
      lx -= VT;
      ++ly;
    }
  }
}

// The radiograph crop (RadRenderer_kernels.cu:85-116) over the tile and the
// chain's halo, four pixels at a time so that sixteen texels are in flight;
// 0 outside the image and where a pixel maps outside the radiograph.  The
// texels and the interpolation are bilinear_at's.
template <class T>
__device__ __forceinline__ void rad_band(const T* __restrict__ rad, float scale, int W, int Hr, const Region& g,
                                         int halo, const int* tcx, const float* tax, const int* tcy, const float* tay,
                                         float* out)
{
  for_units(band(g, halo), [&](int ry, int rx) {
    const int ky = tcy[ry];
    const bool row = ky != kNoTexel && (g.in || (g.y0 + ry >= 0 && g.y0 + ry < g.h));
    const float ay = tay[ry];
    const T *ra = rad + (size_t)min(max(ky, 0), Hr - 1) * W, *rb = rad + (size_t)min(max(ky + 1, 0), Hr - 1) * W;
    float o[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int kx = tcx[rx + i];
      const bool at = row && kx != kNoTexel && (g.in || (g.x0 + rx + i >= 0 && g.x0 + rx + i < g.w));
      o[i] = 0.f;
      if (at) {
        const int xa = min(max(kx, 0), W - 1), xb = min(max(kx + 1, 0), W - 1);
        const float ax = tax[rx + i];
        // rounded before they are used, as image_texel's are
        const float v00 = __fmul_rn(__ldg(ra + xa), scale), v01 = __fmul_rn(__ldg(ra + xb), scale);
        const float v10 = __fmul_rn(__ldg(rb + xa), scale), v11 = __fmul_rn(__ldg(rb + xb), scale);
        const float r0 = fmaf(ax, v01 - v00, v00), r1 = fmaf(ax, v11 - v10, v10);
        o[i] = 1.0f - fmaf(ay, r1 - r0, r0);
      }
    }
    *reinterpret_cast<float4*>(out + ry * g.P + rx) = make_float4(o[0], o[1], o[2], o[3]);
  });
}

// BackgroundRenderer's mask (BackgroundRenderer_kernels.cu:88-120) over the
// tile's DRR: 0 where the background image lies below its threshold.  The
// film-plane mapping once per column and row, in FP64, as the radiograph's and
// in its tables (free after its chain's barriers): per pixel it was half of
// the kernel (64 candidates under SAD at 771 x 645 with a background: 980 us
// with k_sad, 447 here).  A call: inlined, tiles without a background lost 2 %
// to spilled registers.
__device__ __noinline__ void background_mask(const ViewDev& V, const IV& r, const double* rcp, Region g, float* fdrr)
{
  extern __shared__ float smem[];
  int* tcx = (int*)(smem + view_tail_floats(g.EY));
  float* tax = (float*)(tcx + VT);
  int* tcy = (int*)(tax + VT);
  float* tay = (float*)(tcy + VT);
  const int x0 = g.x0 + g.EX, y0 = g.y0 + g.EY;
  for (int i = threadIdx.x; i < 2 * VT; i += VNT) {
    const bool row = i >= VT;
    const int j = row ? i - VT : i;
    int q;
    float a = 0.f;
    const bool ok = row ? image_axis(r.vp[1], r.vp[3], y0 + j, r.h, rcp[1], V.ipf[1], V.ipf[3], rcp[3], V.bg_h, true, q, a)
                        : image_axis(r.vp[0], r.vp[2], x0 + j, r.w, rcp[0], V.ipf[0], V.ipf[2], rcp[2], V.bg_w, false, q, a);
    (row ? tcy : tcx)[j] = ok ? q : kNoTexel;
    (row ? tay : tax)[j] = a;
  }
  __syncthreads();
  // the words that this thread's pass over the masks reads
  for_tile([&](int i, int ly, int lx) {
    const int kx = tcx[lx], ky = tcy[ly];
    if (fdrr[i] != 0.0f && !(kx != kNoTexel && ky != kNoTexel &&
                             V.bg_thr <= bilinear_at(V.bg, 32, V.bg_w, V.bg_h, kx, tax[lx], ky, tay[ly])))
      fdrr[i] = 0.0f;
  });
}

// One 48 x 48 output tile after another from a queue.  What bounds it is
// instruction issue (60 %) and, at 24 warps per SM, the barriers between its
// stages.  On 300 candidates x 2 views of 1024^2 with the four-filter chain:
// 3.58 ms with one column per unit and the FP64 quotients by division, 2.84
// with four columns, 2.63 with the radiograph's texels fetched sixteen at a
// time and the masked pixels kept by their value instead of a flag; one
// candidate of two 256^2 views (latency alone: FP64 chains of one warp,
// round trips to L2, code met for the first time): 61 and 50 us by the moments'
// fields dealt to lanes.  The last thread grabs the next tile while this one is
// filtered, and warp 0 alone finishes a tile (its FP64 moments, the view's
// merge, the item's cost) while the other warps go on to the next.
__global__ void __launch_bounds__(VNT, ASC_VIEW_MINBLOCKS)
    k_view(const SceneDev* __restrict__ sc, Bufs b, double* __restrict__ cost, double* __restrict__ view_cost_out)
{
  extern __shared__ float smem[];
  __shared__ int s_tile[2], s_k[2];  // this tile's and the next one's
  __shared__ float red[8 * 6 * 2];
  __shared__ double ds[6], dc[3];
  __shared__ float s_mean[2];
  __shared__ double s_rcp[4];  // 1 / w, 1 / h of the crop; 1 / the image's width and height on the film plane
  __shared__ float wsh[32];
  __shared__ unsigned s_keep[VNT / 32];
  const int ns = sc->slots, ftiles = b.C->ftiles;
  const bool grabs = threadIdx.x == VNT - 1;
  if (grabs) {
    const int tl = atomicAdd(&b.C->fnext, 1);
    s_tile[0] = tl;
    s_k[0] = tl < ftiles ? b.ftile_iv[tl] : 0;
  }
  __syncthreads();
  for (int turn = 0;; turn ^= 1) {
    const int tile = s_tile[turn], k = s_k[turn];
    if (tile >= ftiles) return;
    int next = 0, next_k = 0;
    if (grabs) {
      next = atomicAdd(&b.C->fnext, 1);
      next_k = next < ftiles ? b.ftile_iv[next] : 0;
    }
    const IV& r = b.iv[k];
    const int t = tile - b.foff[k];
    const int tx0 = (t % r.ftx) * VT, ty0 = (t / r.ftx) * VT;
    const ViewDev& V = sc->views[r.view];
    // this view's halo lays out the shared memory
    const int H = max(V.h_drr, V.h_rad), EX = view_ex(H), P = view_pitch(H), rows = view_rows(H);
    const int size = rows * P;
    float* buf = smem + 4;           // two stage buffers
    float* fdrr = buf + 2 * size;  // VT x VT final DRR, then f = DRR * mask
    // per region column / row: the radiograph texel pair and weight of the
    // film-plane mapping (image_axis; kNoTexel where the pixel maps outside)
    int* tcx = (int*)(smem + view_tail_floats(H));
    float* tax = (float*)(tcx + P);
    int* tcy = (int*)(tax + P);
    float* tay = (float*)(tcy + rows);
    const int rx0 = tx0 - EX, ry0 = ty0 - H;
    const Region g{rx0, ry0, P, EX, H, r.w, r.h, tx0 >= H && ry0 >= 0 && tx0 + VT + H <= r.w && ry0 + rows <= r.h};
    const float* drr = b.drr + r.pix;
    // ---- DRR region; a region of zeros filters to zeros (every filter maps
    // 0 to 0), so its tile masks out entirely and adds nothing to the moments
    bool live;
    {
      // the region's words copied asynchronously (all in flight at once;
      // zero-filled outside the image), then tested for a nonzero DRR
      const Band d = band(g, V.h_drr);
      for_band(d, [&](int ry, int rx) {
        const bool in = g.in || inside(g, ry, rx);
        const float* src = in ? drr + (long long)(g.y0 + ry) * g.w + g.x0 + rx : drr;
        const unsigned dst = (unsigned)__cvta_generic_to_shared(buf + ry * P + rx);
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(dst), "l"(src), "r"(in ? 4 : 0)
                     : "memory");
      });
      asm volatile("cp.async.commit_group;\n" ::: "memory");
      // meanwhile the reciprocals of the mapping's divisors
      if (threadIdx.x < 4) {
        const double v = threadIdx.x == 0 ? (double)r.w
                                          : (threadIdx.x == 1 ? (double)r.h : (double)V.ipf[threadIdx.x == 2 ? 2 : 3]);
        s_rcp[threadIdx.x] = reciprocal(v);
      }
      asm volatile("cp.async.wait_group 0;\n" ::: "memory");
      if (grabs) {  // for after this tile's last barrier
        s_tile[turn ^ 1] = next;
        s_k[turn ^ 1] = next_k;
      }
      bool nz = false;  // of the words that this thread copied
      for_band(d, [&](int ry, int rx) { nz |= buf[ry * P + rx] != 0.f; });
      live = __syncthreads_or(nz);
    }
    float mf = 0.f, mg = 0.f;
    if (live) {
      // the film-plane mapping of the region's columns and rows, in FP64
      // (visible to the radiograph band after the chain's barriers)
      for (int i = threadIdx.x; i < P + rows; i += VNT) {
        const bool row = i >= P;
        const int j = row ? i - P : i;
        int q;
        float a = 0.f;
        const bool ok = row ? image_axis(r.vp[1], r.vp[3], g.y0 + j, r.h, s_rcp[1], V.ipf[1], V.ipf[3], s_rcp[3], V.rad_h,
                                         true, q, a)
                            : image_axis(r.vp[0], r.vp[2], g.x0 + j, r.w, s_rcp[0], V.ipf[0], V.ipf[2], s_rcp[2], V.rad_w,
                                         false, q, a);
        (row ? tcy : tcx)[j] = ok ? q : kNoTexel;
        (row ? tay : tax)[j] = a;
      }
      // ---- DRR chain
      {
        const float* res = run_chain(V.fdrr, V.n_drr, V.h_drr, buf, size, wsh, g) + H * P + EX;
        for (int i = threadIdx.x; i < VT * VT / 4; i += VNT) {
          const int ly = i / (VT / 4), lx = 4 * (i % (VT / 4));
          *reinterpret_cast<float4*>(fdrr + ly * VT + lx) = lds4(res + ly * P + lx);
        }
        __syncthreads();
      }
      // ---- radiograph crop and its chain
      float* gres;
      {
        if (V.rad_bps == 16)
          rad_band((const unsigned short*)V.rad, 1.0f / 65535.0f, V.rad_w, V.rad_h, g, V.h_rad, tcx, tax, tcy, tay, buf);
        else
          rad_band((const unsigned char*)V.rad, 1.0f / 255.0f, V.rad_w, V.rad_h, g, V.h_rad, tcx, tax, tcy, tay, buf);
        __syncthreads();
        gres = run_chain(V.frad, V.n_rad, V.h_rad, buf, size, wsh, g) + H * P + EX;
      }
      // ---- masks and moments (Tracker.cpp:744-770), two passes over the
      // tile: f = DRR * mask over fdrr, g = rad * mask over the chain result
      const unsigned n = (unsigned)g.w * (unsigned)g.h;
      const bool tree = sc->coverage == ASC_SUM_TREE && tree_needed(n);  // else every pixel counts
      int shift = 0;
      if (tree) {
        shift = tree_mask(n, s_keep);
        __syncthreads();
      }
      const bool sad = sc->cf_model != 0;
      // per tile: the pixels with mask 1 and their sums of f and g.  The
      // mask is 0 or 1 and f, g are 0 where it is 0, so these are also the
      // covered pixels' sums of mask, f and g, and a pixel with f != 0 is one
      // under the mask.  Plain FP32 suffices for them: an error in a tile's
      // mean moves the centred moments only at second order; the products are
      // the sums that need compensating.
      if (V.bg && V.bg_thr >= 0.f) background_mask(V, r, s_rcp, g, fdrr);
      float2* fg = b.fg + r.pix;
      float s[3] = {0.f, 0.f, 0.f};
      for_tile([&](int i, int ly, int lx) {
        const int x = tx0 + lx, y = ty0 + ly;
        float f = 0.f, gm = 0.f;
        const bool at = x < g.w && y < g.h;
        if (at && (!tree || tree_kept(s_keep, (unsigned)(y * g.w + x), shift))) {
          const float d = fdrr[i], gg = gres[ly * P + lx];
          const float m = d != 0.0f ? 1.0f : 0.0f;
          f = d * m;
          gm = gg * m;
          if (m > 0.5f) {
            s[0] += 1.f;
            s[1] += f;
            s[2] += gm;
          }
        }
        fdrr[i] = f;
        gres[ly * P + lx] = gm;
        // SAD needs the view's global means first: keep f and g for k_sad
        if (sad && at) fg[(long long)y * g.w + x] = make_float2(f, gm);
      });
      // the sums, and the tile's FP32 centres from them
      block_means(s, red, ds + 3, s_mean);
      mf = s_mean[0];
      mg = s_mean[1];
      DFs c[3] = {};  // compensated co-moments about (mf, mg)
      if (!sad)
        for_tile([&](int i, int ly, int lx) {
          const float f = fdrr[i];
          if (f == 0.f) return;
          const float a = f - mf, bb = gres[ly * P + lx] - mg;
          dfs_add_prod(c[0], a, a);
          dfs_add_prod(c[1], bb, bb);
          dfs_add_prod(c[2], a, bb);
        });
      if (threadIdx.x < 3) ds[threadIdx.x] = ds[3 + threadIdx.x];  // read past the next barrier
      block_sum_dfs<3>(c, red, dc);
    }
    if (threadIdx.x >= 32) continue;
    // ---- warp 0: the tile's moments; the last tile of a view merges its
    // tiles, the last view of an item sums the view costs
    const int lane = threadIdx.x, nt = r.ftx * r.fty;
    bool last = false;
    if (live)
      tile_moments(ds, dc, mf, mg, b.part + tile);
    else if (lane < 9)
      ((double*)(b.part + tile))[lane] = 0.0;  // zeros add nothing
    __threadfence();
    __syncwarp();
    if (lane == 0) {
      last = atomicAdd(&b.ivt[k], 1u) == (unsigned)nt - 1;
    }
    if (!__shfl_sync(FULL_WARP, (int)last, 0)) continue;
    __threadfence();
    const Moments m = merge_moments(b.part + b.foff[k], nt);
    if (lane != 0) continue;
    if (sc->cf_model) {
      // HDist_kernels.cu:111-115: the means over the mask sum; k_sad takes
      // the view from here and reuses its tile tickets
      b.hmean[k] = make_double2(m.sf / m.sm, m.sg / m.sm);
      b.ivt[k] = 0;
      continue;
    }
    b.vcost[k] = 1.0 - moments_ncc(m);
    __threadfence();
    const int item = k / ns;
    if (atomicAdd(&b.itt[item], 1u) == (unsigned)ns - 1) {
      __threadfence();
      finish_item(sc, b, item, cost, view_cost_out);
    }
  }
}

// ---------------------------------------------------------------- k_sad
// cf_model 1 (HDist_kernels.cu:111-203): per view, sum over mask > 0.5 of
// |(f - mean f) - (g - mean g)| with the means k_view left in hmean.  The
// mask is 0 or 1 and a DRR pixel under it is non-zero, so f != 0 marks the
// pixels under the mask; tiles k_view found without such pixels are skipped.
// Tile partials in FP32, the view's sum in FP64 by the view's last tile.
__global__ void __launch_bounds__(256) k_sad(const SceneDev* __restrict__ sc, Bufs b, double* __restrict__ cost,
                                             double* __restrict__ view_cost_out)
{
  __shared__ float red[8];
  __shared__ double dred[8];
  __shared__ bool s_last;
  const int nv = sc->slots, ftiles = b.C->ftiles;
  for (int tile = blockIdx.x; tile < ftiles; tile += gridDim.x) {
    const int k = b.ftile_iv[tile];
    const IV& r = b.iv[k];
    const int t = tile - b.foff[k];
    const int tx0 = (t % r.ftx) * VT, ty0 = (t / r.ftx) * VT;
    float a = 0.f;
    if (b.part[tile].n > 0) {
      const double2 mu = b.hmean[k];
      const float mf = (float)mu.x, mg = (float)mu.y;
      for (int i = threadIdx.x; i < VT * VT; i += blockDim.x) {
        const int x = tx0 + i % VT, y = ty0 + i / VT;
        if (x < r.w && y < r.h) {
          const float2 v = b.fg[r.pix + (long long)y * r.w + x];
          if (v.x != 0.f) a += fabsf((v.x - mf) - (v.y - mg));
        }
      }
    }
    for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = a;
    __syncthreads();
    if (threadIdx.x == 0) {
      float tot = 0.f;
      for (int w = 0; w < (int)(blockDim.x >> 5); ++w) tot += red[w];
      b.tsad[tile] = tot;
      __threadfence();
      s_last = atomicAdd(&b.ivt[k], 1u) == (unsigned)(r.ftx * r.fty) - 1;
    }
    __syncthreads();
    if (s_last) {
      __threadfence();
      const int nt = r.ftx * r.fty, base = b.foff[k];
      double d = 0.0;
      for (int i = threadIdx.x; i < nt; i += blockDim.x) d += (double)__ldcg(b.tsad + base + i);
      for (int o = 16; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
      if ((threadIdx.x & 31) == 0) dred[threadIdx.x >> 5] = d;
      __syncthreads();
      if (threadIdx.x == 0) {
        double vc = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) vc += dred[w];
        b.vcost[k] = vc;
        __threadfence();
        const int item = k / nv;
        if (atomicAdd(&b.itt[item], 1u) == (unsigned)nv - 1) {
          __threadfence();
          finish_item(sc, b, item, cost, view_cost_out);
        }
      }
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------- PSO
struct Swarm {
  double* x;    // [bone][particle][6]
  double* v;
  double* pbx;
  double* pbc;
  double* gx;   // [bone][6]
  double* gc;   // [bone]
  int* iter;
  int* frozen;  // [bone] the swarm stalled: its particles stay put
  int* bone;    // item -> bone
  double* manip;  // item -> x
};

__device__ __forceinline__ double urand(unsigned long long seed, unsigned long long ctr)
{
  unsigned long long z = seed + 0x9e3779b97f4a7c15ull * (ctr + 1);
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  z ^= z >> 31;
  return (double)(z >> 11) * (1.0 / 9007199254740992.0);
}

__global__ void k_pso_init(Swarm s, int nb, int np, double lo, double hi, unsigned long long seed)
{
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nb * np) return;
  int p = i % np;
  for (int d = 0; d < 6; ++d) {
    double x = p == 0 ? 0.0 : lo + urand(seed, (unsigned long long)i * 6 + d) * (hi - lo);
    s.x[6 * i + d] = x;
    s.v[6 * i + d] = 0.0;
    s.pbx[6 * i + d] = x;
  }
  s.pbc[i] = 1e300;
  if (p == 0) {
    int b = i / np;
    for (int d = 0; d < 6; ++d) s.gx[6 * b + d] = 0.0;
    s.gc[b] = 1e300;
    s.frozen[b] = 0;
  }
  if (i == 0) *s.iter = 0;
}

// Synchronous velocity/position update (the rule of PSO.cpp:83-109 with
// runtime w, c1, c2) for every particle of every swarm.
__global__ void k_pso_update(Swarm s, int nb, int np, double w, double c1, double c2, unsigned long long seed)
{
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nb * np) return;
  int b = i / np;
  s.bone[i] = b;
  if (s.frozen[b]) {  // re-scored where it is: the same cost, no best changes
    for (int d = 0; d < 6; ++d) s.manip[6 * i + d] = s.x[6 * i + d];
    return;
  }
  unsigned long long it = (unsigned long long)*s.iter + 1;
  for (int d = 0; d < 6; ++d) {
    unsigned long long c = ((it * (unsigned long long)(nb * np) + i) * 6 + d) * 2;
    double rp = urand(seed, c), rg = urand(seed, c + 1);
    double x = s.x[6 * i + d];
    double vv = w * s.v[6 * i + d] + c1 * rp * (s.pbx[6 * i + d] - x) + c2 * rg * (s.gx[6 * b + d] - x);
    s.v[6 * i + d] = vv;
    s.x[6 * i + d] = x + vv;
    s.manip[6 * i + d] = x + vv;
  }
}

// pBest / gBest update after an iteration's costs (one block per swarm).
__global__ void k_pso_best(Swarm s, int nb, int np, const double* cost)
{
  int b = blockIdx.x;
  __shared__ double bc[256];
  __shared__ int bi[256];
  double best = 1e300;
  int arg = -1;
  for (int p = threadIdx.x; p < np; p += blockDim.x) {
    int i = b * np + p;
    double c = cost[i];
    if (c < s.pbc[i]) {
      s.pbc[i] = c;
      for (int d = 0; d < 6; ++d) s.pbx[6 * i + d] = s.x[6 * i + d];
    }
    if (c < best || (c == best && arg >= 0 && p < arg)) {
      best = c;
      arg = p;
    }
  }
  bc[threadIdx.x] = best;
  bi[threadIdx.x] = arg;
  __syncthreads();
  for (int st = blockDim.x / 2; st > 0; st >>= 1) {
    if (threadIdx.x < st) {
      double o = bc[threadIdx.x + st];
      int oi = bi[threadIdx.x + st];
      if (o < bc[threadIdx.x] || (o == bc[threadIdx.x] && oi >= 0 && (bi[threadIdx.x] < 0 || oi < bi[threadIdx.x]))) {
        bc[threadIdx.x] = o;
        bi[threadIdx.x] = oi;
      }
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    if (bi[0] >= 0 && bc[0] < s.gc[b]) {
      s.gc[b] = bc[0];
      for (int d = 0; d < 6; ++d) s.gx[6 * b + d] = s.x[6 * (b * np + bi[0]) + d];
    }
    if (b == 0) *s.iter += 1;
  }
}

}  // namespace

// ---------------------------------------------------------------- host side

// asc_engine_eval_host's staging, pinned host memory sized for max_items.
struct HostIO {
  void* base = nullptr;
  double *manip = nullptr, *cost = nullptr, *vcost = nullptr;
  int *bone = nullptr, *error = nullptr;
};

// What the captured swarm iteration holds as launch arguments.
struct SwarmKey {
  int particles, skip;
  double w, c1, c2;
  uint64_t seed;
  // a NaN setting matches nothing and is captured anew
  bool operator==(const SwarmKey& o) const
  {
    return particles == o.particles && skip == o.skip && w == o.w && c1 == o.c1 && c2 == o.c2 && seed == o.seed;
  }
};

struct asc_engine_s {
  SceneDev host;
  SceneDev* dev = nullptr;
  int max_items = 0, n_views = 0, n_bones = 0;
  Bufs b{};
  size_t smem = 0;
  int sms = 152;
  int view_blocks = 1;  // resident k_view blocks per SM (the occupancy limit)
  // launch shapes (asc_engine_set_launch): the defaults, or the tuning
  // table's entry for this engine's workload class
  asc_launch_config launch{ASC_RAY_MINBLOCKS, 0, 3};
  // k_view blocks per SM: the configured count, at most the occupancy limit
  int view_grid() const
  {
    const int want = launch.view_blocks_per_sm;
    return want > 0 ? std::min(want, view_blocks) : view_blocks;
  }
  bool prof = false;
  cudaEvent_t ev[4] = {nullptr, nullptr, nullptr, nullptr};
  // after the last asc_engine_eval on a stream of the caller's: what reads
  // the counters waits for it (the other evaluations end in a wait)
  cudaEvent_t done = nullptr;
  // device PSO: swarm state, the captured iteration and a private stream
  double* sw_buf = nullptr;
  int* sw_iter = nullptr;
  int* sw_frozen = nullptr;
  cudaGraphExec_t pso_exec = nullptr;
  SwarmKey pso_key{};
  cudaStream_t own_stream = nullptr;
  int* d_bone = nullptr;
  double* d_manip = nullptr;
  double* d_cost = nullptr;
  HostIO io;
  // plain per-pose path: the reference's Tracker buffers (Tracker.cpp:292-298)
  std::vector<asc_view_desc> vdesc;
  std::vector<asc_bone_desc> bdesc;
  float *p_drr = nullptr, *p_rad = nullptr, *p_mask = nullptr, *p_tmp = nullptr, *p_bgr = nullptr;
  double* p_res = nullptr;
  std::vector<void*> allocs;
  // clearance grids of bones replaced by asc_engine_set_bone, per (bone,
  // slot), with their capacity in bytes
  uint8_t* clr_own[MAX_BONES][MAX_SLOTS] = {};
  size_t clr_cap[MAX_BONES][MAX_SLOTS] = {};
  ~asc_engine_s()
  {
    for (void* p : allocs) cudaFree(p);
    if (io.base) cudaFreeHost(io.base);
    for (auto& row : clr_own)
      for (uint8_t* p : row)
        if (p) cudaFree(p);
    for (cudaEvent_t x : ev)
      if (x) cudaEventDestroy(x);
    if (done) cudaEventDestroy(done);
    if (pso_exec) cudaGraphExecDestroy(pso_exec);
    if (own_stream) cudaStreamDestroy(own_stream);
  }
  template <class T>
  cudaError_t alloc(T*& p, size_t n)
  {
    cudaError_t e = cudaMalloc((void**)&p, std::max<size_t>(n, 1) * sizeof(T));
    if (e == cudaSuccess) allocs.push_back((void*)p);
    return e;
  }
};

static int prep_filters(const asc_filter_desc* in, int n, FilterDev* out, int* halo)
{
  if (n < 0 || n > MAX_FILTERS) return ASC_ERR_RANGE;
  int H = 0, m = 0;
  for (int i = 0; i < n; ++i) {
    const asc_filter_desc& f = in[i];
    if (!f.enabled) continue;  // View::filter copies through a disabled filter
    FilterDev d;
    memset(&d, 0, sizeof d);
    d.kind = f.kind;
    d.p0 = f.p0;
    d.p1 = f.p1;
    d.p2 = f.p2;
    if (f.kind == 1) {
      d.K = 3;
      d.R = 1;
    } else if (f.kind == 0) {
      d.K = (int)f.p2;
      if (d.K < 1) return ASC_ERR_ARG;
      d.R = std::max(d.K / 2, (d.K - 1) / 2);
    } else if (f.kind == 3 || f.kind == 4) {
      d.K = gauss_1d(f.p0, d.g, 32);
      if (d.K < 0) return ASC_ERR_RANGE;
      if (d.K == 1) continue;  // identity
      if (f.kind == 4) d.p1 = f.p1 < 1 ? 1 : f.p1;
      d.R = d.K / 2;
    } else {
      return ASC_ERR_ARG;
    }
    out[m++] = d;
    H += d.R;
  }
  *halo = H;
  return m;
}

static int fill_view(ViewDev& d, const asc_view_desc& v)
{
  memcpy(d.cam, v.frame, sizeof d.cam);
  frame_inverse(v.frame, d.cam_inv);
  memcpy(d.ip, v.image_plane, sizeof d.ip);
  memcpy(d.cvp, v.viewport, sizeof d.cvp);
  for (int j = 0; j < 4; ++j) d.ipf[j] = (float)v.viewport[j];
  if (!v.radiograph) return ASC_ERR_ARG;
  int bps;
  d.rad = image_data(v.radiograph, &d.rad_w, &d.rad_h, &bps);
  d.rad_bps = bps;
  if (bps == 32) return ASC_ERR_ARG;
  d.bg = nullptr;
  d.bg_thr = v.bg_threshold;
  if (v.background) {
    d.bg = (const float*)image_data(v.background, &d.bg_w, &d.bg_h, &bps);
    if (bps != 32) return ASC_ERR_ARG;
  }
  int n = prep_filters(v.drr_filters, v.n_drr_filters, d.fdrr, &d.h_drr);
  if (n < 0) return n;
  d.n_drr = n;
  n = prep_filters(v.rad_filters, v.n_rad_filters, d.frad, &d.h_rad);
  if (n < 0) return n;
  d.n_rad = n;
  if (!view_fits(std::max(d.h_drr, d.h_rad))) return ASC_ERR_RANGE;
  return ASC_OK;
}

static void set_base(BoneDev& B, const double* xyzypr) { memcpy(B.base, xyzypr, sizeof B.base); }

namespace {
void apply_tuning(asc_engine_s* e);  // the tuning table's launch shapes, below

// k_view's dynamic shared-memory limit is an attribute of the function, one
// per device for the whole process: it only ever grows here, so an engine
// with a narrower filter chain never lowers it below what an earlier engine
// launches with.
std::mutex g_view_smem_mu;
size_t g_view_smem[64] = {};

cudaError_t ensure_view_smem(size_t bytes)
{
  int dev = 0;
  cudaError_t err = cudaGetDevice(&dev);
  if (err) return err;
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> l(g_view_smem_mu);
  if (bytes <= g_view_smem[dev]) return cudaSuccess;
  err = cudaFuncSetAttribute(k_view, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (!err) g_view_smem[dev] = bytes;
  return err;
}
}

ASC_API int asc_engine_create(int n_views, const asc_view_desc* views, int n_bones, const asc_bone_desc* bones,
                              int rw, int rh, int max_items, int coverage, int cf_model, asc_engine* out)
{
  if (!views || !bones || !out || n_views < 1 || n_views > MAX_VIEWS || n_bones < 1 || n_bones > MAX_BONES ||
      rw < 1 || rh < 1 || max_items < 1 || (coverage != ASC_SUM_TREE && coverage != ASC_SUM_FULL))
    return ASC_ERR_ARG;
  if (cf_model != 0 && cf_model != 1) return ASC_ERR_ARG;
  Gate g(device_gate());
  // set-up work runs on a private stream, so that creating an engine does not
  // wait for other engines' work
  cudaStream_t cs = nullptr;
  if (cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking)) return ASC_ERR_CUDA;
  struct StreamGuard {
    cudaStream_t s;
    ~StreamGuard() { cudaStreamDestroy(s); }
  } cs_guard{cs};
  auto* e = new asc_engine_s();
  SceneDev& S = e->host;
  memset(&S, 0, sizeof S);
  S.n_views = n_views;
  S.n_bones = n_bones;
  S.rw = rw;
  S.rh = rh;
  S.coverage = coverage;
  S.cf_model = cf_model;
  S.slots = std::min(n_views, MAX_SLOTS);
  S.halo = 0;
  for (int v = 0; v < n_views; ++v) {
    int rc = fill_view(S.views[v], views[v]);
    if (rc) {
      delete e;
      return rc;
    }
    S.views[v].rw = rw;
    S.views[v].rh = rh;
    S.halo = std::max({S.halo, S.views[v].h_drr, S.views[v].h_rad});
  }
  for (int i = 0; i < n_bones; ++i) {
    auto* vh = (asc_volume_host*)bones[i].volume;
    if (!vh) {
      delete e;
      return ASC_ERR_ARG;
    }
    BoneDev& B = S.bones[i];
    B.vol = vh->dev;
    memcpy(B.inv_scale, vh->inv_scale, sizeof B.inv_scale);
    memcpy(B.inv_trans, vh->inv_trans, sizeof B.inv_trans);
    memcpy(B.pivot, bones[i].pivot, sizeof B.pivot);
    frame_inverse(B.pivot, B.pivot_inv);
    set_base(B, bones[i].base_pose);
    B.visible = 1;
    B.n_slots = S.slots;  // bone i is scored in views 0 .. slots - 1
    for (int j = 0; j < S.slots; ++j) {
      B.view_of[j] = j;
      B.step[j] = bones[i].step[j];
      B.scale[j] = bones[i].step[j] * vh->dev.norm / bones[i].intensity[j];
      B.cut[j] = make_cutoff(bones[i].cutoff[j], vh->dev.norm, vh->dev.gmax);
      uint8_t* clr = nullptr;
      if (e->alloc(clr, clearance_cells(vh->dev))) {
        delete e;
        return ASC_ERR_NOMEM;
      }
      int rc = build_clearance(vh->dev, occupancy_threshold(B.cut[j]), clr, cs);
      if (rc) {
        delete e;
        return rc;
      }
      B.clr[j] = clr;
    }
  }
  e->max_items = max_items;
  e->n_views = n_views;
  e->n_bones = n_bones;
  size_t n_iv = (size_t)max_items * S.slots;
  size_t tiles = (size_t)((rw + VT - 1) / VT) * ((rh + VT - 1) / VT);
  cudaError_t err = e->alloc(e->dev, 1);
  if (!err) err = e->alloc(e->b.iv, n_iv);
  if (!err) err = e->alloc(e->b.roff, n_iv + 1);
  if (!err) err = e->alloc(e->b.foff, n_iv + 1);
  if (!err) err = e->alloc(e->b.drr, n_iv * (size_t)rw * rh);
  if (!err) err = e->alloc(e->b.part, n_iv * tiles);
  if (!err) err = e->alloc(e->b.ftile_iv, n_iv * tiles);
  if (!err && cf_model) err = e->alloc(e->b.fg, n_iv * (size_t)rw * rh);
  if (!err && cf_model) err = e->alloc(e->b.hmean, n_iv);
  if (!err && cf_model) err = e->alloc(e->b.tsad, n_iv * tiles);
  if (!err) err = e->alloc(e->b.vcost, n_iv);
  if (!err) err = e->alloc(e->b.ivt, n_iv);
  if (!err) err = e->alloc(e->b.itt, (size_t)max_items);
  // at most every ray tile of a full batch
  const size_t ray_tiles = n_iv * (size_t)((rw + RTX - 1) / RTX) * ((rh + RTY - 1) / RTY);
  if (!err) err = e->alloc(e->b.fixb, ray_tiles * BEAMS);
  if (!err) err = e->alloc(e->b.rtile_iv, ray_tiles);
  if (!err) err = e->alloc(e->b.C, 1);
  if (!err) err = e->alloc(e->d_bone, (size_t)max_items);
  if (!err) err = e->alloc(e->d_manip, (size_t)max_items * 6);
  if (!err) err = e->alloc(e->d_cost, (size_t)max_items);
  if (!err) err = cudaMallocHost(&e->io.base, (max_items * (size_t)(7 + S.slots)) * sizeof(double) +
                                                   (max_items + (size_t)1) * sizeof(int));
  if (!err) {
    HostIO& io = e->io;
    io.manip = (double*)io.base;
    io.cost = io.manip + 6 * (size_t)max_items;
    io.vcost = io.cost + max_items;
    io.bone = (int*)(io.vcost + n_iv);
    io.error = io.bone + max_items;
  }
  if (!err) err = cudaEventCreateWithFlags(&e->done, cudaEventDisableTiming);
  const size_t npix = (size_t)rw * rh;
  if (!err) err = e->alloc(e->p_drr, npix);
  if (!err) err = e->alloc(e->p_rad, npix);
  if (!err) err = e->alloc(e->p_mask, npix);
  if (!err) err = e->alloc(e->p_tmp, npix);
  if (!err) err = e->alloc(e->p_bgr, npix);
  if (!err) err = e->alloc(e->p_res, 1);
  if (!err) err = cudaMemcpyAsync(e->dev, &S, sizeof S, cudaMemcpyHostToDevice, cs);
  if (!err) err = cudaMemsetAsync(e->b.C, 0, sizeof(Counters), cs);
  if (err) {
    delete e;
    return cuda_status(err);
  }
  e->vdesc.assign(views, views + n_views);
  e->bdesc.assign(bones, bones + n_bones);
  if (cudaStreamSynchronize(cs)) {
    delete e;
    return ASC_ERR_CUDA;
  }
  e->smem = view_smem_floats(S.halo) * sizeof(float);
  int dev = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&e->sms, cudaDevAttrMultiProcessorCount, dev);
  err = ensure_view_smem(e->smem);
  if (!err) err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&e->view_blocks, k_view, VNT, e->smem);
  if (err) {
    delete e;
    return cuda_status(err);
  }
  e->view_blocks = std::max(e->view_blocks, 1);
  apply_tuning(e);
  *out = e;
  return ASC_OK;
}

ASC_API int asc_engine_destroy(asc_engine e)
{
  if (!e) return ASC_ERR_ARG;
  Gate g(device_gate());
  cudaDeviceSynchronize();
  delete e;
  return ASC_OK;
}

ASC_API int asc_engine_set_base_pose(asc_engine e, int bone, const double xyzypr[6])
{
  if (!e || !xyzypr || bone < 0 || bone >= e->n_bones) return ASC_ERR_ARG;
  set_base(e->host.bones[bone], xyzypr);
  Gate g(device_gate());
  ASC_CUDA(cudaMemcpy(&e->dev->bones[bone].base, xyzypr, 6 * sizeof(double), cudaMemcpyHostToDevice));
  return ASC_OK;
}

ASC_API int asc_engine_set_visible(asc_engine e, int bone, int visible)
{
  if (!e || bone < 0 || bone >= e->n_bones) return ASC_ERR_ARG;
  e->host.bones[bone].visible = visible ? 1 : 0;
  Gate g(device_gate());
  ASC_CUDA(cudaMemcpy(&e->dev->bones[bone].visible, &e->host.bones[bone].visible, sizeof(int),
                      cudaMemcpyHostToDevice));
  return ASC_OK;
}

ASC_API int asc_engine_set_radiograph(asc_engine e, int view, asc_image rad)
{
  if (!e || !rad || view < 0 || view >= e->n_views) return ASC_ERR_ARG;
  ViewDev& d = e->host.views[view];
  int bps;
  const void* data = image_data(rad, &d.rad_w, &d.rad_h, &bps);
  if (bps == 32) return ASC_ERR_ARG;
  d.rad = data;
  d.rad_bps = bps;
  e->vdesc[view].radiograph = rad;  // the plain path and the image exports read it there
  Gate g(device_gate());
  ASC_CUDA(cudaMemcpy(&e->dev->views[view], &d, sizeof d, cudaMemcpyHostToDevice));
  return ASC_OK;
}

ASC_API int asc_engine_set_view(asc_engine e, int view, const asc_view_desc* desc, int rw, int rh)
{
  if (!e || !desc || view < 0 || view >= e->n_views || rw < 1 || rh < 1 || rw > e->host.rw || rh > e->host.rh)
    return ASC_ERR_ARG;
  ViewDev d;
  memset(&d, 0, sizeof d);
  int rc = fill_view(d, *desc);
  if (rc) return rc;
  d.rw = rw;
  d.rh = rh;
  Gate g(device_gate());
  const int halo = std::max(d.h_drr, d.h_rad);
  const size_t need = view_smem_floats(halo) * sizeof(float);
  if (need > e->smem) {  // a wider filter chain than the engine's views had so far
    int blocks = 0;
    ASC_CUDA(ensure_view_smem(need));
    ASC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, k_view, VNT, need));
    e->smem = need;
    e->view_blocks = std::max(blocks, 1);
    e->host.halo = std::max(e->host.halo, halo);
    if (e->pso_exec) {  // its k_view node holds the old launch shape
      cudaGraphExecDestroy(e->pso_exec);
      e->pso_exec = nullptr;
    }
  }
  e->host.views[view] = d;
  e->vdesc[view] = *desc;
  ASC_CUDA(cudaMemcpy(&e->dev->views[view], &d, sizeof d, cudaMemcpyHostToDevice));
  return ASC_OK;
}

ASC_API int asc_engine_set_bone(asc_engine e, int bone, const asc_bone_desc* desc, int n_views, const int* views)
{
  if (!e || !desc || !desc->volume || bone < 0 || bone >= e->n_bones || n_views < 1 || n_views > e->host.slots ||
      !views)
    return ASC_ERR_ARG;
  for (int j = 0; j < n_views; ++j)
    if (views[j] < 0 || views[j] >= e->n_views) return ASC_ERR_ARG;
  auto* vh = (asc_volume_host*)desc->volume;
  BoneDev B = e->host.bones[bone];
  B.vol = vh->dev;
  memcpy(B.inv_scale, vh->inv_scale, sizeof B.inv_scale);
  memcpy(B.inv_trans, vh->inv_trans, sizeof B.inv_trans);
  memcpy(B.pivot, desc->pivot, sizeof B.pivot);
  frame_inverse(B.pivot, B.pivot_inv);
  set_base(B, desc->base_pose);
  B.visible = 1;
  B.n_slots = n_views;
  Gate g(device_gate());
  const size_t grid = clearance_cells(vh->dev);
  for (int j = 0; j < n_views; ++j) {
    B.view_of[j] = views[j];
    B.step[j] = desc->step[j];
    B.scale[j] = desc->step[j] * vh->dev.norm / desc->intensity[j];
    B.cut[j] = make_cutoff(desc->cutoff[j], vh->dev.norm, vh->dev.gmax);
    uint8_t*& clr = e->clr_own[bone][j];
    if (e->clr_cap[bone][j] < grid) {
      if (clr) cudaFree(clr);
      clr = nullptr;
      e->clr_cap[bone][j] = 0;
      ASC_CUDA(cudaMalloc(&clr, grid));
      e->clr_cap[bone][j] = grid;
    }
    int rc = build_clearance(vh->dev, occupancy_threshold(B.cut[j]), clr, nullptr);
    if (rc) return rc;
    B.clr[j] = clr;
  }
  ASC_CUDA(cudaStreamSynchronize(nullptr));
  e->host.bones[bone] = B;
  e->bdesc[bone] = *desc;
  ASC_CUDA(cudaMemcpy(&e->dev->bones[bone], &B, sizeof B, cudaMemcpyHostToDevice));
  return ASC_OK;
}

// ---- the tuning table: launch shapes per workload class, written by the
// project's autotuner (autoscoper_gb300/tune.py) and read at engine creation.
// A class is (ceil log2 of the render pixels, ceil log2 of the largest
// volume's voxels, views); a line of the table holds
//   rpx vox views ray_blocks_per_sm view_blocks_per_sm ray_shape
// ('#' starts a comment).  An engine takes the entry of its render size and
// view count with the nearest volume class; without one it keeps the defaults.
namespace {
struct TuneEntry {
  int rpx, vox, views;
  asc_launch_config cfg;
};
std::mutex g_tune_mu;
std::vector<TuneEntry> g_tune;

int ceil_log2(double x)
{
  int k = 0;
  while ((double)(1ull << k) < x && k < 62) ++k;
  return k;
}

void workload_class(const asc_engine_s* e, int out[3])
{
  double vox = 0;
  for (int b = 0; b < e->n_bones; ++b) {
    const DevVolume& V = e->host.bones[b].vol;
    vox = std::max(vox, (double)V.nx * V.ny * V.nz);
  }
  out[0] = ceil_log2((double)e->host.rw * e->host.rh);
  out[1] = ceil_log2(vox);
  out[2] = e->n_views;
}

void apply_tuning(asc_engine_s* e)
{
  int c[3];
  workload_class(e, c);
  std::lock_guard<std::mutex> l(g_tune_mu);
  const TuneEntry* best = nullptr;
  for (const TuneEntry& t : g_tune)
    if (t.rpx == c[0] && t.views == c[2] && (!best || std::abs(t.vox - c[1]) < std::abs(best->vox - c[1])))
      best = &t;
  if (best) e->launch = best->cfg;
}
}  // namespace

ASC_API int asc_tuning_load(const char* path)
{
  if (!path) return ASC_ERR_ARG;
  FILE* f = fopen(path, "r");
  if (!f) return ASC_ERR_ARG;
  std::vector<TuneEntry> t;
  char line[512];
  int rc = ASC_OK;
  while (fgets(line, sizeof line, f)) {
    char* hash = strchr(line, '#');
    if (hash) *hash = 0;
    TuneEntry x;
    int n = sscanf(line, "%d %d %d %d %d %d", &x.rpx, &x.vox, &x.views, &x.cfg.ray_blocks_per_sm,
                   &x.cfg.view_blocks_per_sm, &x.cfg.ray_shape);
    if (n <= 0) continue;  // blank or comment
    if (n != 6 || x.cfg.ray_blocks_per_sm < 1 || x.cfg.ray_blocks_per_sm > ASC_RAY_MINBLOCKS ||
        x.cfg.view_blocks_per_sm < 0 || x.cfg.ray_shape < 2 || x.cfg.ray_shape > 4) {
      rc = ASC_ERR_ARG;
      break;
    }
    t.push_back(x);
  }
  fclose(f);
  if (rc) {
    set_error_message("asc_tuning_load: a line is not 'rpx vox views ray_blocks view_blocks ray_shape'");
    return rc;
  }
  std::lock_guard<std::mutex> l(g_tune_mu);
  g_tune = t;
  return ASC_OK;
}

ASC_API int asc_engine_workload_class(asc_engine e, int out[3])
{
  if (!e || !out) return ASC_ERR_ARG;
  workload_class(e, out);
  return ASC_OK;
}

ASC_API int asc_engine_set_launch(asc_engine e, const asc_launch_config* cfg)
{
  if (!e || !cfg || cfg->ray_blocks_per_sm < 1 || cfg->ray_blocks_per_sm > ASC_RAY_MINBLOCKS ||
      cfg->view_blocks_per_sm < 0 || cfg->ray_shape < 2 || cfg->ray_shape > 4)
    return ASC_ERR_ARG;
  Gate g(device_gate());
  e->launch = *cfg;
  if (e->pso_exec) {  // the captured iteration holds the old launch shapes
    cudaGraphExecDestroy(e->pso_exec);
    e->pso_exec = nullptr;
  }
  return ASC_OK;
}

ASC_API int asc_engine_get_launch(asc_engine e, asc_launch_config* cfg, int* view_blocks_max)
{
  if (!e || !cfg) return ASC_ERR_ARG;
  *cfg = e->launch;
  if (view_blocks_max) *view_blocks_max = e->view_blocks;
  return ASC_OK;
}

static int engine_launch(asc_engine e, int n, const int* bone, const double* manip, double* cost, double* vcost,
                         cudaStream_t s, bool capturing = false, int* error = nullptr)
{
  const bool prof = e->prof && !capturing;
  if (prof) ASC_CUDA(cudaEventRecord(e->ev[0], s));
  k_setup<<<n, SETUP_THREADS, 0, s>>>(e->dev, n, bone, manip, e->b, cost, vcost, error);
  if (prof) ASC_CUDA(cudaEventRecord(e->ev[1], s));
  k_ray<<<e->sms * e->launch.ray_blocks_per_sm, NRAY, 0, s>>>(e->dev, e->b, g_empty_skip, e->launch.ray_shape);
  k_ray_fix<<<e->sms * 4, FIX_THREADS, 0, s>>>(e->dev, e->b, e->launch.ray_shape);
  if (prof) ASC_CUDA(cudaEventRecord(e->ev[2], s));
  k_view<<<e->sms * e->view_grid(), VNT, e->smem, s>>>(e->dev, e->b, cost, vcost);
  if (e->host.cf_model) k_sad<<<e->sms * 8, 256, 0, s>>>(e->dev, e->b, cost, vcost);
  if (prof) ASC_CUDA(cudaEventRecord(e->ev[3], s));
  ASC_LAUNCH_CHECK();
  return ASC_OK;
}

ASC_API int asc_engine_profile(asc_engine e, int enable)
{
  if (!e) return ASC_ERR_ARG;
  if (enable && !e->ev[0])
    for (int i = 0; i < 4; ++i) ASC_CUDA(cudaEventCreate(&e->ev[i]));
  e->prof = enable != 0;
  return ASC_OK;
}

// The last evaluation's counters, its samples counted here if they are asked
// for.  The evaluation may be on a stream that nothing orders before the
// default stream, so its event is waited for; and two callers would count into
// one word, so one at a time.
static int read_counters(asc_engine e, Counters& C, bool samples)
{
  ASC_CUDA(cudaEventSynchronize(e->done));
  Gate g(device_gate());
  if (samples) {
    ASC_CUDA(cudaMemset(&e->b.C->samples, 0, sizeof C.samples));
    k_count_samples<<<e->sms * 8, NRAY>>>(e->b);
    ASC_LAUNCH_CHECK();
  }
  ASC_CUDA(cudaMemcpy(&C, e->b.C, sizeof C, cudaMemcpyDeviceToHost));
  return ASC_OK;
}

ASC_API int asc_engine_stats(asc_engine e, float ms[3], unsigned long long* samples, unsigned long long* pixels)
{
  if (!e) return ASC_ERR_ARG;
  if (ms) {
    if (!e->ev[0]) return ASC_ERR_STATE;
    ASC_CUDA(cudaEventSynchronize(e->ev[3]));
    for (int i = 0; i < 3; ++i) ASC_CUDA(cudaEventElapsedTime(&ms[i], e->ev[i], e->ev[i + 1]));
  }
  if (!samples && !pixels) return ASC_OK;
  Counters C;
  int rc = read_counters(e, C, samples != nullptr);
  if (rc) return rc;
  if (samples) *samples = C.samples;
  if (pixels) *pixels = C.pixels;
  return ASC_OK;
}

ASC_API int asc_engine_exact_rays(asc_engine e, int* n)
{
  if (!e || !n) return ASC_ERR_ARG;
  Counters C;
  int rc = read_counters(e, C, false);
  if (rc) return rc;
  *n = C.nfix;
  return ASC_OK;
}

ASC_API int asc_engine_counters(asc_engine e, unsigned long long out[4])
{
  if (!e || !out) return ASC_ERR_ARG;
  Counters C;
  int rc = read_counters(e, C, true);
  if (rc) return rc;
  out[0] = C.samples;
  out[1] = C.pixels;
  out[2] = C.marched;
  out[3] = C.slots;
  return ASC_OK;
}

ASC_API int asc_engine_eval(asc_engine e, int n, const int* bone, const double* manip, double* cost, double* vcost,
                            void* stream)
{
  if (!e || !bone || !manip || !cost || n < 1 || n > e->max_items) return ASC_ERR_ARG;
  cudaStream_t s = S(stream);
  int rc = engine_launch(e, n, bone, manip, cost, vcost, s);
  if (rc || !s) return rc;
  // a captured evaluation runs when its graph does: no event of this call's
  cudaStreamCaptureStatus capture;
  ASC_CUDA(cudaStreamIsCapturing(s, &capture));
  if (capture == cudaStreamCaptureStatusNone) ASC_CUDA(cudaEventRecord(e->done, s));
  return ASC_OK;
}

ASC_API int asc_engine_eval_host(asc_engine e, int n, const int* bone, const double* manip, double* cost,
                                 double* vcost, void* stream)
{
  if (!e || !bone || !manip || !cost || n < 1 || n > e->max_items) return ASC_ERR_ARG;
  // the candidates and the results pass through pinned host memory that the
  // kernels read and write themselves: they are a few KB, and two copies in,
  // three out of pageable memory and a launch to gather the view costs took
  // 39 us of a simplex step's 249
  cudaStream_t s = S(stream);
  const HostIO& io = e->io;
  memcpy(io.bone, bone, n * sizeof(int));
  memcpy(io.manip, manip, n * 6 * sizeof(double));
  int rc = engine_launch(e, n, io.bone, io.manip, io.cost, vcost ? io.vcost : nullptr, s, false, io.error);
  if (rc) return rc;
  ASC_CUDA(cudaStreamSynchronize(s));
  memcpy(cost, io.cost, n * sizeof(double));
  if (vcost) memcpy(vcost, io.vcost, (size_t)n * e->host.slots * sizeof(double));
  return *io.error ? *io.error : ASC_OK;
}

ASC_API int asc_engine_debug(asc_engine e, const float** drr, const int** layout)
{
  if (!e) return ASC_ERR_ARG;
  if (drr) *drr = e->b.drr;
  if (layout) *layout = (const int*)e->b.iv;
  return ASC_OK;
}

ASC_API int asc_engine_pso_stall(asc_engine e, int np, int n_iter, int max_stall, double w, double c1, double c2,
                                 double lo, double hi, uint64_t seed, double* best_manip, double* best_cost,
                                 long long* evals, int* iterations, void* stream)
{
  if (!e || np < 1 || n_iter < 1 || max_stall < 0 || !best_manip || !best_cost) return ASC_ERR_ARG;
  const int nb = e->n_bones, n = nb * np;
  if (n > e->max_items) return ASC_ERR_RANGE;
  cudaStream_t s = S(stream);
  if (!s) {  // one private non-blocking stream per engine
    if (!e->own_stream) ASC_CUDA(cudaStreamCreateWithFlags(&e->own_stream, cudaStreamNonBlocking));
    s = e->own_stream;
  }
  // swarm state: allocated once per engine, sized for max_items particles
  if (!e->sw_buf) {
    Gate g(device_gate());
    const size_t cap = (size_t)e->max_items, nbm = (size_t)e->n_bones;
    cudaError_t err = e->alloc(e->sw_buf, cap * 6 * 3 + cap + nbm * 6 + nbm);
    if (!err) err = e->alloc(e->sw_iter, 1);
    if (!err) err = e->alloc(e->sw_frozen, nbm);
    if (err) return cuda_status(err);
  }
  Swarm sw;
  sw.x = e->sw_buf;
  sw.v = sw.x + (size_t)n * 6;
  sw.pbx = sw.v + (size_t)n * 6;
  sw.pbc = sw.pbx + (size_t)n * 6;
  sw.gx = sw.pbc + n;
  sw.gc = sw.gx + nb * 6;
  sw.iter = e->sw_iter;
  sw.frozen = e->sw_frozen;
  sw.bone = e->d_bone;
  sw.manip = e->d_manip;
  const int tb = 128, gb = (n + tb - 1) / tb;
  k_pso_init<<<gb, tb, 0, s>>>(sw, nb, np, lo, hi, seed);
  cudaError_t err = cudaGetLastError();
  // one iteration = update -> setup -> ray -> view -> best, captured once per
  // SwarmKey and replayed n_iter times
  const SwarmKey key{np, g_empty_skip, w, c1, c2, seed};
  if (!err && (!e->pso_exec || !(key == e->pso_key))) {
    if (e->pso_exec) {
      cudaGraphExecDestroy(e->pso_exec);
      e->pso_exec = nullptr;
    }
    cudaGraph_t graph = nullptr;
    Gate g(device_gate());
    err = cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal);
    if (!err) {
      k_pso_update<<<gb, tb, 0, s>>>(sw, nb, np, w, c1, c2, seed);
      engine_launch(e, n, e->d_bone, e->d_manip, e->d_cost, nullptr, s, true);
      k_pso_best<<<nb, 256, 0, s>>>(sw, nb, np, e->d_cost);
      err = cudaStreamEndCapture(s, &graph);
    }
    if (!err) err = cudaGraphInstantiate(&e->pso_exec, graph, 0);
    if (graph) cudaGraphDestroy(graph);
    if (!err) e->pso_key = key;
  }
  long long scored = 0;
  int it = 0;
  if (max_stall == 0) {
    for (; !err && it < n_iter; ++it) err = cudaGraphLaunch(e->pso_exec, s);
    scored = (long long)n * it;
  } else {
    // the stall rule of PSO.cpp:271-285 per swarm, read back after every
    // iteration: |gBest change| < 1e-4 counts a stall, > 1e-3 resets the
    // count, max_stall stalls in a row stop that swarm (it is frozen, and
    // the iterations end when every swarm is)
    std::vector<double> gc(nb), prev(nb, 1e300);
    std::vector<int> stall(nb, 0), frozen(nb, 0);
    int live = nb;
    for (; !err && it < n_iter && live > 0; ++it) {
      err = cudaGraphLaunch(e->pso_exec, s);
      scored += (long long)np * live;
      if (!err) err = cudaMemcpyAsync(gc.data(), sw.gc, nb * sizeof(double), cudaMemcpyDeviceToHost, s);
      if (!err) err = cudaStreamSynchronize(s);
      for (int b = 0; !err && b < nb; ++b) {
        if (frozen[b]) continue;
        const double d = std::fabs(gc[b] - prev[b]);
        if (d < 1e-4)
          ++stall[b];
        else if (d > 1e-3)
          stall[b] = 0;
        prev[b] = gc[b];
        if (stall[b] == max_stall) {
          frozen[b] = 1;
          --live;
          err = cudaMemcpyAsync(sw.frozen + b, &frozen[b], sizeof(int), cudaMemcpyHostToDevice, s);
        }
      }
    }
  }
  if (!err) err = cudaMemcpyAsync(best_manip, sw.gx, nb * 6 * sizeof(double), cudaMemcpyDeviceToHost, s);
  if (!err) err = cudaMemcpyAsync(best_cost, sw.gc, nb * sizeof(double), cudaMemcpyDeviceToHost, s);
  if (!err) err = cudaStreamSynchronize(s);
  if (evals) *evals = scored;
  if (iterations) *iterations = it;
  return err ? cuda_status(err) : ASC_OK;
}

ASC_API int asc_engine_pso(asc_engine e, int np, int n_iter, double w, double c1, double c2, double lo, double hi,
                           uint64_t seed, double* best_manip, double* best_cost, long long* evals, void* stream)
{
  return asc_engine_pso_stall(e, np, n_iter, 0, w, c1, c2, lo, hi, seed, best_manip, best_cost, evals, nullptr,
                              stream);
}

// ---------------------------------------------------------------- plain path
// Tracker::trackFrame (Tracker.cpp:583-773) one pose at a time over the plain
// per-operator kernels: the same launch sequence as the reference (ray cast,
// DRR filters, radiograph crop, radiograph filters, masks, three multiplies,
// NCC) with the NCC read back to the host after every view.  This is the
// drop-in form the batched engine is measured against.
static int chain_plain(const asc_filter_desc* fl, int nf, float*& cur, float*& other, int w, int h, cudaStream_t s)
{
  for (int i = 0; i < nf; ++i) {
    if (fl[i].enabled) {
      int rc = launch_filter(fl[i], cur, other, w, h, s);
      if (rc) return rc;
      std::swap(cur, other);
    }
  }
  return ASC_OK;
}

// One view of one bone at `xyzypr` over `vp`: the folded camera->volume
// matrix (Tracker.cpp:603-612 with RayCaster::setInvModelView).
static void view_matrix(const ViewDev& V, const BoneDev& B, const double* xyzypr, float m[12])
{
  double f[12], mv[12], imv[12], imv16[16];
  frame_from_xyzypr(xyzypr, f);
  frame_mul(V.cam_inv, f, mv);
  frame_inverse(mv, imv);
  frame_row_matrix(imv, imv16);
  fold_matrix(imv16, B.inv_scale, B.inv_trans, m);
}

// Whether every bone is scored in every view, slot j being view j (the
// layout asc_engine_create makes for up to MAX_SLOTS views).  The plain
// per-pose path and the image exports read the bones' per-view settings by
// view and need it; engines whose bones asc_engine_set_bone moved to other
// views serve batched evaluations only.
static bool identity_slots(const asc_engine_s* e)
{
  if (e->host.slots != e->n_views) return false;
  for (int b = 0; b < e->n_bones; ++b) {
    const BoneDev& B = e->host.bones[b];
    if (B.n_slots != e->n_views) return false;
    for (int j = 0; j < B.n_slots; ++j)
      if (B.view_of[j] != j) return false;
  }
  return true;
}

// RayCaster::render (RayCaster.cpp:123-143) of one bone into `out`: zeros
// for a hidden volume.
static int render_bone(const BoneDev& B, const asc_bone_desc& BD, int v, const float* m, const float* vpf,
                       float* out, int w, int h, cudaStream_t s)
{
  if (!B.visible) {
    ASC_CUDA(cudaMemsetAsync(out, 0, (size_t)w * h * sizeof(float), s));
    return ASC_OK;
  }
  return raycast_launch(B.vol, g_empty_skip ? B.clr[v] : nullptr, m, vpf, BD.step[v], BD.intensity[v], BD.cutoff[v],
                        out, false, w, h, s);
}

ASC_API int asc_engine_eval_plain(asc_engine e, int n, const int* bone, const double* manip, double* cost,
                                  double* view_cost, void* stream)
{
  if (!e || !bone || !manip || !cost || n < 1) return ASC_ERR_ARG;
  if (!identity_slots(e)) return ASC_ERR_STATE;
  cudaStream_t s = S(stream);
  const SceneDev& S_ = e->host;
  const int nv = e->n_views;
  for (int it = 0; it < n; ++it) {
    int bi = bone[it];
    if (bi < 0 || bi >= e->n_bones) return ASC_ERR_ARG;
    const BoneDev& B = S_.bones[bi];
    const asc_bone_desc& BD = e->bdesc[bi];
    double base[12], man[12], t1[12], t2[12], xyz[6];
    frame_from_xyzypr(B.base, base);
    frame_from_axis_angle(manip + 6 * it, man);
    frame_mul(base, B.pivot_inv, t1);
    frame_mul(t1, man, t2);
    frame_mul(t2, B.pivot, t1);
    frame_to_xyzypr(t1, xyz);
    frame_from_xyzypr(xyz, t1);
    double total = 0.0;
    for (int v = 0; v < nv; ++v) {
      const ViewDev& V = S_.views[v];
      const asc_view_desc& VD = e->vdesc[v];
      double mv[12], imv[12], imv16[16], vp[4];
      float m[12];
      frame_mul(V.cam_inv, t1, mv);
      frame_inverse(mv, imv);
      frame_row_matrix(imv, imv16);
      fold_matrix(imv16, B.inv_scale, B.inv_trans, m);
      double vc;
      if (!calculate_viewport(mv, V.cam, V.ip, B.inv_scale, B.inv_trans, vp)) {
        vc = 9999.0;
      } else {
        double fw = vp[2] * S_.rw / V.cvp[2], fh = vp[3] * S_.rh / V.cvp[3];
        unsigned w = fw > 0 ? (unsigned)fw : 0u, h = fh > 0 ? (unsigned)fh : 0u;
        if (w > (unsigned)S_.rw || h > (unsigned)S_.rh) return ASC_ERR_RANGE;
        if (w == 0 || h == 0) {
          vc = S_.cf_model ? 0.0 : 1.0 - 1e5;
        } else {
          float vpf[4] = {(float)vp[0], (float)vp[1], (float)vp[2], (float)vp[3]};
          int rc = render_bone(B, BD, v, m, vpf, e->p_drr, w, h, s);
          float *d = e->p_drr, *o = e->p_tmp;
          if (!rc) rc = chain_plain(VD.drr_filters, VD.n_drr_filters, d, o, w, h, s);
          // the DRR chain ping-pongs p_drr/p_tmp and leaves one of them free (o);
          // the radiograph chain ping-pongs p_rad/o; p_mask stays free
          if (!rc) rc = asc_rad_render(VD.radiograph, V.ipf, vpf, e->p_rad, w, h, s);
          float *r = e->p_rad, *ro = o;
          if (!rc) rc = chain_plain(VD.rad_filters, VD.n_rad_filters, r, ro, w, h, s);
          float* mask = e->p_mask;
          float* bgm = nullptr;  // no background: a mask of ones
          if (!rc && VD.background && VD.bg_threshold >= 0) {
            bgm = e->p_bgr;
            rc = asc_background_render(VD.background, V.ipf, vpf, VD.bg_threshold, bgm, w, h, s);
          }
          if (!rc) rc = mask_images(d, r, bgm, mask, d, r, (size_t)w * h, s);
          double res = 0;
          if (!rc)
            rc = S_.cf_model ? asc_hdist(d, r, mask, w * h, S_.coverage, e->p_res, s)
                             : asc_ncc(d, r, mask, w * h, S_.coverage, e->p_res, s);
          if (!rc) {
            cudaError_t err = cudaMemcpyAsync(&res, e->p_res, sizeof(double), cudaMemcpyDeviceToHost, s);
            if (!err) err = cudaStreamSynchronize(s);
            if (err) rc = cuda_status(err);
          }
          if (rc) return rc;
          vc = S_.cf_model ? res : 1.0 - res;  // Tracker.cpp:762-770
        }
      }
      if (view_cost) view_cost[it * nv + v] = vc;
      total += vc;
    }
    cost[it] = total < 0 ? 9999.0 : total;
  }
  return ASC_OK;
}

// ---------------------------------------------------------------- Tracker::optimize
namespace {

struct EvalCtx {
  asc_engine e;
  cudaStream_t s;
  long long evals;
};

// Batch cost for asc_amoeba_batch: candidate i belongs to simplex (bone) who[i].
int engine_batch_cost(int n, const int* who, const double* x, double* y, void* ctx)
{
  EvalCtx* c = (EvalCtx*)ctx;
  const int cap = c->e->max_items;
  for (int i0 = 0; i0 < n; i0 += cap) {
    const int m = std::min(cap, n - i0);
    int rc = asc_engine_eval_host(c->e, m, who + i0, x + 6 * (size_t)i0, y + i0, nullptr, c->s);
    if (rc) return rc;
  }
  c->evals += n;
  return ASC_OK;
}

// The pose base * V^-1 * manip * V as xyzypr (Tracker.cpp:479-483, :558-562).
void compose_pose(const BoneDev& B, const double* base6, const double* manip, double* out)
{
  double base[12], man[12], t1[12], t2[12];
  frame_from_xyzypr(base6, base);
  frame_from_axis_angle(manip, man);
  frame_mul(base, B.pivot_inv, t1);
  frame_mul(t1, man, t2);
  frame_mul(t2, B.pivot, t1);
  frame_to_xyzypr(t1, out);
}

}  // namespace

ASC_API int asc_engine_optimize_frame_ex(asc_engine e, const asc_opt_params* p, double* pose_out, double* raw_out,
                                         double* cost_out, long long* evals_out, void* stream)
{
  if (!e || !p || !pose_out) return ASC_ERR_ARG;
  const int nb = e->n_bones;
  if (nb * 7 > e->max_items) return ASC_ERR_RANGE;
  cudaStream_t s = S(stream);
  if (!s) {  // the engine's private stream, so that engines on other threads overlap
    if (!e->own_stream) ASC_CUDA(cudaStreamCreateWithFlags(&e->own_stream, cudaStreamNonBlocking));
    s = e->own_stream;
  }
  EvalCtx ctx{e, s, 0};
  std::vector<int> bones(nb);
  for (int b = 0; b < nb; ++b) bones[b] = b;
  // the frame's pose as read from the key curves (the engine's base poses)
  std::vector<double> xyzypr(6 * nb);
  for (int b = 0; b < nb; ++b)
    for (int j = 0; j < 6; ++j) xyzypr[6 * b + j] = e->host.bones[b].base[j];
  // init_ncc = minimizationFunc(0) (Tracker.cpp:441-443)
  std::vector<double> zero(6 * nb, 0.0), init(nb), fin(nb);
  int rc = engine_batch_cost(nb, bones.data(), zero.data(), init.data(), &ctx);
  if (rc) return rc;
  if (p->method == 0) {
    // PSO, then move the pose to the swarm's best: the key curves take the
    // stored (rounded) pose, which the simplex evaluates around, while the
    // final composition starts from the unrounded one (Tracker.cpp:445-491)
    std::vector<double> best(6 * nb), bc(nb);
    long long ev = 0;
    rc = asc_engine_pso_stall(e, p->n_particles, p->n_iter, p->max_stall, p->w, p->c1, p->c2, p->lo, p->hi, p->seed,
                              best.data(), bc.data(), &ev, nullptr, (void*)s);
    if (rc) return rc;
    ctx.evals += ev;
    for (int b = 0; b < nb; ++b) {
      double np[6], st[6];
      compose_pose(e->host.bones[b], xyzypr.data() + 6 * b, best.data() + 6 * b, np);
      keycurve_store(np, st);
      for (int j = 0; j < 6; ++j) xyzypr[6 * b + j] = np[j];
      rc = asc_engine_set_base_pose(e, b, st);
      if (rc) return rc;
    }
  }
  // Downhill Simplex from the offsets (Tracker.cpp:493-515), all bones at once
  const int mp = 7;
  std::vector<double> P((size_t)nb * mp * 6, 0.0), Y((size_t)nb * mp);
  std::vector<int> who((size_t)nb * mp);
  for (int b = 0; b < nb; ++b)
    for (int i = 0; i < mp; ++i) {
      who[b * mp + i] = b;
      if (i > 0) P[((size_t)b * mp + i) * 6 + (i - 1)] = p->offsets[i - 1];
    }
  rc = engine_batch_cost(nb * mp, who.data(), P.data(), Y.data(), &ctx);
  if (rc) return rc;
  std::vector<int> iters(nb);
  rc = asc_amoeba_batch(engine_batch_cost, &ctx, nb, P.data(), Y.data(), 6, p->ftol, iters.data());
  if (rc) return rc;
  // final_ncc = minimizationFunc(P[1]); keep the start of the simplex if not better (Tracker.cpp:517-525)
  std::vector<double> vert0(6 * nb);
  for (int b = 0; b < nb; ++b)
    for (int j = 0; j < 6; ++j) vert0[6 * b + j] = P[(size_t)b * mp * 6 + j];
  rc = engine_batch_cost(nb, bones.data(), vert0.data(), fin.data(), &ctx);
  if (rc) return rc;
  for (int b = 0; b < nb; ++b) {
    const bool take = p->method != 0 || fin[b] < init[b];
    double manip[6] = {0, 0, 0, 0, 0, 0};
    if (take)
      for (int j = 0; j < 6; ++j) manip[j] = vert0[6 * b + j];
    double np[6], st[6];
    compose_pose(e->host.bones[b], xyzypr.data() + 6 * b, manip, np);
    keycurve_store(np, st);
    rc = asc_engine_set_base_pose(e, b, st);
    if (rc) return rc;
    for (int j = 0; j < 6; ++j) pose_out[6 * b + j] = st[j];
    if (raw_out)
      for (int j = 0; j < 6; ++j) raw_out[6 * b + j] = np[j];
    if (cost_out) cost_out[b] = take ? fin[b] : init[b];
  }
  if (evals_out) *evals_out = ctx.evals;
  return ASC_OK;
}

ASC_API int asc_engine_optimize_frame(asc_engine e, const asc_opt_params* p, double* pose_out, double* cost_out,
                                      long long* evals_out, void* stream)
{
  return asc_engine_optimize_frame_ex(e, p, pose_out, nullptr, cost_out, evals_out, stream);
}

ASC_API int asc_keycurve_store(const double pose[6], double out[6])
{
  if (!pose || !out) return ASC_ERR_ARG;
  keycurve_store(pose, out);
  return ASC_OK;
}

ASC_API int asc_engine_track(asc_engine e, int n_frames, const asc_image* rads, const asc_track_params* tp,
                             double* poses, double* costs, long long* evals_out, void* stream)
{
  if (!e || n_frames < 1 || !rads || !tp || !poses || tp->repeats < 1 || (tp->dframe != 1 && tp->dframe != -1) ||
      tp->guess < 0 || tp->guess > 2)
    return ASC_ERR_ARG;
  const int nb = e->n_bones, nv = e->n_views, d = tp->dframe;
  long long evals = 0;
  for (int i = 0; i < n_frames; ++i) {
    const int f = d > 0 ? i : n_frames - 1 - i;
    double* pf = poses + (size_t)f * nb * 6;
    for (int v = 0; v < nv; ++v) {
      int rc = asc_engine_set_radiograph(e, v, rads[(size_t)f * nv + v]);
      if (rc) return rc;
    }
    // initial guess (Tracker.cpp:388-426); i frames are already tracked in
    // this direction.  Without a guess the frame starts from its key curve
    // value: its own key, or for an unkeyed frame the last tracked frame's
    // pose (a key curve holds its last key beyond it)
    for (int b = 0; b < nb; ++b) {
      const double* prev = poses + ((size_t)(f - d) * nb + b) * 6;
      double g[6];
      if (tp->guess == 2 && i > 1) {
        double a[12], c[12], x[12];
        frame_from_xyzypr(poses + ((size_t)(f - 2 * d) * nb + b) * 6, a);
        frame_from_xyzypr(prev, c);
        frame_linear_extrap(a, c, x);
        frame_to_xyzypr(x, g);
        keycurve_store(g, pf + 6 * b);
      } else if (tp->guess == 1 && i > 0) {
        keycurve_store(prev, pf + 6 * b);
      } else if (i > 0 && !(tp->keyed && tp->keyed[f])) {
        for (int j = 0; j < 6; ++j) pf[6 * b + j] = prev[j];
      }
    }
    for (int r = 0; r < tp->repeats; ++r) {
      for (int b = 0; b < nb; ++b) {
        int rc = asc_engine_set_base_pose(e, b, pf + 6 * b);
        if (rc) return rc;
      }
      long long ev = 0;
      int rc = asc_engine_optimize_frame(e, &tp->opt, pf, costs ? costs + (size_t)f * nb : nullptr, &ev, stream);
      if (rc) return rc;
      evals += ev;
    }
  }
  if (evals_out) *evals_out = evals;
  return ASC_OK;
}

ASC_API int asc_engine_optimize_curves(asc_engine e, const asc_pose_curve* curves, int frame, int n_frames,
                                       const asc_track_params* tp, double* costs, long long* evals_out, void* stream)
{
  if (!e || !curves || !tp || tp->repeats < 0 || tp->guess < 0 || frame < 0 || frame >= n_frames)
    return ASC_ERR_ARG;
  const int nb = e->n_bones, d = tp->dframe;
  for (int b = 0; b < nb; ++b)
    if (!curves[b]) return ASC_ERR_ARG;
  // initial guess (Tracker.cpp:386-426), written into the curves at `frame`
  const int behind = d > 0 ? frame : n_frames - frame - 1;
  for (int b = 0; b < nb; ++b) {
    double p1[6], p2[6], g[6];
    if (tp->guess == 2 && behind > 1) {
      double a[12], c[12], x[12];
      asc_pose_curve_eval(curves[b], frame - 2 * d, p1);
      asc_pose_curve_eval(curves[b], frame - d, p2);
      frame_from_xyzypr(p1, a);
      frame_from_xyzypr(p2, c);
      frame_linear_extrap(a, c, x);
      frame_to_xyzypr(x, g);
      asc_pose_curve_insert(curves[b], frame, g, ASC_CURVE_ALL);
    } else if (tp->guess == 1 && behind > 0) {
      asc_pose_curve_eval(curves[b], frame - d, g);
      asc_pose_curve_insert(curves[b], frame, g, ASC_CURVE_ALL);
    }
  }
  // repeats (Tracker.cpp:428-572): from the curves' pose at the frame, the
  // optimized pose inserted back
  long long evals = 0;
  std::vector<double> stored(6 * nb), raw(6 * nb);
  for (int r = 0; r < tp->repeats; ++r) {
    for (int b = 0; b < nb; ++b) {
      double base[6];
      asc_pose_curve_eval(curves[b], frame, base);
      int rc = asc_engine_set_base_pose(e, b, base);
      if (rc) return rc;
    }
    long long ev = 0;
    int rc = asc_engine_optimize_frame_ex(e, &tp->opt, stored.data(), raw.data(), costs, &ev, stream);
    if (rc) return rc;
    evals += ev;
    for (int b = 0; b < nb; ++b) asc_pose_curve_insert(curves[b], frame, raw.data() + 6 * b, ASC_CURVE_ALL);
  }
  if (evals_out) *evals_out = evals;
  return ASC_OK;
}

// ---------------------------------------------------------------- images
ASC_API int asc_engine_render_drr(asc_engine e, int view, const double* poses, const double* viewport, float* out,
                                  void* stream)
{
  if (!e || !poses || !out || view < 0 || view >= e->n_views) return ASC_ERR_ARG;
  if (!identity_slots(e)) return ASC_ERR_STATE;
  cudaStream_t s = S(stream);
  const ViewDev& V = e->host.views[view];
  const asc_view_desc& VD = e->vdesc[view];
  const double full[4] = {-V.cvp[2] / 2, -V.cvp[3] / 2, V.cvp[2], V.cvp[3]};
  const double* vp = viewport ? viewport : full;
  // the render size of the viewport (Tracker.cpp:617-621), at most the buffer
  const double fw = vp[2] * e->host.rw / V.cvp[2], fh = vp[3] * e->host.rh / V.cvp[3];
  const int w = fw > 0 ? std::min((int)fw, e->host.rw) : 0, h = fh > 0 ? std::min((int)fh, e->host.rh) : 0;
  if (w == 0 || h == 0) return ASC_OK;
  const float vpf[4] = {(float)vp[0], (float)vp[1], (float)vp[2], (float)vp[3]};
  // View::renderDrr (View.cpp:201-231): each bone's DRR merged (sum clamped
  // to 1) into a zeroed buffer, then the view's DRR filters.  The first DRR is the merge with zeros
  bool any = false;
  for (int b = 0; b < e->n_bones; ++b) {
    const BoneDev& B = e->host.bones[b];
    const asc_bone_desc& BD = e->bdesc[b];
    float m[12];
    view_matrix(V, B, poses + 6 * b, m);
    if (!B.visible) continue;  // its zeros leave the merge unchanged
    int rc = raycast_launch(B.vol, g_empty_skip ? B.clr[view] : nullptr, m, vpf, BD.step[view], BD.intensity[view],
                            BD.cutoff[view], e->p_mask, any, w, h, s);
    if (rc) return rc;
    any = true;
  }
  if (!any) ASC_CUDA(cudaMemsetAsync(e->p_mask, 0, (size_t)w * h * sizeof(float), s));
  float *d = e->p_mask, *o = e->p_tmp;
  int rc = chain_plain(VD.drr_filters, VD.n_drr_filters, d, o, w, h, s);
  if (!rc) ASC_CUDA(cudaMemcpyAsync(out, d, (size_t)w * h * sizeof(float), cudaMemcpyDeviceToDevice, s));
  return rc;
}

ASC_API int asc_engine_image_data(asc_engine e, int view, int bone, const double pose[6], float* rad, float* drr,
                                  float* mask, int* width, int* height, void* stream)
{
  if (!e || !pose || !rad || !drr || !mask || view < 0 || view >= e->n_views || bone < 0 || bone >= e->n_bones)
    return ASC_ERR_ARG;
  if (!identity_slots(e)) return ASC_ERR_STATE;
  cudaStream_t s = S(stream);
  const ViewDev& V = e->host.views[view];
  const asc_view_desc& VD = e->vdesc[view];
  const BoneDev& B = e->host.bones[bone];
  const asc_bone_desc& BD = e->bdesc[bone];
  // Tracker::getImageData (Tracker.cpp:865-925): the whole image, viewport
  // (-w/2, -h/2, w, h) of the camera's, at the render size
  const double vp[4] = {-V.cvp[2] / 2, -V.cvp[3] / 2, V.cvp[2], V.cvp[3]};
  const int w = e->host.rw, h = e->host.rh;
  const float vpf[4] = {(float)vp[0], (float)vp[1], (float)vp[2], (float)vp[3]};
  float m[12];
  view_matrix(V, B, pose, m);
  int rc = render_bone(B, BD, view, m, vpf, e->p_drr, w, h, s);
  float *d = e->p_drr, *o = e->p_tmp;
  if (!rc) rc = chain_plain(VD.drr_filters, VD.n_drr_filters, d, o, w, h, s);
  if (!rc) rc = asc_rad_render(VD.radiograph, V.ipf, vpf, e->p_rad, w, h, s);
  float *r = e->p_rad, *ro = o;
  if (!rc) rc = chain_plain(VD.rad_filters, VD.n_rad_filters, r, ro, w, h, s);
  float* bgm = nullptr;
  if (!rc && VD.background && VD.bg_threshold >= 0) {
    bgm = e->p_bgr;
    rc = asc_background_render(VD.background, V.ipf, vpf, VD.bg_threshold, bgm, w, h, s);
  }
  if (!rc) rc = mask_images(d, r, bgm, mask, drr, rad, (size_t)w * h, s);
  if (rc) return rc;
  if (width) *width = w;
  if (height) *height = h;
  return ASC_OK;
}

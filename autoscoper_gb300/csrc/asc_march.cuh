// Ray march of the DRR ray caster: device volume layout, double-float ray
// set-up and the FP32 march.  Self-contained so that it also compiles as
// host C++ (tests/cpp/host_march.cpp provides the few intrinsics).
#pragma once

namespace asc {

// --------------------------------------------------------------------------
// Device volume.  Voxels are stored "x-paired": a word for voxel x holds
// voxel x in its low half and voxel x+1 in its high half, so that one 32-bit
// word carries both x taps of a trilinear sample.  The grid is padded by PAD
// voxels on every side with copies of the edge voxels, which is
// clamp-to-edge addressing (cutil_create_tex_obj.h:18-23) built into the
// layout: the taps of any sample inside the volume box need no per-sample
// clamping.  The halves are u16 integers (ASC_STORE_U16), IEEE half
// (ASC_STORE_F16) or bfloat16 (ASC_STORE_BF16), all holding the stored
// integer value; `norm` (1/65535 or 1/255) turns a raw value into the
// normalized float that cudaReadModeNormalizedFloat would return.
// --------------------------------------------------------------------------
constexpr int PAD = 2;
// Each voxel holds two words, the x-pairs of rows y and y+1 ("quads"), so
// that one 8-byte load fetches four taps of a sample and a sample takes two
// loads (ASC_QUADS=0 builds the one-word pair layout, four loads a sample).
#ifndef ASC_QUADS
#define ASC_QUADS 1
#endif
constexpr int QROWS = ASC_QUADS ? 2 : 1;  // x-pairs (rows y, y+1) per voxel

// 32-bit words per voxel: an x-pair is one word of two 16-bit halves, or two
// FP32 words (ASC_STORE_F32).
__host__ __device__ inline int voxel_words(int storage) { return (storage == ASC_STORE_F32 ? 2 : 1) * QROWS; }

struct DevVolume {
  const uint32_t* pairs;  // (nz + 2 PAD) slices of (ny + 2 PAD) rows of (nx + 2 PAD) voxels
  int nx, ny, nz;         // voxels of the volume itself
  int px, pxy;            // padded row and slice pitch in voxels
  int storage;
  float norm;
  float gmax;  // largest step between neighbouring stored voxels along an axis (raw units)
};

inline size_t padded_words(int nx, int ny, int nz, int storage)
{
  return (size_t)voxel_words(storage) * (nx + 2 * PAD) * (ny + 2 * PAD) * (nz + 2 * PAD);
}

// Fills the padded layout from stored values v(x, y, z) of an nx x ny x nz
// volume (host side): 16-bit halves, or FP32 bits for ASC_STORE_F32.
template <class F>
inline void pack_pairs(int nx, int ny, int nz, int storage, F v, uint32_t* out)
{
  const int px = nx + 2 * PAD, py = ny + 2 * PAD, pz = nz + 2 * PAD, wpv = voxel_words(storage);
  auto cl = [](int i, int n) { return i < 0 ? 0 : (i > n - 1 ? n - 1 : i); };
  for (int zp = 0; zp < pz; ++zp)
    for (int yp = 0; yp < py; ++yp)
      for (int xp = 0; xp < px; ++xp) {
        const int z = cl(zp - PAD, nz), x0 = cl(xp - PAD, nx), x1 = cl(xp - PAD + 1, nx);
        uint32_t* o = out + (((size_t)zp * py + yp) * px + xp) * wpv;
        for (int r = 0; r < QROWS; ++r) {
          const int y = cl(yp - PAD + r, ny);
          if (storage == ASC_STORE_F32) {
            o[2 * r] = v(x0, y, z);
            o[2 * r + 1] = v(x1, y, z);
          } else {
            o[r] = v(x0, y, z) | (v(x1, y, z) << 16);
          }
        }
      }
}

// The largest step between neighbouring voxels along an axis, max |v(p + e_i)
// - v(p)|, of stored values v(x, y, z) (host side).  Bounds the slope of the
// trilinear interpolant along every axis, so it turns a sample's position
// error into a value error (Cutoff).  The clamp-to-edge apron adds no steps.
template <class F>
inline float volume_gmax(int nx, int ny, int nz, F v)
{
  float g = 0.f;
  for (int z = 0; z < nz; ++z)
    for (int y = 0; y < ny; ++y)
      for (int x = 0; x < nx; ++x) {
        const float a = v(x, y, z);
        if (x + 1 < nx) g = std::max(g, std::fabs(v(x + 1, y, z) - a));
        if (y + 1 < ny) g = std::max(g, std::fabs(v(x, y + 1, z) - a));
        if (z + 1 < nz) g = std::max(g, std::fabs(v(x, y, z + 1) - a));
      }
  return g;
}

template <int STORE>
__device__ __forceinline__ void unpack(uint32_t w, float& lo, float& hi)
{
  if (STORE == ASC_STORE_BF16) {
    lo = __uint_as_float(w << 16);
    hi = __uint_as_float(w & 0xffff0000u);
  } else if (STORE == ASC_STORE_F16) {
    __half2_raw r;
    r.x = (unsigned short)(w & 0xffffu);
    r.y = (unsigned short)(w >> 16);
    float2 f = __half22float2(*reinterpret_cast<__half2*>(&r));
    lo = f.x;
    hi = f.y;
  } else {
    // u16 -> float without a conversion unit: 2^23 + v is exact in FP32.
    lo = __uint_as_float(0x4b000000u | (w & 0xffffu)) - 8388608.0f;
    hi = __uint_as_float(0x4b000000u | (w >> 16)) - 8388608.0f;
  }
}

// Linear interpolation between the two halves of a paired word with weight
// a on the high half.  For u16 halves the values stay biased by 2^23: the
// biased values, their difference and the removal of the bias are exact in
// FP32, so this equals fmaf(a, hi - lo, lo) of the unbiased values.
template <int STORE>
__device__ __forceinline__ float lerp_pair(uint32_t w, float a)
{
  if (STORE == ASC_STORE_U16) {
    // 2^23 + v: the half's two bytes under the exponent byte 0x4b
    const float lo = __uint_as_float(__byte_perm(w, 0x4b000000u, 0x7610)),
                hi = __uint_as_float(__byte_perm(w, 0x4b000000u, 0x7632));
    return fmaf(a, hi - lo, lo - 8388608.0f);
  } else {
    float lo, hi;
    unpack<STORE>(w, lo, hi);
    return fmaf(a, hi - lo, lo);
  }
}

// Raw value of padded voxel i (the low half of its first x-pair).
template <int STORE>
__device__ __forceinline__ float voxel_value(const DevVolume& V, size_t i)
{
  const uint32_t w = V.pairs[(size_t)voxel_words(STORE) * i];
  if constexpr (STORE == ASC_STORE_F32) {
    return __uint_as_float(w);
  } else {
    float lo, hi;
    unpack<STORE>(w, lo, hi);
    return lo;
  }
}

// The eight taps of a sample whose lower taps are voxel i, as its four
// x-pairs (rows y, y+1 of slices z, z+1) in the storage's own form, and their
// linear interpolation along x with weight a.
template <int STORE>
struct Taps {
  uint32_t w[4];
};
template <>
struct Taps<ASC_STORE_F32> {
  float2 p[4];
};

template <int STORE>
__device__ __forceinline__ Taps<STORE> fetch_taps(const uint32_t* __restrict__ P, unsigned i, unsigned px,
                                                  unsigned pxy)
{
  Taps<STORE> t;
  if constexpr (STORE == ASC_STORE_F32) {
#if ASC_QUADS
    const float4* Q = reinterpret_cast<const float4*>(P);
    const float4 a = __ldg(Q + i), c = __ldg(Q + i + pxy);
    t.p[0] = make_float2(a.x, a.y);
    t.p[1] = make_float2(a.z, a.w);
    t.p[2] = make_float2(c.x, c.y);
    t.p[3] = make_float2(c.z, c.w);
#else
    const float2* Q = reinterpret_cast<const float2*>(P);
    t.p[0] = __ldg(Q + i);
    t.p[1] = __ldg(Q + i + px);
    t.p[2] = __ldg(Q + i + pxy);
    t.p[3] = __ldg(Q + i + pxy + px);
#endif
  } else {
#if ASC_QUADS
    const uint2* Q = reinterpret_cast<const uint2*>(P);
    const uint2 a = __ldg(Q + i), c = __ldg(Q + i + pxy);
    t.w[0] = a.x;
    t.w[1] = a.y;
    t.w[2] = c.x;
    t.w[3] = c.y;
#else
    t.w[0] = __ldg(P + i);
    t.w[1] = __ldg(P + i + px);
    t.w[2] = __ldg(P + i + pxy);
    t.w[3] = __ldg(P + i + pxy + px);
#endif
  }
  return t;
}

template <int STORE>
__device__ __forceinline__ float lerp_tap(const Taps<STORE>& t, int k, float a)
{
  if constexpr (STORE == ASC_STORE_F32)
    return fmaf(a, t.p[k].y - t.p[k].x, t.p[k].x);
  else
    return lerp_pair<STORE>(t.w[k], a);
}

// ---- two samples at once.  The packed FP32 operations of sm_100 and later
// (fma.rn.f32x2, add.f32x2) apply one IEEE operation to each half, so every
// value below equals, bit for bit, the scalar expression cited beside it.
__device__ __forceinline__ float2 bcast2(float a) { return make_float2(a, a); }
// a - b with one rounding
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __ffma2_rn(b, bcast2(-1.0f), a); }

// lerp_tap of tap word k of samples A (x) and B (y), weights a.  The u16
// halves of every other word go through the conversion unit, which then needs
// no bias taken off (two issue slots a pair of samples less), the rest through
// byte permutations: the unit converts 16 values a clock and SM, so with all
// eight words of a pair it bounds the march itself.  k_ray on 300 candidates x
// 2 views of 1024^2: 12.23 ms with no word converted, 11.92 with half of them,
// 12.52 with all.
template <int STORE>
__device__ __forceinline__ float2 lerp_tap2(const Taps<STORE>& A, const Taps<STORE>& B, int k, float2 a)
{
  float2 lo, hi;
  if constexpr (STORE == ASC_STORE_F32) {
    lo = make_float2(A.p[k].x, B.p[k].x);
    hi = make_float2(A.p[k].y, B.p[k].y);
  } else if constexpr (STORE == ASC_STORE_U16) {
    if ((k & 1) == 0) {
      lo = make_float2((float)(unsigned short)A.w[k], (float)(unsigned short)B.w[k]);
      hi = make_float2((float)(unsigned short)(A.w[k] >> 16), (float)(unsigned short)(B.w[k] >> 16));
      return __ffma2_rn(a, sub2(hi, lo), lo);
    }
    // lerp_pair: fmaf(a, hi - lo, lo - 2^23) of the biased halves
    lo = make_float2(__uint_as_float(__byte_perm(A.w[k], 0x4b000000u, 0x7610)),
                     __uint_as_float(__byte_perm(B.w[k], 0x4b000000u, 0x7610)));
    hi = make_float2(__uint_as_float(__byte_perm(A.w[k], 0x4b000000u, 0x7632)),
                     __uint_as_float(__byte_perm(B.w[k], 0x4b000000u, 0x7632)));
    return __ffma2_rn(a, sub2(hi, lo), __fadd2_rn(lo, bcast2(-8388608.0f)));
  } else {
    unpack<STORE>(A.w[k], lo.x, hi.x);
    unpack<STORE>(B.w[k], lo.y, hi.y);
  }
  return __ffma2_rn(a, sub2(hi, lo), lo);  // fmaf(a, hi - lo, lo)
}

// The trilinear values of samples A and B (march_block's accumulate)
template <int STORE>
__device__ __forceinline__ float2 trilinear2(const Taps<STORE>& A, const Taps<STORE>& B, float2 wx, float2 wy,
                                             float2 wz)
{
  const float2 e00 = lerp_tap2<STORE>(A, B, 0, wx), e10 = lerp_tap2<STORE>(A, B, 1, wx);
  const float2 e01 = lerp_tap2<STORE>(A, B, 2, wx), e11 = lerp_tap2<STORE>(A, B, 3, wx);
  const float2 f0 = __ffma2_rn(wy, sub2(e10, e00), e00);  // fmaf(wy, e10 - e00, e00)
  const float2 f1 = __ffma2_rn(wy, sub2(e11, e01), e01);
  return __ffma2_rn(wz, sub2(f1, f0), f0);                // fmaf(wz, f1 - f0, f0)
}

// ---- double-float arithmetic: a value is the unevaluated sum h + l of two
// FP32 numbers (Dekker/Knuth error-free transformations with FMA), 44 to 48
// significant bits.  Used once per ray so that sample positions match FP64.
struct df {
  float h, l;
};

__device__ __forceinline__ df df_two_sum(float a, float b)
{
  const float s = __fadd_rn(a, b);
  const float bb = __fadd_rn(s, -a);
  return {s, __fadd_rn(__fadd_rn(a, -__fadd_rn(s, -bb)), __fadd_rn(b, -bb))};
}

__device__ __forceinline__ df df_fast(float a, float b)  // requires |a| >= |b|
{
  const float s = __fadd_rn(a, b);
  return {s, __fadd_rn(b, -__fadd_rn(s, -a))};
}

// Sum with an exact sum of the high parts and the low parts added in FP32
// (Dekker's addition): relative error ~2^-44 of the larger operand.  Every
// use here needs absolute accuracy in coordinates and ray parameters whose
// magnitudes are at most ~1e4 (voxels, samples): ~1e-9 at worst, far below
// the FP32 rounding of the sample positions the march then uses.
__device__ __forceinline__ df df_add(df a, df b)
{
  df s = df_two_sum(a.h, b.h);
  s.l = __fadd_rn(s.l, __fadd_rn(a.l, b.l));
  return df_fast(s.h, s.l);
}

__device__ __forceinline__ df df_neg(df a) { return {-a.h, -a.l}; }

__device__ __forceinline__ df df_mulf(df a, float b)
{
  const float p = __fmul_rn(a.h, b);
  float e = fmaf(a.h, b, -p);
  e = fmaf(a.l, b, e);
  return df_fast(p, e);
}

__device__ __forceinline__ df df_mul(df a, df b)
{
  const float p = __fmul_rn(a.h, b.h);
  float e = fmaf(a.h, b.h, -p);
  e = fmaf(a.h, b.l, e);
  e = fmaf(a.l, b.h, e);
  return df_fast(p, e);
}

__device__ __forceinline__ df df_div(df a, df b)
{
  const float q1 = __fdiv_rn(a.h, b.h);
  df r = df_add(a, df_neg(df_mulf(b, q1)));
  const float q2 = __fdiv_rn(r.h, b.h);
  r = df_add(r, df_neg(df_mulf(b, q2)));
  const float q3 = __fdiv_rn(r.h, b.h);
  return df_add(df_fast(q1, q2), df{q3, 0.f});
}

__device__ __forceinline__ df df_sqrt(df a)
{
  const float s = __fsqrt_rn(a.h);
  if (!(s > 0.f)) return {s, 0.f};
  const df e = df_add(a, df_neg(df_mul(df{s, 0.f}, df{s, 0.f})));
  return df_fast(s, __fdiv_rn(e.h, 2.0f * s));
}

__device__ __forceinline__ bool df_lt(df a, df b) { return a.h < b.h || (a.h == b.h && a.l < b.l); }

// 1/a and 1/sqrt(a) in double-float: one Newton step from the FP32 value
// (relative error of the FP32 start squared, ~1e-13).
__device__ __forceinline__ df df_rcp(df a)
{
  const float r = __frcp_rn(a.h);
  const df e = df_add(df{1.0f, 0.f}, df_neg(df_mulf(a, r)));  // 1 - a r
  return df_fast(r, __fmul_rn(r, e.h));
}

__device__ __forceinline__ df df_rsqrt(df a)
{
  const float r = rsqrtf(a.h);
  const df r2 = df_mul(df{r, 0.f}, df{r, 0.f});
  const df e = df_add(df{1.0f, 0.f}, df_neg(df_mul(a, r2)));  // 1 - a r^2
  return df_fast(r, __fmul_rn(0.5f * r, e.h));
}

// A float value as a double-float from a double (host or device).
__device__ __host__ __forceinline__ void df_split(double d, float& h, float& l)
{
  h = (float)d;
  l = (float)(d - (double)h);
}

// The cutoff test of the march (RayCaster_kernels.cu:189: density += s >
// cutoff ? step * s : 0), on raw voxel values.  The reference compares
// raw / vmax with c (vmax 65535 or 255); the exact threshold is c x vmax,
// kept as the double-float (th, tl); the FP32 march compares with raw = c /
// norm.
//
// An FP32 sample v differs from the exact trilinear value at its exact
// position by at most
//   u (3 |v| + 11 G)                   the seven lerps' roundings (the taps
//                                      lie within 3 G of v)
//   + G u (9 + 130 (|dX| + |dY| + |dZ|))  the position per axis: the
//                                      fraction's rounding, the FMA of the
//                                      sample offset (values below 1 + 64 |d|)
//                                      and the offset times the dropped low
//                                      part of d; the interpolant's slope
//                                      along an axis is at most G
// with u = 2^-24, G = DevVolume::gmax and d the per-sample step of each axis
// in voxels; raw differs from c x vmax by at most 2 u |raw|.  So a sample
// with |v - raw| >= t0 + t1 (|dX| + |dY| + |dZ|), t0 = u (8 |raw| + 24 G) +
// 1e-6 and t1 = 140 u G, lies on the same side of the threshold in FP32 as
// exactly (3 u |raw| of t0 cover the roundings of the band's ends).  The
// march decides such samples in FP32 and flags the rest (the band); a
// flagged march is redone with the samples in the band decided from their
// double-float position and a double-float trilinear value against (th, tl)
// (sample_above).
//
// When |raw| <= 2 t0 the band is dropped (t0 = t1 = 0, the samples above
// raw, i.e. at or above the next float hi0, counted): a sample decided the
// other way then adds or leaves out at most |raw| + t0, a few times the FP32
// error every counted sample carries, and a cutoff of 0 keeps its empty
// cells (a band reaching below 0 would leave none).
//
// The clearance grids are built at raw - t0 (<= c x vmax): a sample whose
// voxels all lie at or below it is one that the exact test leaves out.
struct Cutoff {
  float raw;      // c / norm, the FP32 threshold
  float hi0;      // raw, or with the band dropped the next float above it
  float t0, t1;   // the band's half-width: t0 + t1 (|dX| + |dY| + |dZ|)
  float th, tl;   // c x vmax as a double-float
};

__host__ __device__ inline Cutoff make_cutoff(float c, float norm, float gmax)
{
  Cutoff k;
  k.raw = c / norm;
  const float u = 5.9604645e-8f;  // 2^-24
  k.t0 = u * (8.0f * fabsf(k.raw) + 24.0f * gmax) + 1e-6f;
  k.t1 = 140.0f * u * gmax;
  k.hi0 = k.raw;
  if (!(fabsf(k.raw) > 2.0f * k.t0)) {
    k.t0 = k.t1 = 0.f;
    k.hi0 = nextafterf(k.raw, INFINITY);
  }
  const double vmax = (double)(int)(1.0f / norm + 0.5f);
  df_split((double)c * vmax, k.th, k.tl);
  return k;
}

// The clearance grids' threshold (Cutoff).
__host__ __device__ inline float occupancy_threshold(const Cutoff& k) { return k.raw - k.t0; }

// The band of a ray with per-sample steps dX, dY, dZ: samples in (lo, hi)
// are decided exactly, samples at or above hi count.
__host__ __device__ inline void cutoff_bounds(const Cutoff& k, float dX, float dY, float dZ, float& lo, float& hi)
{
  const float tol = fmaf(k.t1, fabsf(dX) + fabsf(dY) + fabsf(dZ), k.t0);
  lo = k.raw - tol;
  hi = k.hi0 + tol;
}

// Per-ray set-up of cuda_volume_render_kernel (RayCaster_kernels.cu:144-186)
// for pixel (x, y) of an image over viewport `vp`, with camera->volume matrix
// m (3x4 row-major, normalisation folded), in double-float: the reference's
// FP32 set-up misplaces the far intersection by ~1e-7 of its length, which
// shifts every sample of the ray; here positions agree with FP64 to ~1e-6
// voxel.  (sxh, sxl) and (syh, syl) are vp[2] / w and vp[3] / h as
// double-floats, so that u = vp[0] + x vp[2] / w.  Sample k (k = 0 .. K-1)
// sits at t = far - k, texel coordinates (X - k dX, Y - k dY, Z - k dZ) with
// texel centres at integers.
struct RaySetup {
  int K;
  df X, Y, Z, dX, dY, dZ;
  float tf;  // far, in samples from the camera (sample k sits at tf - k)
};

__device__ __forceinline__ bool ray_setup(const float* m, const float* vp, int x, int y, df sx, df sy, float step,
                                          int nx, int ny, int nz, RaySetup& r)
{
  const df u = df_add(df{vp[0], 0.f}, df_mulf(sx, (float)x));
  const df v = df_add(df{vp[1], 0.f}, df_mulf(sy, (float)y));
  const df sc = df_mulf(df_rsqrt(df_add(df_add(df_mul(u, u), df_mul(v, v)), df{4.0f, 0.f})), step);
  const df l0 = df_mul(u, sc), l1 = df_mul(v, sc), l2 = df_mulf(sc, -2.0f);
  df d[3];
  for (int i = 0; i < 3; ++i)
    d[i] = df_add(df_add(df_mulf(l0, m[4 * i]), df_mulf(l1, m[4 * i + 1])), df_mulf(l2, m[4 * i + 2]));
  const float o[3] = {m[3], m[7], m[11]};
  const float lo[3] = {0.0f, 0.0f, -1.0f}, hi[3] = {1.0f, 1.0f, 0.0f};
  df tn = {-3.0e38f, 0.f}, tf = {3.0e38f, 0.f};
  for (int i = 0; i < 3; ++i) {
    if (d[i].h == 0.f) {  // parallel to the slab
      if (!(o[i] > lo[i] && o[i] < hi[i])) return false;
      continue;
    }
    const df rd = df_rcp(d[i]);
    df a = df_mul(df_two_sum(lo[i], -o[i]), rd);
    df b = df_mul(df_two_sum(hi[i], -o[i]), rd);
    if (df_lt(b, a)) {
      const df c = a;
      a = b;
      b = c;
    }
    if (df_lt(tn, a)) tn = a;
    if (df_lt(b, tf)) tf = b;
  }
  if (!df_lt(tn, tf)) return false;  // also a miss for NaN
  if (tn.h < 0.f) tn = df{0.f, 0.f};
  // samples t = far - k > near: K = #{k >= 0 : k < far - near}
  const df D = df_add(tf, df_neg(tn));
  // t -= 1 stops making progress at 2^24; the reference would spin forever on
  // such a degenerate ray, here it counts as a miss.
  if (!(D.h < 8388608.0f)) return false;
  if (D.h < 0.f || (D.h == 0.f && D.l <= 0.f)) {
    r.K = 0;
  } else {
    const float c = ceilf(D.h);
    r.K = (int)c + ((c == D.h && D.l > 0.f) ? 1 : 0);
  }
  // texture coordinates (p.x, 1 - p.y, -p.z) at t = far, minus the half texel
  const df p0 = df_add(df{o[0], 0.f}, df_mul(tf, d[0]));
  const df p1 = df_add(df{o[1], 0.f}, df_mul(tf, d[1]));
  const df p2 = df_add(df{o[2], 0.f}, df_mul(tf, d[2]));
  r.X = df_add(df_mulf(p0, (float)nx), df{-0.5f, 0.f});
  r.Y = df_add(df_mulf(df_add(df{1.0f, 0.f}, df_neg(p1)), (float)ny), df{-0.5f, 0.f});
  r.Z = df_add(df_mulf(df_neg(p2), (float)nz), df{-0.5f, 0.f});
  r.dX = df_mulf(d[0], (float)nx);   // X decreases by dX per sample (t decreases)
  r.dY = df_mulf(d[1], -(float)ny);
  r.dZ = df_mulf(d[2], -(float)nz);
  r.tf = tf.h;
  return true;
}

// ---- clearance grids: where a march may skip.
//
// For one cutoff, cell (cx, cy, cz) covers the texel coordinates
// [2c, 2c + 2) of each axis and holds (a byte) its distance, in voxels and in
// the maximum norm, to the nearest voxel above the threshold, CLEAR_MAX when
// there is none nearer.  A sample at X blends voxel v only where |X - v| < 1 on every
// axis, so every sample within max-norm distance e - 1 of any point of a cell
// of clearance e is a blend of voxels at or below the threshold, hence itself
// at or below it (each FP32 lerp stays between its ends): it adds exactly
// nothing to the DRR (RayCaster_kernels.cu:189) and need not be sampled.
// Coordinates outside the grid take the nearest cell, which lies nearer to
// every voxel than they do.
//
// Why a distance and not an occupancy bit: one byte answers for a whole box
// of positions (a warp's beam over an interval, below), so a warp finds its
// occupied intervals with one load per interval, where a walk of each ray
// through 8-voxel cells took ~1250 warp instructions.  Cells of 2 voxels
// leave at most 2 voxels of slack per query and an eighth of a byte per voxel.
constexpr int CLEAR_CELL = 2, CLEAR_MAX = 15;
__host__ __device__ __forceinline__ int clear_dim(int n) { return (n + CLEAR_CELL - 1) / CLEAR_CELL; }

#ifdef __CUDA_ARCH__
__device__ __forceinline__ float approx_rcp(float x)  // one instruction, ~1 ulp: for positions that carry a margin
{
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
#else
__device__ __forceinline__ float approx_rcp(float x) { return 1.0f / x; }
#endif

// 2^23 + floor(x / CLEAR_CELL) as the bits of a float (0 <= x < 2^23): the
// directed rounding of one FMA.
__device__ __forceinline__ unsigned cell_bits(float x)
{
#ifdef __CUDA_ARCH__
  return __float_as_uint(__fmaf_rd(1.0f / CLEAR_CELL, x, 8388608.0f));
#else
  return __float_as_uint(8388608.0f + floorf(x * (1.0f / CLEAR_CELL)));
#endif
}

// The clearance at a texel position of an nx x ny x nz volume: the cell
// clamped to the grid (a position above n - 1 lies in the last cell's reach),
// the three biases of its index taken off at once (mod 2^32).
__device__ __forceinline__ float clearance_at(const uint8_t* __restrict__ clr, int nx, int ny, int nz, float X, float Y,
                                              float Z)
{
  const unsigned BM = 0x4b000000u, gx = (unsigned)clear_dim(nx), gxy = gx * (unsigned)clear_dim(ny);
  const unsigned cx = cell_bits(fminf(fmaxf(X, 0.f), (float)(nx - 1)));
  const unsigned cy = cell_bits(fminf(fmaxf(Y, 0.f), (float)(ny - 1)));
  const unsigned cz = cell_bits(fminf(fmaxf(Z, 0.f), (float)(nz - 1)));
  return __uint_as_float(BM | __ldg(clr + (cz * gxy + cy * gx + cx - BM * (gxy + gx + 1u)))) - 8388608.0f;
}

// One ray of a beam in FP32: texel coordinates O + t D at t samples from the
// camera (O the same for every ray of an image), and the t-range
// (near, far) in which it crosses the volume's box widened by `err` voxels,
// which bounds the FP32 error of O + t D there.
struct BeamRay {
  float O[3], D[3];
  float near, far, err;
};

__device__ __forceinline__ BeamRay beam_ray(const float* m, const float* vp, float sx, float sy, float x, float y,
                                            float step, float nx, float ny, float nz)
{
  BeamRay b;
  const float u = fmaf(sx, x, vp[0]), v = fmaf(sy, y, vp[1]);
  const float il = step * rsqrtf(fmaf(u, u, fmaf(v, v, 4.0f)));
  const float l0 = u * il, l1 = v * il, l2 = -2.0f * il;
  b.D[0] = nx * fmaf(m[0], l0, fmaf(m[1], l1, m[2] * l2));
  b.D[1] = -ny * fmaf(m[4], l0, fmaf(m[5], l1, m[6] * l2));
  b.D[2] = -nz * fmaf(m[8], l0, fmaf(m[9], l1, m[10] * l2));
  b.O[0] = fmaf(m[3], nx, -0.5f);
  b.O[1] = fmaf(1.0f - m[7], ny, -0.5f);
  b.O[2] = fmaf(-m[11], nz, -0.5f);
  const float n[3] = {nx, ny, nz};
  b.err = 0.02f + 2.0e-6f * (fmaxf(fabsf(b.O[0]), fmaxf(fabsf(b.O[1]), fabsf(b.O[2]))) + fmaxf(nx, fmaxf(ny, nz)));
  b.near = 0.f;
  b.far = 3.0e38f;
  for (int i = 0; i < 3; ++i) {
    const float r = approx_rcp(b.D[i]);
    const float p = (-0.5f - b.err - b.O[i]) * r, q = (n[i] - 0.5f + b.err - b.O[i]) * r;
    b.near = fmaxf(b.near, fminf(p, q));
    b.far = fminf(b.far, fmaxf(p, q));
  }
  return b;
}

// Whether the beam of all rays with directions within w (per axis) of D,
// between t = tc - half and tc + half, may hold a sample above the threshold.
// wide: no clearance could clear it, it reaches too far from its middle.
__device__ __forceinline__ bool beam_occupied(const uint8_t* __restrict__ clr, int nx, int ny, int nz, const float* O,
                                              const float* D, const float* w, float tc, float half, float err,
                                              bool& wide)
{
  float h = 0.f;
  for (int i = 0; i < 3; ++i) h = fmaxf(h, fmaf(tc + half, w[i], half * fabsf(D[i])));
  const float need = h + 1.0f + err;
  wide = wide || need > (float)CLEAR_MAX;
  const float e = clearance_at(clr, nx, ny, nz, fmaf(tc, D[0], O[0]), fmaf(tc, D[1], O[1]), fmaf(tc, D[2], O[2]));
  return !(e >= need);
}

// The march re-bases its FP32 coordinates every REBASE samples (march_block).
#ifndef ASC_REBASE
#define ASC_REBASE 64
#endif
constexpr int REBASE = ASC_REBASE;

// Whether every sample of a ray has its taps in the padded grid whatever the
// rounding: its first and last sample lie within a voxel of the volume's box,
// hence all between them do, and the apron's second voxel exceeds what FP32
// positions (march_block) are off by on an axis of at most 2^16 voxels.  Rays that
// ray_setup cut to the box meet it.
__device__ __forceinline__ bool ray_inside(const DevVolume& V, const RaySetup& r)
{
  const float l = (float)(r.K - 1);
  const float X = fmaf(-l, r.dX.h, r.X.h), Y = fmaf(-l, r.dY.h, r.Y.h), Z = fmaf(-l, r.dZ.h, r.Z.h);
  return fminf(fminf(fminf(r.X.h, X), fminf(r.Y.h, Y)), fminf(r.Z.h, Z)) >= -1.0f && fmaxf(r.X.h, X) <= (float)V.nx &&
         fmaxf(r.Y.h, Y) <= (float)V.ny && fmaxf(r.Z.h, Z) <= (float)V.nz && max(max(V.nx, V.ny), V.nz) <= 65536;
}

// Integer base and FP32 fraction of coordinate C - k dC.  The march re-bases
// at every multiple of REBASE samples, so that the fraction stays small
// (|fraction| < 1 + REBASE |d|, exact to a few 1e-6 voxel) and a sample's
// coordinates depend on its index k alone.
__device__ __forceinline__ void coord_base(df C, df dC, float k, int& base_i, float& frac)
{
  const df c = df_add(C, df_neg(df_mulf(dC, k)));
  const float fl = floorf(c.h);
  base_i = (int)fminf(fmaxf(fl, -1.0e6f), 1.0e6f);
  frac = __fadd_rn(__fadd_rn(c.h, -fl), c.l);
}

// Whether sample k of a ray lies above the cutoff, computed exactly enough
// to agree with FP64: the position and the trilinear value in double-float,
// against the threshold (th, tl) (Cutoff).  Decides the samples in the band.
template <int STORE>
__device__ __forceinline__ bool sample_above(const DevVolume& V, const RaySetup& r, int k, const Cutoff& cut)
{
  const float kf = (float)k;
  const df C[3] = {df_add(r.X, df_neg(df_mulf(r.dX, kf))), df_add(r.Y, df_neg(df_mulf(r.dY, kf))),
                   df_add(r.Z, df_neg(df_mulf(r.dZ, kf)))};
  int b[3];
  df f[3];
  for (int i = 0; i < 3; ++i) {
    float fl = floorf(C[i].h);
    if (fl == C[i].h && C[i].l < 0.f) fl -= 1.0f;  // h + l lies just below the integer h
    fl = fminf(fmaxf(fl, -1.0f), 1.0e6f);
    b[i] = (int)fl;
    f[i] = df_two_sum(__fadd_rn(C[i].h, -fl), C[i].l);  // C - floor(C): h - floor(h) is exact
  }
  const unsigned px = (unsigned)V.px, pxy = (unsigned)V.pxy;
  const unsigned imax = ASC_QUADS ? (unsigned)(V.nz + 2 * PAD - 1) * pxy - 1u
                                  : (unsigned)(V.nz + 2 * PAD - 1) * pxy - px - 1u;
  const unsigned i = min((unsigned)(b[2] + PAD) * pxy + (unsigned)(b[1] + PAD) * px + (unsigned)(b[0] + PAD), imax);
  const Taps<STORE> t = fetch_taps<STORE>(V.pairs, i, px, pxy);
  df e[4];
  for (int q = 0; q < 4; ++q) {
    float lo, hi;
    if constexpr (STORE == ASC_STORE_F32) {
      lo = t.p[q].x;
      hi = t.p[q].y;
    } else {
      unpack<STORE>(t.w[q], lo, hi);
    }
    e[q] = df_add(df{lo, 0.f}, df_mulf(f[0], __fadd_rn(hi, -lo)));  // raw values: hi - lo is exact
  }
  const df f0 = df_add(e[0], df_mul(f[1], df_add(e[1], df_neg(e[0]))));
  const df f1 = df_add(e[2], df_mul(f[1], df_add(e[3], df_neg(e[2]))));
  const df v = df_add(f0, df_mul(f[2], df_add(f1, df_neg(f0))));
  return df_lt(df{cut.th, cut.tl}, v);
}

// Samples kb + js .. kb + je of one march block (kb a multiple of REBASE) of
// cuda_volume_render_kernel's loop (RayCaster_kernels.cu:187-195; t = far -
// k).  Returns the block's FP32 sum of raw samples above the cutoff (at most
// REBASE of them, so its relative error stays below ~4e-6 and typically near
// 1e-7; the blocks are combined in double-float); a sample at or below the
// cutoff leaves it untouched, so trimming samples that add nothing changes no
// bit.
//
// lo, hi: the cutoff's band for this ray (cutoff_bounds): samples at or
// above hi count, samples in (lo, hi) need the exact test.  EXACT false: a
// sample in the band marks the block, whose sum then comes back negated with
// its sign bit set (-0 for an empty sum; a sum of samples above a cutoff >= 0
// is never negative otherwise, see block_flagged), and the ray must be
// marched again with EXACT true, which decides those samples with
// sample_above.  cut is read only with EXACT.
//
// inside: ray_inside(), on which the taps' index needs no clamp; false: the
// samples one at a time, clamped, to the same bits.
//
// PAIRS: sample pairs whose loads are in flight together.  One where other
// warps cover the loads; more where few warps are resident (they take registers).
template <int STORE, bool EXACT, int PAIRS = 1>
__device__ __forceinline__ float march_block(const DevVolume& V, const RaySetup& r, int kb, int js, int je,
                                              float lo, float hi, const Cutoff& cut, bool inside = false)
{
  const uint32_t* __restrict__ P = V.pairs;
  const unsigned px = (unsigned)V.px, pxy = (unsigned)V.pxy;
  const float dXh = r.dX.h, dYh = r.dY.h, dZh = r.dZ.h;
  int bix, biy, biz;
  float fx, fy, fz;
  const float kbf = (float)kb;
  coord_base(r.X, r.dX, kbf, bix, fx);
  coord_base(r.Y, r.dY, kbf, biy, fy);
  coord_base(r.Z, r.dZ, kbf, biz, fz);
  // Lower tap and weight per axis at fraction X (|X| < 2^22): t = M + X
  // rounded down is M + floor(X), so floor(X) = bits(t) - bits(M) and the
  // weight X - floor(X) in [0, 1) is exact.  The word of the lower taps has
  // padded index (base + PAD + floor) per axis, i.e. bits(tz) pxy + bits(ty)
  // px + bits(tx) + i_base in unsigned (mod 2^32) arithmetic, i_base folding
  // the bases, the padding and bits(M).
  const float M = 12582912.0f;  // 1.5 * 2^23
  const unsigned BM = 0x4b400000u;
  const unsigned i_base = ((unsigned)(biz + PAD) - BM) * pxy + ((unsigned)(biy + PAD) - BM) * px +
                          ((unsigned)(bix + PAD) - BM);
  const unsigned imax = ASC_QUADS ? (unsigned)(V.nz + 2 * PAD - 1) * pxy - 1u
                                  : (unsigned)(V.nz + 2 * PAD - 1) * pxy - px - 1u;
  float acc = 0.f;
  // the largest sample not counted (below hi): above lo once a sample fell
  // in the band (one max, predicated on the test that decides the add)
  float nearf = -3.0e38f;
  // the cutoff test of sample kb + jj with value v: adds v when above
  auto take = [&](float v, float jj) {
    if constexpr (EXACT) {
      if (v >= hi) {
        acc += v;
      } else if (v > lo) {
        if (sample_above<STORE>(V, r, kb + (int)jj, cut)) acc += v;
      }
    } else {
      if (v >= hi)
        acc += v;
      else
        nearf = fmaxf(nearf, v);
    }
  };
  // the taps' voxel index and weights of sample j (j * the low part of d
  // stays below 1e-6 voxel for j < REBASE)
  auto locate = [&](float jj, float& ax, float& ay, float& az) {
    const float X = fmaf(-jj, dXh, fx), Y = fmaf(-jj, dYh, fy), Z = fmaf(-jj, dZh, fz);
    const float tx = __fadd_rd(X, M), ty = __fadd_rd(Y, M), tz = __fadd_rd(Z, M);
    ax = __fadd_rn(X, -__fadd_rn(tx, -M));
    ay = __fadd_rn(Y, -__fadd_rn(ty, -M));
    az = __fadd_rn(Z, -__fadd_rn(tz, -M));
    return min(__float_as_uint(tz) * pxy + __float_as_uint(ty) * px + __float_as_uint(tx) + i_base, imax);
  };
  // Samples two at a time (jj and jj + 1) in packed pairs, both samples'
  // loads issued together; the samples add in order.  The positions are
  // scalar FMAs (the same values as locate's): packed ones would hold six
  // more registers, which the march, at 64 per thread, spills.
  auto locate2 = [&](float jj, float2& wx, float2& wy, float2& wz, unsigned& ia, unsigned& ib) {
    const float j1 = jj + 1.0f;
    const float2 X = make_float2(fmaf(-jj, dXh, fx), fmaf(-j1, dXh, fx));
    const float2 Y = make_float2(fmaf(-jj, dYh, fy), fmaf(-j1, dYh, fy));
    const float2 Z = make_float2(fmaf(-jj, dZh, fz), fmaf(-j1, dZh, fz));
    const float2 tx = __fadd2_rd(X, bcast2(M)), ty = __fadd2_rd(Y, bcast2(M)), tz = __fadd2_rd(Z, bcast2(M));
    wx = sub2(X, __fadd2_rn(tx, bcast2(-M)));
    wy = sub2(Y, __fadd2_rn(ty, bcast2(-M)));
    wz = sub2(Z, __fadd2_rn(tz, bcast2(-M)));
    ia = __float_as_uint(tz.x) * pxy + __float_as_uint(ty.x) * px + __float_as_uint(tx.x) + i_base;
    ib = __float_as_uint(tz.y) * pxy + __float_as_uint(ty.y) * px + __float_as_uint(tx.y) + i_base;
  };
  float j = (float)js;
  const float last = (float)je;
  if (inside) {
    if constexpr (PAIRS > 1) {
      for (; j <= last - (2.0f * PAIRS - 1.0f); j += 2.0f * PAIRS) {
        float2 wx[PAIRS], wy[PAIRS], wz[PAIRS];
        Taps<STORE> A[PAIRS], B[PAIRS];
#pragma unroll
        for (int p = 0; p < PAIRS; ++p) {
          unsigned ia, ib;
          locate2(j + (float)(2 * p), wx[p], wy[p], wz[p], ia, ib);
          A[p] = fetch_taps<STORE>(P, ia, px, pxy);
          B[p] = fetch_taps<STORE>(P, ib, px, pxy);
        }
#pragma unroll
        for (int p = 0; p < PAIRS; ++p) {
          const float2 v = trilinear2<STORE>(A[p], B[p], wx[p], wy[p], wz[p]);
          take(v.x, j + (float)(2 * p));
          take(v.y, j + (float)(2 * p + 1));
        }
      }
    }
#pragma unroll 1
    for (; j < last; j += 2.0f) {
      float2 wx, wy, wz;
      unsigned ia, ib;
      locate2(j, wx, wy, wz, ia, ib);
      const Taps<STORE> A = fetch_taps<STORE>(P, ia, px, pxy), B = fetch_taps<STORE>(P, ib, px, pxy);
      const float2 v = trilinear2<STORE>(A, B, wx, wy, wz);
      take(v.x, j);
      take(v.y, j + 1.0f);
    }
  }
#pragma unroll 1
  for (; j <= last; j += 1.0f) {
    float ax, ay, az;
    const Taps<STORE> t = fetch_taps<STORE>(P, locate(j, ax, ay, az), px, pxy);
    const float e00 = lerp_tap<STORE>(t, 0, ax);
    const float e10 = lerp_tap<STORE>(t, 1, ax);
    const float e01 = lerp_tap<STORE>(t, 2, ax);
    const float e11 = lerp_tap<STORE>(t, 3, ax);
    const float f0 = fmaf(ay, e10 - e00, e00);
    const float f1 = fmaf(ay, e11 - e01, e01);
    const float v = fmaf(az, f1 - f0, f0);
    take(v, j);
  }
  return !EXACT && nearf > lo ? -acc - 0.0f : acc;
}

// Whether a march block's sum carries the band's mark (march_block).
__device__ __forceinline__ bool block_flagged(float p) { return (__float_as_uint(p) >> 31) != 0u; }

// Adds a block's sum to the ray's double-float total; blocks that added
// nothing leave it untouched.
__device__ __forceinline__ void add_block(df& total, float p)
{
  if (p != 0.f) total = df_add(total, df{p, 0.f});
}

}  // namespace asc

#ifndef __CUDACC__
#include "asc_walk.cuh"
#endif

// Plain per-operator kernels of the registration cost path and their C ABI:
// one launch per reference operator call, the drop-in form of
// libautoscoper/src/gpu/cuda/*.  The batched engine (asc_engine.cu) reuses
// the same device functions.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include "asc_internal.cuh"
#include "asc_clear.cuh"
#include "asc_rays.cuh"

namespace asc {

static thread_local std::string g_last_error;

void set_cuda_error(cudaError_t e) { g_last_error = cudaGetErrorString(e); }
void set_error_message(const char* msg) { g_last_error = msg; }

int cuda_status(cudaError_t e)
{
  set_cuda_error(e);
  (void)cudaGetLastError();  // clear a non-sticky error so the context stays usable
  return e == cudaErrorMemoryAllocation ? ASC_ERR_NOMEM : ASC_ERR_CUDA;
}

int gauss_1d(float radius, float* g, int cap)
{
  if (radius < 0) radius = 0;
  int R = (int)(3 * radius);  // float -> int truncation as GaussianFilter.cpp:79
  int K = 2 * R + 1;
  if (K == 1) return 1;
  if (K > cap) return -1;
  double e[128], sum = 0;
  for (int i = 0; i < K; ++i) {
    e[i] = pow(2.71828, -pow((double)(i - R), 2) / (2 * radius));
    sum += e[i];
  }
  for (int i = 0; i < K; ++i) g[i] = (float)(e[i] / sum);
  return K;
}

// ---------------------------------------------------------------- kernels

// cuda_volume_render_kernel (RayCaster_kernels.cu:144-195) for one image: a
// warp, and a block, per beam of 8 x 4 pixels (ray_beam): most beams meet
// nothing, and in a block of several the done ones would hold their warps' places until the
// last is done.  Rays with a sample in the cutoff's band are marched again,
// exactly, by their warp.  merge: the DRR is added to what `out` holds, held to 1.
struct RayArgs {
  float m[12];
  float vp[4];
  float step, scale;
  Cutoff cut;
  float sx[2], sy[2];  // vp[2] / w and vp[3] / h as double-floats
};

// One image fills few warps, so two pairs of samples are in flight per lane
// (96 registers): a 256 x 128 x 128 bone over 1024^2 58 us against 70 with one pair,
// and 98-155 with a thread per ray walking by itself.
constexpr int RAYCAST_PAIRS = 2;
__global__ void __launch_bounds__(32, 20) k_raycast(DevVolume V, const uint8_t* __restrict__ clr,
                                                    const __grid_constant__ RayArgs a, float* __restrict__ out,
                                                    int merge, int y0, int w, int h)
{
  __shared__ RaySlots<32> S;
  __shared__ float s_v[EXACT_FLOATS];
  const int lane = threadIdx.x;
  const int x = blockIdx.x * 8 + (lane & 7), y = y0 + blockIdx.y * 4 + (lane >> 3);
  const bool valid = x < w && y < h;
  const RayScene s{a.m, a.vp, df{a.sx[0], a.sx[1]}, df{a.sy[0], a.sy[1]}, a.step, clr, w, h};
  const Beam b = beam_mask(V, s, min(x, w - 1), min(y, h - 1));
  if (!b.mask && merge) return;  // adds nothing (a DRR lies in [0, 1])
  float d = 0.f;
  if (b.mask) {
    unsigned marched = 0, slots = 0;
    d = ray_beam<RAYCAST_PAIRS>(V, s, a.cut, make_float4(a.cut.raw - a.cut.t0, a.cut.hi0 + a.cut.t0, a.cut.t1, 0.f), S, x, y, valid, b,
                 marched, slots);
    for (unsigned m = __ballot_sync(FULL_WARP, valid && d != d); m; m &= m - 1) {
      const int q = __ffs(m) - 1;
      const int rx = __shfl_sync(FULL_WARP, x, q), ry = __shfl_sync(FULL_WARP, y, q);
      const float e = march_exact(V, s, a.cut, rx, ry, s_v);
      if (lane == q) d = e;
    }
  }
  if (!valid) return;
  float* o = out + (size_t)y * w + x;
  d = fminf(fmaxf(d * a.scale, 0.f), 1.f);
  *o = merge ? fminf(*o + d, 1.0f) : d;
}

// image_render_kernel (RadRenderer_kernels.cu:85-116) and
// background_render_kernel (BackgroundRenderer_kernels.cu:88-120).
struct ImgArgs {
  float ip[4], vp[4];
  double rw, rh, riw, rih;  // reciprocals of the image's and the image plane's sizes (image_axis)
  float threshold;
  int mode;  // 0 radiograph, 1 background mask
};

// 64 x 32 pixels per block of 256.  What bounds it is FP64: the film-plane
// mapping of a block's columns and rows (image_axis, 16 issue cycles an
// operation and warp), shared by its pixels, so the blocks are large.
// 1024^2: 24 us with 32 x 8 pixels per block and FP64 divisions, 10 here.
constexpr int IW = 64, IH = 32;
__global__ void __launch_bounds__(256) k_image_render(const void* __restrict__ img, int bps, int W, int H,
                                                      const __grid_constant__ ImgArgs a, float* __restrict__ out, int w,
                                                      int h)
{
  __shared__ int s_k[IW + IH];
  __shared__ float s_a[IW + IH];
  const int t = threadIdx.x, x0 = blockIdx.x * IW, y0 = blockIdx.y * IH;
  if (t < IW + IH) {
    const bool row = t >= IW;
    const int j = row ? y0 + (t - IW) : x0 + t;
    int k = 0;
    float wgt = 0.f;
    const bool ok =
        row ? j < h && image_axis(a.vp[1], a.vp[3], j, h, a.rh, a.ip[1], a.ip[3], a.rih, H, true, k, wgt)
            : j < w && image_axis(a.vp[0], a.vp[2], j, w, a.rw, a.ip[0], a.ip[2], a.riw, W, false, k, wgt);
    s_k[t] = ok ? k : INT_MIN;
    s_a[t] = wgt;
  }
  __syncthreads();
  const int lx = t % IW, x = x0 + lx, kx = s_k[lx];
  const float ax = s_a[lx];
  if (x >= w) return;
#pragma unroll
  for (int ly = t / IW; ly < IH; ly += 256 / IW) {
    const int y = y0 + ly, ky = s_k[IW + ly];
    if (y >= h) return;
    float r = 0.f;
    if (kx != INT_MIN && ky != INT_MIN) {
      const float v = bilinear_at(img, bps, W, H, kx, ax, ky, s_a[IW + ly]);
      r = a.mode == 0 ? 1.0f - v : (a.threshold <= v ? 1.0f : 0.0f);
    }
    out[(size_t)y * w + x] = r;
  }
}

// Elementwise operators (DRRBackground / Mult / Merger / Compositor kernels).
__global__ void k_elementwise(int op, const float* __restrict__ a, const float* __restrict__ b,
                              const float* __restrict__ c, float* __restrict__ d, size_t n, float val)
{
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    switch (op) {
      case 0: d[i] = a[i] != 0.0f ? 1.0f : 0.0f; break;
      case 1: d[i] = a[i] * b[i]; break;
      case 2: d[i] = fminf(a[i] + b[i], 1.0f); break;
      case 3: {
        float multi = c[i] < 0.5f ? 0.0f : 1.0f;
        float s1 = a[i], s2 = b[i];
        d[3 * i + 0] = s1;
        d[3 * i + 1] = multi * (s1 / 2.0f + s2 / 2.0f);
        d[3 * i + 2] = s2;
        break;
      }
      default: d[i] = val; break;
    }
  }
}

// trackFrame's masks (mask_images), where four elementwise launches moved 44 bytes a pixel instead of 24.
__global__ void __launch_bounds__(256) k_mask(const float* drr, const float* rad, const float* bg, float* mask,
                                              float* drr_out, float* rad_out, size_t n)
{
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const float d = drr[i], r = rad[i], seen = d != 0.0f ? 1.0f : 0.0f, m = bg ? bg[i] * seen : seen;
    mask[i] = m;
    rad_out[i] = r * m;
    drr_out[i] = d * m;
  }
}

int mask_images(const float* drr, const float* rad, const float* bg, float* mask, float* drr_out, float* rad_out,
                size_t n, cudaStream_t s)
{
  if (n == 0) return ASC_OK;
  k_mask<<<(int)std::min<size_t>((n + 255) / 256, 152 * 16), 256, 0, s>>>(drr, rad, bg, mask, drr_out, rad_out, n);
  ASC_LAUNCH_CHECK();
  return ASC_OK;
}

// ---- 2-D stencil filters, 32x32 output tiles staged in shared memory ----
// Out-of-image positions of the staged tile hold 0, so a tap that falls
// outside the image contributes nothing: the "skip" rule of the reference's
// Gaussian/Sharpen (GaussianFilter_kernels.cu:66-89) and, because the
// weights are an outer product, the 2-D sum splits exactly into a
// horizontal and a vertical pass.
constexpr int FT = 32;  // output tile edge

struct StencilArgs {
  int kind;    // 0 contrast, 1 sobel (k_filter alone), 3 gaussian, 4 sharpen
  int K;       // taps per axis (gaussian / sharpen) or window (contrast)
  float p0, p1, p2;
  float g[64];
};

__global__ void __launch_bounds__(256) k_stencil(const float* __restrict__ in, float* __restrict__ out, int w, int h,
                                                 StencilArgs a)
{
  extern __shared__ float sm[];
  const int R = a.K / 2;
  const int E = FT + 2 * R;  // staged edge
  float* tile = sm;           // E x E
  float* hp = sm + E * E;     // E rows x FT (horizontal pass)
  const int x0 = blockIdx.x * FT - R, y0 = blockIdx.y * FT - R;
  for (int i = threadIdx.x; i < E * E; i += blockDim.x) {
    int ty = i / E, tx = i % E, gx = x0 + tx, gy = y0 + ty;
    tile[i] = (gx >= 0 && gx < w && gy >= 0 && gy < h) ? __ldg(in + (size_t)gy * w + gx) : 0.0f;
  }
  __syncthreads();
  if (a.kind == 3 || a.kind == 4) {
    for (int i = threadIdx.x; i < E * FT; i += blockDim.x) {
      int ty = i / FT, tx = i % FT;
      float s = 0.f;
      for (int k = 0; k < a.K; ++k) s = fmaf(a.g[k], tile[ty * E + tx + k], s);
      hp[i] = s;
    }
    __syncthreads();
  }
  for (int i = threadIdx.x; i < FT * FT; i += blockDim.x) {
    int ty = i / FT, tx = i % FT;
    int gx = blockIdx.x * FT + tx, gy = blockIdx.y * FT + ty;
    if (gx >= w || gy >= h) continue;
    float f = tile[(ty + R) * E + tx + R], r;
    if (a.kind == 3 || a.kind == 4) {
      float blur = 0.f;
      for (int k = 0; k < a.K; ++k) blur = fmaf(a.g[k], hp[(ty + k) * FT + tx], blur);
      if (a.kind == 3) {
        r = fminf(fmaxf(blur, 0.f), 1.f);
      } else {
        r = fabsf(f - blur) > a.p2 ? fminf(fmaxf(f + a.p1 * (f - blur), 0.f), 1.f) : f;
      }
    } else {
      // Contrast: box mean over the in-image part of the window
      // (ContrastFilter_kernels.cu:64-80), then axy^(a-b) * f^b.
      int size = a.K;
      int i0 = max(gy - size / 2, 0), i1 = min(gy + (size + 1) / 2, h);
      int j0 = max(gx - size / 2, 0), j1 = min(gx + (size + 1) / 2, w);
      float s = 0.f;
      for (int yy = i0; yy < i1; ++yy)
        for (int xx = j0; xx < j1; ++xx) s += tile[(yy - y0) * E + (xx - x0)];
      float axy = s / (float)((i1 - i0) * (j1 - j0));
      r = axy > 0.01f ? powf(axy, a.p0 - a.p1) * powf(f, a.p1) : 0.0f;
    }
    out[(size_t)gy * w + gx] = r;
  }
}

// The filters of usual size with the taps and the staged tile's edges known to
// the compiler: no index division by the edge, the taps from the constant
// bank, and a warp's lanes on 32 columns of four rows, whose windows overlap
// (a 7-tap vertical pass reads 10 words for 4 outputs).  The same operations per pixel, in the same order,
// as k_stencil.  Sobel stages its neighbours outside the image as the edge's.
// What bounds them is launch and load latency (4 MB in and out of L2 at 1021 x
// 983, and for Contrast its two powf): Contrast 18.0, Sharpen 12.1, Gaussian
// 12.4, Sobel 10.0 us with k_stencil; 13.2, 7.4, 7.6 and 6.0 here.
constexpr int FR = 4;  // rows per warp
template <int KIND, int K>
__global__ void __launch_bounds__(256) k_filter(const float* __restrict__ in, float* __restrict__ out, int w, int h,
                                                const __grid_constant__ StencilArgs a)
{
  constexpr int R = K / 2, E = FT + 2 * R;
  constexpr bool BLUR = KIND == 3 || KIND == 4;
  __shared__ float tile[E][E + 1];
  __shared__ float hp[BLUR ? E : 1][FT];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int x0 = blockIdx.x * FT - R, y0 = blockIdx.y * FT - R;
#pragma unroll
  for (int j = 0; j < (E + 7) / 8; ++j) {
    const int ty = warp + 8 * j;
    if (ty < E)
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const int tx = lane + 32 * c;
        if (tx < E) {
          int x = x0 + tx, y = y0 + ty;
          float v = 0.f;
          if (KIND == 1) {
            x = min(max(x, 0), w - 1);
            y = min(max(y, 0), h - 1);
          }
          if (KIND == 1 || (x >= 0 && x < w && y >= 0 && y < h)) v = __ldg(in + (size_t)y * w + x);
          tile[ty][tx] = v;
        }
      }
  }
  __syncthreads();
  if (BLUR) {
#pragma unroll
    for (int j = 0; j < (E + 7) / 8; ++j) {
      const int ty = warp + 8 * j;
      if (ty < E) {
        float s = 0.f;
#pragma unroll
        for (int k = 0; k < K; ++k) s = fmaf(a.g[k], tile[ty][lane + k], s);
        hp[ty][lane] = s;
      }
    }
    __syncthreads();
  }
  const int gx = blockIdx.x * FT + lane, gy0 = blockIdx.y * FT + warp * FR;
  if (gx >= w) return;
  float col[BLUR ? K + FR - 1 : 1];
  if (BLUR)
#pragma unroll
    for (int t = 0; t < K + FR - 1; ++t) col[t] = hp[warp * FR + t][lane];
#pragma unroll
  for (int t = 0; t < FR; ++t) {
    const int gy = gy0 + t, ty = warp * FR + t;
    if (gy >= h) return;
    const float f = tile[ty + R][lane + R];
    float r;
    if (BLUR) {
      float blur = 0.f;
#pragma unroll
      for (int k = 0; k < K; ++k) blur = fmaf(a.g[k], col[t + k], blur);
      if (KIND == 3)
        r = fminf(fmaxf(blur, 0.f), 1.f);
      else
        r = fabsf(f - blur) > a.p2 ? fminf(fmaxf(f + a.p1 * (f - blur), 0.f), 1.f) : f;
    } else if (KIND == 1) {
      const float p00 = tile[ty][lane], p01 = tile[ty][lane + 1], p02 = tile[ty][lane + 2];
      const float p10 = tile[ty + 1][lane], p12 = tile[ty + 1][lane + 2];
      const float p20 = tile[ty + 2][lane], p21 = tile[ty + 2][lane + 1], p22 = tile[ty + 2][lane + 2];
      const float horz = p02 + 2 * p12 + p22 - p00 - 2 * p10 - p20;
      const float vert = p00 + 2 * p01 + p02 - p20 - 2 * p21 - p22;
      const float grad = sqrtf(horz * horz + vert * vert);
      const float s = a.p1 < 0.5f ? a.p0 * grad + 2.0f * a.p1 * f : 2.0f * (1.0f - a.p1) * a.p0 * grad + f;
      r = fminf(fmaxf(s, 0.f), 1.f);
    } else {
      float s = 0.f;
#pragma unroll
      for (int yy = 0; yy < K; ++yy)
#pragma unroll
        for (int xx = 0; xx < K; ++xx) s += tile[ty + yy][lane + xx];  // 0 outside the image
      float axy;
      if (K == 3 && gx > 0 && gx < w - 1 && gy > 0 && gy < h - 1) {
        axy = ninth(s);
      } else {
        const int ny = min(gy + (K + 1) / 2, h) - max(gy - R, 0), nx = min(gx + (K + 1) / 2, w) - max(gx - R, 0);
        axy = s / (float)(ny * nx);
      }
      r = axy > 0.01f ? powf(axy, a.p0 - a.p1) * powf(f, a.p1) : 0.0f;
    }
    out[(size_t)gy * w + gx] = r;
  }
}

using FilterKernel = void (*)(const float*, float*, int, int, StencilArgs);
template <int KIND>
static FilterKernel blur_kernel(int K)
{
  switch (K) {
    case 3: return k_filter<KIND, 3>;
    case 5: return k_filter<KIND, 5>;
    case 7: return k_filter<KIND, 7>;
    case 9: return k_filter<KIND, 9>;
    case 11: return k_filter<KIND, 11>;
    case 13: return k_filter<KIND, 13>;
  }
  return nullptr;  // k_stencil
}

// ---- cost reductions ----
constexpr int RB = 256;          // threads per reduction block
constexpr int RE = 16;           // elements per thread
constexpr int RCHUNK = RB * RE;  // elements per block

template <class T>
__device__ __forceinline__ T warp_sum(T v)
{
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Block-wide sum of up to 6 floats (pairwise: shuffle tree, then warps).
template <int N>
__device__ __forceinline__ void block_sum(float (&v)[N], float* red)
{
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
  for (int k = 0; k < N; ++k) v[k] = warp_sum(v[k]);
  __syncthreads();
  if (lane == 0)
#pragma unroll
    for (int k = 0; k < N; ++k) red[warp * N + k] = v[k];
  __syncthreads();
  if (warp == 0) {
#pragma unroll
    for (int k = 0; k < N; ++k) {
      float x = lane < nw ? red[lane * N + k] : 0.f;
      v[k] = warp_sum(x);
    }
    if (lane == 0)
#pragma unroll
      for (int k = 0; k < N; ++k) red[k] = v[k];
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < N; ++k) v[k] = red[k];
  __syncthreads();
}

struct ReduceScratch {
  Moments* part;        // one per block
  double* means;        // hdist: (mF, mG)
  unsigned* ticket;     // last-block election
};

// NCC (Ncc_kernels.cu:116-213) in one launch: each block computes the
// moments of its 4096 elements in two passes over registers, the last block
// to finish merges all partials in FP64 and writes the correlation.  What
// bounds it is latency: the load, two compensated block sums, then the FP64
// tail of the last block.
//
// NT: threads per block.  1024 of 4 elements, each block sum finished by a
// warp per value and one warp merging, where the blocks are one wave (two of
// them on an SM): 120 000 pixels take 16 us, and 31 with 256 threads of 16
// elements and a pairwise merge.  Beyond a wave 256 threads of 16 elements:
// eight blocks on an SM cover one another's latencies, and the last block's
// warps share the partials (asc_ncc_host of 2048^2 pixels: 117 us with 1024
// threads and one warp merging, 71 here; of 4096^2: 392 and 157).  The
// chunks, and with them the FP32 centres, are the same.
template <int N, int NT>
__device__ __forceinline__ void wide_sum_dfs(DFs (&v)[N], float2 (*red)[NT / 32], double* out)
{
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < N; ++k) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      DFs b = {__shfl_xor_sync(FULL_WARP, v[k].h, o), __shfl_xor_sync(FULL_WARP, v[k].l, o)};
      dfs_merge(v[k], b);
    }
    if (lane == 0) red[k][warp] = make_float2(v[k].h, v[k].l);
  }
  __syncthreads();
  if (warp < N) {
    const float2 p = lane < NT / 32 ? red[warp][lane] : make_float2(0.f, 0.f);
    const double t = warp_sum_d((double)p.x + (double)p.y);
    if (lane == 0) out[warp] = t;
  }
  __syncthreads();
}

// The partials of nb blocks merged by the W warps of one, in two levels; warp
// 0's result holds.  Writes over part[0 .. W).
template <int W>
__device__ __forceinline__ Moments merge_block(Moments* part, int nb)
{
  const int warp = threadIdx.x >> 5;
  const Moments m = merge_moments<4>(part + warp, (nb - warp + W - 1) / W, W);
  __syncthreads();  // every partial is read
  if ((threadIdx.x & 31) == 0) part[warp] = m;
  __threadfence();
  __syncthreads();
  return merge_moments(part, W);
}

template <int NT>
__global__ void __launch_bounds__(NT) k_ncc(const float* __restrict__ f, const float* __restrict__ g,
                                            const float* __restrict__ mask, unsigned n, int tree, ReduceScratch sc,
                                            double* __restrict__ result)
{
  constexpr int NE = RCHUNK / NT;
  __shared__ float2 red[6][NT / 32];
  __shared__ double ds[6], dc[3];
  __shared__ float s_mean[2];
  __shared__ unsigned s_keep[8];
  float fv[NE], gv[NE], mv[NE];
  unsigned flags = 0;  // bit k: covered and mask > 0.5
  const size_t base = (size_t)blockIdx.x * RCHUNK + threadIdx.x;
#pragma unroll
  for (int k = 0; k < NE; ++k) {
    const size_t i = base + (size_t)k * NT;
    fv[k] = gv[k] = mv[k] = 0.f;
    if (i < n) {
      fv[k] = __ldg(f + i);
      gv[k] = __ldg(g + i);
      mv[k] = __ldg(mask + i);
    }
  }
  int shift = 0;
  if (tree) {
    if (threadIdx.x < 256) shift = tree_mask(n, s_keep);
    for (unsigned m = n; threadIdx.x >= 256 && m > 256u; m = (m + 255u) >> 8) shift += 8;
    __syncthreads();
  }
  DFs s[6] = {};  // sm, sf, sg (covered), n, sf, sg (masked)
#pragma unroll
  for (int k = 0; k < NE; ++k) {
    const size_t i = base + (size_t)k * NT;
    if (i < n && (!tree || tree_kept(s_keep, (unsigned)i, shift))) {
      dfs_add(s[0], mv[k]);
      dfs_add(s[1], fv[k]);
      dfs_add(s[2], gv[k]);
      if (mv[k] > 0.5f) {
        flags |= 1u << k;
        dfs_add(s[3], 1.f);
        dfs_add(s[4], fv[k]);
        dfs_add(s[5], gv[k]);
      }
    }
  }
  wide_sum_dfs<6, NT>(s, red, ds);
  if (threadIdx.x < 2) s_mean[threadIdx.x] = ds[3] > 0 ? (float)(ds[4 + threadIdx.x] / ds[3]) : 0.f;
  __syncthreads();
  const float mf = s_mean[0], mg = s_mean[1];
  DFs c[3] = {};
#pragma unroll
  for (int k = 0; k < NE; ++k)
    if (flags & (1u << k)) {
      float a = fv[k] - mf, b = gv[k] - mg;
      dfs_add_prod(c[0], a, a);
      dfs_add_prod(c[1], b, b);
      dfs_add_prod(c[2], a, b);
    }
  wide_sum_dfs<3, NT>(c, red, dc);
  constexpr bool ONE_WARP = NT == 1024;  // merges alone
  __shared__ bool s_last;
  if (ONE_WARP && threadIdx.x >= 32) return;
  if (threadIdx.x < 32) {
    tile_moments(ds, dc, mf, mg, sc.part + blockIdx.x);
    __threadfence();
    __syncwarp();
    if (threadIdx.x == 0) s_last = atomicAdd(sc.ticket, 1u) == gridDim.x - 1;
  }
  if (ONE_WARP)
    __syncwarp();
  else
    __syncthreads();
  if (!s_last) return;
  __threadfence();
  Moments m;
  if constexpr (ONE_WARP)
    m = merge_moments(sc.part, gridDim.x);
  else
    m = merge_block<NT / 32>(sc.part, gridDim.x);
  if (threadIdx.x == 0) {
    *result = moments_ncc(m);
    *sc.ticket = 0;
  }
}

// The launch for n elements, the same for asc_ncc and asc_ncc_noalloc.
constexpr unsigned NCC_WAVE = 2 * 152;  // blocks of 1024 threads that run at once
void launch_ncc(const float* f, const float* g, const float* mask, unsigned n, int tree, ReduceScratch sc,
                double* result, cudaStream_t s)
{
  const unsigned blocks = (unsigned)(((size_t)n + RCHUNK - 1) / RCHUNK);
  if (blocks <= NCC_WAVE)
    k_ncc<1024><<<blocks, 1024, 0, s>>>(f, g, mask, n, tree, sc, result);
  else
    k_ncc<256><<<blocks, 256, 0, s>>>(f, g, mask, n, tree, sc, result);
}

// The sums over all blocks of the N values that thread 0 holds in v, for the
// SAD kernels: true in the last block, with the sums in its thread 0.  Up to 64
// blocks warp 0 adds their values by itself and the other warps leave; more
// are shared by the block's threads, whose loads one warp would wait for one
// after the other (asc_hdist_host of 2048^2 pixels: 90 us, 48 here; of
// 4096^2: 380 and 161).
template <int N>
__device__ __forceinline__ bool sum_blocks(const float (&v)[N], ReduceScratch sc, double (&sum)[N])
{
  __shared__ bool s_last;
  __shared__ double s_sum[RB / 32][N];
  const int nb = gridDim.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = nb > 64 ? RB / 32 : 1;
  if (warp >= nw) return false;
  if (threadIdx.x == 0) {
    double* p = (double*)(sc.part + blockIdx.x);
#pragma unroll
    for (int k = 0; k < N; ++k) p[k] = v[k];
    __threadfence();
    s_last = atomicAdd(sc.ticket, 1u) == gridDim.x - 1;
  }
  if (nw > 1)
    __syncthreads();
  else
    __syncwarp();
  if (!s_last) return false;
  __threadfence();
#pragma unroll
  for (int k = 0; k < N; ++k) sum[k] = 0.0;
#pragma unroll 4
  for (int i = threadIdx.x; i < nb; i += 32 * nw)
#pragma unroll
    for (int k = 0; k < N; ++k) sum[k] += __ldcg((const double*)(sc.part + i) + k);
  warp_sums(sum);
  if (nw > 1) {
    if (lane == 0)
#pragma unroll
      for (int k = 0; k < N; ++k) s_sum[warp][k] = sum[k];
    __syncthreads();
    if (threadIdx.x == 0)
#pragma unroll
      for (int k = 0; k < N; ++k)
        for (int w = 1; w < nw; ++w) sum[k] += s_sum[w][k];
  }
  return true;
}

// SAD ("hdist", HDist_kernels.cu:111-203): pass 1 computes the masked means
// (as k_ncc's covered sums), pass 2 sums |(f-mF)-(g-mG)| over mask > 0.5.
__global__ void __launch_bounds__(RB) k_hdist_means(const float* __restrict__ f, const float* __restrict__ g,
                                                    const float* __restrict__ mask, unsigned n, int tree,
                                                    ReduceScratch sc)
{
  __shared__ float red[(RB / 32) * 3];
  __shared__ unsigned s_keep[RB / 32];
  float s[3] = {0, 0, 0};
  const size_t base = (size_t)blockIdx.x * RCHUNK + threadIdx.x;
  int shift = 0;
  if (tree) {
    shift = tree_mask(n, s_keep);
    __syncthreads();
  }
#pragma unroll
  for (int k = 0; k < RE; ++k) {
    size_t i = base + (size_t)k * RB;
    if (i < n && (!tree || tree_kept(s_keep, (unsigned)i, shift))) {
      s[0] += __ldg(mask + i);
      s[1] += __ldg(f + i);
      s[2] += __ldg(g + i);
    }
  }
  block_sum<3>(s, red);
  double sum[3];
  if (sum_blocks(s, sc, sum) && threadIdx.x == 0) {
    sc.means[0] = sum[1] / sum[0];
    sc.means[1] = sum[2] / sum[0];
    *sc.ticket = 0;
  }
}

__global__ void __launch_bounds__(RB) k_hdist_sad(const float* __restrict__ f, const float* __restrict__ g,
                                                  const float* __restrict__ mask, unsigned n, int tree,
                                                  ReduceScratch sc, double* __restrict__ result)
{
  __shared__ float red[RB / 32];
  __shared__ unsigned s_keep[RB / 32];
  const float mF = (float)sc.means[0], mG = (float)sc.means[1];
  float s[1] = {0};
  const size_t base = (size_t)blockIdx.x * RCHUNK + threadIdx.x;
  int shift = 0;
  if (tree) {
    shift = tree_mask(n, s_keep);
    __syncthreads();
  }
#pragma unroll
  for (int k = 0; k < RE; ++k) {
    size_t i = base + (size_t)k * RB;
    if (i < n && (!tree || tree_kept(s_keep, (unsigned)i, shift)) && __ldg(mask + i) > 0.5f)
      s[0] += fabsf((__ldg(f + i) - mF) - (__ldg(g + i) - mG));
  }
  block_sum<1>(s, red);
  double sum[1];
  if (sum_blocks(s, sc, sum) && threadIdx.x == 0) {
    *result = sum[0];
    *sc.ticket = 0;
  }
}

template <int STORE>
__global__ void __launch_bounds__(CLEAR_THREADS) k_clearance(DevVolume V, float cutoff_raw, uint8_t* __restrict__ clr)
{
  extern __shared__ __align__(8) unsigned char clear_sm[];
  ClearWork& w = *reinterpret_cast<ClearWork*>(clear_sm);
  const int t = threadIdx.x, cx = blockIdx.x * CB, cy = blockIdx.y * CB, cz = blockIdx.z * CB;
#pragma unroll 4
  for (int i = t >> 5; i < CLEAR_Z * CLEAR_Y / 2; i += CLEAR_THREADS / 32) clear_load<STORE>(V, cutoff_raw, w, i, cx, cy, cz);
  __syncthreads();
  uint2 acc = make_uint2(0u, 0u);
  unsigned n[3] = {0u, 0u, 0u};
#pragma unroll 1
  for (int round = 0; CLEAR_ROUND * round <= CLEAR_REACH; ++round) {
    clear_reach(w, t, round, acc);
    __syncthreads();
    clear_count(w, t, round, n);
    __syncthreads();
  }
  clear_bytes(w, t, n);
  __syncthreads();
  clear_store(w, t, V, cx, cy, cz, clr);
}

int g_empty_skip = 1;

int build_clearance(const DevVolume& V, float cutoff_raw, uint8_t* clr, cudaStream_t s)
{
  const auto kernel = V.storage == ASC_STORE_F32    ? k_clearance<ASC_STORE_F32>
                      : V.storage == ASC_STORE_BF16 ? k_clearance<ASC_STORE_BF16>
                      : V.storage == ASC_STORE_F16  ? k_clearance<ASC_STORE_F16>
                                                    : k_clearance<ASC_STORE_U16>;
  ASC_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(ClearWork)));
  const dim3 grid((clear_dim(V.nx) + CB - 1) / CB, (clear_dim(V.ny) + CB - 1) / CB, (clear_dim(V.nz) + CB - 1) / CB);
  kernel<<<grid, CLEAR_THREADS, sizeof(ClearWork), s>>>(V, cutoff_raw, clr);
  ASC_LAUNCH_CHECK();
  return ASC_OK;
}

// ---------------------------------------------------------------- host side

ClearanceCache::~ClearanceCache()
{
  if (grid) cudaFree(grid);
  for (uint8_t* p : kept) cudaFree(p);
  if (built) cudaEventDestroy(built);
  for (Reader& r : reader)
    if (r.cast) cudaEventDestroy(r.cast);
}

namespace {
// While a stream of this thread is captured: lets the thread allocate and
// work on other streams.
struct RelaxedCapture {
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  const bool on;
  explicit RelaxedCapture(bool capturing) : on(capturing)
  {
    if (on) cudaThreadExchangeStreamCaptureMode(&mode);
  }
  ~RelaxedCapture()
  {
    if (on) cudaThreadExchangeStreamCaptureMode(&mode);
  }
};
}  // namespace

int ClearanceCache::use(const DevVolume& V, float cut, cudaStream_t s, bool capturing)
{
  RelaxedCapture relaxed(capturing);
  if (!built) ASC_CUDA(cudaEventCreateWithFlags(&built, cudaEventDisableTiming));
  if (cutoff == cut) {
    // a graph may run on any stream, so its grid is complete before it is captured
    ASC_CUDA(capturing ? cudaEventSynchronize(built) : cudaStreamWaitEvent(s, built));
    return ASC_OK;
  }
  cutoff = NAN;
  if (captured) {
    kept.push_back(grid);
    grid = nullptr;
    captured = false;
  }
  if (!grid) {
    Gate g(device_gate());
    readers = 0;
    ASC_CUDA(cudaMalloc(&grid, clearance_cells(V)));
  }
  struct Own {  // what a captured cast reads is built now, not by the graph
    cudaStream_t s = nullptr;
    ~Own()
    {
      if (s) cudaStreamDestroy(s);
    }
  } own;
  if (capturing) {
    ASC_CUDA(cudaStreamCreateWithFlags(&own.s, cudaStreamNonBlocking));
    s = own.s;
  }
  for (int i = 0; i < readers; ++i) ASC_CUDA(cudaStreamWaitEvent(s, reader[i].cast));
  int rc = build_clearance(V, cut, grid, s);
  if (rc) return rc;
  ASC_CUDA(cudaEventRecord(built, s));
  if (capturing) ASC_CUDA(cudaStreamSynchronize(s));
  readers = 0;
  cutoff = cut;
  return ASC_OK;
}

int ClearanceCache::read(cudaStream_t s, bool capturing)
{
  if (capturing) {
    captured = true;
    return ASC_OK;
  }
  int i = 0;
  while (i < readers && reader[i].stream != s) ++i;
  if (i == MAX_READERS) i = oldest++ % MAX_READERS;
  Reader& r = reader[i];
  if (!r.cast) ASC_CUDA(cudaEventCreateWithFlags(&r.cast, cudaEventDisableTiming));
  // The new record stands for the old one too: stream order where s is the same
  // stream (a wait would cost a cast of 8 us another 0.8), else a wait.  The
  // per-thread default stream is one name of many streams.
  if (i < readers && (r.stream != s || s == cudaStreamPerThread)) ASC_CUDA(cudaStreamWaitEvent(s, r.cast));
  ASC_CUDA(cudaEventRecord(r.cast, s));
  r.stream = s;
  readers = std::max(readers, i + 1);
  return ASC_OK;
}

int launch_filter(const asc_filter_desc& f, const float* in, float* out, int w, int h, cudaStream_t s)
{
  if (w <= 0 || h <= 0) return ASC_OK;
  StencilArgs a;
  memset(&a, 0, sizeof a);
  a.kind = f.kind;
  a.p0 = f.p0;
  a.p1 = f.p1;
  a.p2 = f.p2;
  int R;
  if (f.kind == 1) {
    a.K = 3;
    R = 1;
  } else if (f.kind == 0) {
    a.K = (int)f.p2;
    if (a.K < 1) return ASC_ERR_ARG;
    R = std::max(a.K / 2, (a.K - 1) / 2);
    if (R > 16) return ASC_ERR_RANGE;
  } else if (f.kind == 3 || f.kind == 4) {
    a.K = gauss_1d(f.p0, a.g, 64);
    if (a.K < 0) return ASC_ERR_RANGE;
    if (a.K == 1) {
      ASC_CUDA(cudaMemcpyAsync(out, in, (size_t)w * h * sizeof(float), cudaMemcpyDeviceToDevice, s));
      return ASC_OK;
    }
    if (f.kind == 4) a.p1 = f.p1 < 1 ? 1 : f.p1;  // SharpenFilter::set_contrast
    R = a.K / 2;
  } else {
    return ASC_ERR_ARG;
  }
  const dim3 grid((w + FT - 1) / FT, (h + FT - 1) / FT);
  const FilterKernel fast = f.kind == 1   ? k_filter<1, 3>
                            : f.kind == 3 ? blur_kernel<3>(a.K)
                            : f.kind == 4 ? blur_kernel<4>(a.K)
                            : a.K == 3    ? k_filter<0, 3>
                            : a.K == 5    ? k_filter<0, 5>
                                          : nullptr;
  if (fast) {
    fast<<<grid, 256, 0, s>>>(in, out, w, h, a);
    ASC_LAUNCH_CHECK();
    return ASC_OK;
  }
  int E = FT + 2 * R;
  size_t smem = (size_t)(E * E + E * FT) * sizeof(float);
  static std::once_flag once;
  std::call_once(once, [] { cudaFuncSetAttribute(k_stencil, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024); });
  k_stencil<<<grid, 256, smem, s>>>(in, out, w, h, a);
  ASC_LAUNCH_CHECK();
  return ASC_OK;
}

// Per-process reduction scratch sized by asc_ncc_init (the reference keeps
// module globals too, Ncc_kernels.cu:50-57).  It lives on the device that was
// current when it was sized; every read or change of it holds g_red_mu.
static std::mutex g_red_mu;
static Moments* g_part = nullptr;
static double* g_means = nullptr;
static unsigned* g_ticket = nullptr;
static unsigned g_max_n = 0;
static int g_red_dev = -1;

std::recursive_mutex& device_gate()
{
  static std::recursive_mutex m;
  return m;
}

static int ncc_init_locked(unsigned max_n);

// The scratch for n elements on the current device, copied out under the
// lock: a thread that grows it frees the old buffers only after taking the
// lock (and cudaFree waits for the kernels still using them).  Scratch sized
// on another device is ASC_ERR_STATE: like the reference's module globals it
// serves one device per process.
static int ensure_scratch(unsigned n, ReduceScratch* out)
{
  std::lock_guard<std::mutex> l(g_red_mu);
  int dev = 0;
  ASC_CUDA(cudaGetDevice(&dev));
  if (g_part && dev != g_red_dev) {
    set_error_message("asc_ncc/asc_hdist: the reduction scratch belongs to another device (asc_ncc_init there)");
    return ASC_ERR_STATE;
  }
  if (!(n <= g_max_n && g_part)) {
    int rc = ncc_init_locked(n);
    if (rc) return rc;
  }
  *out = ReduceScratch{g_part, g_means, g_ticket};
  return ASC_OK;
}

}  // namespace asc

using namespace asc;

// ---------------------------------------------------------------- C ABI

ASC_API const char* asc_version(void) { return "autoscoper_gb300 0.1 (sm_103a)"; }

ASC_API const char* asc_status_string(int st)
{
  switch (st) {
    case ASC_OK: return "ok";
    case ASC_ERR_ARG: return "bad argument";
    case ASC_ERR_CUDA: return "CUDA error";
    case ASC_ERR_EMPTY: return "empty volume";
    case ASC_ERR_RANGE: return "size out of range";
    case ASC_ERR_NOMEM: return "out of device memory";
    case ASC_ERR_TIMEOUT: return "device wait timed out";
    case ASC_ERR_STATE: return "call out of order";
  }
  return "unknown status";
}

ASC_API const char* asc_last_error(void) { return g_last_error.c_str(); }

ASC_API int asc_set_option(int option, int value)
{
  if (option == ASC_OPT_EMPTY_SKIP) {
    g_empty_skip = value != 0;
    return ASC_OK;
  }
  return ASC_ERR_ARG;
}

ASC_API int asc_malloc(void** p, size_t bytes)
{
  if (!p) return ASC_ERR_ARG;
  Gate g(device_gate());
  ASC_CUDA(cudaMalloc(p, bytes ? bytes : 1));
  return ASC_OK;
}
ASC_API int asc_free(void* p)
{
  Gate g(device_gate());
  ASC_CUDA(cudaFree(p));
  return ASC_OK;
}
ASC_API int asc_memcpy_h2d(void* d, const void* s, size_t n, void* st)
{
  ASC_CUDA(cudaMemcpyAsync(d, s, n, cudaMemcpyHostToDevice, S(st)));
  return ASC_OK;
}
ASC_API int asc_memcpy_d2h(void* d, const void* s, size_t n, void* st)
{
  ASC_CUDA(cudaMemcpyAsync(d, s, n, cudaMemcpyDeviceToHost, S(st)));
  ASC_CUDA(cudaStreamSynchronize(S(st)));
  return ASC_OK;
}
ASC_API int asc_memcpy_d2d(void* d, const void* s, size_t n, void* st)
{
  ASC_CUDA(cudaMemcpyAsync(d, s, n, cudaMemcpyDeviceToDevice, S(st)));
  return ASC_OK;
}
ASC_API int asc_memset(void* d, int v, size_t n, void* st)
{
  ASC_CUDA(cudaMemsetAsync(d, v, n, S(st)));
  return ASC_OK;
}
ASC_API int asc_stream_sync(void* st)
{
  ASC_CUDA(cudaStreamSynchronize(S(st)));
  return ASC_OK;
}
ASC_API int asc_device_sync(void)
{
  Gate g(device_gate());
  ASC_CUDA(cudaDeviceSynchronize());
  return ASC_OK;
}
ASC_API int asc_set_device(int d)
{
  ASC_CUDA(cudaSetDevice(d));
  return ASC_OK;
}
ASC_API int asc_stream_create(void** s)
{
  if (!s) return ASC_ERR_ARG;
  ASC_CUDA(cudaStreamCreateWithFlags((cudaStream_t*)s, cudaStreamNonBlocking));
  return ASC_OK;
}
ASC_API int asc_stream_destroy(void* s)
{
  ASC_CUDA(cudaStreamDestroy(S(s)));
  return ASC_OK;
}
ASC_API int asc_event_create(void** e)
{
  if (!e) return ASC_ERR_ARG;
  ASC_CUDA(cudaEventCreate((cudaEvent_t*)e));
  return ASC_OK;
}
ASC_API int asc_event_record(void* e, void* s)
{
  ASC_CUDA(cudaEventRecord((cudaEvent_t)e, S(s)));
  return ASC_OK;
}
ASC_API int asc_event_elapsed(void* a, void* b, float* ms)
{
  if (!ms) return ASC_ERR_ARG;
  ASC_CUDA(cudaEventSynchronize((cudaEvent_t)b));
  ASC_CUDA(cudaEventElapsedTime(ms, (cudaEvent_t)a, (cudaEvent_t)b));
  return ASC_OK;
}
ASC_API int asc_event_destroy(void* e)
{
  ASC_CUDA(cudaEventDestroy((cudaEvent_t)e));
  return ASC_OK;
}
ASC_API int asc_host_alloc(void** p, size_t n)
{
  if (!p) return ASC_ERR_ARG;
  Gate g(device_gate());
  ASC_CUDA(cudaMallocHost(p, n ? n : 1));
  return ASC_OK;
}
ASC_API int asc_host_free(void* p)
{
  Gate g(device_gate());
  ASC_CUDA(cudaFreeHost(p));
  return ASC_OK;
}
ASC_API int asc_mem_info(size_t* free_bytes, size_t* total_bytes)
{
  if (!free_bytes || !total_bytes) return ASC_ERR_ARG;
  ASC_CUDA(cudaMemGetInfo(free_bytes, total_bytes));
  return ASC_OK;
}

// ---- volumes (VolumeDescription.cpp:152-305) ----
template <class T>
static void describe(const T* data, int W, int H, int D, const int* flip, std::vector<T>& crop, int mn[3], int mx[3],
                     T& vmin, T& vmax)
{
  std::vector<T> fl((size_t)W * H * D);
  for (int k = 0; k < D; ++k)
    for (int i = 0; i < H; ++i)
      for (int j = 0; j < W; ++j) {
        int x = flip[0] ? W - 1 - j : j, y = flip[1] ? H - 1 - i : i, z = flip[2] ? D - 1 - k : k;
        fl[(size_t)z * W * H + (size_t)y * W + x] = data[(size_t)k * W * H + (size_t)i * W + j];
      }
  mn[0] = W; mn[1] = H; mn[2] = D;
  mx[0] = mx[1] = mx[2] = 0;
  size_t p = 0;
  for (int k = 0; k < D; ++k) {
    bool col = false;
    for (int i = 0; i < H; ++i) {
      bool row = false;
      for (int j = 0; j < W; ++j, ++p)
        if (fl[p] != T(0)) {
          mn[0] = std::min(mn[0], j);
          mx[0] = std::max(mx[0], j);
          row = true;
        }
      if (row) {
        mn[1] = std::min(mn[1], i);
        mx[1] = std::max(mx[1], i);
        col = true;
      }
    }
    if (col) {
      mn[2] = std::min(mn[2], k);
      mx[2] = std::max(mx[2], k);
    }
  }
  if (mn[0] > mx[0] || mn[1] > mx[1] || mn[2] > mx[2]) return;
  vmin = std::numeric_limits<T>::max();
  vmax = std::numeric_limits<T>::min();
  crop.clear();
  crop.reserve((size_t)(mx[0] - mn[0] + 1) * (mx[1] - mn[1] + 1) * (mx[2] - mn[2] + 1));
  for (int k = mn[2]; k <= mx[2]; ++k)
    for (int i = mn[1]; i <= mx[1]; ++i)
      for (int j = mn[0]; j <= mx[0]; ++j) {
        T v = fl[(size_t)k * W * H + (size_t)i * W + j];
        vmin = std::min(vmin, v);
        vmax = std::max(vmax, v);
        crop.push_back(v);
      }
}

// A voxel as stored: a 16-bit half (u16, IEEE half, bfloat16) or FP32 bits.
static uint32_t to_store(unsigned v, int storage)
{
  if (storage == ASC_STORE_F16) return __half_as_ushort(__float2half_rn((float)v));
  if (storage == ASC_STORE_BF16) return __bfloat16_as_ushort(__float2bfloat16_rn((float)v));
  if (storage == ASC_STORE_F32) {
    const float f = (float)v;
    uint32_t b;
    memcpy(&b, &f, 4);
    return b;
  }
  return (uint16_t)v;
}

ASC_API int asc_volume_create(const void* data, int W, int H, int D, int bps, const double scale[3],
                              const int flip[3], int storage, asc_volume* out)
{
  if (!data || !out || !scale || W <= 0 || H <= 0 || D <= 0) return ASC_ERR_ARG;
  if (bps != 8 && bps != 16) return ASC_ERR_ARG;
  if (storage < ASC_STORE_U16 || storage > ASC_STORE_F32) return ASC_ERR_ARG;
  static const int noflip[3] = {0, 0, 0};
  if (!flip) flip = noflip;
  int mn[3], mx[3];
  std::vector<unsigned> vals;
  unsigned vmin = 0, vmax = 0;
  if (bps == 8) {
    std::vector<uint8_t> crop;
    uint8_t a = 0, b = 0;
    describe((const uint8_t*)data, W, H, D, flip, crop, mn, mx, a, b);
    vals.assign(crop.begin(), crop.end());
    vmin = a; vmax = b;
  } else {
    std::vector<uint16_t> crop;
    uint16_t a = 0, b = 0;
    describe((const uint16_t*)data, W, H, D, flip, crop, mn, mx, a, b);
    vals.assign(crop.begin(), crop.end());
    vmin = a; vmax = b;
  }
  if (mn[0] > mx[0] || mn[1] > mx[1] || mn[2] > mx[2]) return ASC_ERR_EMPTY;
  // the march indexes the padded grid in 32-bit arithmetic
  if ((double)(mx[0] - mn[0] + 1 + 2 * PAD) * (mx[1] - mn[1] + 1 + 2 * PAD) * (mx[2] - mn[2] + 1 + 2 * PAD) >=
      2147483648.0)
    return ASC_ERR_RANGE;
  auto* v = new asc_volume_host();
  int dims[3] = {mx[0] - mn[0] + 1, mx[1] - mn[1] + 1, mx[2] - mn[2] + 1};
  float norm = bps == 8 ? 255.0f : 65535.0f;
  v->min_value = vmin / norm;
  v->max_value = vmax / norm;
  float sc[3] = {(float)scale[0], (float)scale[1], (float)scale[2]};
  v->trans_center[0] = -sc[0] * 0.5 * (mn[0] + mx[0]);
  v->trans_center[1] = -sc[1] * 0.5 * (mn[1] + mx[1]);
  v->trans_center[2] = sc[2] * 0.5 * (mn[2] + mx[2]);
  for (int a = 0; a < 3; ++a) {
    v->inv_scale[a] = 1.0f / (float)(sc[a] * dims[a]);
    v->dims[a] = dims[a];
  }
  v->inv_trans[0] = -mn[0] / (float)dims[0];
  v->inv_trans[1] = -((H - mx[1] - 1) / (float)dims[1]);
  v->inv_trans[2] = mn[2] / (float)dims[2];
  v->bps = bps;
  // x-paired words on the padded grid (see DevVolume)
  const size_t nwords = padded_words(dims[0], dims[1], dims[2], storage);
  std::vector<uint32_t> pairs(nwords);
  const int dx = dims[0], dxy = dims[0] * dims[1];
  pack_pairs(dims[0], dims[1], dims[2], storage,
             [&](int x, int y, int z) { return to_store(vals[(size_t)z * dxy + (size_t)y * dx + x], storage); },
             pairs.data());
  Gate g(device_gate());
  cudaError_t e = cudaMalloc(&v->pairs, nwords * sizeof(uint32_t));
  if (e == cudaSuccess) e = cudaMemcpy(v->pairs, pairs.data(), nwords * sizeof(uint32_t), cudaMemcpyHostToDevice);
  if (e != cudaSuccess) {
    if (v->pairs) cudaFree(v->pairs);
    delete v;
    return cuda_status(e);
  }
  const int px = dims[0] + 2 * PAD, pxy = px * (dims[1] + 2 * PAD);
  // the stored values' largest neighbour step (the march's cutoff band)
  const float gmax = volume_gmax(dims[0], dims[1], dims[2], [&](int x, int y, int z) {
    const uint32_t w = to_store(vals[(size_t)z * dxy + (size_t)y * dx + x], storage);
    if (storage == ASC_STORE_F16) return __half2float(__ushort_as_half((unsigned short)w));
    if (storage == ASC_STORE_BF16) return __bfloat162float(__ushort_as_bfloat16((unsigned short)w));
    if (storage == ASC_STORE_F32) {
      float f;
      memcpy(&f, &w, 4);
      return f;
    }
    return (float)w;
  });
  v->dev = DevVolume{v->pairs, dims[0], dims[1], dims[2], px, pxy, storage, 1.0f / norm, gmax};
  *out = (asc_volume)v;
  return ASC_OK;
}

ASC_API int asc_volume_info(asc_volume vol, float inv_scale[3], float inv_trans[3], double trans_center[3],
                            float* min_value, float* max_value, int dims[3])
{
  auto* v = (asc_volume_host*)vol;
  if (!v) return ASC_ERR_ARG;
  for (int a = 0; a < 3; ++a) {
    if (inv_scale) inv_scale[a] = v->inv_scale[a];
    if (inv_trans) inv_trans[a] = v->inv_trans[a];
    if (trans_center) trans_center[a] = v->trans_center[a];
    if (dims) dims[a] = v->dims[a];
  }
  if (min_value) *min_value = v->min_value;
  if (max_value) *max_value = v->max_value;
  return ASC_OK;
}

ASC_API int asc_volume_destroy(asc_volume vol)
{
  auto* v = (asc_volume_host*)vol;
  if (!v) return ASC_ERR_ARG;
  Gate g(device_gate());
  cudaFree(v->pairs);
  delete v;
  return ASC_OK;
}

namespace asc {
int raycast_launch(const DevVolume& V, const uint8_t* clr, const float* m12, const float* vp, float step,
                   float intensity, float cutoff, float* out, bool merge, int w, int h, cudaStream_t s)
{
  RayArgs a;
  memcpy(a.m, m12, sizeof a.m);
  memcpy(a.vp, vp, sizeof a.vp);
  a.step = step;
  // density = step * sum(norm * raw) / intensity; cutoff compares normalized samples
  a.scale = step * V.norm / intensity;
  a.cut = make_cutoff(cutoff, V.norm, V.gmax);
  df_split((double)vp[2] / (double)w, a.sx[0], a.sx[1]);
  df_split((double)vp[3] / (double)h, a.sy[0], a.sy[1]);
  // the grid's rows reach 65535: taller images take several launches
  for (int y0 = 0; y0 < h; y0 += 4 * 65535) {
    const dim3 grid((w + 7) / 8, std::min((h - y0 + 3) / 4, 65535));
    k_raycast<<<grid, 32, 0, s>>>(V, clr, a, out, merge, y0, w, h);
  }
  ASC_LAUNCH_CHECK();
  return ASC_OK;
}
}  // namespace asc

ASC_API int asc_raycast(asc_volume vol, const double imv[16], const float vp[4], float step, float intensity,
                        float cutoff, int visible, float* out, int w, int h, void* stream)
{
  auto* v = (asc_volume_host*)vol;
  if (!v) return ASC_ERR_STATE;  // RayCaster::render without a volume
  if (!imv || !vp || !out || w < 0 || h < 0) return ASC_ERR_ARG;
  if (w == 0 || h == 0) return ASC_OK;
  if (!visible) {
    ASC_CUDA(cudaMemsetAsync(out, 0, (size_t)w * h * sizeof(float), S(stream)));
    return ASC_OK;
  }
  float m[12];
  fold_matrix(imv, v->inv_scale, v->inv_trans, m);
  const float cut = occupancy_threshold(make_cutoff(cutoff, v->dev.norm, v->dev.gmax));
  cudaStream_t s = S(stream);
  if (!g_empty_skip)
    return raycast_launch(v->dev, nullptr, m, vp, step, intensity, cutoff, out, false, w, h, s);
  cudaStreamCaptureStatus capture;
  ASC_CUDA(cudaStreamIsCapturing(s, &capture));
  const bool capturing = capture != cudaStreamCaptureStatusNone;
  std::lock_guard<std::mutex> lock(v->clr.mu);
  int rc = v->clr.use(v->dev, cut, s, capturing);
  if (!rc) rc = raycast_launch(v->dev, v->clr.grid, m, vp, step, intensity, cutoff, out, false, w, h, s);
  return rc ? rc : v->clr.read(s, capturing);
}

// ---- images ----
struct asc_image_s {
  void* data;
  int w, h, bps;
};

ASC_API int asc_image_create(const void* data, int w, int h, int bps, asc_image* out)
{
  if (!data || !out || w <= 0 || h <= 0 || (bps != 8 && bps != 16 && bps != 32)) return ASC_ERR_ARG;
  auto* im = new asc_image_s{nullptr, w, h, bps};
  size_t bytes = (size_t)w * h * (bps / 8);
  Gate g(device_gate());
  cudaError_t e = cudaMalloc(&im->data, bytes);
  if (e == cudaSuccess) e = cudaMemcpy(im->data, data, bytes, cudaMemcpyHostToDevice);
  if (e != cudaSuccess) {
    if (im->data) cudaFree(im->data);
    delete im;
    return cuda_status(e);
  }
  *out = im;
  return ASC_OK;
}

ASC_API int asc_image_update(asc_image im, const void* data, void* st)
{
  if (!im || !data) return ASC_ERR_ARG;
  ASC_CUDA(cudaMemcpyAsync(im->data, data, (size_t)im->w * im->h * (im->bps / 8), cudaMemcpyHostToDevice, S(st)));
  return ASC_OK;
}

ASC_API int asc_image_destroy(asc_image im)
{
  if (!im) return ASC_ERR_ARG;
  Gate g(device_gate());
  cudaFree(im->data);
  delete im;
  return ASC_OK;
}

// Video::create_background_image (Video.cpp:147-218): per pixel, the largest
// normalized value over the frames (8, 16 or 32 bits per sample).
__global__ void k_background_max(const void* __restrict__ img, int bps, size_t n, float* __restrict__ out)
{
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    float v;
    if (bps == 8)
      v = (float)__ldg((const unsigned char*)img + i) / 255.0f;
    else if (bps == 16)
      v = (float)__ldg((const unsigned short*)img + i) / 65535.0f;
    else
      v = (float)__ldg((const unsigned*)img + i) / 4294967295.0f;
    if (v > out[i]) out[i] = v;
  }
}

ASC_API int asc_background_from_frames(const asc_image* frames, int n, float* out, void* st)
{
  if (!frames || !out || n < 2) return ASC_ERR_ARG;  // the reference wants two images at least
  const int w = frames[0]->w, h = frames[0]->h;
  for (int i = 0; i < n; ++i)
    if (!frames[i] || frames[i]->w != w || frames[i]->h != h || frames[i]->bps == 32) return ASC_ERR_ARG;
  const size_t px = (size_t)w * h;
  ASC_CUDA(cudaMemsetAsync(out, 0, px * sizeof(float), S(st)));
  const int blocks = (int)std::min<size_t>((px + 255) / 256, 4096);
  for (int i = 0; i < n; ++i) k_background_max<<<blocks, 256, 0, S(st)>>>(frames[i]->data, frames[i]->bps, px, out);
  ASC_LAUNCH_CHECK();
  return ASC_OK;
}

namespace asc {
const void* image_data(asc_image im, int* w, int* h, int* bps)
{
  *w = im->w;
  *h = im->h;
  *bps = im->bps;
  return im->data;
}
}  // namespace asc

static int image_render(asc_image im, const float ip[4], const float vp[4], int mode, float thr, float* out, int w,
                        int h, void* stream)
{
  if (!im || !ip || !vp || !out || w < 0 || h < 0) return ASC_ERR_ARG;
  if (w == 0 || h == 0) return ASC_OK;
  ImgArgs a;
  memcpy(a.ip, ip, sizeof a.ip);
  memcpy(a.vp, vp, sizeof a.vp);
  a.threshold = thr;
  a.mode = mode;
  a.rw = reciprocal((double)w);
  a.rh = reciprocal((double)h);
  a.riw = reciprocal((double)ip[2]);
  a.rih = reciprocal((double)ip[3]);
  const dim3 g((w + IW - 1) / IW, (h + IH - 1) / IH);
  k_image_render<<<g, 256, 0, S(stream)>>>(im->data, im->bps, im->w, im->h, a, out, w, h);
  ASC_LAUNCH_CHECK();
  return ASC_OK;
}

ASC_API int asc_rad_render(asc_image im, const float ip[4], const float vp[4], float* out, int w, int h, void* st)
{
  return image_render(im, ip, vp, 0, 0.f, out, w, h, st);
}

ASC_API int asc_background_render(asc_image im, const float ip[4], const float vp[4], float thr, float* out, int w,
                                  int h, void* st)
{
  return image_render(im, ip, vp, 1, thr, out, w, h, st);
}

// ---- elementwise ----
static int elementwise(int op, const float* a, const float* b, const float* c, float* d, size_t n, float val,
                       void* st)
{
  if (!d || (op <= 3 && !a) || ((op == 1 || op == 2 || op == 3) && !b) || (op == 3 && !c)) return ASC_ERR_ARG;
  if (n == 0) return ASC_OK;
  int blocks = (int)std::min<size_t>((n + 255) / 256, 152 * 16);
  k_elementwise<<<blocks, 256, 0, S(st)>>>(op, a, b, c, d, n, val);
  ASC_LAUNCH_CHECK();
  return ASC_OK;
}

ASC_API int asc_drr_background(const float* s, float* d, int w, int h, void* st)
{
  if (w < 0 || h < 0) return ASC_ERR_ARG;
  return elementwise(0, s, nullptr, nullptr, d, (size_t)w * h, 0.f, st);
}
ASC_API int asc_multiply(const float* a, const float* b, float* d, int w, int h, void* st)
{
  if (w < 0 || h < 0) return ASC_ERR_ARG;
  return elementwise(1, a, b, nullptr, d, (size_t)w * h, 0.f, st);
}
ASC_API int asc_merge(const float* a, const float* b, float* d, int w, int h, void* st)
{
  if (w < 0 || h < 0) return ASC_ERR_ARG;
  return elementwise(2, a, b, nullptr, d, (size_t)w * h, 0.f, st);
}
ASC_API int asc_composite(const float* a, const float* b, const float* c, const float*, float* d, int w, int h,
                          void* st)
{
  if (w < 0 || h < 0) return ASC_ERR_ARG;
  return elementwise(3, a, b, c, d, (size_t)w * h, 0.f, st);
}
ASC_API int asc_fill(float* d, size_t n, float v, void* st) { return elementwise(4, nullptr, nullptr, nullptr, d, n, v, st); }

// ---- filters ----
static int filter(int kind, const float* in, float* out, int w, int h, float p0, float p1, float p2, void* st)
{
  if (!in || !out || w < 0 || h < 0 || in == out) return ASC_ERR_ARG;
  asc_filter_desc f = {kind, 1, p0, p1, p2};
  return launch_filter(f, in, out, w, h, S(st));
}
ASC_API int asc_sobel(const float* in, float* out, int w, int h, float scale, float blend, void* st)
{
  return filter(1, in, out, w, h, scale, blend, 0.f, st);
}
ASC_API int asc_contrast(const float* in, float* out, int w, int h, float alpha, float beta, int size, void* st)
{
  return filter(0, in, out, w, h, alpha, beta, (float)size, st);
}
ASC_API int asc_gaussian(const float* in, float* out, int w, int h, float radius, void* st)
{
  return filter(3, in, out, w, h, radius, 0.f, 0.f, st);
}
ASC_API int asc_sharpen(const float* in, float* out, int w, int h, float radius, float contrast, float threshold,
                        void* st)
{
  return filter(4, in, out, w, h, radius, contrast, threshold, st);
}

// ---- reductions ----
ASC_API int asc_ncc_init(unsigned max_n)
{
  std::lock_guard<std::mutex> l(g_red_mu);
  return ncc_init_locked(max_n);
}

int asc::ncc_init_locked(unsigned max_n)
{
  Gate g(device_gate());
  if (g_part) cudaFree(g_part);
  if (g_means) cudaFree(g_means);
  if (g_ticket) cudaFree(g_ticket);
  g_part = nullptr;
  g_means = nullptr;
  g_ticket = nullptr;
  g_max_n = 0;
  if (max_n == 0) return ASC_OK;
  const size_t nb = ((size_t)max_n + RCHUNK - 1) / RCHUNK;
  ASC_CUDA(cudaMalloc(&g_part, nb * sizeof(Moments)));
  ASC_CUDA(cudaMalloc(&g_means, 2 * sizeof(double)));
  ASC_CUDA(cudaMalloc(&g_ticket, sizeof(unsigned)));
  ASC_CUDA(cudaMemset(g_ticket, 0, sizeof(unsigned)));
  g_max_n = max_n;
  ASC_CUDA(cudaGetDevice(&g_red_dev));
  return ASC_OK;
}

ASC_API int asc_ncc(const float* f, const float* g, const float* m, unsigned n, int coverage, double* res, void* st)
{
  if (!f || !g || !m || !res || n == 0 || (coverage != ASC_SUM_TREE && coverage != ASC_SUM_FULL)) return ASC_ERR_ARG;
  ReduceScratch sc;
  int rc = ensure_scratch(n, &sc);
  if (rc) return rc;
  int tree = coverage == ASC_SUM_TREE && tree_needed(n);
  launch_ncc(f, g, m, n, tree, sc, res, S(st));
  ASC_LAUNCH_CHECK();
  return ASC_OK;
}

ASC_API int asc_hdist(const float* f, const float* g, const float* m, unsigned n, int coverage, double* res,
                      void* st)
{
  if (!f || !g || !m || !res || n == 0 || (coverage != ASC_SUM_TREE && coverage != ASC_SUM_FULL)) return ASC_ERR_ARG;
  ReduceScratch sc;
  int rc = ensure_scratch(n, &sc);
  if (rc) return rc;
  int tree = coverage == ASC_SUM_TREE && tree_needed(n);
  unsigned nb = (n + RCHUNK - 1) / RCHUNK;
  k_hdist_means<<<nb, RB, 0, S(st)>>>(f, g, m, n, tree, sc);
  k_hdist_sad<<<nb, RB, 0, S(st)>>>(f, g, m, n, tree, sc, res);
  ASC_LAUNCH_CHECK();
  return ASC_OK;
}

static int host_result(int rc, double* dev, double* out, void* st)
{
  if (rc == ASC_OK) {
    cudaError_t e = cudaMemcpyAsync(out, dev, sizeof(double), cudaMemcpyDeviceToHost, S(st));
    if (e == cudaSuccess) e = cudaStreamSynchronize(S(st));
    if (e != cudaSuccess) rc = cuda_status(e);
  }
  Gate g(device_gate());
  cudaFree(dev);
  return rc;
}

ASC_API int asc_ncc_host(const float* f, const float* g, const float* m, unsigned n, int coverage, double* out,
                         void* st)
{
  if (!out) return ASC_ERR_ARG;
  double* dev = nullptr;
  {
    Gate g(device_gate());
    ASC_CUDA(cudaMalloc(&dev, sizeof(double)));
  }
  return host_result(asc_ncc(f, g, m, n, coverage, dev, st), dev, out, st);
}

ASC_API int asc_hdist_host(const float* f, const float* g, const float* m, unsigned n, int coverage, double* out,
                           void* st)
{
  if (!out) return ASC_ERR_ARG;
  double* dev = nullptr;
  {
    Gate g(device_gate());
    ASC_CUDA(cudaMalloc(&dev, sizeof(double)));
  }
  return host_result(asc_hdist(f, g, m, n, coverage, dev, st), dev, out, st);
}

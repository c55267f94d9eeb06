// denoise.cuh — argent's built-in à-trous denoiser on the device
// (crates/argent-post/src/denoise.rs:535-700): an edge-avoiding à-trous
// wavelet filter (Dammertz et al. 2010) with SVGF-style luminance edge
// stopping (Schied et al. 2017), 5 passes of the 5x5 B3-spline kernel with
// holes 1, 2, 4, 8, 16, albedo demodulation, normal and albedo weights.
//
// Every per-pixel sum runs in argent's order (kernel taps in index order,
// borders renormalised) and the library has no FMA contraction, so the
// result differs from argent's only through expf (CUDA against the host's).
// One image: all buffers are w*h, row-major; colours are 3 floats per pixel.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

namespace dn {

#define DN_PASSES 5
#define DN_SIGMA_LUM 4.0f
#define DN_INV_SIGMA_ALBEDO2 100.0f  // 1 / 0.01
#define DN_DEMOD_FLOOR 0.02f

__device__ __forceinline__ float clean_radiance(float v) { return isfinite(v) ? fmaxf(v, 0.0f) : 0.0f; }
__device__ __forceinline__ float clean_unit(float v, float lo) {
  return isfinite(v) ? fminf(fmaxf(v, lo), 1.0f) : 0.0f;
}
__device__ __forceinline__ float lum(float r, float g, float b) { return 0.2126f * r + 0.7152f * g + 0.0722f * b; }

// Per pixel, so that a tap is one 16-byte load of the signal, one of the
// guides, and two small ones:
//   sig     demodulated colour, luminance
//   guide   albedo, normal x
//   nyz     normal y, z
// and the variance apart (the passes rewrite it with the signal).

// denoise.rs:675-704: guides, demodulated signal and its luminance.
template <bool ALBEDO, bool NORMAL>
__global__ void k_dn_prep(const float* color, const float* albedo, const float* normal, uint32_t np, float4* sig,
                          float4* guide, float2* nyz) {
  for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < np; p += gridDim.x * blockDim.x) {
    size_t o = 3 * (size_t)p;
    float s[3], a[3] = {0.0f, 0.0f, 0.0f}, n[3] = {0.0f, 0.0f, 0.0f};
    for (int c = 0; c < 3; ++c) s[c] = clean_radiance(color[o + c]);
    if (ALBEDO) {
      for (int c = 0; c < 3; ++c) {
        a[c] = clean_unit(albedo[o + c], 0.0f);
        s[c] = s[c] / fmaxf(a[c], DN_DEMOD_FLOOR);
      }
    }
    if (NORMAL) {
      float v[3];
      for (int c = 0; c < 3; ++c) v[c] = isfinite(normal[o + c]) ? normal[o + c] : 0.0f;
      float len = sqrtf(v[0] * v[0] + v[1] * v[1] + v[2] * v[2]);
      for (int c = 0; c < 3; ++c) n[c] = len > 1e-6f ? v[c] / len : 0.0f;
      nyz[p] = make_float2(n[1], n[2]);
    }
    if (ALBEDO) guide[p] = make_float4(a[0], a[1], a[2], n[0]);
    sig[p] = make_float4(s[0], s[1], s[2], lum(s[0], s[1], s[2]));
  }
}

// blur_sep (denoise.rs:547-578) with three taps at one pixel: the rows'
// horizontal sums, then their vertical one; the weight sum of the taps inside
// the image renormalises each.  at(x, y) gives the value of a pixel.  A weight
// sum of 1 needs no division.
template <class F>
__device__ __forceinline__ float blur3(F at, int x, int y, int w, int h, float k0, float k1) {
  const float k[3] = {k0, k1, k0};
  float acc = 0.0f, ws = 0.0f;
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const int yy = y + j - 1;
    if (yy < 0 || yy >= h) continue;
    float ra = 0.0f, rw = 0.0f;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const int xx = x + i - 1;
      if (xx >= 0 && xx < w) {
        ra += k[i] * at(xx, yy);
        rw += k[i];
      }
    }
    acc += k[j] * (rw == 1.0f ? ra : ra / rw);
    ws += k[j];
  }
  return ws == 1.0f ? acc : acc / ws;
}

// noise_variance's residual (denoise.rs:582-586): 9/8 (v - mean)^2, the mean
// over 3 x 3 pixels.
__global__ void __launch_bounds__(256) k_dn_resid(const float4* sig, uint32_t w, uint32_t h, float* out) {
  const uint32_t tx = (w + 31) / 32;  // tiles per row
  const int x = (int)(blockIdx.x % tx * 32 + (threadIdx.x & 31)), y = (int)(blockIdx.x / tx * 8 + (threadIdx.x >> 5));
  if (x >= (int)w || y >= (int)h) return;
  float mean = blur3([&](int xx, int yy) { return sig[(size_t)yy * w + xx].w; }, x, y, (int)w, (int)h, 1.0f, 1.0f);
  float d = sig[(size_t)y * w + x].w - mean;
  out[(size_t)y * w + x] = 1.125f * d * d;
}

// blur_sep with five unit taps, both directions: a tile's rows, two above
// and below it, summed horizontally into shared memory, then vertically.
__global__ void __launch_bounds__(256) k_dn_box5(const float* src, float* dst, uint32_t w, uint32_t h) {
  __shared__ float rows[12][32];
  const uint32_t tx = (w + 31) / 32;
  const int x = (int)(blockIdx.x % tx * 32 + (threadIdx.x & 31)), y0 = (int)(blockIdx.x / tx * 8);
  for (int r = (int)(threadIdx.x >> 5); r < 12; r += 8) {
    const int y = y0 + r - 2;
    if (x < (int)w && y >= 0 && y < (int)h) {
      float acc = 0.0f, ws = 0.0f;
#pragma unroll
      for (int i = -2; i <= 2; ++i)
        if (x + i >= 0 && x + i < (int)w) {
          acc += src[(size_t)y * w + (x + i)];
          ws += 1.0f;
        }
      rows[r][threadIdx.x & 31] = acc / ws;
    }
  }
  __syncthreads();
  const int y = y0 + (int)(threadIdx.x >> 5);
  if (x >= (int)w || y >= (int)h) return;
  float acc = 0.0f, ws = 0.0f;
#pragma unroll
  for (int j = -2; j <= 2; ++j)
    if (y + j >= 0 && y + j < (int)h) {
      acc += rows[(int)(threadIdx.x >> 5) + 2 + j][threadIdx.x & 31];
      ws += 1.0f;
    }
  dst[(size_t)y * w + x] = acc / ws;
}

__device__ __forceinline__ float pow128(float d) {
  // powi(d, 128): seven squarings, as binary exponentiation does it.
  float x = d;
#pragma unroll
  for (int i = 0; i < 7; ++i) x = x * x;
  return x;
}

// atrous_pass (denoise.rs:593-650), with the variance's 3-tap blur at the
// pixel and, in the last pass (LAST), the remodulation by the albedo
// (denoise.rs:705-711), written as 3 floats per pixel.  Blocks are tiles of
// 32 x 8 pixels, so that the rows of taps a block shares come from L1.  Bound
// by the instructions of the 25 taps (an expf each); with eleven 4-byte loads
// per tap from planar arrays, two launches of blur before it and blocks of
// one row, a pass took 251 us at 1920 x 1080 (ncu, cold), now 150-184;
// the whole filter 1.40 ms and 20 launches, now 0.91 ms and 8.
template <bool ALBEDO, bool NORMAL, bool LAST>
__global__ void __launch_bounds__(256) k_dn_atrous(const float4* __restrict__ sig, const float* __restrict__ var,
                                                   const float4* __restrict__ guide,
                                                   const float2* __restrict__ nyz, uint32_t w, uint32_t h, int step,
                                                   float4* out, float* out_var, float* out_rgb) {
  const float B3[5] = {1.0f / 16.0f, 1.0f / 4.0f, 3.0f / 8.0f, 1.0f / 4.0f, 1.0f / 16.0f};
  const uint32_t tx = (w + 31) / 32;  // tiles per row
  const int x = (int)(blockIdx.x % tx * 32 + (threadIdx.x & 31)), y = (int)(blockIdx.x / tx * 8 + (threadIdx.x >> 5));
  if (x >= (int)w || y >= (int)h) return;
  const size_t p = (size_t)y * w + x;
  const float lp = sig[p].w;
  const float vb = blur3([&](int xx, int yy) { return var[(size_t)yy * w + xx]; }, x, y, (int)w, (int)h, 0.25f, 0.5f);
  const float inv_sl = 1.0f / (DN_SIGMA_LUM * sqrtf(fmaxf(vb, 0.0f)) + 1e-10f);
  float4 gp = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  float2 np2 = make_float2(0.0f, 0.0f);
  if (ALBEDO) gp = guide[p];
  if (NORMAL) np2 = nyz[p];
  const bool np_zero = gp.w == 0.0f && np2.x == 0.0f && np2.y == 0.0f;
  float acc[3] = {0, 0, 0}, ws = 0.0f, wv = 0.0f;
  for (int ky = 0; ky < 5; ++ky) {
    int qy = y + (ky - 2) * step;
    if (qy < 0 || qy >= (int)h) continue;
    float hy = B3[ky];
#pragma unroll
    for (int kx = 0; kx < 5; ++kx) {
      int qx = x + (kx - 2) * step;
      if (qx < 0 || qx >= (int)w) continue;
      float hx = B3[kx];
      size_t q = (size_t)qy * w + qx;
      const float4 s = sig[q];
      float e = fabsf(s.w - lp) * inv_sl;
      float4 g = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      if (ALBEDO) {
        g = guide[q];
        float d0 = gp.x - g.x, d1 = gp.y - g.y, d2 = gp.z - g.z;
        e += (d0 * d0 + d1 * d1 + d2 * d2) * DN_INV_SIGMA_ALBEDO2;
      }
      float wgt = hx * hy * expf(-e);
      if (NORMAL) {
        const float2 n = nyz[q];
        bool nq_zero = g.w == 0.0f && n.x == 0.0f && n.y == 0.0f;
        if (!np_zero && !nq_zero) {
          float d = fmaxf(gp.w * g.w + np2.x * n.x + np2.y * n.y, 0.0f);
          wgt *= pow128(d);
        }
      }
      acc[0] += wgt * s.x;
      acc[1] += wgt * s.y;
      acc[2] += wgt * s.z;
      ws += wgt;
      wv += wgt * wgt * var[q];
    }
  }
  float r[3] = {acc[0] / ws, acc[1] / ws, acc[2] / ws};
  if (LAST) {
    if (ALBEDO) {
      r[0] = r[0] * fmaxf(gp.x, DN_DEMOD_FLOOR);
      r[1] = r[1] * fmaxf(gp.y, DN_DEMOD_FLOOR);
      r[2] = r[2] * fmaxf(gp.z, DN_DEMOD_FLOOR);
    }
    for (int c = 0; c < 3; ++c) out_rgb[3 * p + c] = r[c];
  } else {
    out[p] = make_float4(r[0], r[1], r[2], lum(r[0], r[1], r[2]));
    out_var[p] = wv / (ws * ws);
  }
}

}  // namespace dn

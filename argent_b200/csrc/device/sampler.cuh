// sampler.cuh — argent's per-sample dimension stream on the device
// (crates/argent-core/src/sampler.rs:5-100).
//
// Dimensions below 256 of samples with index < 2^16 come from an
// Owen-scrambled Sobol sequence evaluated four dimensions at a time; the rest
// come from argent's PCG-XSH-RR stream.  argent gets the Sobol values from the
// sobol_burley 0.5.0 crate, which is not vendored.  This file implements the
// published method instead (Burley 2020, "Practical Hash-based Owen
// Scrambling", JCGT 9(4)): index shuffling by nested uniform scrambling, the
// first four Sobol dimensions, and an independent scramble per 4-dimension
// set (padding).  The direction numbers of those four dimensions come from
// the primitive polynomials x+1, x^2+x+1 and x^3+x+1.
#pragma once
#include <cstdint>

#include "dev_math.cuh"
#include "tables.cuh"

namespace dev {

#define ARGENT_SOBOL_MAX_DIM 256u


__device__ __forceinline__ uint32_t hash32(uint32_t x) {
  x ^= x >> 16;
  x *= 0x7feb352du;
  x ^= x >> 15;
  x *= 0x846ca68bu;
  x ^= x >> 16;
  return x;
}
__device__ __forceinline__ uint32_t lk_permutation(uint32_t x, uint32_t seed) {
  x += seed;
  x ^= x * 0x6c50b47cu;
  x ^= x * 0xb82f1e52u;
  x ^= x * 0xc7afe638u;
  x ^= x * 0x8d22f6e6u;
  return x;
}
__device__ __forceinline__ uint32_t nested_uniform_scramble(uint32_t x, uint32_t seed) {
  return __brev(lk_permutation(__brev(x), seed));
}
__device__ __forceinline__ uint32_t hash_combine(uint32_t seed, uint32_t v) {
  return seed ^ (v + 0x9e3779b9u + (seed << 6) + (seed >> 2));
}
__device__ __forceinline__ uint32_t sobol_dim(uint32_t index, int d) {
  const uint32_t* t = &d_sobol_bytes[d][0][0];
  return __ldg(t + (index & 0xffu)) ^ __ldg(t + 256 + ((index >> 8) & 0xffu)) ^
         __ldg(t + 512 + ((index >> 16) & 0xffu)) ^ __ldg(t + 768 + (index >> 24));
}
// The first N of the four values of padding set `set`.  Dimension 0 is the
// van der Corput sequence, whose generator matrix reverses the index's bits:
// the reversal cancels the scramble's own (the tables serve the others).
template <int N>
__device__ __forceinline__ void sample_4d(uint32_t index, uint32_t set, uint32_t seed, float* out) {
  uint32_t sseed = hash_combine(seed, hash32(set));
  uint32_t shuffled = nested_uniform_scramble(index, sseed);
#pragma unroll
  for (int d = 0; d < N; ++d) {
    uint32_t dseed = hash_combine(sseed, hash32((uint32_t)d + 1u));
    uint32_t x = d == 0 ? __brev(lk_permutation(shuffled, dseed))
                        : nested_uniform_scramble(sobol_dim(shuffled, d), dseed);
    out[d] = (float)(x >> 8) * (1.0f / 16777216.0f);
  }
}

// argent's dimension stream is drawn in sets of four dimensions, as the
// callers need them: a path's camera sample takes dimensions 0..4, bounce d
// the eight from 8 + 8 d.  A set is Sobol or PCG as a whole (256 is a
// multiple of four), and PCG values come in the order of the dimensions, so
// the values are those of argent's one-by-one draws.  (argent clamps Sobol
// values to 0.99999994; 24-bit values never exceed it.)
struct Sampler {
  uint32_t index, seed;
  uint64_t rng;

  __device__ __forceinline__ void init(uint32_t pixel_seed, uint32_t sample_index) {
    index = sample_index;
    seed = pixel_seed;
    rng = (((uint64_t)pixel_seed << 32) | (uint64_t)sample_index) ^ 0x9e3779b97f4a7c15ull;
  }
  // Resume a path: the PCG state travels with the path between kernels.
  __device__ __forceinline__ void resume(uint32_t pixel_seed, uint32_t sample_index, uint64_t rng_state) {
    index = sample_index;
    seed = pixel_seed;
    rng = rng_state;
  }
  __device__ __forceinline__ float next_random() {
    rng = rng * 6364136223846793005ull + 1442695040888963407ull;
    uint64_t x = ((rng >> 18) ^ rng) >> 27;
    uint32_t rot = (uint32_t)(rng >> 59);
    uint32_t v = __funnelshift_r((uint32_t)x, (uint32_t)x, rot);
    return (float)(v >> 8) * (1.0f / 16777216.0f);
  }
  // The first N dimensions of set `set` (dimensions 4 set .. 4 set + N - 1).
  template <int N>
  __device__ __forceinline__ void draw(uint32_t set, float* out) {
    if (set < ARGENT_SOBOL_MAX_DIM / 4u && index < (1u << 16)) {
      sample_4d<N>(index, set, seed, out);
    } else {
#pragma unroll
      for (int d = 0; d < N; ++d) out[d] = next_random();
    }
  }
};

// sampler.rs:103-108
__device__ __forceinline__ float tent(float u, float r) {
  float uu = 2.0f * u;
  if (uu < 1.0f) return r * (sqrtf(uu) - 1.0f);
  return r * (1.0f - sqrtf(2.0f - uu));
}
// sampler.rs:111-124
__device__ __forceinline__ void disk(float u, float v, float* ox, float* oy) {
  float a = 2.0f * u - 1.0f;
  float b = 2.0f * v - 1.0f;
  if (a == 0.0f && b == 0.0f) {
    *ox = 0.0f;
    *oy = 0.0f;
    return;
  }
  float r, phi;
  if (fabsf(a) > fabsf(b)) {
    r = a;
    phi = (ARGENT_PI_F / 4.0f) * (b / a);
  } else {
    r = b;
    phi = (ARGENT_PI_F / 2.0f) - (ARGENT_PI_F / 4.0f) * (a / b);
  }
  float s, c;
  sincosf(phi, &s, &c);
  *ox = r * c;
  *oy = r * s;
}
// sampler.rs:127-132
__device__ __forceinline__ V3 cosine_hemisphere(float u, float v) {
  float x, y;
  disk(u, v, &x, &y);
  float z = sqrtf(fmaxf(1.0f - x * x - y * y, 0.0f));
  return V3{x, y, z};
}

}  // namespace dev

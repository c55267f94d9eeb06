// The device code compiled for the CPU: what the headers under
// argent_b200/csrc use of CUDA, in plain C++.  Tests put this folder first in
// the include path, so `#include <cuda_runtime.h>` finds this file.
//
// A launch runs its blocks one after the other, each thread of a block as a
// thread of its own.  Warp collectives (shuffles, ballots) and __syncthreads
// meet at barriers, so every lane of a warp has to take the same ones, as the
// kernels do; a lane that returned is dropped from them.  Arithmetic is the
// host's IEEE arithmetic without contraction, which is what the library's
// build (--fmad=false) rounds like.
#pragma once
#include <atomic>
#include <barrier>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <memory>
#include <mutex>
#include <thread>
#include <vector>

#define __device__
#define __host__
#define __global__
#define __constant__ inline
#define __shared__ static
#define __forceinline__ inline
#define __noinline__
#define __launch_bounds__(...)
#define __restrict__

struct uint2 { uint32_t x, y; };
struct int2 { int32_t x, y; };
struct alignas(16) uint4 { uint32_t x, y, z, w; };
struct float2 { float x, y; };
struct float3 { float x, y, z; };
struct alignas(16) float4 { float x, y, z, w; };
inline uint2 make_uint2(uint32_t x, uint32_t y) { return {x, y}; }
inline int2 make_int2(int32_t x, int32_t y) { return {x, y}; }
inline uint4 make_uint4(uint32_t x, uint32_t y, uint32_t z, uint32_t w) { return {x, y, z, w}; }
inline float2 make_float2(float x, float y) { return {x, y}; }
inline float4 make_float4(float x, float y, float z, float w) { return {x, y, z, w}; }

typedef int cudaError_t;
typedef void* cudaStream_t;
typedef void* cudaEvent_t;
typedef void* cudaMemPool_t;
typedef void* cudaGraphExec_t;
inline int cudaFree(void*) { return 0; }

struct Dim { unsigned x = 0, y = 0, z = 0; };
inline thread_local Dim threadIdx, blockIdx;
inline Dim blockDim, gridDim;

namespace host_emulation {
struct Warp {
  std::barrier<> meet;
  uint64_t slot[32] = {};
  bool live[32] = {};
  explicit Warp(int n) : meet(n) {}
};
inline thread_local Warp* warp;
inline std::unique_ptr<std::barrier<>> block;

template <class F>
void launch(unsigned blocks, unsigned threads, F kernel) {
  blockDim.x = threads;
  gridDim.x = blocks;
  for (unsigned b = 0; b < blocks; ++b) {
    std::vector<std::unique_ptr<Warp>> warps;
    for (unsigned w = 0; w < (threads + 31) / 32; ++w) {
      const unsigned n = std::min(32u, threads - 32 * w);
      warps.push_back(std::make_unique<Warp>((int)n));
      for (unsigned i = 0; i < n; ++i) warps[w]->live[i] = true;
    }
    block = std::make_unique<std::barrier<>>((int)threads);
    std::vector<std::thread> ts;
    for (unsigned t = 0; t < threads; ++t)
      ts.emplace_back([&, t] {
        threadIdx.x = t;
        blockIdx.x = b;
        warp = warps[t / 32].get();
        kernel();
        warp->live[t & 31] = false;
        warp->meet.arrive_and_drop();
        block->arrive_and_drop();
      });
    for (auto& t : ts) t.join();
  }
}

// Every lane's value to `pick`, between two meetings of the warp.
template <class T, class F>
auto exchange(T v, F pick) {
  static_assert(sizeof(T) <= 8);
  Warp& w = *warp;
  uint64_t bits = 0;
  std::memcpy(&bits, &v, sizeof v);
  w.slot[threadIdx.x & 31] = bits;
  w.meet.arrive_and_wait();
  auto r = pick([&](unsigned lane) {
    T x;
    std::memcpy(&x, &w.slot[lane & 31], sizeof x);
    return x;
  });
  w.meet.arrive_and_wait();
  return r;
}
}  // namespace host_emulation

inline void __syncthreads() { host_emulation::block->arrive_and_wait(); }
inline int __syncthreads_or(int p) {
  static std::atomic<int> any;
  if (p) any = 1;
  __syncthreads();
  const int r = any;
  __syncthreads();
  any = 0;
  __syncthreads();
  return r;
}
inline void __threadfence() { std::atomic_thread_fence(std::memory_order_seq_cst); }

#define HE_LANE (threadIdx.x & 31u)
template <class T>
T __shfl_sync(unsigned, T v, int src) {
  return host_emulation::exchange(v, [&](auto at) { return at((unsigned)src); });
}
template <class T>
T __shfl_xor_sync(unsigned, T v, int m) {
  return host_emulation::exchange(v, [&](auto at) { return at(HE_LANE ^ (unsigned)m); });
}
template <class T>
T __shfl_up_sync(unsigned, T v, unsigned d) {
  return host_emulation::exchange(v, [&](auto at) { return at(HE_LANE >= d ? HE_LANE - d : HE_LANE); });
}
template <class T>
T __shfl_down_sync(unsigned, T v, unsigned d) {
  return host_emulation::exchange(v, [&](auto at) { return at(HE_LANE + d < 32 ? HE_LANE + d : HE_LANE); });
}
inline unsigned __ballot_sync(unsigned, int p) {
  auto* w = host_emulation::warp;
  return host_emulation::exchange((uint32_t)(p != 0), [&](auto at) {
    unsigned r = 0;
    for (unsigned i = 0; i < 32; ++i) r |= w->live[i] && at(i) ? 1u << i : 0u;
    return r;
  });
}
inline unsigned __match_any_sync(unsigned, unsigned v) {
  auto* w = host_emulation::warp;
  return host_emulation::exchange((uint32_t)v, [&](auto at) {
    unsigned r = 0;
    for (unsigned i = 0; i < 32; ++i) r |= w->live[i] && at(i) == v ? 1u << i : 0u;
    return r;
  });
}
inline unsigned __activemask() { return __ballot_sync(~0u, 1); }
inline unsigned __reduce_or_sync(unsigned, unsigned v) {
  return host_emulation::exchange((uint32_t)v, [&](auto at) {
    unsigned r = 0;
    for (unsigned i = 0; i < 32; ++i) r |= at(i);
    return r;
  });
}
inline unsigned __reduce_max_sync(unsigned, unsigned v) {
  return host_emulation::exchange((uint32_t)v, [&](auto at) {
    unsigned r = 0;
    for (unsigned i = 0; i < 32; ++i) r = std::max<unsigned>(r, at(i));
    return r;
  });
}

template <class T, class U>
T atomicAdd(T* p, U v) {
  return std::atomic_ref<T>(*p).fetch_add((T)v);
}
template <class T, class U>
T atomicOr(T* p, U v) {
  return std::atomic_ref<T>(*p).fetch_or((T)v);
}
template <class T, class U>
T atomicMax(T* p, U v) {
  std::atomic_ref<T> a(*p);
  T o = a.load();
  while (o < (T)v && !a.compare_exchange_weak(o, (T)v)) {
  }
  return o;
}
template <class T, class U>
T atomicMin(T* p, U v) {
  std::atomic_ref<T> a(*p);
  T o = a.load();
  while (o > (T)v && !a.compare_exchange_weak(o, (T)v)) {
  }
  return o;
}

template <class T>
T __ldg(const T* p) { return *p; }
template <class T>
T __ldcg(const T* p) { return *p; }
template <class T>
T __ldcs(const T* p) { return *p; }
template <class T>
void __stcs(T* p, T v) { *p = v; }

inline uint32_t __float_as_uint(float f) { uint32_t u; std::memcpy(&u, &f, 4); return u; }
inline float __uint_as_float(uint32_t u) { float f; std::memcpy(&f, &u, 4); return f; }
inline int __float_as_int(float f) { return (int)__float_as_uint(f); }
inline float __int_as_float(int i) { return __uint_as_float((uint32_t)i); }
inline int __popc(uint32_t v) { return __builtin_popcount(v); }
inline int __ffs(uint32_t v) { return __builtin_ffs((int)v); }
inline int __clz(uint32_t v) { return v ? __builtin_clz(v) : 32; }
inline int __clzll(uint64_t v) { return v ? __builtin_clzll(v) : 64; }
inline uint32_t __brev(uint32_t v) {
  uint32_t r = 0;
  for (int i = 0; i < 32; ++i) r |= ((v >> i) & 1u) << (31 - i);
  return r;
}
inline uint32_t __byte_perm(uint32_t a, uint32_t b, uint32_t s) {
  const uint64_t x = ((uint64_t)b << 32) | a;
  uint32_t r = 0;
  for (int i = 0; i < 4; ++i) r |= (uint32_t)((x >> (8 * ((s >> (4 * i)) & 7u))) & 0xffu) << (8 * i);
  return r;
}
inline uint32_t __funnelshift_r(uint32_t lo, uint32_t hi, uint32_t s) {
  return (uint32_t)((((uint64_t)hi << 32) | lo) >> (s & 31u));
}
inline float __fadd_rn(float a, float b) { return a + b; }
inline float __fsub_rn(float a, float b) { return a - b; }
inline float __fmul_rn(float a, float b) { return a * b; }
inline float __fdiv_rn(float a, float b) { return a / b; }
inline float __frcp_rn(float a) { return 1.0f / a; }
inline float __fsqrt_rn(float a) { return std::sqrt(a); }
inline float __fmul_ru(float a, float b) {  // the product is exact in double
  const float r = (float)((double)a * b);
  return (double)r < (double)a * b ? std::nextafter(r, INFINITY) : r;
}
inline float __fmaf_rn(float a, float b, float c) { return std::fma(a, b, c); }
inline double __dadd_rn(double a, double b) { return a + b; }
inline double __dsub_rn(double a, double b) { return a - b; }
inline double __dmul_rn(double a, double b) { return a * b; }
template <class A, class B>
auto min(A a, B b) { return a < b ? a : b; }
template <class A, class B>
auto max(A a, B b) { return a > b ? a : b; }
using std::isfinite;
using std::signbit;

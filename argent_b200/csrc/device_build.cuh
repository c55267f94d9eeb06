// device_build.cuh — the piece BVH built on the device, for fast piece
// swaps (argent builds on the host at every prepare, bvh.rs:117-146).
//
// A linear BVH (Karras 2012, "Maximizing parallelism in the construction of
// BVHs, octrees, and k-d trees"): 63-bit Morton codes of the triangle
// centroids, a radix sort, the binary radix tree (one thread per internal
// node), boxes bottom-up, then the same collapse to 8-wide nodes the host
// builder does (open the interior child of largest area until 8 children;
// subtrees of at most 4 triangles become leaves), level by level, writing
// the same 80-byte node and 48-byte triangle layouts (host/bvh_build.h) with
// the same conservative plane quantisation.  The traversal takes either
// builder's tree: every closest hit is the minimum of (t, triangle index) over
// the triangles that are tested and pass, which is the same for both but for
// hits of edge-on triangles outside their own boxes (device/traverse.cuh).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

namespace db {

#define DB_LEAF_MAX 4
#define DB_ERR_EXTENT 1u
#define DB_ERR_QUANT 2u

struct Bin {
  float* lo;  // 3 per node
  float* hi;
  uint32_t* first;
  uint32_t* last;
  int32_t* left;
  int32_t* right;
  int32_t* parent;
  uint32_t* flag;
};

// Floats as unsigned words of the same order, for atomicMin and atomicMax.
__device__ __forceinline__ uint32_t ordered(float f) {
  uint32_t u = __float_as_uint(f);
  return u & 0x80000000u ? ~u : u | 0x80000000u;
}
__device__ __forceinline__ float unordered(uint32_t u) {
  return __uint_as_float(u & 0x80000000u ? u & 0x7fffffffu : ~u);
}

#define DB_BAD_INDEX 1u
#define DB_BAD_POSITION 2u

// A piece's arrays as the kernels read them, from the caller's: vertices and
// normals in 16 bytes, triangles with their material slot.  info[0] collects
// what is wrong with them, info[1] the highest material slot; info[2..7] start
// the centroid bounds.
__global__ void __launch_bounds__(256) k_piece_pack(const float* __restrict__ pos, const float* __restrict__ nrm,
                                                    const uint32_t* __restrict__ tri,
                                                    const uint16_t* __restrict__ mat, uint32_t nv, uint32_t nt,
                                                    float4* pos4, float4* nrm4, uint4* tidx, uint32_t* info) {
  const uint32_t t0 = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
  uint32_t bad = 0, top = 0;
  if (t0 < 6) info[2 + t0] = t0 < 3 ? 0xffffffffu : 0u;
  for (uint64_t i = t0; i < nv; i += stride) {  // nv may be near 2^32, where a 32-bit i would wrap
    const float x = pos[3 * i], y = pos[3 * i + 1], z = pos[3 * i + 2];
    if (!(isfinite(x) && isfinite(y) && isfinite(z))) bad |= DB_BAD_POSITION;
    pos4[i] = make_float4(x, y, z, 0.0f);
    if (nrm) nrm4[i] = make_float4(nrm[3 * i], nrm[3 * i + 1], nrm[3 * i + 2], 0.0f);
  }
  for (uint32_t i = t0; i < nt; i += stride) {
    const uint32_t a = tri[3 * (size_t)i], b = tri[3 * (size_t)i + 1], c = tri[3 * (size_t)i + 2];
    const uint32_t m = mat ? mat[i] : 0u;
    if (a >= nv || b >= nv || c >= nv) bad |= DB_BAD_INDEX;
    top = max(top, m);
    tidx[i] = make_uint4(a, b, c, m);
  }
  bad = __reduce_or_sync(0xffffffffu, bad);
  top = __reduce_max_sync(0xffffffffu, top);
  if ((threadIdx.x & 31) == 0) {
    if (bad) atomicOr(info, bad);
    if (top) atomicMax(info + 1, top);
  }
}

// Per triangle: box and centroid; the centroid bounds (ordered words, three
// minima and three maxima).  Launched with 256 threads per block.
__global__ void __launch_bounds__(256) k_tri_boxes(const float4* pos, const uint4* tri, uint32_t n, float* tlo,
                                                   float* thi, float* cen, uint32_t* bounds) {
  __shared__ float slo[3][256], shi[3][256];
  float clo[3] = {INFINITY, INFINITY, INFINITY}, chi[3] = {-INFINITY, -INFINITY, -INFINITY};
  for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
    uint4 q = tri[t];
    float4 a = pos[q.x], b = pos[q.y], c = pos[q.z];
    float lo[3] = {fminf(fminf(a.x, b.x), c.x), fminf(fminf(a.y, b.y), c.y), fminf(fminf(a.z, b.z), c.z)};
    float hi[3] = {fmaxf(fmaxf(a.x, b.x), c.x), fmaxf(fmaxf(a.y, b.y), c.y), fmaxf(fmaxf(a.z, b.z), c.z)};
    for (int k = 0; k < 3; ++k) {
      tlo[3 * (size_t)t + k] = lo[k];
      thi[3 * (size_t)t + k] = hi[k];
      float m = 0.5f * lo[k] + 0.5f * hi[k];
      cen[3 * (size_t)t + k] = m;
      clo[k] = fminf(clo[k], m);
      chi[k] = fmaxf(chi[k], m);
    }
  }
  for (int k = 0; k < 3; ++k) {
    slo[k][threadIdx.x] = clo[k];
    shi[k][threadIdx.x] = chi[k];
  }
  __syncthreads();
  for (int s = blockDim.x / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s)
      for (int k = 0; k < 3; ++k) {
        slo[k][threadIdx.x] = fminf(slo[k][threadIdx.x], slo[k][threadIdx.x + s]);
        shi[k][threadIdx.x] = fmaxf(shi[k][threadIdx.x], shi[k][threadIdx.x + s]);
      }
    __syncthreads();
  }
  if (threadIdx.x < 3) {
    atomicMin(bounds + threadIdx.x, ordered(slo[threadIdx.x][0]));
    atomicMax(bounds + 3 + threadIdx.x, ordered(shi[threadIdx.x][0]));
  }
}

__device__ __forceinline__ uint64_t spread21(uint32_t v) {
  uint64_t x = v & 0x1fffffu;
  x = (x | x << 32) & 0x1f00000000ffffull;
  x = (x | x << 16) & 0x1f0000ff0000ffull;
  x = (x | x << 8) & 0x100f00f00f00f00full;
  x = (x | x << 4) & 0x10c30c30c30c30c3ull;
  x = (x | x << 2) & 0x1249249249249249ull;
  return x;
}

// 63-bit Morton code of each centroid within the centroid bounds.  (With
// per-block partial bounds that every thread reduced for itself, this took
// 302 us for 500k triangles, a fifth of the build's kernels.)
__global__ void k_morton(const float* cen, uint32_t n, const uint32_t* bounds, uint64_t* keys, uint32_t* vals) {
  float lo[3], hi[3];
  for (int k = 0; k < 3; ++k) {
    lo[k] = unordered(bounds[k]);
    hi[k] = unordered(bounds[3 + k]);
  }
  for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
    uint32_t q[3];
    for (int k = 0; k < 3; ++k) {
      float ext = hi[k] - lo[k];
      float u = ext > 0.0f ? (cen[3 * (size_t)t + k] - lo[k]) / ext : 0.0f;
      u = fminf(fmaxf(u, 0.0f), 1.0f);
      q[k] = (uint32_t)fminf(u * 2097152.0f, 2097151.0f);
    }
    keys[t] = (spread21(q[0]) << 2) | (spread21(q[1]) << 1) | spread21(q[2]);
    vals[t] = t;
  }
}

// Karras' common-prefix length of sorted keys i and j (-1 outside the
// array; equal keys fall back to the indices).
__device__ __forceinline__ int delta(const uint64_t* keys, int64_t n, int64_t i, int64_t j) {
  if (j < 0 || j >= n) return -1;
  uint64_t a = keys[i], b = keys[j];
  if (a == b) return 64 + __clz((uint32_t)(i ^ j));
  return __clzll(a ^ b);
}

// Internal node i of the binary radix tree (Karras 2012, Fig. 4).  Binary
// ids: internal nodes 0 .. n-2, leaf k (sorted position k) at n-1+k.
__global__ void k_radix_tree(const uint64_t* keys, uint32_t n, Bin bn) {
  int64_t N = n;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < N - 1; i += (int64_t)gridDim.x * blockDim.x) {
    int d = delta(keys, N, i, i + 1) - delta(keys, N, i, i - 1) >= 0 ? 1 : -1;
    int dmin = delta(keys, N, i, i - d);
    int64_t lmax = 2;
    while (delta(keys, N, i, i + lmax * d) > dmin) lmax *= 2;
    int64_t l = 0;
    for (int64_t t = lmax / 2; t >= 1; t /= 2)
      if (delta(keys, N, i, i + (l + t) * d) > dmin) l += t;
    int64_t j = i + l * d;
    int dnode = delta(keys, N, i, j);
    int64_t s = 0, t = l;
    do {
      t = (t + 1) / 2;
      if (delta(keys, N, i, i + (s + t) * d) > dnode) s += t;
    } while (t > 1);
    int64_t gamma = i + s * d + (d < 0 ? -1 : 0);
    int64_t lo = i < j ? i : j, hi = i < j ? j : i;
    int32_t left = (lo == gamma) ? (int32_t)(N - 1 + gamma) : (int32_t)gamma;
    int32_t right = (hi == gamma + 1) ? (int32_t)(N - 1 + gamma + 1) : (int32_t)(gamma + 1);
    bn.left[i] = left;
    bn.right[i] = right;
    bn.first[i] = (uint32_t)lo;
    bn.last[i] = (uint32_t)hi;
    bn.parent[left] = (int32_t)i;
    bn.parent[right] = (int32_t)i;
  }
}

// Boxes bottom-up: each leaf writes its box and climbs; the second child to
// arrive at a node computes the node's box and continues.
__global__ void k_boxes_up(const float* tlo, const float* thi, const uint32_t* vals, uint32_t n, Bin bn) {
  for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
    uint32_t leaf = n - 1 + k, t = vals[k];
    for (int a = 0; a < 3; ++a) {
      bn.lo[3 * (size_t)leaf + a] = tlo[3 * (size_t)t + a];
      bn.hi[3 * (size_t)leaf + a] = thi[3 * (size_t)t + a];
    }
    bn.first[leaf] = k;
    bn.last[leaf] = k;
    bn.left[leaf] = -1;
    bn.right[leaf] = -1;
    __threadfence();
    int32_t p = n > 1 ? bn.parent[leaf] : -1;
    while (p >= 0) {
      if (atomicAdd(bn.flag + p, 1u) == 0) break;
      int32_t l = bn.left[p], r = bn.right[p];
      for (int a = 0; a < 3; ++a) {
        bn.lo[3 * (size_t)p + a] = fminf(__ldcg(bn.lo + 3 * (size_t)l + a), __ldcg(bn.lo + 3 * (size_t)r + a));
        bn.hi[3 * (size_t)p + a] = fmaxf(__ldcg(bn.hi + 3 * (size_t)l + a), __ldcg(bn.hi + 3 * (size_t)r + a));
      }
      __threadfence();
      p = p == 0 ? -1 : bn.parent[p];
    }
  }
}

// host/bvh_build.h decode_plane: origin + q * 2^(e-127), one rounding.
__device__ __forceinline__ float decode_plane(float origin, uint32_t q, uint32_t e) {
  return __fadd_rn(origin, __fmul_rn((float)q, __uint_as_float(e << 23)));
}
// Largest q with decode(q) <= v (host/bvh_build.cpp quant_lo).
__device__ uint32_t quant_lo(float origin, float v, uint32_t e) {
  double qd = floor(((double)v - (double)origin) / (double)__uint_as_float(e << 23));
  int q = (int)fmin(fmax(qd, 0.0), 255.0);
  while (q > 0 && decode_plane(origin, (uint32_t)q, e) > v) --q;
  while (q < 255 && decode_plane(origin, (uint32_t)(q + 1), e) <= v) ++q;
  return (uint32_t)q;
}
// Smallest q with decode(q) >= v; false when no byte reaches v.
__device__ bool quant_hi(float origin, float v, uint32_t e, uint32_t* out) {
  double qd = ceil(((double)v - (double)origin) / (double)__uint_as_float(e << 23));
  int q = (int)fmin(fmax(qd, 0.0), 255.0);
  while (q < 255 && decode_plane(origin, (uint32_t)q, e) < v) ++q;
  while (q > 0 && decode_plane(origin, (uint32_t)(q - 1), e) >= v) --q;
  if (decode_plane(origin, (uint32_t)q, e) < v) return false;
  *out = (uint32_t)q;
  return true;
}

struct Collapse {
  const int2* in;  // (wide node, binary node) of this level
  const uint32_t* n_in;
  int2* out;
  uint32_t* n_out;
  uint32_t* node_count;
  uint32_t* tri_count;
  uint4* nodes;  // 5 per wide node
  float4* tris;  // 3 per triangle
  const float4* pos;
  const uint4* tri;
  const uint32_t* vals;
  uint32_t* err;
};

__device__ __forceinline__ bool leafish(const Bin& bn, uint32_t n, int32_t b) {
  return (uint32_t)b >= n - 1 || bn.last[b] - bn.first[b] + 1 <= DB_LEAF_MAX;
}
__device__ __forceinline__ float half_area(const Bin& bn, int32_t b) {
  float e0 = bn.hi[3 * (size_t)b] - bn.lo[3 * (size_t)b], e1 = bn.hi[3 * (size_t)b + 1] - bn.lo[3 * (size_t)b + 1],
        e2 = bn.hi[3 * (size_t)b + 2] - bn.lo[3 * (size_t)b + 2];
  return e0 * e1 + e1 * e2 + e2 * e0;
}

// One level of the collapse: each item fills one wide node from the binary
// subtree below it (host/bvh_build.cpp Collapser::fill) and queues its
// interior children for the next level.  Eight lanes per item, a lane per
// child: a level is as slow as one item's chain of loads, and a lone thread
// walked the children's areas, boxes and double-precision quantisation one
// after the other (60 to 120 us a level at any number of items, now 24 to 45;
// 500k triangles have eight levels).  The level's length is read on the
// device, so levels follow each other without a copy to the host.
__global__ void __launch_bounds__(128) k_collapse(Collapse c, Bin bn, uint32_t n) {
  const unsigned full = 0xffffffffu;
  const unsigned lane = threadIdx.x & 31u, me = lane & 7u, g0 = lane & 24u;
  const uint32_t n_in = *c.n_in;
  const uint32_t warps = gridDim.x * (blockDim.x >> 5), warp = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  for (uint32_t base = warp * 4; base < n_in; base += warps * 4) {
    const uint32_t it = base + (lane >> 3);
    const bool on = it < n_in;
    int2 item = on ? c.in[it] : make_int2(0, 0);
    // This lane's child: its binary node, whether it may be opened, and its
    // half area if so (-1 otherwise).
    int32_t kid = -1;
    float area = -1.0f;
    int nk = 0;
    auto take = [&](int32_t b) {
      kid = b;
      // A box that overflows (its piece is refused below) can have no number as
      // its area, which must not enter the lanes' maximum: they would disagree.
      const float a = leafish(bn, n, b) ? -1.0f : half_area(bn, b);
      area = a >= 0.0f ? a : -1.0f;
    };
    if (on) {
      if (leafish(bn, n, item.y)) {
        nk = 1;
        if (me == 0) take(item.y);
      } else {
        nk = 2;
        if (me == 0) take(bn.left[item.y]);
        if (me == 1) take(bn.right[item.y]);
      }
    }
    for (;;) {
      // The first of the largest areas among the children that can be opened.
      float best_a = area;
      unsigned best = me;
#pragma unroll
      for (int i = 1; i < 8; i <<= 1) {
        const float oa = __shfl_xor_sync(full, best_a, i);
        const unsigned ob = __shfl_xor_sync(full, best, i);
        if (oa > best_a || (oa == best_a && ob < best)) {
          best_a = oa;
          best = ob;
        }
      }
      const bool open = on && nk < 8 && best_a > -1.0f;
      if (__ballot_sync(full, open) == 0) break;
      const int32_t opened = __shfl_sync(full, kid, (int)(g0 + best));
      const int32_t up_kid = __shfl_up_sync(full, kid, 1);
      const float up_area = __shfl_up_sync(full, area, 1);
      if (open) {
        if (me == best) {
          take(bn.left[opened]);
        } else if (me == best + 1) {
          take(bn.right[opened]);
        } else if (me > best + 1) {
          kid = up_kid;
          area = up_area;
        }
        ++nk;
      }
    }
    const bool have = on && (int)me < nk;
    float klo[3] = {INFINITY, INFINITY, INFINITY}, khi[3] = {-INFINITY, -INFINITY, -INFINITY};
    uint32_t first = 0, last = 0;
    bool leaf = false;
    if (have) {
      leaf = leafish(bn, n, kid);
      first = bn.first[kid];
      last = bn.last[kid];
      for (int a = 0; a < 3; ++a) {
        klo[a] = bn.lo[3 * (size_t)kid + a];
        khi[a] = bn.hi[3 * (size_t)kid + a];
      }
    }
    float lo[3], hi[3];
    for (int a = 0; a < 3; ++a) {
      lo[a] = klo[a];
      hi[a] = khi[a];
#pragma unroll
      for (int i = 1; i < 8; i <<= 1) {
        lo[a] = fminf(lo[a], __shfl_xor_sync(full, lo[a], i));
        hi[a] = fmaxf(hi[a], __shfl_xor_sync(full, hi[a], i));
      }
    }
    // The axes' exponents: a lane per axis.
    uint32_t ex = 0;
    if (on && me < 3) {
      const float l = me == 0 ? lo[0] : me == 1 ? lo[1] : lo[2], h = me == 0 ? hi[0] : me == 1 ? hi[1] : hi[2];
      float ext = h - l;
      int ee = -120;
      if (ext > 0.0f) {
        int x;
        frexp((double)ext / 255.0, &x);
        ee = x;
      }
      ee = max(ee, -120);
      if (ee > 60) {
        atomicOr(c.err, DB_ERR_EXTENT);
        ee = 60;
      }
      uint32_t qh;
      while (ee <= 60 && !quant_hi(l, h, (uint32_t)(ee + 127), &qh)) ++ee;
      if (ee > 60) {
        atomicOr(c.err, DB_ERR_QUANT);
        ee = 60;
      }
      ex = (uint32_t)(ee + 127);
    }
    uint32_t e[3];
    for (int a = 0; a < 3; ++a) e[a] = __shfl_sync(full, ex, (int)g0 + a);
    // Bases of the item's interior children and triangles.
    const unsigned im = (__ballot_sync(full, have && !leaf) >> g0) & 0xffu;
    const unsigned pm = (__ballot_sync(full, have) >> g0) & 0xffu;
    const uint32_t cnt = have && leaf ? last - first + 1u : 0u;
    uint32_t toff = cnt;  // inclusive sum over the lanes before and this one
#pragma unroll
    for (int i = 1; i < 8; i <<= 1) {
      const uint32_t x = __shfl_up_sync(full, toff, i);
      if ((int)me >= i) toff += x;
    }
    const uint32_t n_tri = __shfl_sync(full, toff, (int)g0 + 7), n_int = (uint32_t)__popc(im);
    toff -= cnt;
    uint32_t child_base = 0, tri_base = 0, out_base = 0;
    if (on && me == 0) {
      if (n_int) {
        child_base = atomicAdd(c.node_count, n_int);
        out_base = atomicAdd(c.n_out, n_int);
      }
      if (n_tri) tri_base = atomicAdd(c.tri_count, n_tri);
    }
    child_base = __shfl_sync(full, child_base, (int)g0);
    tri_base = __shfl_sync(full, tri_base, (int)g0);
    out_base = __shfl_sync(full, out_base, (int)g0);
    // This child's planes: lo x, y, z then hi x, y, z (absent: inside out).
    uint32_t q[6] = {255, 255, 255, 0, 0, 0};
    if (have) {
      for (int a = 0; a < 3; ++a) {
        q[a] = quant_lo(lo[a], klo[a], e[a]);
        q[3 + a] = 255;
        if (!quant_hi(lo[a], khi[a], e[a], &q[3 + a])) atomicOr(c.err, DB_ERR_QUANT);
      }
      if (leaf) {
        for (uint32_t s = first; s <= last; ++s) {
          uint32_t t = c.vals[s];
          uint4 ti = c.tri[t];
          float4 a = c.pos[ti.x], b = c.pos[ti.y], d = c.pos[ti.z];
          size_t o = 3 * (size_t)(tri_base + toff + (s - first));
          c.tris[o] = make_float4(a.x, a.y, a.z, __uint_as_float(t));
          c.tris[o + 1] = make_float4(__fsub_rn(b.x, a.x), __fsub_rn(b.y, a.y), __fsub_rn(b.z, a.z), 0.0f);
          c.tris[o + 2] = make_float4(__fsub_rn(d.x, a.x), __fsub_rn(d.y, a.y), __fsub_rn(d.z, a.z), 0.0f);
        }
      } else {
        const uint32_t slot = (uint32_t)__popc(im & ((1u << me) - 1u));
        c.out[out_base + slot] = make_int2((int)(child_base + slot), kid);
      }
    }
    // Packed words: each lane's byte (and leaf count) into its place.
    const uint32_t sh = 8 * (me & 3);
    uint32_t counts = cnt ? (cnt - 1u) << (4 * me) : 0u;
#pragma unroll
    for (int i = 1; i < 8; i <<= 1) counts |= __shfl_xor_sync(full, counts, i);
    uint32_t pw[6][2];
#pragma unroll
    for (int a = 0; a < 6; ++a) {
      uint32_t x = q[a] << sh;  // halves of the group: lanes 0-3 and 4-7
      x |= __shfl_xor_sync(full, x, 1);
      x |= __shfl_xor_sync(full, x, 2);
      pw[a][0] = __shfl_sync(full, x, (int)g0);
      pw[a][1] = __shfl_sync(full, x, (int)g0 + 4);
    }
    if (on && me < 5) {
      uint4 w;
      if (me == 0)
        w = make_uint4(__float_as_uint(lo[0]), __float_as_uint(lo[1]), __float_as_uint(lo[2]),
                       e[0] | (e[1] << 8) | (e[2] << 16) | (im << 24));
      else if (me == 1)
        w = make_uint4(child_base, tri_base, counts, pm);
      else if (me == 2)
        w = make_uint4(pw[0][0], pw[0][1], pw[1][0], pw[1][1]);
      else if (me == 3)
        w = make_uint4(pw[2][0], pw[2][1], pw[3][0], pw[3][1]);
      else
        w = make_uint4(pw[4][0], pw[4][1], pw[5][0], pw[5][1]);
      c.nodes[5 * (size_t)item.x + me] = w;
    }
  }
}

}  // namespace db

// What the tree builders share: a triangle's box, order-preserving keys, chunks of a
// level's nodes.
#pragma once
#include <cuda_runtime.h>
#include <math_constants.h>

#include "mt_common.h"

namespace mt {
namespace {

constexpr int kSmallTris = 256;   // triangles of a subtree that one warp finishes
constexpr int kSmallWarps = 4;    // such warps per block
constexpr int kChunk = 2048;      // triangles of a large node per block

// order-preserving float <-> int keys for integer min/max
__device__ __forceinline__ int fkey(float f) {
  const int b = __float_as_int(f);
  return b >= 0 ? b : b ^ 0x7FFFFFFF;
}
__device__ __forceinline__ float fval(int k) { return __int_as_float(k >= 0 ? k : k ^ 0x7FFFFFFF); }

// A triangle's box and its id; two 16-byte accesses.
struct Prim {
  float lo[3];
  int id;
  float hi[3];
  int pad;
};
static_assert(sizeof(Prim) == 32, "two float4");
__device__ __forceinline__ float centroid(const Prim& p, int a) { return 0.5f * (p.lo[a] + p.hi[a]); }
__device__ __forceinline__ void load_prim(const Prim* p, Prim& r) {
  const float4 a = reinterpret_cast<const float4*>(p)[0], b = reinterpret_cast<const float4*>(p)[1];
  r.lo[0] = a.x; r.lo[1] = a.y; r.lo[2] = a.z; r.id = __float_as_int(a.w);
  r.hi[0] = b.x; r.hi[1] = b.y; r.hi[2] = b.z; r.pad = 0;
}
__device__ __forceinline__ void store_prim(Prim* p, const Prim& r) {
  reinterpret_cast<float4*>(p)[0] = make_float4(r.lo[0], r.lo[1], r.lo[2], __int_as_float(r.id));
  reinterpret_cast<float4*>(p)[1] = make_float4(r.hi[0], r.hi[1], r.hi[2], 0.f);
}
// The box of face f (CNormalBVH.java:82-100: comparisons, so a coordinate that is not a number is left out).
__device__ __forceinline__ void tri_prim(const float4* __restrict__ pts, const Face& f, int id, Prim& r) {
  const float4 p[3] = {pts[f.vx], pts[f.vy], pts[f.vz]};
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    float lo = CUDART_INF_F, hi = -CUDART_INF_F;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const float v = a == 0 ? p[k].x : a == 1 ? p[k].y : p[k].z;
      if (v < lo) lo = v;
      if (v > hi) hi = v;
    }
    r.lo[a] = lo;
    r.hi[a] = hi;
  }
  r.id = id;
  r.pad = 0;
}
// The node a chunk of the level belongs to: the last one whose first chunk is not
// after it (the list's chunk0 ascend).
template <class N>
__device__ __forceinline__ int node_of_chunk(const N* nodes, int n, int chunk) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (nodes[mid].chunk0 <= chunk) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

}  // namespace
}  // namespace mt

// A surface-area-heuristic tree over the scene's triangles, built on the GPU for
// the 4-wide FP16 nodes (precision 3).
//
// The reference's tree splits every node at the middle of its centroid bound. A
// quantised format may be any tree over the same leaves (its boxes contain the
// triangles' boxes, so a ray reaches the same triangles), and splits that
// minimise area x triangles on each side give shallower work where triangle sizes
// differ: the stadium's ground plane of large triangles around a small sphere
// takes 9.8 node visits per camera ray against 20.0, the 1M soup 39.1 against
// 41.8.
//
// Binned splits (Wald, "On fast Construction of SAH-based Bounding Volume
// Hierarchies", RT 2007), in two phases:
//   nodes of more than 256 triangles, level by level: k_bins counts and bounds
//     the centroid bins of every node (blocks over chunks of one node's triangles,
//     bins in shared memory, one flush per block), k_split picks each node's split
//     and writes its record, k_part moves the triangles to their side;
//   the subtrees of at most 256 triangles, one warp each, down to the leaves with
//     the triangles' boxes in shared memory (k_small): no launches or global
//     passes for the many small levels.
// Records are numbered in preorder (left child r + 1, right child r + k for a left
// child of k triangles), as the reference tree's are, so k_quad_fp16 reads either
// tree.
//
// Any-order partition: a block reserves its place on each side with one atomic, so
// triangles of a node keep no order; only nodes whose centroids coincide, split by
// position, depend on it.
#include <cuda_runtime.h>
#include <math_constants.h>

#include <algorithm>
#include <cstring>

#include "mt_build.cuh"
#include "mt_internal.h"

namespace mt {
namespace {

constexpr int kBins = 16;         // bins per axis of a large node
constexpr int kSmallBins = 10;    // 3 axes x 10 bins: one per lane
constexpr int kPartThreads = 256;

// A node being split: its triangles, its record, its centroid bound.
struct Node {
  int start, end, rec, depth;
  int cmn[3], cmx[3];   // fkey
  int chunk0;           // its first chunk of the level
  int dim, bin;         // the split: centroid bin < bin goes left; dim -1: by position
  int nl;               // triangles going left
  int cur[2];           // places taken on each side (k_part)
  int next[2];          // large children in the next level's list, or -1
};
struct Small {
  int start, count, rec, depth, buf;
};
struct Bin {
  int n, lo[3], hi[3];
};
struct Heads {  // list lengths and flags in device memory
  int nodes[2], chunks[2];
  int smalls, depth;
};

// The bin of centroid c in the bound (mn, mx); any float gives a valid bin.
template <int K>
__device__ __forceinline__ int bin_of(float c, float mn, float mx) {
  const int b = (int)((c - mn) * ((float)K / (mx - mn)));
  return min(max(b, 0), K - 1);
}
__device__ __forceinline__ float half_area(const float* lo, const float* hi) {
  const float x = hi[0] - lo[0], y = hi[1] - lo[1], z = hi[2] - lo[2];
  return x * y + y * z + z * x;
}

__global__ void k_start(Node* nodes, Small* smalls, Heads* h, int n) {
  if (threadIdx.x || blockIdx.x) return;
  Node r{};
  r.end = n;
  for (int a = 0; a < 3; ++a) {
    r.cmn[a] = fkey(CUDART_INF_F);
    r.cmx[a] = fkey(-CUDART_INF_F);
  }
  nodes[0] = r;
  Heads z{};
  if (n > kSmallTris) {
    z.nodes[0] = 1;
    z.chunks[0] = (n + kChunk - 1) / kChunk;
  } else {
    z.smalls = 1;
    smalls[0] = Small{0, n, 0, 0, 0};
  }
  *h = z;
}

// Triangle boxes (the leaf boxes of the reference tree: k_prims of mt_bvh.cu) and the
// root's centroid bound.
__global__ void __launch_bounds__(kPartThreads)
    k_boxes(const float4* __restrict__ tris, const float4* __restrict__ pts, const Face* __restrict__ faces, int n,
            Prim* __restrict__ out, Node* root) {
  const int k = blockIdx.x * kPartThreads + threadIdx.x;
  int mn[3], mx[3];
  for (int a = 0; a < 3; ++a) {
    mn[a] = fkey(CUDART_INF_F);
    mx[a] = fkey(-CUDART_INF_F);
  }
  if (k < n) {
    Prim r;
    tri_prim(pts, faces[__float_as_int(tris[3 * (size_t)k].w)], k, r);
    store_prim(out + k, r);
    for (int a = 0; a < 3; ++a) mn[a] = mx[a] = fkey(centroid(r, a));
  }
  for (int a = 0; a < 3; ++a) {
    mn[a] = __reduce_min_sync(0xffffffffu, mn[a]);
    mx[a] = __reduce_max_sync(0xffffffffu, mx[a]);
  }
  __shared__ int s[kPartThreads / 32][6];
  if ((threadIdx.x & 31) == 0)
    for (int a = 0; a < 3; ++a) {
      s[threadIdx.x >> 5][a] = mn[a];
      s[threadIdx.x >> 5][3 + a] = mx[a];
    }
  __syncthreads();
  if (threadIdx.x < 6) {
    int v = s[0][threadIdx.x];
    for (int w = 1; w < kPartThreads / 32; ++w)
      v = threadIdx.x < 3 ? min(v, s[w][threadIdx.x]) : max(v, s[w][threadIdx.x]);
    if (threadIdx.x < 3) atomicMin(&root->cmn[threadIdx.x], v);
    else atomicMax(&root->cmx[threadIdx.x - 3], v);
  }
}

// Bins of the level's nodes: one block per chunk.
__global__ void __launch_bounds__(kPartThreads)
    k_bins(const Prim* __restrict__ prims, const Node* __restrict__ nodes, const Heads* __restrict__ h, int level,
           Bin* __restrict__ bins) {
  __shared__ Bin sb[3 * kBins];
  __shared__ int s_node;
  if ((int)blockIdx.x >= h->chunks[level & 1]) return;
  if (threadIdx.x == 0) s_node = node_of_chunk(nodes, h->nodes[level & 1], blockIdx.x);
  for (int i = threadIdx.x; i < 3 * kBins; i += kPartThreads) {
    Bin b;
    b.n = 0;
    for (int a = 0; a < 3; ++a) {
      b.lo[a] = fkey(CUDART_INF_F);
      b.hi[a] = fkey(-CUDART_INF_F);
    }
    sb[i] = b;
  }
  __syncthreads();
  const Node& nd = nodes[s_node];
  const int p0 = nd.start + ((int)blockIdx.x - nd.chunk0) * kChunk, p1 = min(nd.end, p0 + kChunk);
  float mn[3], mx[3];
  for (int a = 0; a < 3; ++a) {
    mn[a] = fval(nd.cmn[a]);
    mx[a] = fval(nd.cmx[a]);
  }
  for (int p = p0 + threadIdx.x; p < p1; p += kPartThreads) {
    Prim r;
    load_prim(prims + p, r);
    int lo[3], hi[3];
    for (int a = 0; a < 3; ++a) {
      lo[a] = fkey(r.lo[a]);
      hi[a] = fkey(r.hi[a]);
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      Bin& b = sb[a * kBins + bin_of<kBins>(centroid(r, a), mn[a], mx[a])];
      atomicAdd(&b.n, 1);
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        // most boxes lie inside their bin's: a read is cheaper than a lost atomic
        if (lo[q] < b.lo[q]) atomicMin(&b.lo[q], lo[q]);
        if (hi[q] > b.hi[q]) atomicMax(&b.hi[q], hi[q]);
      }
    }
  }
  __syncthreads();
  Bin* out = bins + (size_t)s_node * 3 * kBins;
  for (int i = threadIdx.x; i < 3 * kBins; i += kPartThreads) {
    const Bin b = sb[i];
    if (b.n == 0) continue;
    atomicAdd(&out[i].n, b.n);
    for (int a = 0; a < 3; ++a) {
      atomicMin(&out[i].lo[a], b.lo[a]);
      atomicMax(&out[i].hi[a], b.hi[a]);
    }
  }
}

__device__ __forceinline__ void empty_bin(Bin& b) {
  b.n = 0;
  for (int a = 0; a < 3; ++a) {
    b.lo[a] = fkey(CUDART_INF_F);
    b.hi[a] = fkey(-CUDART_INF_F);
  }
}
__global__ void k_bins_init(Bin* bins, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) empty_bin(bins[i]);
}

__device__ __forceinline__ void write_record(float4* recs, int rec, const float* llo, const float* lhi,
                                             const float* rlo, const float* rhi, int lref, int rref) {
  float4* R = recs + 4 * (size_t)rec;
  R[0] = make_float4(llo[0], lhi[0], llo[1], lhi[1]);
  R[1] = make_float4(rlo[0], rhi[0], rlo[1], rhi[1]);
  R[2] = make_float4(llo[2], lhi[2], rlo[2], rhi[2]);
  R[3] = make_float4(__int_as_float(lref), __int_as_float(rref), 0.f, 0.f);
}

// Each node's split, its record and its children's places: one thread per axis of a
// node (32 threads, 10 nodes). Leaves the node's bins empty for the next level.
__global__ void __launch_bounds__(32)
    k_split(Node* __restrict__ nodes, Bin* __restrict__ bins, float4* __restrict__ recs, int level,
            Node* __restrict__ next, int next_cap, Small* __restrict__ smalls, int small_cap, Heads* h) {
  const int lane = threadIdx.x, nnodes = h->nodes[level & 1];
  if ((int)blockIdx.x * 10 >= nnodes) return;
  const int a = lane % 3, s = blockIdx.x * 10 + lane / 3;
  const bool on = lane < 30 && s < nnodes;
  float best = CUDART_INF_F;
  int bbin = -1, bnl = 0;
  Bin* B = bins + ((size_t)(on ? s : 0) * 3 + a) * kBins;
  const int total = on ? nodes[s].end - nodes[s].start : 0;
  if (on) {
    // suffix areas, then a prefix sweep
    float ra[kBins];
    float lo[3], hi[3];
    for (int q = 0; q < 3; ++q) {
      lo[q] = CUDART_INF_F;
      hi[q] = -CUDART_INF_F;
    }
#pragma unroll
    for (int b = kBins - 1; b > 0; --b) {
      for (int q = 0; q < 3; ++q) {
        lo[q] = fminf(lo[q], fval(B[b].lo[q]));
        hi[q] = fmaxf(hi[q], fval(B[b].hi[q]));
      }
      ra[b] = half_area(lo, hi);
    }
    for (int q = 0; q < 3; ++q) {
      lo[q] = CUDART_INF_F;
      hi[q] = -CUDART_INF_F;
    }
    int nl = 0;
#pragma unroll
    for (int b = 1; b < kBins; ++b) {
      nl += B[b - 1].n;
      for (int q = 0; q < 3; ++q) {
        lo[q] = fminf(lo[q], fval(B[b - 1].lo[q]));
        hi[q] = fmaxf(hi[q], fval(B[b - 1].hi[q]));
      }
      if (nl == 0 || nl == total) continue;
      const float cost = half_area(lo, hi) * (float)nl + ra[b] * (float)(total - nl);
      if (cost < best) {
        best = cost;
        bbin = b;
        bnl = nl;
      }
    }
  }
  // the node's best axis (the lowest of equals)
  const float b0 = __shfl_sync(0xffffffffu, best, lane - a), b1 = __shfl_sync(0xffffffffu, best, min(31, lane - a + 1)),
              b2 = __shfl_sync(0xffffffffu, best, min(31, lane - a + 2));
  int dim = 0;
  float bc = b0;
  if (b1 < bc) { bc = b1; dim = 1; }
  if (b2 < bc) { bc = b2; dim = 2; }
  bbin = __shfl_sync(0xffffffffu, bbin, min(31, lane - a + dim));
  bnl = __shfl_sync(0xffffffffu, bnl, min(31, lane - a + dim));
  if (!on || a != 0) return;
  Node& nd = nodes[s];
  float llo[3], lhi[3], rlo[3], rhi[3];
  for (int q = 0; q < 3; ++q) {
    llo[q] = rlo[q] = CUDART_INF_F;
    lhi[q] = rhi[q] = -CUDART_INF_F;
  }
  B = bins + ((size_t)s * 3 + dim) * kBins;
  const bool split = bbin > 0;
  for (int b = 0; b < kBins; ++b) {
    const bool left = !split || b < bbin, right = !split || b >= bbin;
    for (int q = 0; q < 3; ++q) {
      const float l = fval(B[b].lo[q]), u = fval(B[b].hi[q]);
      if (left) {
        llo[q] = fminf(llo[q], l);
        lhi[q] = fmaxf(lhi[q], u);
      }
      if (right) {
        rlo[q] = fminf(rlo[q], l);
        rhi[q] = fmaxf(rhi[q], u);
      }
    }
  }
  for (int b = 0; b < 3 * kBins; ++b) empty_bin(bins[(size_t)s * 3 * kBins + b]);
  // no split (coinciding centroids, or areas that are not numbers): half by position,
  // each half in the whole node's box
  nd.dim = split ? dim : -1;
  nd.bin = bbin;
  nd.nl = split ? bnl : total / 2;
  nd.cur[0] = nd.cur[1] = 0;
  const int nl = nd.nl, nr = total - nl;
  const int mid = nd.start + nl;
  const int cs[2] = {nd.start, mid}, cn[2] = {nl, nr}, cr[2] = {nd.rec + 1, nd.rec + nl};
  for (int c = 0; c < 2; ++c) {
    nd.next[c] = -1;
    if (cn[c] > kSmallTris) {
      const int k = atomicAdd(&h->nodes[(level + 1) & 1], 1);
      if (k < next_cap) {
        Node x{};
        x.start = cs[c];
        x.end = cs[c] + cn[c];
        x.rec = cr[c];
        x.depth = nd.depth + 1;
        for (int q = 0; q < 3; ++q) {
          x.cmn[q] = fkey(CUDART_INF_F);
          x.cmx[q] = fkey(-CUDART_INF_F);
        }
        next[k] = x;
        nd.next[c] = k;
      }
    } else if (cn[c] > 1) {
      const int k = atomicAdd(&h->smalls, 1);
      if (k < small_cap) smalls[k] = Small{cs[c], cn[c], cr[c], nd.depth + 1, (level + 1) & 1};
    }
  }
  // a child of one triangle is a leaf: k_part writes its ref
  write_record(recs, nd.rec, llo, lhi, rlo, rhi, nl > 1 ? cr[0] : -1, nr > 1 ? cr[1] : -1);
  atomicMax(&h->depth, nd.depth + 1);
}

// First chunks of the next level's nodes (one block; a level has at most n / kSmallTris nodes).
__global__ void __launch_bounds__(1024) k_chunks(Node* nodes, Heads* h, int level) {
  __shared__ int sh[32];
  __shared__ int carry;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  const int n = h->nodes[level & 1];
  for (int i0 = 0; i0 < n; i0 += 1024) {
    const int i = i0 + threadIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int v = i < n ? (nodes[i].end - nodes[i].start + kChunk - 1) / kChunk : 0;
    int x = v;
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) sh[warp] = x;
    __syncthreads();
    int before = carry;
    for (int w = 0; w < warp; ++w) before += sh[w];
    if (i < n) nodes[i].chunk0 = before + x - v;
    __syncthreads();
    if (threadIdx.x == 1023) carry = before + x;
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    h->chunks[level & 1] = carry;
    h->nodes[(level + 1) & 1] = 0;
  }
}

// Triangles to their side, and the children's centroid bounds: one block per chunk.
__global__ void __launch_bounds__(kPartThreads)
    k_part(const Prim* __restrict__ in, Prim* __restrict__ out, Node* nodes, const Heads* __restrict__ h, int level,
           Node* next, float4* __restrict__ recs) {
  __shared__ int s_node, s_base[2], s_warp[2][kPartThreads / 32], s_c[2][6];
  if ((int)blockIdx.x >= h->chunks[level & 1]) return;
  if (threadIdx.x == 0) s_node = node_of_chunk(nodes, h->nodes[level & 1], blockIdx.x);
  if (threadIdx.x < 12) s_c[threadIdx.x / 6][threadIdx.x % 6] = fkey(threadIdx.x % 6 < 3 ? CUDART_INF_F : -CUDART_INF_F);
  __syncthreads();
  Node& nd = nodes[s_node];
  const int p0 = nd.start + ((int)blockIdx.x - nd.chunk0) * kChunk, p1 = min(nd.end, p0 + kChunk);
  const int dim = nd.dim, mid = nd.start + nd.nl;
  const float mn = dim >= 0 ? fval(nd.cmn[dim]) : 0.f, mx = dim >= 0 ? fval(nd.cmx[dim]) : 0.f;
  constexpr int kPer = kChunk / kPartThreads;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned sides = 0, have = 0;  // bit i: this thread's i-th triangle goes right / exists
  int cnt[2] = {0, 0};
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    const int p = p0 + i * kPartThreads + threadIdx.x;
    if (p >= p1) continue;
    int side;
    if (dim < 0) {
      side = p < mid ? 0 : 1;
    } else {
      const Prim* q = in + p;
      side = bin_of<kBins>(0.5f * (q->lo[dim] + q->hi[dim]), mn, mx) < nd.bin ? 0 : 1;
    }
    have |= 1u << i;
    sides |= (unsigned)side << i;
    ++cnt[side];
  }
  // each thread's first place on either side
  int at[2];
  for (int s = 0; s < 2; ++s) {
    int x = cnt[s];
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) s_warp[s][warp] = x;
    at[s] = x - cnt[s];
  }
  __syncthreads();
  if (threadIdx.x < 2) {
    int t = 0;
    for (int w = 0; w < kPartThreads / 32; ++w) {
      const int v = s_warp[threadIdx.x][w];
      s_warp[threadIdx.x][w] = t;
      t += v;
    }
    s_base[threadIdx.x] = t ? atomicAdd(&nd.cur[threadIdx.x], t) : 0;
  }
  __syncthreads();
  for (int s = 0; s < 2; ++s) at[s] += s_warp[s][warp] + s_base[s] + (s ? mid : nd.start);
  int c[2][6];
  for (int s = 0; s < 2; ++s)
    for (int k = 0; k < 6; ++k) c[s][k] = fkey(k < 3 ? CUDART_INF_F : -CUDART_INF_F);
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    if (!(have >> i & 1u)) continue;
    Prim r;
    load_prim(in + p0 + i * kPartThreads + threadIdx.x, r);
    const int s = sides >> i & 1u;
    const int q = s ? at[1]++ : at[0]++;
    store_prim(out + q, r);
    if ((s ? nd.end - mid : nd.nl) == 1) reinterpret_cast<int*>(recs + 4 * (size_t)nd.rec + 3)[s] = ~r.id;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const int v = fkey(centroid(r, a));
      if (s) {
        c[1][a] = min(c[1][a], v);
        c[1][3 + a] = max(c[1][3 + a], v);
      } else {
        c[0][a] = min(c[0][a], v);
        c[0][3 + a] = max(c[0][3 + a], v);
      }
    }
  }
  for (int s = 0; s < 2; ++s) {
    if (nd.next[s] < 0) continue;  // the same for the whole block
    for (int k = 0; k < 6; ++k) {
      const int v = k < 3 ? __reduce_min_sync(0xffffffffu, c[s][k]) : __reduce_max_sync(0xffffffffu, c[s][k]);
      if (lane == 0) {
        if (k < 3) atomicMin(&s_c[s][k], v);
        else atomicMax(&s_c[s][k], v);
      }
    }
  }
  __syncthreads();
  if (threadIdx.x < 12) {
    const int s = threadIdx.x / 6, k = threadIdx.x % 6;
    if (nd.next[s] >= 0) {
      Node& x = next[nd.next[s]];
      if (k < 3) atomicMin(&x.cmn[k], s_c[s][k]);
      else atomicMax(&x.cmx[k - 3], s_c[s][k]);
    }
  }
}

// One warp per subtree of 2..kSmallTris triangles. Bounded by its serial chain of nodes
// (a node reads its triangles once for the centroid bound, once for the bins, once
// for the partition), so many warps run side by side: 28 bytes of shared memory per
// triangle hold the boxes, the order is a byte per triangle.
struct SmallMem {
  float lo[3][kSmallTris], hi[3][kSmallTris];
  int slot[kSmallTris];
  unsigned char ord[kSmallTris], tmp[kSmallTris];
  int stack[10][4];
};
__global__ void __launch_bounds__(32 * kSmallWarps)
    k_small(const Prim* __restrict__ buf0, const Prim* __restrict__ buf1, const Small* __restrict__ smalls, int cap,
            float4* __restrict__ recs, Heads* h) {
  __shared__ SmallMem mem[kSmallWarps];
  const int lane = threadIdx.x & 31;
  SmallMem& M = mem[threadIdx.x >> 5];
  const int k = blockIdx.x * kSmallWarps + (threadIdx.x >> 5);
  if (k >= min(h->smalls, cap)) return;
  const Small sm = smalls[k];
  const Prim* src = (sm.buf ? buf1 : buf0) + sm.start;
  for (int i = lane; i < sm.count; i += 32) {
    Prim r;
    load_prim(src + i, r);
    for (int a = 0; a < 3; ++a) {
      M.lo[a][i] = r.lo[a];
      M.hi[a][i] = r.hi[a];
    }
    M.slot[i] = r.id;
    M.ord[i] = (unsigned char)i;
  }
  __syncwarp();
  const int axis = min(lane / kSmallBins, 2), mybin = lane % kSmallBins;
  const bool binning = lane < 3 * kSmallBins;
  int start = 0, count = sm.count, rec = sm.rec, depth = sm.depth, sp = 0, deepest = sm.depth;
  for (;;) {
    // the centroid bound
    float mn[3], mx[3];
    for (int a = 0; a < 3; ++a) {
      mn[a] = CUDART_INF_F;
      mx[a] = -CUDART_INF_F;
    }
    for (int i = lane; i < count; i += 32) {
      const int o = M.ord[start + i];
      for (int a = 0; a < 3; ++a) {
        const float c = 0.5f * (M.lo[a][o] + M.hi[a][o]);
        mn[a] = fminf(mn[a], c);
        mx[a] = fmaxf(mx[a], c);
      }
    }
    for (int a = 0; a < 3; ++a) {
      mn[a] = fval(__reduce_min_sync(0xffffffffu, fkey(mn[a])));
      mx[a] = fval(__reduce_max_sync(0xffffffffu, fkey(mx[a])));
    }
    const float amn = axis == 0 ? mn[0] : axis == 1 ? mn[1] : mn[2];
    const float amx = axis == 0 ? mx[0] : axis == 1 ? mx[1] : mx[2];
    // my axis and bin: its triangles' count and box
    float lo[3], hi[3];
    int n = 0;
    for (int q = 0; q < 3; ++q) {
      lo[q] = CUDART_INF_F;
      hi[q] = -CUDART_INF_F;
    }
    for (int i = 0; i < count; ++i) {
      const int o = M.ord[start + i];
      const float bl[3] = {M.lo[0][o], M.lo[1][o], M.lo[2][o]}, bh[3] = {M.hi[0][o], M.hi[1][o], M.hi[2][o]};
      const float c = 0.5f * (axis == 0 ? bl[0] + bh[0] : axis == 1 ? bl[1] + bh[1] : bl[2] + bh[2]);
      if (bin_of<kSmallBins>(c, amn, amx) == mybin) {
        ++n;
        for (int q = 0; q < 3; ++q) {
          lo[q] = fminf(lo[q], bl[q]);
          hi[q] = fmaxf(hi[q], bh[q]);
        }
      }
    }
    // inclusive prefixes and suffixes over the axis's bins
    float pl[3], ph[3], sl[3], su[3];
    int pn = n;
    for (int q = 0; q < 3; ++q) {
      pl[q] = sl[q] = lo[q];
      ph[q] = su[q] = hi[q];
    }
#pragma unroll
    for (int o = 1; o < kSmallBins; o <<= 1) {
      const int yn = __shfl_up_sync(0xffffffffu, pn, o);
      if (mybin >= o) pn += yn;
      for (int q = 0; q < 3; ++q) {
        const float a = __shfl_up_sync(0xffffffffu, pl[q], o), b = __shfl_up_sync(0xffffffffu, ph[q], o);
        const float c = __shfl_down_sync(0xffffffffu, sl[q], o), d = __shfl_down_sync(0xffffffffu, su[q], o);
        if (mybin >= o) {
          pl[q] = fminf(pl[q], a);
          ph[q] = fmaxf(ph[q], b);
        }
        if (mybin + o < kSmallBins) {
          sl[q] = fminf(sl[q], c);
          su[q] = fmaxf(su[q], d);
        }
      }
    }
    // the split after my bin
    float rl[3], rh[3];
    for (int q = 0; q < 3; ++q) {
      rl[q] = __shfl_down_sync(0xffffffffu, sl[q], 1);
      rh[q] = __shfl_down_sync(0xffffffffu, su[q], 1);
    }
    float cost = CUDART_INF_F;
    if (binning && mybin < kSmallBins - 1 && pn > 0 && pn < count) {
      cost = half_area(pl, ph) * (float)pn + half_area(rl, rh) * (float)(count - pn);
      if (!(cost < CUDART_INF_F)) cost = CUDART_INF_F;
    }
    // the lane of the least cost (areas are not negative, so their bits order as they do)
    const unsigned key = __reduce_min_sync(0xffffffffu, __float_as_uint(cost));
    const unsigned who = __ballot_sync(0xffffffffu, __float_as_uint(cost) == key);
    const bool split = __uint_as_float(key) < CUDART_INF_F;
    const int w = __ffs(who) - 1;
    int nl = count / 2, dim = -1, at = 0;
    if (split) {
      nl = __shfl_sync(0xffffffffu, pn, w);
      dim = w / kSmallBins;
      at = w % kSmallBins;
      // stable partition by bin
      const float smn = dim == 0 ? mn[0] : dim == 1 ? mn[1] : mn[2], smx = dim == 0 ? mx[0] : dim == 1 ? mx[1] : mx[2];
      int l = 0, r = 0;
      for (int i0 = 0; i0 < count; i0 += 32) {
        const int i = i0 + lane;
        int o = 0;
        bool left = false;
        if (i < count) {
          o = M.ord[start + i];
          left = bin_of<kSmallBins>(0.5f * (M.lo[dim][o] + M.hi[dim][o]), smn, smx) <= at;
        }
        const unsigned lm = __ballot_sync(0xffffffffu, i < count && left), rm = __ballot_sync(0xffffffffu, i < count && !left);
        const unsigned lt = (1u << lane) - 1u;
        if (i < count) M.tmp[left ? l + __popc(lm & lt) : nl + r + __popc(rm & lt)] = (unsigned char)o;
        l += __popc(lm);
        r += __popc(rm);
      }
      __syncwarp();
      for (int i = lane; i < count; i += 32) M.ord[start + i] = M.tmp[i];
      __syncwarp();
      for (int q = 0; q < 3; ++q) {
        pl[q] = __shfl_sync(0xffffffffu, pl[q], w);
        ph[q] = __shfl_sync(0xffffffffu, ph[q], w);
        rl[q] = __shfl_sync(0xffffffffu, rl[q], w);
        rh[q] = __shfl_sync(0xffffffffu, rh[q], w);
      }
    } else {
      // half by position, each half in the whole node's box (lane 0's suffix from bin 0)
      for (int q = 0; q < 3; ++q) {
        pl[q] = rl[q] = __shfl_sync(0xffffffffu, sl[q], 0);
        ph[q] = rh[q] = __shfl_sync(0xffffffffu, su[q], 0);
      }
    }
    const int nr = count - nl;
    const int lref = nl > 1 ? rec + 1 : ~M.slot[M.ord[start]];
    const int rref = nr > 1 ? rec + nl : ~M.slot[M.ord[start + nl]];
    if (lane == 0) write_record(recs, rec, pl, ph, rl, rh, lref, rref);
    ++depth;
    deepest = max(deepest, depth);
    // the larger child waits, the smaller goes on: at most 8 wait
    const bool lgo = nl > 1, rgo = nr > 1;
    if (lgo && rgo) {
      const bool first = nl <= nr;
      if (lane == 0) {
        M.stack[sp][0] = first ? start + nl : start;
        M.stack[sp][1] = first ? nr : nl;
        M.stack[sp][2] = first ? rec + nl : rec + 1;
        M.stack[sp][3] = depth;
      }
      ++sp;
      const int r0 = rec;
      rec = first ? r0 + 1 : r0 + nl;
      start = first ? start : start + nl;
      count = first ? nl : nr;
    } else if (lgo) {
      ++rec;
      count = nl;
    } else if (rgo) {
      rec += nl;
      start += nl;
      count = nr;
    } else if (sp > 0) {
      --sp;
      __syncwarp();
      start = M.stack[sp][0];
      count = M.stack[sp][1];
      rec = M.stack[sp][2];
      depth = M.stack[sp][3];
    } else {
      break;
    }
    __syncwarp();
  }
  if (lane == 0) atomicMax(&h->depth, deepest);
}

}  // namespace
}  // namespace mt

using namespace mt;

int build_sah_records(mt_scene* s, Workspace& ws, float4** recs_out) {
  *recs_out = nullptr;
  const int n = s->ntri;
  cudaStream_t st = s->ctx->stream;
  const int node_cap = n / kSmallTris + 2, small_cap = n / 2 + 1;
  // records, the triangles twice, the node lists, the small subtrees, the bins, the heads
  auto align = Workspace::round;
  const size_t b_prim = align(sizeof(Prim) * (size_t)n), b_node = align(sizeof(Node) * (size_t)node_cap),
               b_small = align(sizeof(Small) * (size_t)small_cap),
               b_bins = align(sizeof(Bin) * 3 * kBins * (size_t)node_cap), b_head = align(sizeof(Heads));
  int r = ws.get(s->ctx, align(64 * (size_t)(n - 1)) + 2 * b_prim + 2 * b_node + b_small + b_bins + b_head);
  if (r) return r;
  float4* recs = (float4*)ws.take<char>(64 * (size_t)(n - 1));
  char* slab = ws.take<char>(2 * b_prim + 2 * b_node + b_small + b_bins + b_head);
  Prim* prim[2] = {(Prim*)slab, (Prim*)(slab + b_prim)};
  Node* nodes[2] = {(Node*)(slab + 2 * b_prim), (Node*)(slab + 2 * b_prim + b_node)};
  Small* smalls = (Small*)(slab + 2 * b_prim + 2 * b_node);
  Bin* bins = (Bin*)(slab + 2 * b_prim + 2 * b_node + b_small);
  Heads* heads = (Heads*)(slab + 2 * b_prim + 2 * b_node + b_small + b_bins);
  auto blocks = [](size_t m, int t) { return (unsigned)((m + t - 1) / t); };
  k_start<<<1, 1, 0, st>>>(nodes[0], smalls, heads, n);
  k_boxes<<<blocks(n, kPartThreads), kPartThreads, 0, st>>>(s->d_tris, s->d_points, s->d_faces, n, prim[0], nodes[0]);
  // the levels, as in mt_bvh_build_device: without waiting for the host at each
  const int chunk_cap = n / kChunk + node_cap;
  k_bins_init<<<blocks((size_t)node_cap * 3 * kBins, 256), 256, 0, st>>>(bins, node_cap * 3 * kBins);
  Heads hh{};
  int level = 0, until = 0;
  for (int m = n; m > kSmallTris; m = (m + 1) / 2) ++until;
  for (until += 4; n > kSmallTris; until = level + 4) {
    for (; level < until; ++level) {
      const int c = level & 1;
      k_bins<<<chunk_cap, kPartThreads, 0, st>>>(prim[c], nodes[c], heads, level, bins);
      k_split<<<blocks(node_cap, 10), 32, 0, st>>>(nodes[c], bins, recs, level, nodes[c ^ 1], node_cap, smalls,
                                                  small_cap, heads);
      k_part<<<chunk_cap, kPartThreads, 0, st>>>(prim[c], prim[c ^ 1], nodes[c], heads, level, nodes[c ^ 1], recs);
      k_chunks<<<1, 1024, 0, st>>>(nodes[c ^ 1], heads, level + 1);
    }
    if (cudaMemcpyAsync(&hh, heads, sizeof(hh), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess)
      return fail(MT_ERR_CUDA, "surface-area tree: %s", cudaGetErrorString(cudaGetLastError()));
    if (hh.nodes[level & 1] == 0) break;
    if (level > kStackDepth) return MT_OK;  // too deep: the caller keeps the reference tree
  }
  const int nsmall = n > kSmallTris ? std::min(hh.smalls, small_cap) : 1;
  if (nsmall > 0)
    k_small<<<blocks(nsmall, kSmallWarps), 32 * kSmallWarps, 0, st>>>(prim[0], prim[1], smalls, small_cap, recs, heads);
  if (cudaMemcpyAsync(&hh, heads, sizeof(hh), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
      cudaStreamSynchronize(st) != cudaSuccess)
    return fail(MT_ERR_CUDA, "surface-area tree: %s", cudaGetErrorString(cudaGetLastError()));
  if (hh.depth > kStackDepth) return MT_OK;
  *recs_out = recs;
  return MT_OK;
}

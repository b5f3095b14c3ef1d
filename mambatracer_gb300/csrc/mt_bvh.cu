// The reference's BVH built on the GPU.
//
// CNormalBVH.build (src/cl/scene/CNormalBVH.java:45-148) splits a node's
// triangles at the centre of their centroid bound's longest axis (stable
// partition "centroid < split", the middle index when one side would be empty),
// one triangle per leaf, children allocated as adjacent pairs in the order the
// recursion subdivides. The host restatement (mt_bvh_build_host) runs it
// recursively; here it runs level by level over all nodes of a level at once:
//
//   k_count     triangles left of the split, per chunk of a node's triangles
//   k_plan      the counts scanned, per node its split, its records and its
//               children's places
//   k_scatter   a stable partition, and the children's bounds and centroid bounds
//               (exact min/max of order-preserving integer keys)
//
// for nodes of more than 256 triangles; the subtrees below are finished by one
// warp each (k_small), so the many small levels cost no launches and no passes over
// all triangles. The large levels run without the host waiting for each, over
// chunks of 2048 triangles of one node, so a block works for one node and flushes
// its bounds once (a warp at a time, the root's 12 atomics of every warp met at the
// same addresses: 50 us a level). 1M triangles 6.7 -> 1.6 ms, 3.3M 23.5 -> 5.1 ms, 20k
// 1.8 -> 0.52 ms against all levels in the large form, with the host reading each
// level's size.
//
// A node subdivided when the allocation counter reads P gets children P and
// P + 1; its left subtree (k triangles) then allocates 2(k - 1) nodes, so its
// right child is subdivided at P + 2k and its left child at P + 2: every
// node's index follows from its parent's counter and its left sibling's size.
// The result equals the host build element for element (the test compares the
// reference-layout arrays). The traversal layout is written in the same pass:
// interior records in depth-first preorder (an interior node with record R and
// a left child of k triangles has its left child at R + 1 and its right child
// at R + k, since the left subtree holds k - 1 interior nodes), leaf slots = the
// triangles' final positions (the depth-first leaf order), each record holding
// its two children's boxes.
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <math_constants.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "mt_build.cuh"
#include "mt_internal.h"

namespace mt {
namespace {

constexpr int kT = 256;

// A node of more than kSmallTris triangles, being split: its triangles, numbering
// (see the file header), bound and centroid bound.
struct Big {
  int start, end, node, P, parent, depth, rec, prec, side;  // prec: the parent's record, side 0 left 1 right
  int box[12];  // fkey: minimum, maximum, centroid minimum, centroid maximum
  int chunk0;   // its first chunk of the level
  int dim, nl, mid;
  float split;
  int next[2];  // its children: index into the next level's list, or ~index into the small ones
};
struct Small {
  int start, count, node, P, parent, depth, rec, prec, side;
  int box[12];
};
struct Heads {
  int nodes[2], chunks[2];
  int smalls, depth;
};
// Optional reference-layout arrays (7 ints and 8 floats per node).
struct RefOut {
  int* nodes;
  float* bounds;
};

__device__ __forceinline__ void init_box(int* box) {
#pragma unroll
  for (int k = 0; k < 12; ++k) box[k] = fkey((k / 3) % 2 == 0 ? CUDART_INF_F : -CUDART_INF_F);
}
// one triangle's keys in Big::box order
__device__ __forceinline__ void tri_box(const Prim& r, int* v) {
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    v[a] = fkey(r.lo[a]);
    v[3 + a] = fkey(r.hi[a]);
    v[6 + a] = v[9 + a] = fkey(centroid(r, a));
  }
}
__device__ __forceinline__ int merge_key(int k, int a, int b) { return (k / 3) % 2 == 0 ? min(a, b) : max(a, b); }
__device__ __forceinline__ int warp_key(int k, int v) {
  return (k / 3) % 2 == 0 ? __reduce_min_sync(0xffffffffu, v) : __reduce_max_sync(0xffffffffu, v);
}
__device__ __forceinline__ void atomic_key(int k, int* p, int v) {
  if ((k / 3) % 2 == 0) atomicMin(p, v);
  else atomicMax(p, v);
}
// The split of CNormalBVH.build from the centroid bound's keys: the longest axis, its middle.
__device__ __forceinline__ void split_of(const int* box, int* dim, float* split) {
  const float ex = fval(box[9]) - fval(box[6]), ey = fval(box[10]) - fval(box[7]), ez = fval(box[11]) - fval(box[8]);
  *dim = (ex > ey && ex > ez) ? 0 : (ey > ez ? 1 : 2);
  const int d = *dim;
  *split = 0.5f * ((d == 0 ? fval(box[6]) : d == 1 ? fval(box[7]) : fval(box[8])) +
                   (d == 0 ? fval(box[9]) : d == 1 ? fval(box[10]) : fval(box[11])));
}

// A node's box and ref into its parent's record, and its reference-layout entries.
// ref: its record, or ~slot of a leaf's triangle `face`.
__device__ __forceinline__ void link_node(float4* recs, RefOut out, const int* box, int node, int P, int parent, int rec,
                                          int prec, int side, bool leaf, int slot, int face) {
  const float x0 = fval(box[0]), y0 = fval(box[1]), z0 = fval(box[2]);
  const float x1 = fval(box[3]), y1 = fval(box[4]), z1 = fval(box[5]);
  if (prec >= 0) {
    float4* R = recs + 4 * (size_t)prec;
    R[side] = make_float4(x0, x1, y0, y1);
    reinterpret_cast<float2*>(R + 2)[side] = make_float2(z0, z1);
    reinterpret_cast<int*>(R + 3)[side] = leaf ? ~slot : rec;
    reinterpret_cast<int*>(R + 3)[2 + side] = 0;
  }
  if (out.nodes) {
    int* nd = out.nodes + 7 * (size_t)node;
    nd[0] = node;                                                // bound
    nd[1] = prec < 0 ? 0 : side == 0 ? node + 1 : node - 1;      // sibling
    nd[2] = leaf ? 0 : P;                                        // left
    nd[3] = leaf ? 0 : P + 1;                                    // right
    nd[4] = parent;
    nd[5] = leaf ? 1 : 0;                                        // isLeaf
    nd[6] = leaf ? face : 0;                                     // child
  }
  if (out.bounds) {
    float4* bd = reinterpret_cast<float4*>(out.bounds) + 2 * (size_t)node;
    bd[0] = make_float4(x0, y0, z0, 0.f);
    bd[1] = make_float4(x1, y1, z1, 0.f);
  }
}

__global__ void k_start(Big* nodes, Small* smalls, Heads* h, int n) {
  if (threadIdx.x || blockIdx.x) return;
  Heads z{};
  if (n > kSmallTris) {
    Big r{};
    r.end = n;
    r.P = 1;
    r.prec = -1;
    init_box(r.box);
    nodes[0] = r;
    z.nodes[0] = 1;
    z.chunks[0] = (n + kChunk - 1) / kChunk;
  } else {
    Small r{};
    r.count = n;
    r.P = 1;
    r.prec = -1;
    init_box(r.box);
    smalls[0] = r;
    z.smalls = 1;
  }
  *h = z;
}

// Triangle boxes, and the root's bounds into root_box.
__global__ void __launch_bounds__(kT) k_prims(const float4* __restrict__ pts, const Face* __restrict__ faces, int n,
                                              Prim* __restrict__ out, int* root_box) {
  __shared__ int s_box[12];
  if (threadIdx.x < 12) s_box[threadIdx.x] = fkey((threadIdx.x / 3) % 2 == 0 ? CUDART_INF_F : -CUDART_INF_F);
  __syncthreads();
  const int t = blockIdx.x * kT + threadIdx.x;
  int v[12];
  init_box(v);
  if (t < n) {
    Prim r;
    tri_prim(pts, faces[t], t, r);
    store_prim(out + t, r);
    tri_box(r, v);
  }
#pragma unroll
  for (int k = 0; k < 12; ++k) {
    const int w = warp_key(k, v[k]);
    if ((threadIdx.x & 31) == 0) atomic_key(k, &s_box[k], w);
  }
  __syncthreads();
  if (threadIdx.x < 12) atomic_key(threadIdx.x, root_box + threadIdx.x, s_box[threadIdx.x]);
}

// Triangles of each chunk left of their node's split.
__global__ void __launch_bounds__(kT)
    k_count(const Prim* __restrict__ prims, const Big* __restrict__ nodes, const Heads* __restrict__ h, int level,
            int* __restrict__ cnt) {
  __shared__ int s_node, s_warp[kT / 32];
  if ((int)blockIdx.x >= h->chunks[level & 1]) return;
  if (threadIdx.x == 0) s_node = node_of_chunk(nodes, h->nodes[level & 1], blockIdx.x);
  __syncthreads();
  const Big& nd = nodes[s_node];
  int dim;
  float split;
  split_of(nd.box, &dim, &split);
  const int p0 = nd.start + ((int)blockIdx.x - nd.chunk0) * kChunk, p1 = min(nd.end, p0 + kChunk);
  int c = 0;
#pragma unroll
  for (int i = 0; i < kChunk / kT; ++i) {
    const int p = p0 + i * kT + threadIdx.x;
    if (p < p1) c += 0.5f * (prims[p].lo[dim] + prims[p].hi[dim]) < split;
  }
  c = __reduce_add_sync(0xffffffffu, c);
  if ((threadIdx.x & 31) == 0) s_warp[threadIdx.x >> 5] = c;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < kT / 32; ++w) c += s_warp[w];
    cnt[blockIdx.x] = c;
  }
}

// One block: the chunk counts scanned (cnt[i] becomes the triangles left of the
// splits before chunk i, cnt[chunks] the total), every node's split, its link and
// its children in the next lists, and the next level's chunks.
__global__ void __launch_bounds__(1024)
    k_plan(Big* __restrict__ nodes, Big* __restrict__ next, Small* __restrict__ smalls, Heads* h, int level,
           int* __restrict__ cnt, float4* __restrict__ recs, RefOut out) {
  __shared__ int sh[32], s_carry, s_next;
  const int nn = h->nodes[level & 1], nc = h->chunks[level & 1];
  if (nn == 0) {  // the levels ended earlier
    if (threadIdx.x == 0) h->nodes[(level + 1) & 1] = h->chunks[(level + 1) & 1] = 0;
    return;
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) s_carry = s_next = 0;
  __syncthreads();
  // exclusive prefix of v over the block after what s_carry holds; s_carry advances
  auto scan = [&](int v) {
    int x = v;
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) sh[warp] = x;
    __syncthreads();
    int before = s_carry;
    for (int w = 0; w < warp; ++w) before += sh[w];
    __syncthreads();
    if (threadIdx.x == 1023) s_carry = before + x;
    __syncthreads();
    return before + x - v;
  };
  for (int i0 = 0; i0 < nc; i0 += 1024) {
    const int i = i0 + threadIdx.x;
    const int e = scan(i < nc ? cnt[i] : 0);
    if (i < nc) cnt[i] = e;
  }
  if (threadIdx.x == 0) cnt[nc] = s_carry;
  __syncthreads();
  for (int i = threadIdx.x; i < nn; i += 1024) {
    Big& nd = nodes[i];
    const int size = nd.end - nd.start;
    const int nl = cnt[nd.chunk0 + (size + kChunk - 1) / kChunk] - cnt[nd.chunk0];
    split_of(nd.box, &nd.dim, &nd.split);
    const bool kept = nl != 0 && nl != size;  // else the middle index splits, in the old order
    if (!kept) nd.dim = -1;
    nd.nl = nl;
    nd.mid = kept ? nd.start + nl : nd.start + size / 2;
    link_node(recs, out, nd.box, nd.node, nd.P, nd.parent, nd.rec, nd.prec, nd.side, false, 0, 0);
    for (int s = 0; s < 2; ++s) {
      const int cs = s ? nd.mid : nd.start, cn = s ? nd.end - nd.mid : nd.mid - nd.start;
      const int cnode = nd.P + s, cP = s ? nd.P + 2 * (nd.mid - nd.start) : nd.P + 2;
      const int crec = s ? nd.rec + (nd.mid - nd.start) : nd.rec + 1;
      if (cn > kSmallTris) {
        const int k = atomicAdd(&s_next, 1);
        Big c{};
        c.start = cs;
        c.end = cs + cn;
        c.node = cnode;
        c.P = cP;
        c.parent = nd.node;
        c.depth = nd.depth + 1;
        c.rec = crec;
        c.prec = nd.rec;
        c.side = s;
        init_box(c.box);
        next[k] = c;
        nd.next[s] = k;
      } else {
        const int k = atomicAdd(&h->smalls, 1);
        Small c{};
        c.start = cs;
        c.count = cn;
        c.node = cnode;
        c.P = cP;
        c.parent = nd.node;
        // the level's triangles move to the other buffer: bit 30 tells which
        c.depth = (nd.depth + 1) | (((level + 1) & 1) << 30);
        c.rec = crec;
        c.prec = nd.rec;
        c.side = s;
        init_box(c.box);
        smalls[k] = c;
        nd.next[s] = ~k;
      }
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) s_carry = 0;
  __syncthreads();
  const int m = s_next;
  for (int i0 = 0; i0 < m; i0 += 1024) {
    const int i = i0 + threadIdx.x;
    const int e = scan(i < m ? (next[i].end - next[i].start + kChunk - 1) / kChunk : 0);
    if (i < m) next[i].chunk0 = e;
  }
  if (threadIdx.x == 0) {
    h->nodes[(level + 1) & 1] = m;
    h->chunks[(level + 1) & 1] = s_carry;
  }
}

// Triangles to their child's range, each side in its old order, and the children's
// bounds: one block per chunk.
__global__ void __launch_bounds__(kT)
    k_scatter(const Prim* __restrict__ in, Prim* __restrict__ outp, const Big* __restrict__ nodes, Big* next,
              Small* smalls, const Heads* __restrict__ h, int level, const int* __restrict__ cnt) {
  __shared__ int s_node, s_warp[kT / 32], s_box[2][12];
  // k_plan has set the next level's counts only: this level's stay
  if ((int)blockIdx.x >= h->chunks[level & 1]) return;
  if (threadIdx.x == 0) s_node = node_of_chunk(nodes, h->nodes[level & 1], blockIdx.x);
  if (threadIdx.x < 24) s_box[threadIdx.x / 12][threadIdx.x % 12] = fkey((threadIdx.x % 12 / 3) % 2 == 0 ? CUDART_INF_F : -CUDART_INF_F);
  __syncthreads();
  const Big& nd = nodes[s_node];
  const int p0 = nd.start + ((int)blockIdx.x - nd.chunk0) * kChunk, p1 = min(nd.end, p0 + kChunk);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int dim = nd.dim, mid = nd.mid;
  int left = cnt[blockIdx.x] - cnt[nd.chunk0];  // triangles left of the split before this chunk
  int v[2][12];
  init_box(v[0]);
  init_box(v[1]);
  for (int i = 0; i < kChunk / kT; ++i) {
    const int p = p0 + i * kT + threadIdx.x;
    const bool on = p < p1;
    Prim r;
    bool l = false;
    if (on) {
      load_prim(in + p, r);
      const float c = dim == 0 ? centroid(r, 0) : dim == 1 ? centroid(r, 1) : centroid(r, 2);
      l = dim < 0 ? p < mid : c < nd.split;
    }
    const unsigned lm = __ballot_sync(0xffffffffu, l);
    if (lane == 0) s_warp[warp] = __popc(lm);
    __syncthreads();
    int before = left, all = 0;
    for (int w = 0; w < kT / 32; ++w) {
      const int c = s_warp[w];
      if (w < warp) before += c;
      all += c;
    }
    __syncthreads();
    if (on) {
      const int lrank = before + __popc(lm & ((1u << lane) - 1u));
      const int q = dim < 0 ? p : l ? nd.start + lrank : mid + ((p - nd.start) - lrank);
      store_prim(outp + q, r);
      int t[12];
      tri_box(r, t);
      if (l) {
#pragma unroll
        for (int k = 0; k < 12; ++k) v[0][k] = merge_key(k, v[0][k], t[k]);
      } else {
#pragma unroll
        for (int k = 0; k < 12; ++k) v[1][k] = merge_key(k, v[1][k], t[k]);
      }
    }
    left += all;
  }
#pragma unroll
  for (int s = 0; s < 2; ++s)
#pragma unroll
    for (int k = 0; k < 12; ++k) {
      const int w = warp_key(k, v[s][k]);
      if (lane == 0) atomic_key(k, &s_box[s][k], w);
    }
  __syncthreads();
  if (threadIdx.x < 24) {
    const int s = threadIdx.x / 12, k = threadIdx.x % 12, c = nd.next[s];
    atomic_key(k, c >= 0 ? &next[c].box[k] : &smalls[~c].box[k], s_box[s][k]);
  }
}

// The subtrees of at most kSmallTris triangles, one warp each, down to the leaves,
// their triangles' keys in shared memory: a node partitions its triangles in order
// and finds both children's bounds in the same pass. At the end the triangles'
// slots are written in leaf order. Bounded by the chain of a subtree's nodes (a
// few hundred instructions each), so many warps run side by side.
struct SmallMem {
  int key[6][kSmallTris];  // fkey of lo, hi
  int face[kSmallTris];
  unsigned char ord[kSmallTris], tmp[kSmallTris];
  int stack[10][12];
};
__global__ void __launch_bounds__(32 * kSmallWarps)
    k_small(const Prim* __restrict__ buf0, const Prim* __restrict__ buf1, const Small* __restrict__ smalls, Heads* h,
            float4* __restrict__ recs, RefOut out, const float4* __restrict__ pts, const Face* __restrict__ faces,
            float4* __restrict__ tris) {
  __shared__ SmallMem mem[kSmallWarps];
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  SmallMem& M = mem[threadIdx.x >> 5];
  const int w = blockIdx.x * kSmallWarps + (threadIdx.x >> 5);
  if (w >= h->smalls) return;
  const Small sm = smalls[w];
  const int base = sm.start, total = sm.count;
  const Prim* src = (sm.depth >> 30 & 1 ? buf1 : buf0) + base;
  for (int i = lane; i < total; i += 32) {
    Prim r;
    load_prim(src + i, r);
    for (int a = 0; a < 3; ++a) {
      M.key[a][i] = fkey(r.lo[a]);
      M.key[3 + a][i] = fkey(r.hi[a]);
    }
    M.face[i] = r.id;
    M.ord[i] = (unsigned char)i;
  }
  __syncwarp();
  int depth = sm.depth & 0x3FFFFFFF, deepest = depth, sp = 0;
  if (lane == 0)
    link_node(recs, out, sm.box, sm.node, sm.P, sm.parent, sm.rec, sm.prec, sm.side, total < 2, base, M.face[0]);
  int start = 0, count = total, node = sm.node, P = sm.P, rec = sm.rec;
  int cb[6];
  for (int k = 0; k < 6; ++k) cb[k] = sm.box[6 + k];
  while (count > 1) {
    int full[12], dim;
    float split;
    for (int k = 0; k < 6; ++k) full[6 + k] = cb[k];
    split_of(full, &dim, &split);
    auto left_of = [&](int o) { return 0.5f * (fval(M.key[dim][o]) + fval(M.key[3 + dim][o])) < split; };
    int nl = 0;
    for (int i0 = 0; i0 < count; i0 += 32)
      nl += __popc(__ballot_sync(0xffffffffu, i0 + lane < count && left_of(M.ord[start + min(i0 + lane, count - 1)])));
    const bool kept = nl != 0 && nl != count;
    const int half = kept ? nl : count / 2;
    int v[2][12], l0 = 0, r0 = 0;
    init_box(v[0]);
    init_box(v[1]);
    for (int i0 = 0; i0 < count; i0 += 32) {
      const int i = i0 + lane;
      const bool on = i < count;
      const int o = M.ord[start + min(i, count - 1)];
      const bool l = on && (kept ? left_of(o) : i < half);
      const unsigned lm = __ballot_sync(0xffffffffu, l), rm = __ballot_sync(0xffffffffu, on && !l);
      if (on) {
        M.tmp[l ? l0 + __popc(lm & lt) : half + r0 + __popc(rm & lt)] = (unsigned char)o;
        int t[12];
#pragma unroll
        for (int k = 0; k < 6; ++k) t[k] = M.key[k][o];
#pragma unroll
        for (int a = 0; a < 3; ++a) t[6 + a] = t[9 + a] = fkey(0.5f * (fval(t[a]) + fval(t[3 + a])));
        if (l) {
#pragma unroll
          for (int k = 0; k < 12; ++k) v[0][k] = merge_key(k, v[0][k], t[k]);
        } else {
#pragma unroll
          for (int k = 0; k < 12; ++k) v[1][k] = merge_key(k, v[1][k], t[k]);
        }
      }
      l0 += __popc(lm);
      r0 += __popc(rm);
    }
#pragma unroll
    for (int s = 0; s < 2; ++s)
#pragma unroll
      for (int k = 0; k < 12; ++k) v[s][k] = warp_key(k, v[s][k]);
    __syncwarp();
    for (int i = lane; i < count; i += 32) M.ord[start + i] = M.tmp[i];
    __syncwarp();
    const int nr = count - half;
    ++depth;
    deepest = max(deepest, depth);
    if (lane == 0)
      link_node(recs, out, v[0], P, P + 2, node, rec + 1, rec, 0, half < 2, base + start, M.face[M.ord[start]]);
    if (lane == 1)
      link_node(recs, out, v[1], P + 1, P + 2 * half, node, rec + half, rec, 1, nr < 2, base + start + half,
                M.face[M.ord[start + half]]);
    // the larger child waits, the smaller goes on (at most 8 wait); leaves are done
    const bool lgo = half > 1, rgo = nr > 1;
    const bool take_left = lgo && (!rgo || half <= nr);
    if (lgo && rgo) {
      if (lane == 0) {
        int* st = M.stack[sp];
        st[0] = take_left ? start + half : start;
        st[1] = take_left ? nr : half;
        st[2] = take_left ? P + 1 : P;
        st[3] = take_left ? P + 2 * half : P + 2;
        st[4] = take_left ? rec + half : rec + 1;
        st[5] = depth;
        for (int k = 0; k < 6; ++k) st[6 + k] = take_left ? v[1][6 + k] : v[0][6 + k];
      }
      ++sp;
    }
    if (lgo || rgo) {
      const int p0 = P;
      node = take_left ? p0 : p0 + 1;
      P = take_left ? p0 + 2 : p0 + 2 * half;
      rec = take_left ? rec + 1 : rec + half;
      start = take_left ? start : start + half;
      count = take_left ? half : nr;
      for (int k = 0; k < 6; ++k) cb[k] = take_left ? v[0][6 + k] : v[1][6 + k];
    } else if (sp > 0) {
      --sp;
      __syncwarp();
      const int* st = M.stack[sp];
      start = st[0];
      count = st[1];
      node = st[2];
      P = st[3];
      rec = st[4];
      depth = st[5];
      for (int k = 0; k < 6; ++k) cb[k] = st[6 + k];
    } else {
      break;
    }
    __syncwarp();
  }
  if (lane == 0) atomicMax(&h->depth, deepest);
  for (int i = lane; i < total; i += 32) {
    const int f = M.face[M.ord[i]];
    const Face F = faces[f];
    const float4 p1 = pts[F.vx], p2 = pts[F.vy], p3 = pts[F.vz];
    float4* o = tris + 3 * (size_t)(base + i);
    o[0] = make_float4(p1.x, p1.y, p1.z, __int_as_float(f));
    o[1] = make_float4(p2.x - p1.x, p2.y - p1.y, p2.z - p1.z, 0.f);
    o[2] = make_float4(p3.x - p1.x, p3.y - p1.y, p3.z - p1.z, 0.f);
  }
}

// FP16 records from FP32 ones: lower planes rounded down, upper planes up.
__global__ void k_quantize_fp16(const float4* __restrict__ recs, int nrec, uint4* q) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nrec) return;
  const float4* p = recs + 4 * (size_t)i;
  const float4 n0 = p[0], n1 = p[1], n2 = p[2], n3 = p[3];
  auto pair = [](float lo, float hi) {
    __half2 h = __halves2half2(__float2half_rd(lo), __float2half_ru(hi));
    return *reinterpret_cast<unsigned*>(&h);
  };
  q[2 * (size_t)i + 0] = make_uint4(pair(n0.x, n0.y), pair(n0.z, n0.w), pair(n1.x, n1.y), pair(n1.z, n1.w));
  q[2 * (size_t)i + 1] = make_uint4(pair(n2.x, n2.y), pair(n2.z, n2.w), __float_as_uint(n3.x), __float_as_uint(n3.y));
}

// 4-wide FP16 nodes from FP32 records: node r holds, for each child of record r,
// that child's two children when it is interior, else the child (a leaf), with
// the same outward rounding as the FP16 records. The tree's nodes start at node
// `first` of q.
__global__ void k_quad_fp16(const float4* __restrict__ recs, int nrec, int first, uint4* q) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nrec) return;
  auto pair = [](float lo, float hi) {
    __half2 h = __halves2half2(__float2half_rd(lo), __float2half_ru(hi));
    return *reinterpret_cast<unsigned*>(&h);
  };
  // a record's children: boxes (lo/hi per axis) and refs
  auto kids = [&](int r, float box[2][6], int ref[2]) {
    const float4* p = recs + 4 * (size_t)r;
    const float4 n0 = p[0], n1 = p[1], n2 = p[2], n3 = p[3];
    const float b[2][6] = {{n0.x, n0.y, n0.z, n0.w, n2.x, n2.y}, {n1.x, n1.y, n1.z, n1.w, n2.z, n2.w}};
    for (int c = 0; c < 2; ++c)
      for (int k = 0; k < 6; ++k) box[c][k] = b[c][k];
    ref[0] = __float_as_int(n3.x);
    ref[1] = __float_as_int(n3.y);
  };
  float box[2][6];
  int ref[2];
  kids(i, box, ref);
  unsigned w[16];
  int n = 0;
  const unsigned empty_box = pair(INFINITY, -INFINITY);
  for (int c = 0; c < 2; ++c) {
    if (ref[c] >= 0) {
      float gb[2][6];
      int gr[2];
      kids(ref[c], gb, gr);
      for (int g = 0; g < 2; ++g, ++n) {
        for (int a = 0; a < 3; ++a) w[3 * n + a] = pair(gb[g][2 * a], gb[g][2 * a + 1]);
        w[12 + n] = (unsigned)(gr[g] >= 0 ? first + gr[g] : gr[g]);
      }
    } else {
      for (int a = 0; a < 3; ++a) w[3 * n + a] = pair(box[c][2 * a], box[c][2 * a + 1]);
      w[12 + n] = (unsigned)ref[c];
      ++n;
    }
  }
  for (; n < 4; ++n) {
    for (int a = 0; a < 3; ++a) w[3 * n + a] = empty_box;
    w[12 + n] = (unsigned)kQuadEmpty;
  }
  uint4* o = q + 4 * ((size_t)first + i);
  o[0] = make_uint4(w[0], w[1], w[2], w[3]);
  o[1] = make_uint4(w[4], w[5], w[6], w[7]);
  o[2] = make_uint4(w[8], w[9], w[10], w[11]);
  o[3] = make_uint4(w[12], w[13], w[14], w[15]);
}

// Parent links: up[c] = (r, the other child of r) for each record child c of record r.
__global__ void k_up_links(const float4* __restrict__ recs, int nrec, int root, int2* up) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nrec) return;
  const float4 n3 = recs[4 * (size_t)i + 3];
  const int l = __float_as_int(n3.x), r = __float_as_int(n3.y);
  if (l >= 0) up[l] = make_int2(i, r);
  if (r >= 0) up[r] = make_int2(i, l);
  if (i == root) up[i] = make_int2(-1, -1);
}

inline unsigned blocks(size_t n) { return (unsigned)((n + kT - 1) / kT); }

}  // namespace
}  // namespace mt

using namespace mt;

extern "C" int mt_bvh_build_device(mt_scene* s, int32_t* nodes_out, float* bounds_out, int* depth_out) {
  if (!s) return fail(MT_ERR_INVALID, "NULL scene");
  const int n = s->ntri;
  if (n < 1) return fail(MT_ERR_INVALID, "empty scene");
  mt_context* ctx = s->ctx;
  std::lock_guard<std::recursive_mutex> lk(ctx->mu);
  CU(cudaSetDevice(ctx->device));
  int q = quiesce(ctx);
  if (q) return q;
  cudaStream_t st = ctx->stream;
  const size_t nn = 2 * (size_t)n - 1;
  const int nrec = n > 1 ? n - 1 : 0;
  // a level has at most n / kSmallTris large nodes, each with at most two small
  // subtrees below it (levels beyond the limit fail), and no two share a triangle
  const size_t node_cap = (size_t)n / kSmallTris + 2,
               small_cap = std::min((size_t)n, 2 * node_cap * (kStackDepth + 8)) + 1;
  const int chunk_cap = n / kChunk + (int)node_cap;
  auto align = Workspace::round;
  const size_t b_prim = align(sizeof(Prim) * (size_t)n), b_node = align(sizeof(Big) * node_cap),
               b_small = align(sizeof(Small) * small_cap), b_cnt = align(sizeof(int) * ((size_t)chunk_cap + 1)),
               b_ref = nodes_out ? align(28 * nn) : 0, b_bound = bounds_out ? align(32 * nn) : 0;
  Workspace ws;
  float4 *recs = nullptr, *tris = nullptr;
  // the tree's arrays first: they can take the place of the scratch that is kept, not of
  // the scratch in use
  int r = dalloc(ctx, &recs, 4 * (size_t)std::max(nrec, 1));
  if (!r) r = dalloc(ctx, &tris, 3 * (size_t)n);
  if (!r) r = ws.get(ctx, 2 * b_prim + 2 * b_node + b_small + b_cnt + b_ref + b_bound + 256);
  auto fail_all = [&](int code, const char* msg) {
    std::string keep = msg ? std::string(msg) : mt_last_error();
    cudaStreamSynchronize(st);
    ws.release();
    dfree(recs);
    dfree(tris);
    return fail(code, "%s", keep.c_str());
  };
  if (r) return fail_all(r, nullptr);
  auto take = [&](size_t b) { return ws.take<char>(b); };
  Prim* prim[2] = {(Prim*)take(b_prim), nullptr};
  prim[1] = (Prim*)take(b_prim);
  Big* nodes[2] = {(Big*)take(b_node), nullptr};
  nodes[1] = (Big*)take(b_node);
  Small* smalls = (Small*)take(b_small);
  int* cnt = (int*)take(b_cnt);
  RefOut out{};
  if (nodes_out) out.nodes = (int*)take(b_ref);
  if (bounds_out) out.bounds = (float*)take(b_bound);
  Heads* heads = (Heads*)take(256);
  k_start<<<1, 1, 0, st>>>(nodes[0], smalls, heads, n);
  k_prims<<<blocks(n), kT, 0, st>>>(s->d_points, s->d_faces, n, prim[0],
                                    n > kSmallTris ? nodes[0]->box : smalls[0].box);
  // The levels of large nodes, without waiting for the host to see how many are
  // left: as many as an even tree has, then a few at a time. An empty level costs
  // three launches that end at once.
  Heads hh{};
  int level = 0, until = 0;
  for (int m = n; m > kSmallTris; m = (m + 1) / 2) ++until;
  for (until += 2; n > kSmallTris; until = level + 4) {
    for (; level < until; ++level) {
      const int c = level & 1;
      k_count<<<chunk_cap, kT, 0, st>>>(prim[c], nodes[c], heads, level, cnt);
      k_plan<<<1, 1024, 0, st>>>(nodes[c], nodes[c ^ 1], smalls, heads, level, cnt, recs, out);
      k_scatter<<<chunk_cap, kT, 0, st>>>(prim[c], prim[c ^ 1], nodes[c], nodes[c ^ 1], smalls, heads, level, cnt);
    }
    if (cudaMemcpyAsync(&hh, heads, sizeof(hh), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess)
      return fail_all(MT_ERR_CUDA, cudaGetErrorString(cudaGetLastError()));
    if (hh.nodes[level & 1] == 0) break;
    if (level > kStackDepth) return fail_all(MT_ERR_DEPTH, "BVH deeper than the 64-level traversal stack");
  }
  const int nsmall = n > kSmallTris ? hh.smalls : 1;
  k_small<<<(nsmall + kSmallWarps - 1) / kSmallWarps, 32 * kSmallWarps, 0, st>>>(
      prim[0], prim[1], smalls, heads, recs, out, s->d_points, s->d_faces, tris);
  if (cudaMemcpyAsync(&hh, heads, sizeof(hh), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
      (nodes_out && cudaMemcpyAsync(nodes_out, out.nodes, 28 * nn, cudaMemcpyDeviceToHost, st) != cudaSuccess) ||
      (bounds_out && cudaMemcpyAsync(bounds_out, out.bounds, 32 * nn, cudaMemcpyDeviceToHost, st) != cudaSuccess) ||
      cudaStreamSynchronize(st) != cudaSuccess)
    return fail_all(MT_ERR_CUDA, cudaGetErrorString(cudaGetLastError()));
  const int depth = hh.depth;
  if (depth > kStackDepth) return fail_all(MT_ERR_DEPTH, "BVH deeper than the 64-level traversal stack");
  ws.release();
  dfree(s->d_nodes);
  dfree(s->d_tris);
  s->d_nodes = recs;
  s->d_tris = tris;
  s->nrec = nrec;
  s->root_ref = n > 1 ? 0 : ~0;
  s->depth = depth;
  s->has_bvh = 1;
  ++s->version;
  if (depth_out) *depth_out = depth;
  return refresh_qnodes(s);
}

bool traversal_bitstack() {
  static const bool on = [] {
    const char* e = std::getenv("MT_TRAVERSAL");
    return e && std::strcmp(e, "bitstack") == 0;
  }();
  return on;
}

int refresh_qnodes(mt_scene* s) {
  dfree(s->d_qnodes);
  dfree(s->d_quad);
  dfree(s->d_up);
  if (traversal_bitstack() && s->has_bvh && s->nrec > 0) {
    int r = dalloc(s->ctx, &s->d_up, (size_t)s->nrec);
    if (r) return r;
    cudaStream_t st = s->ctx->stream;
    k_up_links<<<blocks(s->nrec), kT, 0, st>>>(s->d_nodes, s->nrec, s->root_ref, s->d_up);
    if (cudaGetLastError() != cudaSuccess || cudaStreamSynchronize(st) != cudaSuccess) {
      dfree(s->d_up);
      return fail(MT_ERR_CUDA, "parent links: %s", cudaGetErrorString(cudaGetLastError()));
    }
  }
  if (int w = refresh_wide(s)) return w;
  if (s->precision == 3 && s->has_bvh && s->nrec > 0) {
    Workspace ws;
    float4* sah = nullptr;
    // nodes over the surface-area tree and over the reference's (the array first, as above);
    // over the latter alone where that tree would be too deep or memory is short
    int r = dalloc(s->ctx, &s->d_quad, 8 * (size_t)s->nrec);
    if (!r) r = build_sah_records(s, ws, &sah);
    if (r == MT_ERR_NOMEM || (!r && !sah)) {
      ws.release();
      dfree(s->d_quad);
      r = dalloc(s->ctx, &s->d_quad, 4 * (size_t)s->nrec);
    }
    cudaError_t e = cudaSuccess;
    if (!r) {
      cudaStream_t st = s->ctx->stream;
      s->quad_again = sah ? s->nrec : 0;
      if (sah) k_quad_fp16<<<blocks(s->nrec), kT, 0, st>>>(sah, s->nrec, 0, s->d_quad);
      k_quad_fp16<<<blocks(s->nrec), kT, 0, st>>>(s->d_nodes, s->nrec, s->quad_again, s->d_quad);
      e = cudaGetLastError();
      const cudaError_t w = cudaStreamSynchronize(st);
      if (e == cudaSuccess) e = w;
    }
    ws.release();
    if (r || e != cudaSuccess) {
      dfree(s->d_quad);
      return r ? r : fail(MT_ERR_CUDA, "4-wide FP16 nodes: %s", cudaGetErrorString(e));
    }
    return MT_OK;
  }
  if (s->precision != 1 || !s->has_bvh || s->nrec == 0) return MT_OK;
  int r = dalloc(s->ctx, &s->d_qnodes, 2 * (size_t)s->nrec);
  if (r) return r;
  cudaStream_t st = s->ctx->stream;
  k_quantize_fp16<<<blocks(s->nrec), kT, 0, st>>>(s->d_nodes, s->nrec, s->d_qnodes);
  if (cudaGetLastError() != cudaSuccess || cudaStreamSynchronize(st) != cudaSuccess) {
    dfree(s->d_qnodes);
    return fail(MT_ERR_CUDA, "FP16 records: %s", cudaGetErrorString(cudaGetLastError()));
  }
  return MT_OK;
}

// Mesh arrays on the device: index checks, the mesh-light list, triangle slots of an
// imported tree. The arrays are read at the GPU's memory rate where one host thread
// took 4 ms for the faces of 500k triangles alone (40 bytes each).
#include <cuda_runtime.h>

#include <climits>
#include <cstring>
#include <vector>

#include "mt_internal.h"
#include "mt_scan.cuh"

namespace mt {
namespace {

using namespace scan;

constexpr int kT = 256;

__device__ __forceinline__ bool in(int i, int n) { return i >= 0 && i < n; }

// The first face with an index out of range, into *bad (INT_MAX: none). nuvs, nnormals:
// 0 when the mesh has none. mat_only: its material alone.
__global__ void __launch_bounds__(kT) k_check_faces(const Face* __restrict__ faces, int n, int npoints, int nuvs,
                                                    int nnormals, int nmat, int mat_only, int* bad) {
  const int i = blockIdx.x * kT + threadIdx.x;
  bool ok = true;
  if (i < n) {
    const Face f = faces[i];
    ok = (f.mat & 0xFFFF) < nmat;
    if (!mat_only)
      ok = ok && in(f.vx, npoints) && in(f.vy, npoints) && in(f.vz, npoints) &&
           (f.uvx <= -1 || (in(f.uvx, nuvs) && in(f.uvy, nuvs) && in(f.uvz, nuvs))) &&
           (f.nx <= -1 || (in(f.nx, nnormals) && in(f.ny, nnormals) && in(f.nz, nnormals)));
  }
  const unsigned wrong = __ballot_sync(0xffffffffu, !ok);
  if (wrong && (threadIdx.x & 31) == 0) atomicMin(bad, i + __ffs(wrong) - 1);
}

// The faces whose material emits, in face order: an ordered compaction.
__global__ void __launch_bounds__(kT)
    k_light_faces(const Face* __restrict__ faces, int n, const unsigned char* __restrict__ emits, int* __restrict__ out,
                  unsigned long long* status, int* words) {  // words: tile counter, count, error
  __shared__ unsigned long long sh[kT / 32 + 1], s_base;
  __shared__ int s_tile;
  if (threadIdx.x == 0) s_tile = atomicAdd(&words[0], 1);
  __syncthreads();
  const int tile = s_tile, i = tile * kT + threadIdx.x;
  const bool keep = i < n && emits[faces[i].mat & 0xFFFF];
  unsigned long long tot;
  const unsigned long long excl = block_rank2<kT>(keep, false, &tot, sh);
  if (threadIdx.x < 32) {
    const unsigned long long b = lookback(status, tile, tot, &words[2]);
    if (threadIdx.x == 0) s_base = b;
  }
  __syncthreads();
  if (keep) out[s_base + excl] = i;
  if (threadIdx.x == 0 && tile == (int)gridDim.x - 1) words[1] = (int)(s_base + tot);
}

// Slot k holds triangle order[k]: p1 with the face id, e1 = p2 - p1, e2 = p3 - p1.
__global__ void k_order_tris(int n, const int* __restrict__ order, const float4* __restrict__ pts,
                             const Face* __restrict__ faces, float4* __restrict__ tris) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const int f = order[k];
  const Face F = faces[f];
  const float4 p1 = pts[F.vx], p2 = pts[F.vy], p3 = pts[F.vz];
  tris[3 * (size_t)k + 0] = make_float4(p1.x, p1.y, p1.z, __int_as_float(f));
  tris[3 * (size_t)k + 1] = make_float4(p2.x - p1.x, p2.y - p1.y, p2.z - p1.z, 0.f);
  tris[3 * (size_t)k + 2] = make_float4(p3.x - p1.x, p3.y - p1.y, p3.z - p1.z, 0.f);
}

unsigned blocks(int n) { return (unsigned)((n + kT - 1) / kT); }

}  // namespace
}  // namespace mt

int first_bad_face(mt_scene* s, int nmat, bool mat_only, int* bad) {
  mt_context* ctx = s->ctx;
  *bad = INT_MAX;
  CU(cudaMemcpyAsync(ctx->d_scratch, bad, 4, cudaMemcpyHostToDevice, ctx->stream));
  mt::k_check_faces<<<mt::blocks(s->ntri), mt::kT, 0, ctx->stream>>>(s->d_faces, s->ntri, s->npoints, s->nuvs, s->nnormals,
                                                                     nmat, mat_only ? 1 : 0, ctx->d_scratch);
  CU(cudaGetLastError());
  CU(cudaMemcpyAsync(bad, ctx->d_scratch, 4, cudaMemcpyDeviceToHost, ctx->stream));
  CU(cudaStreamSynchronize(ctx->stream));
  return MT_OK;
}

namespace {
// The two calls below without scratch, for a device that has none left: the arrays go
// through the host.
int host_light_faces(mt_scene* s, const std::vector<unsigned char>& emits) {
  std::vector<Face> F((size_t)s->ntri);
  CU(cudaMemcpy(F.data(), s->d_faces, F.size() * sizeof(Face), cudaMemcpyDeviceToHost));
  std::vector<int> list;
  for (int i = 0; i < s->ntri; ++i)
    if (emits[F[i].mat & 0xFFFF]) list.push_back(i);
  if (list.empty()) return MT_OK;
  const int r = dalloc(s->ctx, &s->d_light_faces, list.size());
  if (r) return r;
  CU(cudaMemcpy(s->d_light_faces, list.data(), 4 * list.size(), cudaMemcpyHostToDevice));
  s->nlights = (int)list.size();
  return MT_OK;
}
int host_order_triangles(mt_scene* s, const std::vector<int>& order, float4* tris) {
  std::vector<Face> F((size_t)s->ntri);
  std::vector<float4> P((size_t)s->npoints), T(3 * order.size());
  CU(cudaMemcpy(F.data(), s->d_faces, F.size() * sizeof(Face), cudaMemcpyDeviceToHost));
  CU(cudaMemcpy(P.data(), s->d_points, P.size() * sizeof(float4), cudaMemcpyDeviceToHost));
  for (size_t k = 0; k < order.size(); ++k) {
    const Face& f = F[order[k]];
    const float4 p1 = P[f.vx], p2 = P[f.vy], p3 = P[f.vz];
    float id;
    std::memcpy(&id, &order[k], 4);
    T[3 * k + 0] = make_float4(p1.x, p1.y, p1.z, id);
    T[3 * k + 1] = make_float4(p2.x - p1.x, p2.y - p1.y, p2.z - p1.z, 0.f);
    T[3 * k + 2] = make_float4(p3.x - p1.x, p3.y - p1.y, p3.z - p1.z, 0.f);
  }
  CU(cudaMemcpy(tris, T.data(), T.size() * sizeof(float4), cudaMemcpyHostToDevice));
  return MT_OK;
}
}  // namespace

// identifyMeshLights + prefix scan + prepareLightInfo (CLightConfiguration.java:43-87).
int list_light_faces(mt_scene* s, const std::vector<unsigned char>& emits) {
  mt_context* ctx = s->ctx;
  dfree(s->d_light_faces);
  s->nlights = 0;
  bool any = false;
  for (unsigned char e : emits) any |= e != 0;
  if (!any) return MT_OK;
  const size_t tiles = mt::blocks(s->ntri);
  Workspace ws;
  int r = ws.get(ctx, Workspace::round(emits.size()) + Workspace::round(4 * (size_t)s->ntri) + Workspace::round(8 * tiles) +
                          Workspace::round(16));
  if (r == MT_ERR_NOMEM) return host_light_faces(s, emits);
  if (r) return r;
  unsigned char* d_emits = ws.take<unsigned char>(emits.size());
  int* list = ws.take<int>((size_t)s->ntri);
  auto* status = ws.take<unsigned long long>(tiles);
  int* words = ws.take<int>(4);
  int h[4] = {0, 0, 0, 0};
  cudaError_t e = cudaMemcpyAsync(d_emits, emits.data(), emits.size(), cudaMemcpyHostToDevice, ctx->stream);
  if (e == cudaSuccess) e = cudaMemsetAsync(status, 0, 8 * tiles, ctx->stream);
  if (e == cudaSuccess) e = cudaMemsetAsync(words, 0, 16, ctx->stream);
  if (e == cudaSuccess) {
    mt::k_light_faces<<<(unsigned)tiles, mt::kT, 0, ctx->stream>>>(s->d_faces, s->ntri, d_emits, list, status, words);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpyAsync(h, words, 16, cudaMemcpyDeviceToHost, ctx->stream);
  const cudaError_t w = cudaStreamSynchronize(ctx->stream);
  if (e == cudaSuccess) e = w;
  if (e != cudaSuccess) r = fail(MT_ERR_CUDA, "light list: %s", cudaGetErrorString(e));
  else if (h[2]) r = fail(MT_ERR_DEVICE, "light list: device error %d", h[2]);
  if (!r && h[1] > 0) {
    r = dalloc(ctx, &s->d_light_faces, (size_t)h[1]);
    if (!r && (cudaMemcpyAsync(s->d_light_faces, list, 4 * (size_t)h[1], cudaMemcpyDeviceToDevice, ctx->stream) !=
                   cudaSuccess ||
               cudaStreamSynchronize(ctx->stream) != cudaSuccess))
      r = fail(MT_ERR_CUDA, "light list: %s", cudaGetErrorString(cudaGetLastError()));
    if (!r) s->nlights = h[1];
  }
  ws.release();
  // the list's own array may need the kept scratch's bytes
  return r == MT_ERR_NOMEM ? host_light_faces(s, emits) : r;
}

int order_triangles(mt_scene* s, const std::vector<int>& order, float4* tris) {
  mt_context* ctx = s->ctx;
  Workspace ws;
  int r = ws.get(ctx, Workspace::round(4 * order.size()));
  if (r == MT_ERR_NOMEM) return host_order_triangles(s, order, tris);
  if (r) return r;
  int* d = ws.take<int>(order.size());
  cudaError_t e = cudaMemcpyAsync(d, order.data(), 4 * order.size(), cudaMemcpyHostToDevice, ctx->stream);
  if (e == cudaSuccess) {
    mt::k_order_tris<<<mt::blocks((int)order.size()), mt::kT, 0, ctx->stream>>>((int)order.size(), d, s->d_points,
                                                                               s->d_faces, tris);
    e = cudaGetLastError();
  }
  const cudaError_t w = cudaStreamSynchronize(ctx->stream);
  if (e == cudaSuccess) e = w;
  ws.release();
  return e == cudaSuccess ? MT_OK : fail(MT_ERR_CUDA, "triangle slots: %s", cudaGetErrorString(e));
}

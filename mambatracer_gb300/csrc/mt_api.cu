// C-ABI of the GB300 wavefront path tracer (see include/mambatracer.h).
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <type_traits>
#include <cstdlib>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <deque>
#include <mutex>
#include <string>
#include <unordered_map>
#include <vector>

#include "mt_compact.h"
#include "mt_device.cuh"
#include "mt_internal.h"

// ------------------------------------------------------------------ context
namespace {
thread_local std::string g_err;
}

extern "C" const char* mt_last_error(void) { return g_err.c_str(); }

namespace {
// MT_DEVICE_ROOM's account of the library's arrays.
struct DeviceRoom {
  const bool on = std::getenv("MT_DEVICE_ROOM") != nullptr;
  std::mutex mu;
  std::unordered_map<void*, size_t> sizes;
  size_t live = 0, limit = SIZE_MAX;
  std::string seen;
  // bytes the arrays may still grow by (mu held)
  size_t left() {
    const char* e = std::getenv("MT_DEVICE_ROOM");
    if (!e) e = "";
    if (seen != e) {
      seen = e;
      limit = *e ? live + (size_t)std::strtoull(e, nullptr, 10) : SIZE_MAX;
    }
    return limit > live ? limit - live : 0;
  }
};
DeviceRoom& device_room() {
  static DeviceRoom r;
  return r;
}
}  // namespace

namespace mt {
__attribute__((visibility("hidden"))) void set_last_error(const char* msg) { g_err = msg; }
__attribute__((visibility("hidden"))) int fail(int code, const char* fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof(buf), fmt, ap);
  va_end(ap);
  g_err = buf;
  return code;
}

__attribute__((visibility("hidden"))) cudaError_t device_malloc(void** p, size_t bytes) {
  DeviceRoom& r = device_room();
  if (!r.on) return cudaMalloc(p, bytes);
  std::lock_guard<std::mutex> lk(r.mu);
  if (bytes > r.left()) return cudaErrorMemoryAllocation;
  const cudaError_t e = cudaMalloc(p, bytes);
  if (e == cudaSuccess) r.live += r.sizes[*p] = bytes;
  return e;
}
__attribute__((visibility("hidden"))) void device_free(void* p) {
  DeviceRoom& r = device_room();
  if (r.on) {
    std::lock_guard<std::mutex> lk(r.mu);
    r.live -= r.sizes[p];
    r.sizes.erase(p);
  }
  cudaFree(p);
}
__attribute__((visibility("hidden"))) size_t device_left() {
  size_t free = 0, total = 0;
  if (cudaMemGetInfo(&free, &total) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  DeviceRoom& r = device_room();
  if (!r.on) return free;
  std::lock_guard<std::mutex> lk(r.mu);
  return std::min(free, r.left());
}
}  // namespace mt

int quiesce(mt_context* ctx) {
  join_jobs(ctx);
  CU(cudaStreamSynchronize(ctx->stream));
  servers_sync(ctx);
  return MT_OK;
}

void join_jobs(mt_context* ctx) {
  for (mt_job* j : ctx->jobs) {
    for (JobSlot& s : j->slots)
      if (s.done) cudaStreamWaitEvent(ctx->stream, s.done, 0);
    if (j->rdone) cudaStreamWaitEvent(ctx->stream, j->rdone, 0);
  }
}

int Workspace::get(mt_context* c, size_t bytes) {
  ctx = c;
  at = 0;
  own = bytes > kWorkspaceMax;
  if (own) return dalloc(c, &base, bytes);
  if (bytes > c->ws_bytes) {
    // grown in steps, so calls of slowly growing sizes do not allocate each time
    const size_t grown = std::min(kWorkspaceMax, std::max({bytes, 2 * c->ws_bytes, (size_t)1 << 20}));
    cudaStreamSynchronize(c->stream);
    dfree(c->ws);
    c->ws_bytes = 0;
    size_t got = grown;
    int r = dalloc(&c->ws, grown);
    if (r && bytes < grown) r = dalloc(&c->ws, got = bytes);
    if (r) return r;
    c->ws_bytes = got;
  }
  base = c->ws;
  c->ws_used = true;
  return MT_OK;
}

void Workspace::release() {
  if (own) dfree(base);
  else if (base) ctx->ws_used = false;
  base = nullptr;
}

bool drop_workspace(mt_context* c) {
  if (!c->ws || c->ws_used) return false;
  cudaStreamSynchronize(c->stream);
  dfree(c->ws);
  c->ws_bytes = 0;
  return true;
}

size_t overlap_bytes(mt_context* c, size_t most) {
  return std::min(most, (device_left() + (c->ws_used ? 0 : c->ws_bytes)) / 4);
}

void prefault(void* p, size_t bytes, cudaEvent_t ready) {
  // only the process's own pages: pinned memory is mapped, and a device pointer, which
  // the copy that follows refuses, is not the host's to write
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess || a.type != cudaMemoryTypeUnregistered) {
    cudaGetLastError();
    return;
  }
  constexpr size_t kPage = 4096, kStep = 64 * kPage;
  auto* b = static_cast<volatile char*>(p);
  for (size_t o = 0; o < bytes; o += kStep) {
    if (cudaEventQuery(ready) != cudaErrorNotReady) return;
    cudaGetLastError();  // not ready is not an error
    for (size_t q = o; q < std::min(bytes, o + kStep); q += kPage) b[q] = 0;
  }
}

extern "C" const char* mt_version(void) {
  return "mambatracer-gb300 sm_103a fmad=false prec-div prec-sqrt";
}

extern "C" int mt_ctx_create(int device, mt_context** out) {
  if (!out) return fail(MT_ERR_INVALID, "out is NULL");
  *out = nullptr;
  int n = 0;
  CU(cudaGetDeviceCount(&n));
  if (device < 0 || device >= n) return fail(MT_ERR_INVALID, "device %d of %d", device, n);
  CU(cudaSetDevice(device));
  auto* c = new mt_context();
  c->device = device;
  cudaDeviceProp prop;
  cudaError_t e = cudaGetDeviceProperties(&prop, device);
  if (e != cudaSuccess) {
    delete c;
    return fail(MT_ERR_CUDA, "cudaGetDeviceProperties: %s", cudaGetErrorString(e));
  }
  c->num_sms = prop.multiProcessorCount;
  e = cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking);
  if (e != cudaSuccess) {
    delete c;
    return fail(MT_ERR_CUDA, "cudaStreamCreate: %s", cudaGetErrorString(e));
  }
  if (dalloc(&c->d_scratch, 4) != MT_OK) {
    cudaStreamDestroy(c->stream);
    delete c;
    return MT_ERR_NOMEM;
  }
  for (auto& ev : c->ev) cudaEventCreate(&ev);
  cudaEventCreateWithFlags(&c->ready, cudaEventDisableTiming);
  *out = c;
  return MT_OK;
}

extern "C" int mt_ctx_destroy(mt_context* ctx) {
  if (!ctx) return fail(MT_ERR_INVALID, "ctx is NULL");
  cudaSetDevice(ctx->device);
  cudaStreamSynchronize(ctx->stream);
  dfree(ctx->d_scratch);
  dfree(ctx->ws);
  for (auto& p : ctx->pass_streams) {
    for (cudaEvent_t e : {p.fork, p.join, p.done})
      if (e) cudaEventDestroy(e);
    for (cudaStream_t q : {p.stream, p.side})
      if (q) cudaStreamDestroy(q);
  }
  dfree(ctx->cs_status);
  dfree(ctx->cs_words);
  dfree(ctx->d_plain_err);
  for (auto& ev : ctx->ev)
    if (ev) cudaEventDestroy(ev);
  if (ctx->ready) cudaEventDestroy(ctx->ready);
  cudaStreamDestroy(ctx->stream);
  delete ctx;
  return MT_OK;
}

extern "C" int mt_ctx_event_record(mt_context* ctx, int slot) {
  if (!ctx || slot < 0 || slot >= 8) return fail(MT_ERR_INVALID, "bad event slot");
  std::lock_guard<std::recursive_mutex> lk(ctx->mu);
  CU(cudaSetDevice(ctx->device));
  join_jobs(ctx);
  CU(cudaEventRecord(ctx->ev[slot], ctx->stream));
  return MT_OK;
}

extern "C" int mt_ctx_event_elapsed(mt_context* ctx, int a, int b, float* ms) {
  if (!ctx || !ms || a < 0 || a >= 8 || b < 0 || b >= 8) return fail(MT_ERR_INVALID, "bad event slot");
  CU(cudaSetDevice(ctx->device));
  CU(cudaEventSynchronize(ctx->ev[b]));
  CU(cudaEventElapsedTime(ms, ctx->ev[a], ctx->ev[b]));
  return MT_OK;
}

extern "C" int mt_finish(mt_context* ctx) {
  if (!ctx) return fail(MT_ERR_INVALID, "ctx is NULL");
  std::lock_guard<std::recursive_mutex> lk(ctx->mu);
  CU(cudaSetDevice(ctx->device));
  join_jobs(ctx);
  CU(cudaStreamSynchronize(ctx->stream));
  if (ctx->d_plain_err) {
    int e = 0;
    CU(cudaMemcpy(&e, ctx->d_plain_err, 4, cudaMemcpyDeviceToHost));
    if (e) {
      CU(cudaMemset(ctx->d_plain_err, 0, 4));
      return fail(MT_ERR_DEVICE, "a kernel launched by name met %s", e == 1 ? "an index out of range in its buffers"
                                                                           : "a BVH deeper than 64 levels");
    }
  }
  return MT_OK;
}

// ------------------------------------------------------------------ buffers
extern "C" int mt_buf_alloc(mt_context* ctx, size_t bytes, mt_buffer** out) {
  if (!ctx || !out) return fail(MT_ERR_INVALID, "NULL argument");
  std::lock_guard<std::recursive_mutex> lk(ctx->mu);
  CU(cudaSetDevice(ctx->device));
  void* p = nullptr;
  cudaError_t e = device_malloc(&p, bytes ? bytes : 1);
  if (e == cudaErrorMemoryAllocation && drop_workspace(ctx)) e = device_malloc(&p, bytes ? bytes : 1);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(MT_ERR_NOMEM, "cudaMalloc(%zu): %s", bytes, cudaGetErrorString(e));
  }
  CU(cudaMemsetAsync(p, 0, bytes ? bytes : 1, ctx->stream));
  *out = new mt_buffer{ctx, p, bytes};
  return MT_OK;
}

extern "C" int mt_buf_create_from(mt_context* ctx, const void* host, size_t bytes, mt_buffer** out) {
  int r = mt_buf_alloc(ctx, bytes, out);
  if (r != MT_OK) return r;
  return mt_buf_write(*out, 0, host, bytes);
}

extern "C" int mt_buf_write(mt_buffer* b, size_t off, const void* host, size_t bytes) {
  if (!b || (!host && bytes)) return fail(MT_ERR_INVALID, "NULL argument");
  if (off > b->bytes || bytes > b->bytes - off) return fail(MT_ERR_INVALID, "write [%zu,+%zu) past %zu B", off, bytes, b->bytes);
  std::lock_guard<std::recursive_mutex> lk(b->ctx->mu);
  CU(cudaSetDevice(b->ctx->device));
  CU(cudaMemcpyAsync((char*)b->ptr + off, host, bytes, cudaMemcpyHostToDevice, b->ctx->stream));
  CU(cudaStreamSynchronize(b->ctx->stream));
  return MT_OK;
}

extern "C" int mt_buf_read(mt_buffer* b, size_t off, void* host, size_t bytes) {
  if (!b || (!host && bytes)) return fail(MT_ERR_INVALID, "NULL argument");
  if (off > b->bytes || bytes > b->bytes - off) return fail(MT_ERR_INVALID, "read [%zu,+%zu) past %zu B", off, bytes, b->bytes);
  std::lock_guard<std::recursive_mutex> lk(b->ctx->mu);
  CU(cudaSetDevice(b->ctx->device));
  CU(cudaMemcpyAsync(host, (char*)b->ptr + off, bytes, cudaMemcpyDeviceToHost, b->ctx->stream));
  CU(cudaStreamSynchronize(b->ctx->stream));
  return MT_OK;
}

namespace {
__global__ void k_fill32(uint32_t* p, uint32_t v, size_t n) {
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) p[i] = v;
}
}  // namespace

extern "C" int mt_buf_fill32(mt_buffer* b, uint32_t pattern, size_t off, size_t bytes) {
  if (!b) return fail(MT_ERR_INVALID, "NULL buffer");
  if ((off | bytes) & 3) return fail(MT_ERR_INVALID, "offset and size must be multiples of 4");
  if (off > b->bytes || bytes > b->bytes - off) return fail(MT_ERR_INVALID, "fill past the end");
  std::lock_guard<std::recursive_mutex> lk(b->ctx->mu);
  CU(cudaSetDevice(b->ctx->device));
  size_t n = bytes / 4;
  if (n) k_fill32<<<(unsigned)((n + 255) / 256), 256, 0, b->ctx->stream>>>((uint32_t*)((char*)b->ptr + off), pattern, n);
  CU(cudaGetLastError());
  return MT_OK;
}

extern "C" size_t mt_buf_size(const mt_buffer* b) { return b ? b->bytes : 0; }

extern "C" int mt_buf_free(mt_buffer* b) {
  if (!b) return fail(MT_ERR_INVALID, "NULL buffer");
  {
    std::lock_guard<std::recursive_mutex> lk(b->ctx->mu);
    cudaSetDevice(b->ctx->device);
    cudaStreamSynchronize(b->ctx->stream);
    device_free(b->ptr);
  }
  delete b;
  return MT_OK;
}

// ------------------------------------------------------------------- scene
namespace {

bool emitter_host(const Material& m) {
  float s = m.emission_param.x;
  float x = m.emission_color.x * s, y = m.emission_color.y * s, z = m.emission_color.z * s;
  return (0.2989f * x + 0.5866f * y) + 0.1145f * z != 0.0f;
}

// The mesh lights of the scene's materials.
int upload_lights(mt_scene* s) {
  const Material* M = reinterpret_cast<const Material*>(s->h_materials.data());
  std::vector<unsigned char> emits(s->nmat);
  for (int m = 0; m < s->nmat; ++m) emits[m] = emitter_host(M[m]);
  return list_light_faces(s, emits);
}

template <class T>
int upload(mt_context* c, T** d, const void* h, size_t count) {
  dfree(*d);
  int r = dalloc(c, d, count);
  if (r) return r;
  if (h && count) CU(cudaMemcpy(*d, h, count * sizeof(T), cudaMemcpyHostToDevice));
  return MT_OK;
}

void free_env(mt_scene* s) {
  dfree(s->d_env);
  s->env_bytes = 0;
  s->d_env_rgb = nullptr;
  s->d_env_lum = s->d_env_sat = s->d_env_marg = s->d_env_cond = nullptr;
  s->d_env_sat64 = nullptr;
}

void free_scene(mt_scene* s) {
  dfree(s->d_mesh);
  s->d_points = nullptr;
  s->d_uvs = nullptr;
  s->d_normals = nullptr;
  s->d_faces = nullptr;
  dfree(s->d_materials);
  dfree(s->d_light_faces);
  dfree(s->d_nodes);
  dfree(s->d_tris);
  dfree(s->d_qnodes);
  dfree(s->d_wnodes);
  dfree(s->d_wtris);
  dfree(s->d_quad);
  dfree(s->d_up);
  free_env(s);
  dfree(s->d_texels);
  dfree(s->d_tex_ref);
}

// Arrays of a w x h environment map, one allocation: texels, luminance, SATs (with64:
// the FP64 one too) and, unless switched off, the CDF tables of full-map sampling. A
// map of the same shape takes the arrays of the one before.
int alloc_env(mt_scene* s, int w, int h, bool with64) {
  const size_t n = (size_t)w * h;
  size_t marg = 0;
  const size_t cond = map_table_floats(w, h, &marg);
  const bool tables = cdf_tables_enabled();
  auto R = Workspace::round;
  const size_t bytes = R(16 * n) + 2 * R(4 * n) + (with64 ? R(8 * n) : 0) + (tables ? R(4 * marg) + R(4 * cond) : 0);
  if (bytes != s->env_bytes || w != s->env_w || h != s->env_h) {
    free_env(s);
    int r = dalloc(s->ctx, &s->d_env, bytes);
    if (r) return r;
    s->env_bytes = bytes;
  }
  char* at = s->d_env;
  auto take = [&](auto** p, size_t b) {
    *p = reinterpret_cast<std::remove_reference_t<decltype(*p)>>(at);
    at += R(b);
  };
  take(&s->d_env_rgb, 16 * n);
  take(&s->d_env_lum, 4 * n);
  take(&s->d_env_sat, 4 * n);
  s->d_env_sat64 = nullptr;
  s->d_env_marg = s->d_env_cond = nullptr;
  if (with64) take(&s->d_env_sat64, 8 * n);
  if (tables) {
    take(&s->d_env_marg, 4 * marg);
    take(&s->d_env_cond, 4 * cond);
  }
  s->env_w = w;
  s->env_h = h;
  return MT_OK;
}

int build_env_tables(mt_scene* s) {
  if (s->d_env_marg &&
      launch_map_tables(s->ctx->stream, s->d_env_sat, s->env_w, s->env_h, s->d_env_marg, s->d_env_cond))
    return fail(MT_ERR_CUDA, "environment tables: %s", cudaGetErrorString(cudaGetLastError()));
  return MT_OK;
}

// Texel pool (all images back to back) and the per-material table of
// (first texel, width, height, 0) for diffuse, glossy, roughness and mirror.
int upload_textures(mt_scene* s) {
  s->h_tex.resize(4 * (size_t)s->nmat);
  size_t total = 0;
  for (const auto& t : s->h_tex) total += t.argb.size();
  if (total > 0x7FFFFFFFu) return fail(MT_ERR_INVALID, "textures hold %zu texels (at most 2^31 - 1)", total);
  dfree(s->d_texels);
  dfree(s->d_tex_ref);
  s->tex_on = 0;
  if (total == 0) return MT_OK;
  std::vector<int32_t> pool;
  pool.reserve(total);
  std::vector<int4> ref(s->h_tex.size());
  for (size_t i = 0; i < s->h_tex.size(); ++i) {
    const auto& t = s->h_tex[i];
    ref[i] = make_int4(t.argb.empty() ? 0 : (int)pool.size(), t.argb.empty() ? 0 : t.w, t.argb.empty() ? 0 : t.h, 0);
    pool.insert(pool.end(), t.argb.begin(), t.argb.end());
  }
  int r = upload(s->ctx, &s->d_texels, pool.data(), pool.size());
  if (!r) r = upload(s->ctx, &s->d_tex_ref, ref.data(), ref.size());
  if (r) return r;
  s->tex_on = 1;
  return MT_OK;
}

}  // namespace

extern "C" int mt_scene_create(mt_context* ctx, const float* points, int npoints, const float* uvs, int nuvs,
                               const float* normals, int nnormals, const int32_t* faces, int nfaces,
                               const void* materials, int nmaterials, mt_scene** out) {
  if (!ctx || !out || !points || !faces || !materials) return fail(MT_ERR_INVALID, "NULL argument");
  if (npoints <= 0 || nfaces <= 0 || nmaterials <= 0) return fail(MT_ERR_INVALID, "empty scene");
  if (nmaterials > 65536) return fail(MT_ERR_INVALID, "more than 65536 materials (16-bit material index)");
  if ((uvs && nuvs < 0) || (normals && nnormals < 0)) return fail(MT_ERR_INVALID, "negative uv or normal count");
  *out = nullptr;
  std::lock_guard<std::recursive_mutex> lk(ctx->mu);
  CU(cudaSetDevice(ctx->device));
  auto* s = new mt_scene();
  s->ctx = ctx;
  s->npoints = npoints;
  s->nuvs = nuvs;
  s->nnormals = nnormals;
  s->ntri = nfaces;
  s->nmat = nmaterials;
  s->h_materials.assign((const uint8_t*)materials, (const uint8_t*)materials + 144 * (size_t)nmaterials);
  if (!uvs) s->nuvs = 0;
  if (!normals) s->nnormals = 0;
  const size_t b_pts = Workspace::round(16 * (size_t)npoints), b_uvs = Workspace::round(8 * (size_t)std::max(s->nuvs, 1)),
               b_nrm = Workspace::round(16 * (size_t)std::max(s->nnormals, 1));
  int r = dalloc(ctx, &s->d_mesh, b_pts + b_uvs + b_nrm + 40 * (size_t)nfaces);
  if (!r) {
    s->d_points = (float4*)s->d_mesh;
    s->d_uvs = (float2*)(s->d_mesh + b_pts);
    s->d_normals = (float4*)(s->d_mesh + b_pts + b_uvs);
    s->d_faces = (Face*)(s->d_mesh + b_pts + b_uvs + b_nrm);
    cudaError_t e = cudaMemcpyAsync(s->d_points, points, 16 * (size_t)npoints, cudaMemcpyHostToDevice, ctx->stream);
    if (e == cudaSuccess && s->nuvs > 0)
      e = cudaMemcpyAsync(s->d_uvs, uvs, 8 * (size_t)s->nuvs, cudaMemcpyHostToDevice, ctx->stream);
    if (e == cudaSuccess && s->nnormals > 0)
      e = cudaMemcpyAsync(s->d_normals, normals, 16 * (size_t)s->nnormals, cudaMemcpyHostToDevice, ctx->stream);
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(s->d_faces, faces, 40 * (size_t)nfaces, cudaMemcpyHostToDevice, ctx->stream);
    if (e != cudaSuccess) r = fail(MT_ERR_CUDA, "mesh upload: %s", cudaGetErrorString(e));
  }
  int bad = INT_MAX;
  if (!r) r = first_bad_face(s, nmaterials, false, &bad);
  if (!r && bad < nfaces) {
    const Face& f = reinterpret_cast<const Face*>(faces)[bad];
    if (f.vx < 0 || f.vy < 0 || f.vz < 0 || f.vx >= npoints || f.vy >= npoints || f.vz >= npoints)
      r = fail(MT_ERR_INVALID, "face %d: vertex index out of range", bad);
    else if ((f.mat & 0xFFFF) >= nmaterials)
      r = fail(MT_ERR_INVALID, "face %d: material %d of %d", bad, f.mat & 0xFFFF, nmaterials);
    else if (f.uvx > -1 && (f.uvx >= s->nuvs || f.uvy < 0 || f.uvy >= s->nuvs || f.uvz < 0 || f.uvz >= s->nuvs))
      r = fail(MT_ERR_INVALID, "face %d: uv index out of range", bad);
    else
      r = fail(MT_ERR_INVALID, "face %d: normal index out of range", bad);
  }
  if (!r) r = upload(ctx, &s->d_materials, materials, (size_t)nmaterials);
  if (!r) r = upload_lights(s);
  if (r) {
    std::string keep = g_err;
    cudaStreamSynchronize(ctx->stream);  // the caller's arrays are no longer read
    free_scene(s);
    delete s;
    g_err = keep;
    return r;
  }
  *out = s;
  return MT_OK;
}

extern "C" int mt_scene_set_materials(mt_scene* s, const void* materials, int nmaterials) {
  if (!s || !materials || nmaterials <= 0) return fail(MT_ERR_INVALID, "bad argument");
  std::lock_guard<std::recursive_mutex> lk(s->ctx->mu);
  CU(cudaSetDevice(s->ctx->device));
  int q = quiesce(s->ctx);
  if (q) return q;
  int bad = INT_MAX;
  q = first_bad_face(s, nmaterials, true, &bad);
  if (q) return q;
  if (bad < s->ntri) {
    Face f;
    CU(cudaMemcpy(&f, s->d_faces + bad, sizeof(Face), cudaMemcpyDeviceToHost));
    return fail(MT_ERR_INVALID, "face %d needs material %d", bad, f.mat & 0xFFFF);
  }
  ++s->version;
  s->h_materials.assign((const uint8_t*)materials, (const uint8_t*)materials + 144 * (size_t)nmaterials);
  s->nmat = nmaterials;
  int r = upload(s->ctx, &s->d_materials, materials, (size_t)nmaterials);
  if (!r) r = upload_lights(s);
  if (!r) r = upload_textures(s);
  return r;
}

extern "C" int mt_scene_set_texture(mt_scene* s, int material, int kind, const int32_t* argb, int width,
                                    int height) {
  if (!s) return fail(MT_ERR_INVALID, "NULL scene");
  if (material < 0 || material >= s->nmat) return fail(MT_ERR_INVALID, "material %d of %d", material, s->nmat);
  if (kind < 0 || kind > 3) return fail(MT_ERR_INVALID, "texture kind %d (0 diffuse, 1 glossy, 2 roughness, 3 mirror)", kind);
  if (argb && (width <= 0 || height <= 0 || (long long)width * height > 0x7FFFFFFFll))
    return fail(MT_ERR_INVALID, "texture of %d x %d", width, height);
  std::lock_guard<std::recursive_mutex> lk(s->ctx->mu);
  CU(cudaSetDevice(s->ctx->device));
  int q = quiesce(s->ctx);
  if (q) return q;
  ++s->version;
  s->h_tex.resize(4 * (size_t)s->nmat);
  auto& t = s->h_tex[4 * (size_t)material + kind];
  if (argb) {
    t.argb.assign(argb, argb + (size_t)width * height);
    t.w = width;
    t.h = height;
  } else {
    t = mt_scene::HostTex{};
  }
  return upload_textures(s);
}

bool cdf_tables_enabled() {
  const char* v = std::getenv("MT_CDF_TABLES");
  return !(v && std::atoi(v) == 0);
}

extern "C" int mt_scene_light_count(const mt_scene* s) { return s ? s->nlights : -1; }

extern "C" int mt_scene_destroy(mt_scene* s) {
  if (!s) return fail(MT_ERR_INVALID, "NULL scene");
  if (s->refs.load() > 0) return fail(MT_ERR_BUSY, "scene used by %d served requests", s->refs.load());
  {
    std::lock_guard<std::recursive_mutex> lk(s->ctx->mu);
    cudaSetDevice(s->ctx->device);
    quiesce(s->ctx);
    free_scene(s);
  }
  delete s;
  return MT_OK;
}

// ---------------------------------------------------------------- BVH build
// CNormalBVH.build (src/cl/scene/CNormalBVH.java:45-148): recursive split at the
// centre of the centroid bound's longest axis, one triangle per leaf, children
// allocated as adjacent pairs in preorder, node.bound = node index. The
// partition (CNormalBVH.java:132) is an un-vendored library routine; this builder
// uses a stable split "centroid[dim] < split", falling back to the middle index
// when one side would be empty (CNormalBVH.java:135-136).
namespace {
struct Builder {
  const float* pts;
  const Face* faces;
  int n;
  std::vector<int> obj, tmp;
  std::vector<float> tb, cen;
  int32_t* nodes;   // 7 per node
  float* bounds;    // 8 per node
  int ptr = 1, max_depth = 0;

  void init() {
    obj.resize(n);
    tb.resize(6 * (size_t)n);
    cen.resize(3 * (size_t)n);
    for (int t = 0; t < n; ++t) {
      obj[t] = t;
      const Face& f = faces[t];
      const float* p[3] = {pts + 4 * (size_t)f.vx, pts + 4 * (size_t)f.vy, pts + 4 * (size_t)f.vz};
      for (int a = 0; a < 3; ++a) {
        float lo = INFINITY, hi = -INFINITY;
        for (int k = 0; k < 3; ++k) {
          if (p[k][a] < lo) lo = p[k][a];
          if (p[k][a] > hi) hi = p[k][a];
        }
        tb[6 * (size_t)t + a] = lo;
        tb[6 * (size_t)t + 3 + a] = hi;
        cen[3 * (size_t)t + a] = 0.5f * (lo + hi);
      }
    }
  }
  void subdivide(int parent, int start, int end, int depth) {
    // iterative on the right child to bound the C++ stack on deep trees
    for (;;) {
      max_depth = std::max(max_depth, depth);
      float bmn[3] = {INFINITY, INFINITY, INFINITY}, bmx[3] = {-INFINITY, -INFINITY, -INFINITY};
      float cmn[3] = {INFINITY, INFINITY, INFINITY}, cmx[3] = {-INFINITY, -INFINITY, -INFINITY};
      for (int p = start; p < end; ++p) {
        int t = obj[p];
        for (int a = 0; a < 3; ++a) {
          float lo = tb[6 * (size_t)t + a], hi = tb[6 * (size_t)t + 3 + a], c = cen[3 * (size_t)t + a];
          bmn[a] = std::min(bmn[a], lo);
          bmx[a] = std::max(bmx[a], hi);
          cmn[a] = std::min(cmn[a], c);
          cmx[a] = std::max(cmx[a], c);
        }
      }
      int32_t* nd = nodes + 7 * (size_t)parent;
      float* bd = bounds + 8 * (size_t)parent;
      nd[0] = parent;  // bound
      for (int a = 0; a < 3; ++a) {
        bd[a] = bmn[a];
        bd[4 + a] = bmx[a];
      }
      bd[3] = bd[7] = 0.f;
      if (end - start < 2) {
        nd[6] = obj[start];  // child
        nd[5] = 1;           // isLeaf
        return;
      }
      int li = ptr++, ri = ptr++;
      int32_t* ln = nodes + 7 * (size_t)li;
      int32_t* rn = nodes + 7 * (size_t)ri;
      std::memset(ln, 0, 28);
      std::memset(rn, 0, 28);
      ln[4] = parent;  // parent
      rn[4] = parent;
      ln[1] = ri;      // sibling
      rn[1] = li;
      nd[2] = li;      // left
      nd[3] = ri;      // right
      float ex = cmx[0] - cmn[0], ey = cmx[1] - cmn[1], ez = cmx[2] - cmn[2];
      int dim = (ex > ey && ex > ez) ? 0 : (ey > ez ? 1 : 2);
      float split = 0.5f * (cmn[dim] + cmx[dim]);
      int nl = 0;
      for (int p = start; p < end; ++p) nl += cen[3 * (size_t)obj[p] + dim] < split;
      int mid = start + nl;
      if (mid != start && mid != end) {
        tmp.resize(end - start);
        int a = start, b = 0;
        for (int p = start; p < end; ++p) {
          int t = obj[p];
          if (cen[3 * (size_t)t + dim] < split) obj[a++] = t;
          else tmp[b++] = t;
        }
        std::memcpy(obj.data() + mid, tmp.data(), sizeof(int) * (size_t)b);
      } else {
        mid = start + (end - start) / 2;
      }
      subdivide(li, start, mid, depth + 1);
      parent = ri;
      start = mid;
      depth = depth + 1;
    }
  }
};

// Convert the reference node layout into the traversal layout and upload it.
int import_bvh(mt_scene* s, const int32_t* nodes, const float* bounds, int nnodes) {
  const int n = s->ntri;
  if (nnodes != 2 * n - 1) return fail(MT_ERR_INVALID, "%d nodes for %d triangles (want 2N-1)", nnodes, n);
  auto node = [&](int i) { return nodes + 7 * (size_t)i; };
  // A breadth-first pass checks the tree and its depth; a depth-first pass (left
  // before right) numbers the interior records in preorder and the leaf slots
  // in leaf order.
  std::vector<int> rec(nnodes, -1), slot(nnodes, -1), level(nnodes, 0);
  std::vector<int> order;
  order.reserve(n);
  const int32_t* root = node(0);
  int max_level = 0;
  if (!root[5]) {
    std::deque<int> q;
    q.push_back(0);
    int k = 0;
    std::vector<char> seen(nnodes, 0);
    seen[0] = 1;
    while (!q.empty()) {
      int i = q.front();
      q.pop_front();
      const int32_t* nd = node(i);
      for (int c : {nd[2], nd[3]}) {
        if (c <= 0 || c >= nnodes || seen[c]) return fail(MT_ERR_INVALID, "node %d: bad child %d", i, c);
        seen[c] = 1;
        const int32_t* cn = node(c);
        if (cn[0] < 0 || cn[0] >= nnodes) return fail(MT_ERR_INVALID, "node %d: bad bound index %d", c, cn[0]);
        level[c] = level[i] + 1;
        max_level = std::max(max_level, level[c]);
        if (!cn[5]) q.push_back(c);
        else if (cn[6] < 0 || cn[6] >= n) return fail(MT_ERR_INVALID, "leaf %d: bad triangle %d", c, cn[6]);
      }
    }
    std::vector<int> st{0};
    while (!st.empty()) {
      int i = st.back();
      st.pop_back();
      const int32_t* nd = node(i);
      if (nd[5]) {
        slot[i] = (int)order.size();
        order.push_back(nd[6]);
        continue;
      }
      rec[i] = k++;
      st.push_back(nd[3]);
      st.push_back(nd[2]);
    }
  } else {
    if (root[6] < 0 || root[6] >= n) return fail(MT_ERR_INVALID, "root leaf: bad triangle");
    slot[0] = 0;
    order.push_back(root[6]);
  }
  // Deferred-node stack depth needed <= tree depth; the reference's bitstack holds 64 levels.
  if (max_level > kStackDepth) return fail(MT_ERR_DEPTH, "BVH depth %d exceeds %d", max_level, kStackDepth);
  const int nrec = root[5] ? 0 : n - 1;
  std::vector<float4> hn(4 * (size_t)std::max(nrec, 1));
  auto ref_of = [&](int c) { return node(c)[5] ? ~slot[c] : rec[c]; };
  for (int i = 0; i < nnodes; ++i) {
    if (rec[i] < 0) continue;
    const int32_t* nd = node(i);
    const float* bl = bounds + 8 * (size_t)node(nd[2])[0];
    const float* br = bounds + 8 * (size_t)node(nd[3])[0];
    float4* r = hn.data() + 4 * (size_t)rec[i];
    r[0] = make_float4(bl[0], bl[4], bl[1], bl[5]);
    r[1] = make_float4(br[0], br[4], br[1], br[5]);
    r[2] = make_float4(bl[2], bl[6], br[2], br[6]);
    int lr = ref_of(nd[2]), rr = ref_of(nd[3]);
    float lf, rf;
    std::memcpy(&lf, &lr, 4);
    std::memcpy(&rf, &rr, 4);
    r[3] = make_float4(lf, rf, 0.f, 0.f);
  }
  if ((int)order.size() != n) return fail(MT_ERR_INVALID, "BVH reaches %zu of %d triangles", order.size(), n);
  // The new tree beside the old one, which stays when this fails, or, where both do not
  // fit, in its place.
  float4 *recs = nullptr, *tris = nullptr;
  auto make = [&] {
    int r = upload(s->ctx, &recs, hn.data(), hn.size());
    if (!r) r = dalloc(s->ctx, &tris, 3 * (size_t)n);
    if (!r) r = order_triangles(s, order, tris);
    if (r) {
      dfree(recs);
      dfree(tris);
    }
    return r;
  };
  int r = make();
  if (r == MT_ERR_NOMEM && s->has_bvh) {
    s->has_bvh = 0;  // until the new one is there, nothing is rendered
    dfree(s->d_nodes);
    dfree(s->d_tris);
    r = make();
  }
  if (r) return r;
  dfree(s->d_nodes);
  dfree(s->d_tris);
  s->d_nodes = recs;
  s->d_tris = tris;
  s->nrec = nrec;
  s->root_ref = root[5] ? ~0 : 0;
  s->depth = max_level;
  s->has_bvh = 1;
  return MT_OK;
}
}  // namespace

extern "C" int mt_bvh_build(mt_scene* s, int32_t* nodes_out, float* bounds_out, int* depth_out) {
  if (!s) return fail(MT_ERR_INVALID, "NULL scene");
  const int n = s->ntri;
  std::vector<int32_t> nodes(7 * (size_t)(2 * n - 1), 0);
  std::vector<float> bounds(8 * (size_t)(2 * n - 1), 0.f);
  std::vector<float> points(4 * (size_t)s->npoints);
  std::vector<Face> faces((size_t)n);
  {
    std::lock_guard<std::recursive_mutex> lk(s->ctx->mu);
    CU(cudaSetDevice(s->ctx->device));
    CU(cudaMemcpy(points.data(), s->d_points, points.size() * 4, cudaMemcpyDeviceToHost));
    CU(cudaMemcpy(faces.data(), s->d_faces, faces.size() * sizeof(Face), cudaMemcpyDeviceToHost));
  }
  Builder b;
  b.pts = points.data();
  b.faces = faces.data();
  b.n = n;
  b.nodes = nodes.data();
  b.bounds = bounds.data();
  b.init();
  b.subdivide(0, 0, n, 0);
  if (nodes_out) std::memcpy(nodes_out, nodes.data(), nodes.size() * 4);
  if (bounds_out) std::memcpy(bounds_out, bounds.data(), bounds.size() * 4);
  if (depth_out) *depth_out = b.max_depth;
  std::lock_guard<std::recursive_mutex> lk(s->ctx->mu);
  CU(cudaSetDevice(s->ctx->device));
  int q = quiesce(s->ctx);
  if (q) return q;
  ++s->version;
  int r = import_bvh(s, nodes.data(), bounds.data(), 2 * n - 1);
  return r ? r : refresh_qnodes(s);
}

extern "C" int mt_bvh_build_host(const float* points, int npoints, const int32_t* faces, int nfaces,
                                 int32_t* nodes_out, float* bounds_out, int* depth_out) {
  if (!points || !faces || !nodes_out || !bounds_out || npoints <= 0 || nfaces <= 0)
    return fail(MT_ERR_INVALID, "bad argument");
  const Face* F = reinterpret_cast<const Face*>(faces);
  for (int i = 0; i < nfaces; ++i)
    if (F[i].vx < 0 || F[i].vy < 0 || F[i].vz < 0 || F[i].vx >= npoints || F[i].vy >= npoints || F[i].vz >= npoints)
      return fail(MT_ERR_INVALID, "face %d: vertex index out of range", i);
  std::memset(nodes_out, 0, 28 * (size_t)(2 * nfaces - 1));
  std::memset(bounds_out, 0, 32 * (size_t)(2 * nfaces - 1));
  Builder b;
  b.pts = points;
  b.faces = F;
  b.n = nfaces;
  b.nodes = nodes_out;
  b.bounds = bounds_out;
  b.init();
  b.subdivide(0, 0, nfaces, 0);
  if (depth_out) *depth_out = b.max_depth;
  return MT_OK;
}

extern "C" int mt_scene_layout_read(mt_scene* s, void* records_out, void* tris_out, int* nrec_out,
                                    int* root_ref_out) {
  if (!s) return fail(MT_ERR_INVALID, "NULL scene");
  if (!s->has_bvh) return fail(MT_ERR_INVALID, "scene has no BVH");
  std::lock_guard<std::recursive_mutex> lk(s->ctx->mu);
  CU(cudaSetDevice(s->ctx->device));
  CU(cudaStreamSynchronize(s->ctx->stream));
  if (records_out && s->nrec) CU(cudaMemcpy(records_out, s->d_nodes, 64 * (size_t)s->nrec, cudaMemcpyDeviceToHost));
  if (tris_out) CU(cudaMemcpy(tris_out, s->d_tris, 48 * (size_t)s->ntri, cudaMemcpyDeviceToHost));
  if (nrec_out) *nrec_out = s->nrec;
  if (root_ref_out) *root_ref_out = s->root_ref;
  return MT_OK;
}

extern "C" int mt_bvh_import(mt_scene* s, const int32_t* nodes, const float* bounds, int nnodes) {
  if (!s || !nodes || !bounds) return fail(MT_ERR_INVALID, "NULL argument");
  std::lock_guard<std::recursive_mutex> lk(s->ctx->mu);
  CU(cudaSetDevice(s->ctx->device));
  int q = quiesce(s->ctx);
  if (q) return q;
  ++s->version;
  int r = import_bvh(s, nodes, bounds, nnodes);
  return r ? r : refresh_qnodes(s);
}

extern "C" int mt_scene_set_bvh_precision(mt_scene* s, int precision) {
  if (!s) return fail(MT_ERR_INVALID, "NULL scene");
  if (precision < 0 || precision > 3)
    return fail(MT_ERR_INVALID, "BVH precision %d (0 FP32, 1 FP16, 2 wide 8-bit, 3 4-wide FP16)", precision);
  std::lock_guard<std::recursive_mutex> lk(s->ctx->mu);
  CU(cudaSetDevice(s->ctx->device));
  int q = quiesce(s->ctx);
  if (q) return q;
  ++s->version;
  s->precision = precision;
  return refresh_qnodes(s);
}

// -------------------------------------------------------------- environment
extern "C" int mt_env_set(mt_scene* s, const float* rgb, int w, int h) {
  if (!s || !rgb || w <= 0 || h <= 0) return fail(MT_ERR_INVALID, "bad environment map");
  std::lock_guard<std::recursive_mutex> lk(s->ctx->mu);
  CU(cudaSetDevice(s->ctx->device));
  int q = quiesce(s->ctx);
  if (q) return q;
  ++s->version;
  s->env_present = 0;
  int r = alloc_env(s, w, h, true);
  if (r) return r;
  CU(cudaMemcpyAsync(s->d_env_rgb, rgb, 16 * (size_t)w * h, cudaMemcpyHostToDevice, s->ctx->stream));
  if (launch_env_build(s->ctx->stream, s->d_env_rgb, w, h, s->d_env_lum, s->d_env_sat64, s->d_env_sat))
    return fail(MT_ERR_CUDA, "environment build launch: %s", cudaGetErrorString(cudaGetLastError()));
  if ((r = build_env_tables(s))) return r;
  CU(cudaStreamSynchronize(s->ctx->stream));
  s->env_present = 1;
  return MT_OK;
}

extern "C" int mt_env_set_with_sat(mt_scene* s, const float* rgb, const float* lum, const float* sat, int w, int h) {
  if (!s || !rgb || !lum || !sat || w <= 0 || h <= 0) return fail(MT_ERR_INVALID, "bad environment map");
  std::lock_guard<std::recursive_mutex> lk(s->ctx->mu);
  CU(cudaSetDevice(s->ctx->device));
  int q = quiesce(s->ctx);
  if (q) return q;
  ++s->version;
  s->env_present = 0;
  int r = alloc_env(s, w, h, false);
  if (r) return r;
  const size_t n = (size_t)w * h;
  CU(cudaMemcpyAsync(s->d_env_rgb, rgb, 16 * n, cudaMemcpyHostToDevice, s->ctx->stream));
  CU(cudaMemcpyAsync(s->d_env_lum, lum, 4 * n, cudaMemcpyHostToDevice, s->ctx->stream));
  CU(cudaMemcpyAsync(s->d_env_sat, sat, 4 * n, cudaMemcpyHostToDevice, s->ctx->stream));
  if ((r = build_env_tables(s))) return r;
  CU(cudaStreamSynchronize(s->ctx->stream));
  s->env_present = 1;
  return MT_OK;
}

extern "C" int mt_env_clear(mt_scene* s) {
  if (!s) return fail(MT_ERR_INVALID, "NULL scene");
  std::lock_guard<std::recursive_mutex> lk(s->ctx->mu);
  CU(cudaSetDevice(s->ctx->device));
  int q = quiesce(s->ctx);
  if (q) return q;
  ++s->version;
  s->env_present = 0;
  return MT_OK;
}

extern "C" int mt_env_read(mt_scene* s, float* lum, double* sat64, float* sat32) {
  if (!s || !s->env_present) return fail(MT_ERR_INVALID, "no environment map");
  std::lock_guard<std::recursive_mutex> lk(s->ctx->mu);
  CU(cudaSetDevice(s->ctx->device));
  CU(cudaStreamSynchronize(s->ctx->stream));
  size_t n = (size_t)s->env_w * s->env_h;
  if (lum) CU(cudaMemcpy(lum, s->d_env_lum, n * 4, cudaMemcpyDeviceToHost));
  if (sat32) CU(cudaMemcpy(sat32, s->d_env_sat, n * 4, cudaMemcpyDeviceToHost));
  if (sat64) {
    if (!s->d_env_sat64) return fail(MT_ERR_INVALID, "the SAT was given, not built in FP64");
    CU(cudaMemcpy(sat64, s->d_env_sat64, n * 8, cudaMemcpyDeviceToHost));
  }
  return MT_OK;
}

extern "C" int mt_env_grid_config(mt_scene* s, int nu, int nv, int rx, int ry, int enable) {
  if (!s || nu <= 0 || nv <= 0 || nu % rx || nv % ry || enable < 0 || enable > 2) return fail(MT_ERR_INVALID, "bad grid");
  if (!((rx == 8 || rx == 16 || rx == 32) && (ry == 8 || ry == 16 || ry == 32)))
    return fail(MT_ERR_INVALID, "tiles per cell must be 8, 16 or 32 along each axis");
  if ((long long)nu * nv > (1ll << 28)) return fail(MT_ERR_INVALID, "grid of %d x %d is too large", nu, nv);
  std::lock_guard<std::recursive_mutex> lk(s->ctx->mu);
  CU(cudaSetDevice(s->ctx->device));
  int q = quiesce(s->ctx);
  if (q) return q;
  ++s->version;
  s->grid_nu = nu;
  s->grid_nv = nv;
  s->grid_rx = rx;
  s->grid_ry = ry;
  s->grid_on = enable;
  return MT_OK;
}

extern "C" int mt_env_grid_sat(mt_context* ctx, const float* func, float* sat_out, int nu, int nv, int rx, int ry,
                               int fp64) {
  if (!ctx || !func || !sat_out || nu <= 0 || nv <= 0) return fail(MT_ERR_INVALID, "bad argument");
  if (!((rx == 8 || rx == 16 || rx == 32) && (ry == 8 || ry == 16 || ry == 32)) || nu % rx || nv % ry)
    return fail(MT_ERR_INVALID, "tiles per cell must be 8, 16 or 32 and divide the grid");
  std::lock_guard<std::recursive_mutex> lk(ctx->mu);
  CU(cudaSetDevice(ctx->device));
  size_t n = (size_t)nu * nv;
  float *d_func = nullptr, *d_sat = nullptr;
  double* d_sat64 = nullptr;
  int r = dalloc(ctx, &d_func, n);
  if (!r) r = dalloc(ctx, &d_sat, n);
  if (!r && fp64) r = dalloc(ctx, &d_sat64, n);
  if (!r) {
    cudaMemcpyAsync(d_func, func, n * 4, cudaMemcpyHostToDevice, ctx->stream);
    if (launch_grid_sat(ctx->stream, d_func, d_sat, d_sat64, nu, nv, rx, ry, fp64))
      r = fail(MT_ERR_CUDA, "grid SAT launch failed");
    else if (cudaMemcpyAsync(sat_out, d_sat, n * 4, cudaMemcpyDeviceToHost, ctx->stream) != cudaSuccess ||
             cudaStreamSynchronize(ctx->stream) != cudaSuccess)
      r = fail(MT_ERR_CUDA, "grid SAT copy: %s", cudaGetErrorString(cudaGetLastError()));
  }
  dfree(d_func);
  dfree(d_sat);
  dfree(d_sat64);
  return r;
}

// ------------------------------------------------------------- ray queries
namespace {
int query(mt_scene* s, const void* rays, int n, int any, float* t_out, int32_t* prim_out,
          int32_t* counts_out = nullptr) {
  if (!s || (!rays && n) || !prim_out || (!any && !t_out) || n < 0) return fail(MT_ERR_INVALID, "bad argument");
  if (!s->has_bvh) return fail(MT_ERR_INVALID, "scene has no BVH");
  if (n == 0) return MT_OK;
  mt_context* ctx = s->ctx;
  std::lock_guard<std::recursive_mutex> lk(ctx->mu);
  CU(cudaSetDevice(ctx->device));
  const size_t bytes = Workspace::round(80 * (size_t)n) + 2 * Workspace::round(4 * (size_t)n) +
                       (counts_out ? Workspace::round(8 * (size_t)n) : 0);
  Workspace ws;
  int r = ws.get(ctx, bytes);
  if (r) return r;
  float4* d_rays = ws.take<float4>(5 * (size_t)n);
  float* d_t = ws.take<float>((size_t)n);
  int* d_p = ws.take<int>((size_t)n);
  int* d_c = counts_out ? ws.take<int>(2 * (size_t)n) : nullptr;
  cudaMemcpyAsync(d_rays, rays, 80 * (size_t)n, cudaMemcpyHostToDevice, ctx->stream);
  cudaMemsetAsync(ctx->d_scratch, 0, 8, ctx->stream);
  const int lr = counts_out ? launch_count(ctx->stream, s->view(), d_rays, n, any, d_t, d_p, d_c, ctx->d_scratch + 1)
                            : launch_query(ctx->stream, s->view(), d_rays, n, any, d_t, d_p, ctx->d_scratch,
                                           ctx->d_scratch + 1, ctx->num_sms);
  if (lr) r = fail(MT_ERR_CUDA, "query launch: %s", cudaGetErrorString(cudaGetLastError()));
  int err = 0;
  if (!r) {
    cudaEventRecord(ctx->ready, ctx->stream);
    if (!any) prefault(t_out, 4 * (size_t)n, ctx->ready);
    prefault(prim_out, 4 * (size_t)n, ctx->ready);
    if (!any) cudaMemcpyAsync(t_out, d_t, 4 * (size_t)n, cudaMemcpyDeviceToHost, ctx->stream);
    cudaMemcpyAsync(prim_out, d_p, 4 * (size_t)n, cudaMemcpyDeviceToHost, ctx->stream);
    if (counts_out) cudaMemcpyAsync(counts_out, d_c, 8 * (size_t)n, cudaMemcpyDeviceToHost, ctx->stream);
    cudaMemcpyAsync(&err, ctx->d_scratch + 1, 4, cudaMemcpyDeviceToHost, ctx->stream);
  }
  const cudaError_t e = cudaStreamSynchronize(ctx->stream);
  if (!r && e != cudaSuccess) r = fail(MT_ERR_CUDA, "query: %s", cudaGetErrorString(e));
  else if (!r && err) r = fail(MT_ERR_DEVICE, "device error %d", err);
  ws.release();
  return r;
}
}  // namespace

extern "C" int mt_trace_counts(mt_scene* s, const void* rays, int n, int any, float* t_out, int32_t* prim_out,
                               int32_t* counts_out) {
  if (!counts_out) return fail(MT_ERR_INVALID, "NULL counts");
  return query(s, rays, n, any ? 1 : 0, any ? nullptr : t_out, prim_out, counts_out);
}

extern "C" int mt_trace_closest(mt_scene* s, const void* rays, int n, float* t_out, int32_t* prim_out) {
  return query(s, rays, n, 0, t_out, prim_out);
}

extern "C" int mt_tuning_get(mt_tuning* out) {
  if (!out) return fail(MT_ERR_INVALID, "NULL argument");
  const Tuning t = get_tuning();
  *out = mt_tuning{t.closest_minb, t.shadow_minb, t.closest_grid, t.shadow_grid, t.shade_minb, t.refill_steps,
                   t.shadow_stream};
  return MT_OK;
}

extern "C" int mt_tuning_set(const mt_tuning* in) {
  if (!in) return fail(MT_ERR_INVALID, "NULL argument");
  const Tuning t{in->closest_minb, in->shadow_minb, in->closest_grid, in->shadow_grid,
                 in->shade_minb,   in->refill_steps, in->shadow_stream};
  if (!set_tuning(t))
    return fail(MT_ERR_INVALID, "tuning out of range: minb %d/%d (8, 12, 16), grids %d/%d (0..32), shade %d (3..5), "
                                "steps %d (4..1024), shadow_stream %d (0, 1)",
                t.closest_minb, t.shadow_minb, t.closest_grid, t.shadow_grid, t.shade_minb, t.refill_steps,
                t.shadow_stream);
  return MT_OK;
}

extern "C" int mt_trace_any(mt_scene* s, const void* rays, int n, int32_t* occluded_out) {
  return query(s, rays, n, 1, nullptr, occluded_out);
}

extern "C" int mt_trace_closest_dev(mt_scene* s, mt_buffer* rays, int n, mt_buffer* t_out, mt_buffer* prim_out,
                                    float* ms_out) {
  if (!s || !rays || !t_out || !prim_out || n < 0) return fail(MT_ERR_INVALID, "bad argument");
  if (rays->bytes < 80 * (size_t)n || t_out->bytes < 4 * (size_t)n || prim_out->bytes < 4 * (size_t)n)
    return fail(MT_ERR_INVALID, "buffers too small for %d rays", n);
  mt_context* ctx = s->ctx;
  std::lock_guard<std::recursive_mutex> lk(ctx->mu);
  CU(cudaSetDevice(ctx->device));
  cudaEvent_t a, b;
  CU(cudaEventCreate(&a));
  CU(cudaEventCreate(&b));
  cudaMemsetAsync(ctx->d_scratch, 0, 8, ctx->stream);
  cudaEventRecord(a, ctx->stream);
  int r = launch_query(ctx->stream, s->view(), (const float4*)rays->ptr, n, 0, (float*)t_out->ptr, (int*)prim_out->ptr,
                       ctx->d_scratch, ctx->d_scratch + 1, ctx->num_sms);
  cudaEventRecord(b, ctx->stream);
  cudaError_t e = cudaEventSynchronize(b);
  float ms = 0;
  cudaEventElapsedTime(&ms, a, b);
  cudaEventDestroy(a);
  cudaEventDestroy(b);
  if (r || e != cudaSuccess) return fail(MT_ERR_CUDA, "trace: %s", cudaGetErrorString(cudaGetLastError()));
  if (ms_out) *ms_out = ms;
  return MT_OK;
}

// ------------------------------------------------- kernels by name (stubs)
// ------------------------------------------------------------- compaction
extern "C" int mt_compact_isects(mt_context* ctx, const void* isects_in, const int32_t* pixels_in, int n,
                                 void* isects_out, int32_t* pixels_out, int32_t* count_io) {
  if (!ctx || n < 0 || (n > 0 && (!isects_in || !pixels_in || !isects_out || !pixels_out)) || !count_io)
    return fail(MT_ERR_INVALID, "bad argument");
  if (n > (1 << 30)) return fail(MT_ERR_INVALID, "n = %d exceeds 2^30", n);
  std::lock_guard<std::recursive_mutex> lk(ctx->mu);
  CU(cudaSetDevice(ctx->device));
  const size_t tiles = (size_t)(n + kCompactThreads - 1) / kCompactThreads;
  if (tiles > ctx->cs_tiles || !ctx->cs_words) {
    CU(cudaStreamSynchronize(ctx->stream));
    dfree(ctx->cs_status);
    dfree(ctx->cs_words);
    ctx->cs_tiles = 0;
    int r = dalloc(ctx, &ctx->cs_status, tiles ? tiles : 1);
    if (!r) r = dalloc(ctx, &ctx->cs_words, 4);
    if (r) return r;
    ctx->cs_tiles = tiles ? tiles : 1;
  }
  const cudaError_t le = launch_compact_isects(ctx->stream, isects_in, pixels_in, n, isects_out, pixels_out,
                                               count_io, CompactScratch{ctx->cs_status, ctx->cs_words});
  if (le != cudaSuccess) return fail(MT_ERR_CUDA, "compaction launch: %s", cudaGetErrorString(le));
  int err = 0;
  CU(cudaMemcpyAsync(&err, ctx->cs_words + 2, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
  CU(cudaStreamSynchronize(ctx->stream));
  if (err) return fail(MT_ERR_DEVICE, "compaction: device error %d", err);
  return MT_OK;
}

extern "C" void* mt_buf_device_ptr(mt_buffer* b) { return b ? b->ptr : nullptr; }

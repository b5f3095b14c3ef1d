// The preview device's frame in one launch: CDeviceRT.loop
// (src/cl/device/CDeviceRT.java:176-197) runs InitCameraRayData,
// IntersectPrimitives, SetupBSDFRaytrace, backgroundShade, fastShade and
// updateGroupbufferShadeImage (src/cl/kernel/Raytrace.cl) one launch each; here
// a persistent traversal kernel generates each pixel's unjittered camera ray,
// finds its closest hit on the scene's traversal layout and writes the quick
// colour (emission, or diffuse colour x the cosine to the camera) or the gamma-2.2
// environment texel, and the material group, directly.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>

#include "mt_device.cuh"
#include "mt_internal.h"
#include "mt_traverse.cuh"

namespace mt {
namespace {

using namespace dv;

__device__ __forceinline__ int pack_argb(float r, float g, float b, float a) {  // getIntARGB, Util.cl:469-480
  auto q = [](float v) { return (int)(fminf(fmaxf(v, 0.f), 1.f) * 255.0f); };
  return (q(a) << 24) | (q(r) << 16) | (q(g) << 8) | q(b);
}

struct CameraRays {  // InitCameraRayData (Raytrace.cl:1-31)
  PassParams pp;
  __device__ __forceinline__ tr::RayT operator()(int i) const {
    const int id = tile_pixel(i, pp.width, pp.height);
    const int W = pp.width;
    const float px = (float)(id % W), py = (float)(id / W);
    V d = normalize4(mk(pp.cam_a * (2.f * px / pp.dim_w - 1.f), -2.f * py / pp.dim_h + 1.f, -pp.cam_d, 0.f));
    const float* m = pp.cam_m;
    V z = zero4();
    V m0 = mk(m[0], m[1], m[2], m[3]), m1 = mk(m[4], m[5], m[6], m[7]), m2 = mk(m[8], m[9], m[10], m[11]),
      m3 = mk(m[12], m[13], m[14], m[15]);
    V o = mk(dot3(m0, z) + m0.w, dot3(m1, z) + m1.w, dot3(m2, z) + m2.w, dot3(m3, z) + m3.w);
    if (!(o.w == 1.f)) o = mk(o.x / o.w, o.y / o.w, o.z / o.w, 0.f);
    V dw = mk(dot4(m0, d), dot4(m1, d), dot4(m2, d), 0.f);
    return tr::make_ray(make_float4(o.x, o.y, o.z, 0.f), make_float4(dw.x, dw.y, dw.z, 0.f), 0.001f, CUDART_INF_F);
  }
};

struct PreviewOut {  // setupBsdf's cosine, fastShade, backgroundShade, group
  DevScene S;
  DevEnv E;
  int* argb;
  int* group;
  int width, height;
  __device__ __forceinline__ void operator()(int i, const tr::RayT& r, int hit) const {
    const int id = tile_pixel(i, width, height);
    const V d = mk(r.dx, r.dy, r.dz, 0.f);
    if (hit >= 0) {
      Hit H;
      hit_record(S, mk(r.ox, r.oy, r.oz, 0.f), d, r.tmax, hit, H);
      const Frame f = get_frame(H.n);
      const float coeff = local_coord(f, neg(d)).z;
      const Material& P = S.materials[H.mat];
      const float4 ec = P.emission_color;
      float4 dc = P.diffuse_color;
      // textureInitPassRT, CTextureApplyPass.process, updateToTextureColorRT
      // (Raytrace.cl:52-145): the quick colour takes the diffuse texel at the hit's uv
      if (S.tex_on && P.isDiffuseTexture && !is_emitter(P)) {
        const int4 t = __ldg(S.tex_ref + 4 * (size_t)H.mat);
        dc = argb_float4(t.y > 0 ? tex_fetch(S.texels, t, H.u, H.v) : 0);
      }
      const V c = is_emitter(P) ? mk(ec.x, ec.y, ec.z, ec.w) : muls(mk(dc.x, dc.y, dc.z, dc.w), coeff);
      argb[id] = pack_argb(c.x, c.y, c.z, 1.f);
      if (group) group[id] = H.mat;
    } else {
      if (E.present) {
        int x, y;
        sph_xy(E.w, E.h, d, &x, &y);
        const float4 e = E.rgb[sph_index(E.w, E.h, x, y)];
        const float ig = 1.f / 2.2f;
        argb[id] = pack_argb(powf(e.x, ig), powf(e.y, ig), powf(e.z, ig), e.w);
      } else {
        argb[id] = pack_argb(0.f, 0.f, 0.f, 1.f);
      }
      if (group) group[id] = -1;
    }
  }
};

template <int MINB>
__global__ void __launch_bounds__(kTraceThreads, MINB)
    k_preview(DevScene S, DevEnv E, PassParams pp, int n, int* argb, int* group, int* work, int* err) {
  bool overflow = false;
  tr::trace_persistent<false, 32>(S, n, work, CameraRays{pp}, PreviewOut{S, E, argb, group, pp.width, pp.height}, &overflow);
  if (overflow) atomicExch(err, kDevErrStack);
}

}  // namespace
}  // namespace mt

extern "C" int mt_preview_frame(mt_scene* s, const void* camera, int width, int height, int32_t* argb,
                                int32_t* group) {
  if (!s || !camera || !argb) return fail(MT_ERR_INVALID, "NULL argument");
  if (width <= 0 || height <= 0 || (long long)width * height > (1ll << 28))
    return fail(MT_ERR_INVALID, "frame %d x %d", width, height);
  if (!s->has_bvh) return fail(MT_ERR_INVALID, "scene has no BVH");
  mt_context* ctx = s->ctx;
  std::lock_guard<std::recursive_mutex> lk(ctx->mu);
  CU(cudaSetDevice(ctx->device));
  join_jobs(ctx);
  const int n = width * height;
  PassParams pp{};
  camera_constants(camera, width, height, pp);
  pp.width = width;
  pp.height = height;
  Workspace ws;
  if (int r = ws.get(ctx, 2 * Workspace::round((size_t)n * 4))) return r;
  int* d_argb = ws.take<int>((size_t)n);
  int* d_group = group ? ws.take<int>((size_t)n) : nullptr;
  cudaError_t e = cudaMemsetAsync(ctx->d_scratch, 0, 8, ctx->stream);
  // Built for 12 blocks per SM where the rays fill them (40 registers, more warps to
  // hide reads: 1920 x 1080 over 1M triangles 2.02 -> 1.91 ms), for 8 otherwise (300 x 200
  // over 300k 291 -> 282 us). A small frame's rays are spread down to 4 a warp
  // (trace_persistent): 200 x 100 over 300k triangles 290 -> 211 us; from 600 x 400 on the
  // grid is full.
  constexpr int kRaysPerBlock = 4 * (kTraceThreads / 32);
  const bool big = n >= ctx->num_sms * 12 * kTraceThreads;
  int bps = 0;
  if (big) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, mt::k_preview<12>, kTraceThreads, 0);
  else cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, mt::k_preview<8>, kTraceThreads, 0);
  const int grid = std::max(1, std::min(ctx->num_sms * std::max(bps, 1), (n + kRaysPerBlock - 1) / kRaysPerBlock));
  if (big)
    mt::k_preview<12><<<grid, kTraceThreads, 0, ctx->stream>>>(s->view(), s->env_view(), pp, n, d_argb, d_group,
                                                               ctx->d_scratch, ctx->d_scratch + 1);
  else
    mt::k_preview<8><<<grid, kTraceThreads, 0, ctx->stream>>>(s->view(), s->env_view(), pp, n, d_argb, d_group,
                                                              ctx->d_scratch, ctx->d_scratch + 1);
  if (e == cudaSuccess) e = cudaGetLastError();
  int err = 0;
  if (e == cudaSuccess) e = cudaEventRecord(ctx->ready, ctx->stream);
  if (e == cudaSuccess) {
    prefault(argb, (size_t)n * 4, ctx->ready);
    if (group) prefault(group, (size_t)n * 4, ctx->ready);
  }
  if (e == cudaSuccess) e = cudaMemcpyAsync(argb, d_argb, (size_t)n * 4, cudaMemcpyDeviceToHost, ctx->stream);
  if (e == cudaSuccess && group)
    e = cudaMemcpyAsync(group, d_group, (size_t)n * 4, cudaMemcpyDeviceToHost, ctx->stream);
  if (e == cudaSuccess) e = cudaMemcpyAsync(&err, ctx->d_scratch + 1, 4, cudaMemcpyDeviceToHost, ctx->stream);
  const cudaError_t w = cudaStreamSynchronize(ctx->stream);
  ws.release();
  if (e == cudaSuccess) e = w;
  if (e != cudaSuccess) return fail(MT_ERR_CUDA, "preview: %s", cudaGetErrorString(e));
  if (err) return fail(MT_ERR_DEPTH, "BVH deeper than the traversal stack");
  return MT_OK;
}

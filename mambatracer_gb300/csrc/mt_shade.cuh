// The per-path work of a frame: camera ray, hit shading, light and BSDF samples,
// film adds.
#pragma once
#include <cuda_runtime.h>

#include "mt_device.cuh"
#include "mt_kernels.h"

namespace mt {

using namespace dv;

__device__ __forceinline__ void film_add(float4* __restrict__ acc, float4* __restrict__ comp, int pixel, V v, int kahan) {
  if (!abs_valid4(v)) return;  // addAccum, src/cl/kernel/Render.cl:1-7
  V a = acc[pixel];
  if (!kahan) {
    acc[pixel] = add(a, v);
    return;
  }
  V c = comp[pixel];
  V y = sub(v, c);
  V t = add(a, y);
  comp[pixel] = sub(sub(t, a), y);
  acc[pixel] = t;
}

// A contribution of path g to pixel f: added to the film, or kept in the pass's log,
// from which k_replay adds it once the passes before have been added. Either way a
// pixel's sums see the same values in the same order.
__device__ __forceinline__ void contribute(const FrameBufs& fb, int g, int f, V v, int kahan) {
  if (!fb.log) {
    film_add(fb.film, fb.film_c, f, v, kahan);
  } else if (abs_valid4(v)) {
    const int k = fb.log_n[g];
    fb.log[(size_t)k * fb.log_stride + g] = v;
    fb.log_n[g] = k + 1;
  }
}

// The camera ray of pixel id (InitCameraRayDataJitter): origin, world direction.
__device__ __forceinline__ void camera_ray(const PassParams* __restrict__ pp, int id, V* o_out, V* d_out) {
  int32_t sx, sy;
  if (pp->mode == 0) {
    sx = pp->seeds[0];
    sy = pp->seeds[1];
  } else {
    stage_seed(0, 0, &sx, &sy);
  }
  Seed s = gen_seed(sx, sy, pp->frame_count, pp->mode == 0 ? id : pixel_gid(id));
  float r0 = rnd(s), r1 = rnd(s);
  const int W = pp->width;
  float px = (float)(id % W), py = (float)(id / W);
  float j1 = pp->inv_w * (2.f * r0 - 1.f);
  float j2 = pp->inv_h * (2.f * r1 - 1.f);
  V d = normalize4(mk(pp->cam_a * (2.f * px / pp->dim_w - 1.f + j1), -2.f * py / pp->dim_h + 1.f + j2, -pp->cam_d, 0.f));
  const float* m = pp->cam_m;
  V z = zero4();
  V m0 = mk(m[0], m[1], m[2], m[3]), m1 = mk(m[4], m[5], m[6], m[7]), m2 = mk(m[8], m[9], m[10], m[11]),
    m3 = mk(m[12], m[13], m[14], m[15]);
  V o = mk(dot3(m0, z) + m0.w, dot3(m1, z) + m1.w, dot3(m2, z) + m2.w, dot3(m3, z) + m3.w);
  if (!(o.w == 1.f)) o = mk(o.x / o.w, o.y / o.w, o.z / o.w, 0.f);
  V dw = mk(dot4(m0, d), dot4(m1, d), dot4(m2, d), 0.f);
  *o_out = o;
  *d_out = dw;
}
// Queue slot j of a new path g. Its state is InitPathData's constants, which bounce 1
// knows (queue_state).
__device__ __forceinline__ void start_path(FrameBufs& fb, int j, int g, V o, V dw) {
  fb.q_o[0][j] = mk(o.x, o.y, o.z, __int_as_float(g));
  fb.q_d[0][j] = mk(dw.x, dw.y, dw.z, 1.f);
  if (fb.log) fb.log_n[g] = 0;
}

// ----------------------------------------------------------------- shade
// The per-path work, in two phases around the reference's compaction:
//   shade_hit       IntersectPrimitives' hit record, SetupBSDFPath and
//                   LightHitPass (emitter or environment contribution);
//   shade_continue  the texture pass, DirectLight (light sample, BSDF
//                   evaluation, shadow ray) and SampleBSDFRayDirection, then
//                   Russian roulette in benchmark semantics.
struct PathState {
  bool alive;
  int slot;                 // its queue slot
  int pixel;                // its path index: which pixel of which frame
  int fidx;                 // film index of its pixel
  int local;                // its pixel within its frame (the samples' key)
  const PassParams* pp;     // its frame's parameters
  V thr;                    // throughput (from shade_continue on)
  V ps;                     // hitpoint.xyz of the last bounce, lastPdfW
  int spec;                 // lastSpecular: only the camera's ray
  Hit H;
  Bsdf B;
};
struct ShadeOut {
  bool has_shadow;
  V sho, shd, shc, ndir;
};
// What lights the scene, known when a kernel is launched: an instance for each of
// the common cases leaves the other cases' code out. The whole is 130-160 KB of
// instructions, several times what an SM caches, and shading warps stalled on
// instruction fetch more than on anything else.
enum Lights {
  kAnyLights = 0,   // decided at run time
  kGridLights = 1,  // an environment map through the light grid, no mesh lights; CDF tables built
  kMeshLights = 2,  // mesh lights, no environment
  kMapLights = 3,   // an environment map sampled whole, no mesh lights; CDF tables built
};
template <int L> __device__ __forceinline__ bool mesh_lights(const DevScene& S) {
  return L == kAnyLights ? S.nlights > 0 : L == kMeshLights;
}
template <int L> __device__ __forceinline__ bool env_present(const DevEnv& E) {
  return L == kAnyLights ? E.present : L != kMeshLights;
}
template <int L> __device__ __forceinline__ bool grid_on(const DevEnv& E) {
  return L == kAnyLights ? E.grid_on : L == kGridLights;
}

// Which frame a path belongs to: one frame (its parameters, film index = path
// index), or a batch of frames sharing the queues (BatchFrames).
struct OneFrame {
  const PassParams* pp;
  __device__ __forceinline__ void operator()(int g, PathState& P) const {
    P.pp = pp;
    P.fidx = g;
    P.local = g;
  }
};
// Frames of a merged batch pass: frame k holds the paths start[k] .. start[k+1]-1
// (pixel g - start[k] of that frame), its film at film[k] .. and its parameters
// at pp[k].
struct BatchFrames {
  const int* start;  // n + 1
  const int* film;   // n
  const PassParams* pp;
  int n;
  __device__ __forceinline__ void operator()(int g, PathState& P) const {
    int lo = 0, hi = n - 1;  // the last frame with start <= g
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (__ldg(start + mid) <= g) lo = mid;
      else hi = mid - 1;
    }
    P.pp = pp + lo;
    P.local = g - __ldg(start + lo);
    P.fidx = __ldg(film + lo) + P.local;
  }
};

// A path's state in queue slot j at bounce b. It travels with the queue (q_d.w the
// last pdf, q_t the throughput; the last hitpoint is the ray's origin), so a bounce
// reads and writes it in slot order; bounce 1 starts from InitPathData's constants.
__device__ __forceinline__ void queue_state(int b, float4 qo, float4 qd, PathState& P) {
  P.ps = b == 1 ? mk(0.f, 0.f, 0.f, 1.f) : mk(qo.x, qo.y, qo.z, qd.w);
  P.spec = b == 1;
}
__device__ __forceinline__ V queue_thr(const FrameBufs& fb, int b, int j) {
  return b == 1 ? mk(1.f, 1.f, 1.f, 1.f) : __ldg(fb.q_t[(b + 1) & 1] + j);
}

template <int MODE, int L = kAnyLights, class Res = OneFrame>
__device__ __forceinline__ void shade_hit(const DevScene& S, const DevEnv& E, Res res, int b, const FrameBufs& fb,
                                          int j, int count, PathState& P) {
  P.alive = false;
  P.slot = j;
  P.pixel = 0;
  P.ps = zero4();
  P.spec = 0;
  P.B.mat = -1;
  if (j >= count) return;
  float4 qo = __ldg(fb.q_o[(b + 1) & 1] + j);
  float4 qd = __ldg(fb.q_d[(b + 1) & 1] + j);
  const int pixel = __float_as_int(qo.w);
  P.pixel = pixel;
  res(pixel, P);
  const PassParams* __restrict__ pp = P.pp;
  const int kahan = pp->kahan;
  V o = mk(qo.x, qo.y, qo.z, 0.f), d = mk(qd.x, qd.y, qd.z, 0.f);
  const float t = fb.hit_t[j];
  const int prim = fb.hit_prim[j];
  queue_state(b, qo, qd, P);
  if (prim >= 0) {
    hit_record(S, o, d, t, prim, P.H);
    P.B = setup_bsdf(S, d, P.H.n, P.H.mat);
    if (P.B.mat >= 0) {
      const Material& M = S.materials[P.B.mat];
      if ((L == kAnyLights || L == kMeshLights) && is_emitter(M)) {  // LightHitPass emitter branch, Render.cl:76-104
        float pick = 1.f / (float)S.nlights;
        if (MODE == 1 && E.present && S.nlights > 0) pick = pick * 0.5f;
        AreaLight L = get_area_light(S, M, prim);
        float pdfA = 0.f;
        V c = radiance_area(L, d, &pdfA);
        if (zero3(c)) {
          P.alive = true;  // Render.cl:88-89 returns with isect->hit still set
        } else {
          float w = 1.f;
          if (!P.spec) {
            float pdfW = pdf_a_to_w(pdfA, t, P.B.fix.z);
            w = mis2(P.ps.w, pdfW * pick);
          }
          contribute(fb, P.pixel, P.fidx, muls(mul(queue_thr(fb, b, j), c), w), kahan);
        }
      } else {
        P.alive = true;
      }
    }
  } else if (env_present<L>(E)) {  // LightHitPass environment branch, Render.cl:106-123
    float pdfW = 0.f;
    V c;
    if (MODE == 1 && grid_on<L>(E))
      c = radiance_env_grid(E, pp->cam_pos, P.ps, d, &pdfW, pp->grid_accum && !P.spec);
    else
      c = radiance_env(E, d, &pdfW);
    if (!zero3(c)) {
      if (MODE == 1 && mesh_lights<L>(S)) pdfW = pdfW * 0.5f;
      float w = 1.f;
      if (!P.spec) w = mis2(P.ps.w, pdfW);
      contribute(fb, P.pixel, P.fidx, muls(mul(queue_thr(fb, b, j), c), w), kahan);
    }
  }
}

// A path that shade_hit kept going (benchmark semantics), loaded again from its
// queue slot j: the hit record and BSDF set-up are recomputed from the same
// inputs by the same code, so they equal what shade_hit computed.
template <class Res>
__device__ __forceinline__ void shade_load(const DevScene& S, Res res, int b, const FrameBufs& fb, int j,
                                           PathState& P) {
  const float4 qo = __ldg(fb.q_o[(b + 1) & 1] + j);
  const float4 qd = __ldg(fb.q_d[(b + 1) & 1] + j);
  const int pixel = __float_as_int(qo.w);
  P.alive = true;
  P.slot = j;
  P.pixel = pixel;
  res(pixel, P);
  const V o = mk(qo.x, qo.y, qo.z, 0.f), d = mk(qd.x, qd.y, qd.z, 0.f);
  hit_record(S, o, d, __ldg(fb.hit_t + j), __ldg(fb.hit_prim + j), P.H);
  P.B = setup_bsdf(S, d, P.H.n, P.H.mat);
}

// gid: the work-item id the samples are keyed on (mode 0: the compacted slot,
// mode 1: the pixel's id). P ends with the next bounce's state; P.alive turns false when
// Russian roulette ends the path.
template <int MODE, bool TEX, int L = kAnyLights>
__device__ __forceinline__ void shade_continue(const DevScene& S, const DevEnv& E, int b, const FrameBufs& fb,
                                               int gid, PathState& P, ShadeOut& R) {
  const PassParams* __restrict__ pp = P.pp;
  const float fc = pp->frame_count;
  P.thr = queue_thr(fb, b, P.slot);
  R.has_shadow = false;
  R.ndir = zero4();
  Bsdf B = P.B;
  Material tm;  // the path's textured copy of its material
  if (TEX && has_textures(*B.pm)) {
    tm = *B.pm;
    apply_textures(S, B.mat, P.H.u, P.H.v, tm);
    B.pm = &tm;
  }
  int32_t lx, ly, bx, by;
  if (MODE == 0) {
    lx = pp->seeds[2 * (2 * b)];
    ly = pp->seeds[2 * (2 * b) + 1];
    bx = lx;
    by = ly;
  } else {
    stage_seed(b, 1, &lx, &ly);
    stage_seed(b, 2, &bx, &by);
  }
  Seed s = gen_seed(lx, ly, fc, gid);
  V dir = zero4();
  float dist = 0.f, pdfW = 0.f, pick = 1.f;
  V smp;
  smp.x = rnd(s);
  smp.y = rnd(s);
  smp.z = rnd(s);
  smp.w = rnd(s);
  V rad = zero4();
  bool smesh = false, senv = false;
  if (env_present<L>(E) && mesh_lights<L>(S)) {
    float r = rnd(s);
    pick = pick * 0.5f;
    if (r < 0.5f) smesh = true; else senv = true;
  } else if (env_present<L>(E)) {
    senv = true;
  } else if (mesh_lights<L>(S)) {
    smesh = true;
  }
  if (smesh) {
    int li = (int)(rnd(s) * (float)S.nlights);
    li = li < S.nlights ? li : S.nlights - 1;  // rounding of rnd * n for n > 2^22
    int tri = S.light_faces[MODE == 0 ? 0 : li];  // Render.cl:305 reads light 0
    pick = pick * (1.f / (float)S.nlights);
    const Material& Ml = S.materials[__ldg(reinterpret_cast<const int*>(S.faces + tri) + 9) & 0xFFFF];
    AreaLight L = get_area_light(S, Ml, tri);
    rad = illuminate_area(L, P.H.p, smp.x, smp.y, &dir, &dist, &pdfW);
  } else if (senv) {
    if (MODE == 1 && grid_on<L>(E))
      rad = illuminate_env_grid<L != kAnyLights>(E, pp->cam_pos, P.H.p, smp, &dir, &dist, &pdfW);
    else
      rad = illuminate_env<L != kAnyLights>(E, smp, &dir, &dist, &pdfW);
  }
  // BSDF sample
  Seed s2 = gen_seed(bx, by, fc, gid);
  const float s0 = rnd(s2), s1 = rnd(s2), sz = rnd(s2);
  const LobeDir ds = sample_dir(B, s0, s1, sz);
  const bool lit = !zero3(rad);
  float cosL = 0.f;
  LobeDir dl;
  dl.dif = dl.glo = false;
  if (lit) dl = eval_dir(B, dir, &cosL);
  // both directions' values by one copy of the code: first the light's, then the sample's
  V fl = zero4(), f = zero4();
  float bpdf = 0.f, pdf = 0.f;
#pragma unroll 1
  for (int k = 0; k < 2; ++k) {
    LobeDir d = dl;
    if (k) d = ds;
    bpdf = pdf;
    fl = f;
    pdf = 0.f;
    f = lobes(B, d, &pdf);
  }
  if (lit && !zero3(fl)) {
    const float w = mis2(pdfW, bpdf);
    const float sc = (w * cosL / (pick * pdfW));
    R.shc = mk(sc * (rad.x * fl.x) * P.thr.x, sc * (rad.y * fl.y) * P.thr.y, sc * (rad.z * fl.z) * P.thr.z, 1.f);
    R.sho = mk(P.H.p.x, P.H.p.y, P.H.p.z, __int_as_float(fb.log ? P.pixel : P.fidx));
    R.shd = mk(dir.x, dir.y, dir.z, dist - 2.f * 1e-3f);
    R.has_shadow = true;
  }
  float cosO = 0.f;
  f = sample_end(B, ds, f, &R.ndir, &cosO);
  float q = cosO / pdf;
  V thr = mul(P.thr, muls(f, q));
  if (MODE == 1 && pp->rr_depth > 0 && b >= pp->rr_depth) {
    int32_t rx, ry;
    stage_seed(b, 3, &rx, &ry);
    Seed rs = gen_seed(rx, ry, fc, gid);
    float u = rnd(rs);
    float mx = maxf_(thr.x, maxf_(thr.y, thr.z));
    float cont = minf_(0.95f, mx);
    if (!(u < cont)) P.alive = false;
    else thr = divs(thr, cont);
  }
  P.thr = thr;
  P.ps.w = pdf;
}

}  // namespace mt

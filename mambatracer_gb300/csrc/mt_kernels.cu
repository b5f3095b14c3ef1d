// Wavefront frame kernels: raygen, closest-hit traversal, fused shading with
// stable queue compaction, shadow traversal with film resolve.
//
// One pass of CDeviceGI.loop (src/cl/device/CDeviceGI.java:214-271) is
//   k_raygen                       InitCameraRayDataJitter + InitPathData +
//                                  InitIntersection + InitIntDataToIndex
//   per bounce b:
//     k_trace_closest              IntersectPrimitives (traversal part)
//     k_shade                      IntersectPrimitives (hit record) + SetupBSDFPath +
//                                  LightHitPass + CCompact.execute + DirectLight (light
//                                  sample and BSDF evaluation) + SampleBSDFRayDirection
//     k_trace_shadow               DirectLight's testOcclusion + addAccum
// with every queue on the device, so a pass needs no host round trip.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstddef>
#include <cstdlib>

#include "mt_device.cuh"
#include "mt_kernels.h"
#include "mt_shade.cuh"
#include "mt_traverse.cuh"

namespace mt {

using namespace dv;

// ----------------------------------------------------------------- raygen
// InitCameraRayDataJitter (src/cl/kernel/Initialize.cl:129-172) with the
// per-frame camera constants precomputed on the host, plus the path and queue
// resets of InitPathData / InitIntersection / InitIntDataToIndex. Starts the pass's
// control block too (a memset of its own in front of the pass costs 2 us).
__global__ void k_raygen(const PassParams* __restrict__ pp, Ctrl* ctrl, FrameBufs fb) {
  const int N = pp->width * pp->height;
  const int id = blockIdx.x * blockDim.x + threadIdx.x;
  static_assert(offsetof(Ctrl, count) == 0, "count[1] is word 1");
  if (blockIdx.x == 0)
    for (int k = threadIdx.x; k < (int)(sizeof(Ctrl) / 4); k += blockDim.x) reinterpret_cast<int*>(ctrl)[k] = k == 1 ? N : 0;
  if (id >= N) return;
  // reference semantics key samples on the slot, which is the pixel
  const int pixel = pp->mode == 0 ? id : tile_pixel(id, pp->width, pp->height);
  V o, dw;
  camera_ray(pp, pixel, &o, &dw);
  start_path(fb, id, pixel, o, dw);
}

// ----------------------------------------------------------- traversal
namespace {
struct QueueRays {
  const float4* qo;
  const float4* qd;
  __device__ __forceinline__ tr::RayT operator()(int i) const {
    return tr::make_ray(__ldg(qo + i), __ldg(qd + i), 0.001f, CUDART_INF_F);  // initGlobalRay, Util.cl:577-587
  }
};
struct HitOut {
  float* t;
  int* prim;
  __device__ __forceinline__ void operator()(int i, const tr::RayT& r, int hit) const {
    t[i] = r.tmax;
    prim[i] = hit;
  }
};
struct ShadowRays {
  const float4* so;
  const float4* sd;
  __device__ __forceinline__ tr::RayT operator()(int i) const {
    float4 o = __ldg(so + i), d = __ldg(sd + i);
    // initGlobalRayT (Util.cl:590-600); a slot without a shadow ray (pixel < 0)
    // gets an empty interval and ends at the first node
    return tr::make_ray(o, d, 0.0001f, __float_as_int(o.w) >= 0 ? d.w : -CUDART_INF_F);
  }
};
struct ShadowResolve {
  const float4* so;
  const float4* sc;
  FrameBufs fb;
  int kahan;
  unsigned* traced;
  __device__ __forceinline__ void operator()(int i, const tr::RayT&, int hit) const {
    int pixel = __float_as_int(__ldg(so + i).w);
    if (pixel < 0) return;
    ++*traced;
    if (hit < 0) {  // unoccluded: addAccum(&accum[pixel], contrib), Render.cl:456-461
      float4 c = __ldg(sc + i);
      contribute(fb, pixel, pixel, mk(c.x, c.y, c.z, 1.f), kahan);
    }
  }
};
// traversal steps between two refill points of a warp (the default of
// Tuning::refill_steps): measured 576, 588, 608, 614, 608, 595 Mrays/s at 8,
// 16, 32, 64, 128, 256 on the 1M soup
constexpr int kSteps = 64;
}  // namespace

// MINB: resident blocks per SM the register allocation is bounded for (the
// traversal is latency-bound: more resident warps hide more load latency, at
// the price of registers).
// PREC: the BVH format (0 FP32 child boxes, 1 FP16 outward-rounded, 2 the wide
// BVH with 8-bit boxes, 3 4-wide FP16 nodes).
template <int MINB, int PREC>
__global__ void __launch_bounds__(kTraceThreads, MINB) k_trace_closest(DevScene S, Ctrl* ctrl, int b, FrameBufs fb,
                                                                       int steps, int min_lanes) {
  const int count = ctrl->count[b];
  bool overflow = false;
  tr::trace_persistent<false, kSteps, QueueRays, HitOut, PREC>(
      S, count, &ctrl->work[2 * b], QueueRays{fb.q_o[(b + 1) & 1], fb.q_d[(b + 1) & 1]}, HitOut{fb.hit_t, fb.hit_prim},
      &overflow, steps, min_lanes);
  if (overflow) atomicExch(&ctrl->error, kDevErrStack);
}

template <int MINB, int PREC>
__global__ void __launch_bounds__(kTraceThreads, MINB) k_trace_shadow(DevScene S, Ctrl* ctrl, int b, int mode,
                                                                      FrameBufs fb, int kahan, int steps, int min_lanes) {
  // mode 0: shadow slots are the compacted survivor slots (flagged by pixel >= 0)
  const int count = mode == 0 ? ctrl->count[b + 1] : ctrl->shadow[b];
  bool overflow = false;
  unsigned traced = 0;
  tr::trace_persistent<true, kSteps, ShadowRays, ShadowResolve, PREC>(
      S, count, &ctrl->work[2 * b + 1], ShadowRays{fb.s_o, fb.s_d},
      ShadowResolve{fb.s_o, fb.s_c, fb, kahan, &traced}, &overflow, steps, min_lanes);
  unsigned long long tot = traced;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) tot += __shfl_down_sync(0xffffffffu, tot, o);
  if ((threadIdx.x & 31) == 0 && tot) atomicAdd(&ctrl->rays[2], tot);
  if (overflow) atomicExch(&ctrl->error, kDevErrStack);
}

// Adds a finished pass's ray counts into the job's running totals
// [primary, extension, shadow].
__global__ void k_accumulate(const Ctrl* ctrl, int max_depth, int n_pixels, unsigned long long* totals) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  unsigned long long ext = 0;
  for (int b = 2; b <= max_depth; ++b) ext += (unsigned long long)ctrl->count[b];
  // frames of in-flight slots finish concurrently: the totals are shared
  atomicAdd(totals + 0, (unsigned long long)n_pixels);
  atomicAdd(totals + 1, ext);
  atomicAdd(totals + 2, (unsigned long long)ctrl->rays[2]);
  if (ctrl->error) atomicExch(totals + 3, (unsigned long long)ctrl->error);
}

// Adds logged contributions to the film, one thread per pixel: reads what was
// logged and the film once, coalesced.
__global__ void k_replay(Replay R, float4* __restrict__ film, float4* __restrict__ film_c, unsigned long long* totals) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < R.passes) {
    const Ctrl& c = *R.ctrl[i];
    unsigned long long ext = 0;
    for (int b = 2; b <= R.max_depth; ++b) ext += (unsigned long long)c.count[b];
    atomicAdd(totals + 0, (unsigned long long)R.n);
    atomicAdd(totals + 1, ext);
    atomicAdd(totals + 2, c.rays[2]);
    if (c.error) atomicExch(totals + 3, (unsigned long long)c.error);
  }
  if (i >= R.n) return;
  int n[kReplayPasses], any = 0;
#pragma unroll
  for (int p = 0; p < kReplayPasses; ++p) {
    n[p] = p < R.passes ? R.count[p][i] : 0;
    any |= n[p];
  }
  if (!any) return;
  int px = i;
  if (R.frames) {
    PathState P;
    BatchFrames{R.start, R.film, nullptr, R.frames}(i, P);
    px = P.fidx;
  }
  V a = film[px], c = R.kahan ? film_c[px] : zero4();
#pragma unroll
  for (int p = 0; p < kReplayPasses; ++p)
    for (int k = 0; k < n[p]; ++k) {
      const V v = R.log[p][(size_t)k * R.stride + i];
      if (!R.kahan) {
        a = add(a, v);
        continue;
      }
      const V y = sub(v, c), t = add(a, y);
      c = sub(sub(t, a), y);
      a = t;
    }
  film[px] = a;
  if (R.kahan) film_c[px] = c;
}
int launch_replay(cudaStream_t st, const Replay& R, float4* film, float4* film_c, unsigned long long* totals) {
  k_replay<<<(R.n + 255) / 256, 256, 0, st>>>(R, film, film_c, totals);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

// ---------------------------------------------------------------- launchers
namespace {
// Register bounds of the traversal kernels (resident 128-thread blocks per SM):
// measured best on the 1M soup, 12 for closest hits (42 registers, a few bytes
// of spill) and 8 for shadow rays. MT_TRACE_MINB / MT_SHADOW_MINB (8, 12 or 16)
// select another build of either.
int env_minb(const char* name, int dflt) {
  const char* e = std::getenv(name);
  int x = e ? std::atoi(e) : dflt;
  return (x == 8 || x == 12 || x == 16) ? x : dflt;
}
// Persistent traversal grids of a shared pass, in blocks per SM (MT_TRACE_GRID /
// MT_SHADOW_GRID; 0: half of what fits). Frames in flight run their launches
// side by side, so a launch that leaves room on each SM lets another frame's
// kernels run there. Measured on the 1M soup with six frames in flight (blocks
// per SM for closest / shadow rays): 12/8 (all that fits) 613-616 Mrays/s,
// 8/8 637, 8/4 644, 6/4 633-651, 4/4 653, 3/3 651.
int grid_bps(const char* name, int dflt) {
  const char* e = std::getenv(name);
  int x = e ? std::atoi(e) : dflt;
  return x >= 0 && x <= 32 ? x : dflt;
}
// Resident 256-thread blocks per SM the benchmark-semantics shading kernel is
// bounded for (MT_SHADE_MINB: 3, 4 or 5).
int env_shade_minb() {
  const char* e = std::getenv("MT_SHADE_MINB");
  int x = e ? std::atoi(e) : kShadeMinBlocks;
  return (x == 3 || x == 4 || x == 5) ? x : kShadeMinBlocks;
}
int env_steps() {
  const char* e = std::getenv("MT_REFILL_STEPS");
  int x = e ? std::atoi(e) : kSteps;
  return x >= 4 && x <= 1024 ? x : kSteps;
}
// The process's launch shapes: the defaults above, the MT_* knobs, then
// whatever set_tuning installs.
Tuning& tuning_ref() {
  static Tuning t = {env_minb("MT_TRACE_MINB", kTraceMinBlocksClosest), env_minb("MT_SHADOW_MINB", kTraceMinBlocksShadow),
                     grid_bps("MT_TRACE_GRID", 0), grid_bps("MT_SHADOW_GRID", 0), env_shade_minb(), env_steps(),
                     std::getenv("MT_SHADOW_STREAM") && std::atoi(std::getenv("MT_SHADOW_STREAM")) == 0 ? 0 : 1};
  return t;
}
std::atomic<unsigned> g_tuning_version{1};
int trace_grid_bps() { return tuning_ref().closest_grid; }
int shadow_grid_bps() { return tuning_ref().shadow_grid; }
int trace_minb() { return tuning_ref().closest_minb; }
int shadow_minb() { return tuning_ref().shadow_minb; }
int shade_minb() { return tuning_ref().shade_minb; }
template <int MINB>
int trace_blocks_per_sm() {
  int n = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_trace_closest<MINB, 0>, kTraceThreads, 0);
  return n > 0 ? n : 1;
}
// The wide-BVH kernels are built for 8 resident blocks per SM whatever the
// tuning's bound (at 12 or 16 their wide node tests spill registers), and
// refill after an eighth of the binary kernels' steps (a wide step tests eight
// child boxes; measured on the 1M soup at 1080p, refill every 4, 8, 12, 16, 32,
// 64 wide steps: bounce-1 closest hits 1.73, 1.76, 1.81, 1.86, 2.02, 2.21 ms).
constexpr int kWideMinBlocks = 8;
int wide_steps_of(int steps) { return std::max(2, steps / 8); }
int wide_blocks_per_sm() {
  int n = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_trace_closest<kWideMinBlocks, 2>, kTraceThreads, 0);
  return n > 0 ? n : 1;
}
// 4-wide FP16 nodes (built for the tuning's bound like the binary kernels): a
// step visits a node of four child boxes (two binary levels) or tests a triangle.
int quad_steps_of(int steps) { return std::max(2, steps / 2); }
template <int MINB>
void launch_traces(cudaStream_t st, int grid, const DevScene& S, Ctrl* ctrl, int b, int mode, FrameBufs fb, int kahan,
                   bool closest, int min_lanes) {
  const int steps = tuning_ref().refill_steps;
  if (S.bitstack && S.precision <= 1) {
    if (closest) {
      if (S.precision == 1) k_trace_closest<MINB, 5><<<grid, kTraceThreads, 0, st>>>(S, ctrl, b, fb, steps, min_lanes);
      else k_trace_closest<MINB, 4><<<grid, kTraceThreads, 0, st>>>(S, ctrl, b, fb, steps, min_lanes);
    } else {
      if (S.precision == 1) k_trace_shadow<MINB, 5><<<grid, kTraceThreads, 0, st>>>(S, ctrl, b, mode, fb, kahan, steps, min_lanes);
      else k_trace_shadow<MINB, 4><<<grid, kTraceThreads, 0, st>>>(S, ctrl, b, mode, fb, kahan, steps, min_lanes);
    }
    return;
  }
  if (closest) {
    const int f = S.precision;
    if (f == 3)
      k_trace_closest<MINB, 3><<<grid, kTraceThreads, 0, st>>>(S, ctrl, b, fb, quad_steps_of(steps), min_lanes);
    else if (f == 2)
      k_trace_closest<kWideMinBlocks, 2><<<grid, kTraceThreads, 0, st>>>(S, ctrl, b, fb, wide_steps_of(steps), min_lanes);
    else if (f == 1)
      k_trace_closest<MINB, 1><<<grid, kTraceThreads, 0, st>>>(S, ctrl, b, fb, steps, min_lanes);
    else
      k_trace_closest<MINB, 0><<<grid, kTraceThreads, 0, st>>>(S, ctrl, b, fb, steps, min_lanes);
  } else {
    const int f = S.precision;
    if (f == 3)
      k_trace_shadow<MINB, 3><<<grid, kTraceThreads, 0, st>>>(S, ctrl, b, mode, fb, kahan, quad_steps_of(steps), min_lanes);
    else if (f == 2)
      k_trace_shadow<kWideMinBlocks, 2><<<grid, kTraceThreads, 0, st>>>(S, ctrl, b, mode, fb, kahan,
                                                                        wide_steps_of(steps), min_lanes);
    else if (f == 1)
      k_trace_shadow<MINB, 1><<<grid, kTraceThreads, 0, st>>>(S, ctrl, b, mode, fb, kahan, steps, min_lanes);
    else
      k_trace_shadow<MINB, 0><<<grid, kTraceThreads, 0, st>>>(S, ctrl, b, mode, fb, kahan, steps, min_lanes);
  }
}
}  // namespace

Tuning get_tuning() { return tuning_ref(); }

bool shade_split(int n, bool beside) {
  static const int m = [] {
    const char* e = std::getenv("MT_SHADE_SPLIT");
    if (!e) return -1;
    return std::atoi(e) == 0 ? 0 : 1;
  }();
  return m < 0 ? n >= (beside ? 1 << 18 : 1 << 20) : m != 0;
}

bool set_tuning(const Tuning& t) {
  auto minb_ok = [](int x) { return x == 8 || x == 12 || x == 16; };
  if (!minb_ok(t.closest_minb) || !minb_ok(t.shadow_minb) || t.closest_grid < 0 || t.closest_grid > 32 ||
      t.shadow_grid < 0 || t.shadow_grid > 32 || t.shade_minb < 3 || t.shade_minb > 5 || t.refill_steps < 4 ||
      t.refill_steps > 1024 || (t.shadow_stream != 0 && t.shadow_stream != 1))
    return false;
  tuning_ref() = t;
  g_tuning_version.fetch_add(1);
  return true;
}

unsigned tuning_version() { return g_tuning_version.load(); }

// One persistent traversal launch over a queue of at most N rays.
void launch_trace(cudaStream_t st, const DevScene& S, Ctrl* ctrl, int b, int mode, FrameBufs fb, int kahan, bool closest,
                  int N, int num_sms, bool shared, int min_lanes) {
  static int bps[17] = {};
  static int wide_bps = 0;
  const int minb = closest ? trace_minb() : shadow_minb();
  if (bps[minb] == 0)
    bps[minb] = minb == 16 ? trace_blocks_per_sm<16>() : minb == 12 ? trace_blocks_per_sm<12>() : trace_blocks_per_sm<8>();
  if (wide_bps == 0) wide_bps = wide_blocks_per_sm();
  const int fit = S.precision == 2 ? wide_bps : bps[minb];
  const int want = closest ? trace_grid_bps() : shadow_grid_bps();
  const int per_sm = !shared ? fit : want > 0 ? std::min(want, fit) : std::max(1, fit / 2);
  const int grid = std::max(1, std::min(num_sms * per_sm, (N + kTraceThreads - 1) / kTraceThreads));
  if (minb == 16) launch_traces<16>(st, grid, S, ctrl, b, mode, fb, kahan, closest, min_lanes);
  else if (minb == 12) launch_traces<12>(st, grid, S, ctrl, b, mode, fb, kahan, closest, min_lanes);
  else launch_traces<8>(st, grid, S, ctrl, b, mode, fb, kahan, closest, min_lanes);
}

int launch_pass(cudaStream_t st, const DevScene& S, const DevEnv& E, const PassParams* d_pp, int mode, int max_depth,
                int kahan, int width, int height, Ctrl* ctrl, FrameBufs fb, unsigned long long* status,
                size_t status_stride, int num_sms, cudaEvent_t* ev, unsigned long long* totals, bool shared,
                cudaStream_t side, cudaEvent_t fork, cudaEvent_t join, bool two_launches, int min_lanes) {
  const int N = width * height;
  // shadow rays of bounce b beside the extension rays of bounce b + 1 (no
  // per-kernel events): both read only what shading b wrote (in reference
  // semantics both read its survivor count), and shading b + 1, which rewrites
  // the shadow queue and adds to the film after the shadow kernel's adds, waits
  // for them
  const bool split = side && fork && join && !ev && tuning_ref().shadow_stream;
  if (split) shared = true;
  auto trace = [&](bool closest, int b) { launch_trace(st, S, ctrl, b, mode, fb, kahan, closest, N, num_sms, shared, min_lanes); };
  // persistent traversal: one resident wave, or fewer blocks for a small frame
  // (a queue never exceeds the frame's pixels), leaving SMs to other streams
  int e = 0;
  if (ev) cudaEventRecord(ev[e++], st);
  k_raygen<<<(N + 255) / 256, 256, 0, st>>>(d_pp, ctrl, fb);
  if (ev) cudaEventRecord(ev[e++], st);
  for (int b = 1; b <= max_depth; ++b) {
    trace(true, b);
    if (ev) cudaEventRecord(ev[e++], st);
    if (split && b > 1) cudaStreamWaitEvent(st, join, 0);
    if (mode == 0) launch_shade_ref(st, S, E, d_pp, N, ctrl, b, fb, status + (size_t)(b - 1) * status_stride);
    else launch_shade(st, S, E, d_pp, two_launches, shade_minb(), num_sms, N, ctrl, b, fb);
    if (ev) cudaEventRecord(ev[e++], st);
    if (split) {
      cudaEventRecord(fork, st);
      cudaStreamWaitEvent(side, fork, 0);
      launch_trace(side, S, ctrl, b, mode, fb, kahan, false, N, num_sms, shared, min_lanes);
      cudaEventRecord(join, side);
    } else {
      trace(false, b);
    }
    if (ev) cudaEventRecord(ev[e++], st);
  }
  if (split) cudaStreamWaitEvent(st, join, 0);
  if (totals) k_accumulate<<<1, 32, 0, st>>>(ctrl, max_depth, N, totals);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

namespace {
// Camera rays of a merged batch pass: path g is pixel g - start[k] of frame k.
__global__ void k_raygen_batch(BatchFrames B, int total, Ctrl* ctrl, FrameBufs fb) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j == 0) ctrl->count[1] = total;
  if (j >= total) return;
  PathState P;
  B(j, P);
  const int pixel = tile_pixel(P.local, P.pp->width, P.pp->height);
  V o, dw;
  camera_ray(P.pp, pixel, &o, &dw);
  start_path(fb, j, j - P.local + pixel, o, dw);
}
}  // namespace

int launch_batch_pass(cudaStream_t st, const DevScene& S, const DevEnv& E, const int* d_start, const int* d_film,
                      const PassParams* d_pp, int nframes, int total, int max_depth, int kahan, Ctrl* ctrl,
                      FrameBufs fb, int num_sms, unsigned long long* totals, cudaStream_t side, cudaEvent_t fork,
                      cudaEvent_t join, int beside) {
  const BatchFrames B{d_start, d_film, d_pp, nframes};
  const bool split = tuning_ref().shadow_stream, two = shade_split(total, beside > 1);
  const int lanes = tail_lanes(S, beside);
  k_raygen_batch<<<(total + 255) / 256, 256, 0, st>>>(B, total, ctrl, fb);
  // shadow rays beside the next bounce's extension rays, as in launch_pass
  for (int b = 1; b <= max_depth; ++b) {
    launch_trace(st, S, ctrl, b, 1, fb, kahan, true, total, num_sms, split || beside > 1, lanes);
    if (split && b > 1) cudaStreamWaitEvent(st, join, 0);
    launch_shade_batch(st, S, E, d_start, d_film, d_pp, nframes, two, num_sms, total, ctrl, b, fb);
    if (split) {
      cudaEventRecord(fork, st);
      cudaStreamWaitEvent(side, fork, 0);
    }
    launch_trace(split ? side : st, S, ctrl, b, 1, fb, kahan, false, total, num_sms, split || beside > 1, lanes);
    if (split) cudaEventRecord(join, side);
  }
  if (split) cudaStreamWaitEvent(st, join, 0);
  if (totals) k_accumulate<<<1, 32, 0, st>>>(ctrl, max_depth, total, totals);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

// Ray queries on reference-layout rays (80 B): closest or any hit.
namespace {
struct RefRays {
  const float4* rays;
  __device__ __forceinline__ tr::RayT operator()(int i) const {
    const float4* R = rays + 5 * (size_t)i;  // Ray: o, d, inv_d, sign, (extra, tMin, tMax)
    float4 o = __ldg(R + 0), d = __ldg(R + 1), tail = __ldg(R + 4);
    return tr::make_ray(o, d, tail.z, tail.w);
  }
};
struct QueryOut {
  int any;
  float* t;
  int* prim;
  __device__ __forceinline__ void operator()(int i, const tr::RayT& r, int hit) const {
    if (any) {
      prim[i] = hit >= 0 ? 1 : 0;
    } else {
      t[i] = r.tmax;
      prim[i] = hit;
    }
  }
};
}  // namespace

// One kernel a query (both in one took the registers of the larger: a million rays, closest
// and any, 4.10 -> 3.80 ms), the binary records' built for 12 blocks per SM (8, 10, 12, 16:
// 3.80, 3.64, 3.50, 3.86 ms), the others for 8 (4-wide nodes, 50k rays: 8, 10, 12 blocks
// 410, 436, 468 us).
template <int PREC, bool ANY>
__global__ void __launch_bounds__(kTraceThreads, PREC <= 1 ? 12 : 8)
    k_query(DevScene S, const float4* __restrict__ rays, int n, float* __restrict__ t_out, int* __restrict__ prim_out,
            int* work, int* err) {
  bool overflow = false;
  const int steps = PREC == 2 ? kSteps / 8 : PREC == 3 ? kSteps / 2 : kSteps;  // 4, 5: stackless binary
  tr::trace_persistent<ANY, kSteps, RefRays, QueryOut, PREC>(S, n, work, RefRays{rays},
                                                             QueryOut{ANY ? 1 : 0, t_out, prim_out}, &overflow, steps);
  if (overflow) atomicExch(err, kDevErrStack);
}

// Traversal work per ray: the same traversal as k_query, one step at a time,
// counting interior-node visits and triangle tests (counts[2 i], counts[2 i + 1]).
// Binary records: the visits the reference's algorithm makes (a step is one or
// the other, classified before it runs); the wide BVH: its node visits (96-byte
// nodes); 4-wide FP16 nodes: their node visits (64-byte nodes).
template <int PREC, bool ANY>
__global__ void __launch_bounds__(kTraceThreads) k_count(DevScene S, const float4* __restrict__ rays, int n,
                                                         float* __restrict__ t_out, int* __restrict__ prim_out,
                                                         int* __restrict__ counts, int* err) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  tr::RayT r = RefRays{rays}(i);
  bool overflow = false;
  int hit = -1, sp = 0, visits = 0, tests = 0;
  if constexpr (PREC == 2) {
    uint2 stack[kWideStack];
    tr::WideState w;
    tr::wide_init(r, w);
    int cnt[2] = {0, 0};
    while (!tr::wide_steps<ANY>(S, r, w, sp, hit, stack, 1, &overflow, cnt)) {
    }
    visits = cnt[0];
    tests = cnt[1];
  } else {
    typename tr::StackEntry<ANY>::type stack[PREC == 3 ? kQuadStack : kStackDepth], top;
    int ref = S.root_ref;
    const bool finite = tr::ray_is_finite(r);
    if constexpr (PREC >= 4) {
      unsigned long long bits = 0;
      int par = -1, sib = -1;
      for (;;) {
        const bool node = ref >= 0;
        const bool done = tr::bitstack_steps<ANY, PREC - 4>(S, r, ref, bits, par, sib, hit, finite, 1);
        visits += node;
        tests += !node;
        if (done) break;
      }
    } else if constexpr (PREC == 3) {
      int leaf = kQuadEmpty, cnt[2] = {0, 0};
      int tie = tr::kTieNone;
      const float tmax = r.tmax;
      for (;;) {
        if (!tr::quad_steps<ANY>(S, r, ref, leaf, sp, hit, finite, stack, top, 1, &overflow, tie, cnt)) continue;
        if (tie != tr::kTieSeen || overflow) break;
        r.tmax = tmax;
        ref = S.quad_again;
        leaf = kQuadEmpty;
        sp = 0;
        hit = -1;
        tie = tr::kTieAgain;
      }
      visits = cnt[0];
      tests = cnt[1];
    } else {
      for (;;) {
        const bool node = ref >= 0;
        const bool done = tr::trav_steps<ANY, PREC>(S, r, ref, sp, hit, finite, stack, top, 1, &overflow);
        visits += node;
        tests += !node;
        if (done) break;
      }
    }
  }
  if (overflow) atomicExch(err, kDevErrStack);
  QueryOut{ANY ? 1 : 0, t_out, prim_out}(i, r, hit);
  counts[2 * i] = visits;
  counts[2 * i + 1] = tests;
}

int launch_count(cudaStream_t st, const DevScene& S, const float4* rays, int n, int any, float* t_out, int* prim_out,
                 int* counts, int* err) {
  const int g = (n + kTraceThreads - 1) / kTraceThreads;
  if (n <= 0) return 0;
#define MT_COUNT(P)                                                                              \
  if (any) k_count<P, true><<<g, kTraceThreads, 0, st>>>(S, rays, n, t_out, prim_out, counts, err); \
  else k_count<P, false><<<g, kTraceThreads, 0, st>>>(S, rays, n, t_out, prim_out, counts, err);
  const int f = S.bitstack && S.precision <= 1 ? 4 + S.precision : S.precision;
  if (f == 5) {
    MT_COUNT(5)
  } else if (f == 4) {
    MT_COUNT(4)
  } else if (f == 3) {
    MT_COUNT(3)
  } else if (f == 2) {
    MT_COUNT(2)
  } else if (f == 1) {
    MT_COUNT(1)
  } else {
    MT_COUNT(0)
  }
#undef MT_COUNT
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

namespace {
template <int PREC>
void query_kernel(cudaStream_t st, int num_sms, const DevScene& S, const float4* rays, int n, int any, float* t_out,
                  int* prim_out, int* work, int* err) {
  // one resident wave, whatever the number of rays: few rays are spread over it
  int bps = 0;
  if (any) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, k_query<PREC, true>, kTraceThreads, 0);
  else cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, k_query<PREC, false>, kTraceThreads, 0);
  const int grid = num_sms * std::max(bps, 1);
  if (any) k_query<PREC, true><<<grid, kTraceThreads, 0, st>>>(S, rays, n, t_out, prim_out, work, err);
  else k_query<PREC, false><<<grid, kTraceThreads, 0, st>>>(S, rays, n, t_out, prim_out, work, err);
}
}  // namespace

int launch_query(cudaStream_t st, const DevScene& S, const float4* rays, int n, int any, float* t_out, int* prim_out,
                 int* work, int* err, int num_sms) {
  const int f = S.bitstack && S.precision <= 1 ? 4 + S.precision : S.precision;
  if (f == 5) query_kernel<5>(st, num_sms, S, rays, n, any, t_out, prim_out, work, err);
  else if (f == 4) query_kernel<4>(st, num_sms, S, rays, n, any, t_out, prim_out, work, err);
  else if (f == 3) query_kernel<3>(st, num_sms, S, rays, n, any, t_out, prim_out, work, err);
  else if (f == 2) query_kernel<2>(st, num_sms, S, rays, n, any, t_out, prim_out, work, err);
  else if (f == 1) query_kernel<1>(st, num_sms, S, rays, n, any, t_out, prim_out, work, err);
  else query_kernel<0>(st, num_sms, S, rays, n, any, t_out, prim_out, work, err);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

}  // namespace mt

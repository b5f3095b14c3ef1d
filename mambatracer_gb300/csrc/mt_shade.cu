// Shading kernels: hit record, BSDF, lights, queue appends and compaction.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdlib>
#include <type_traits>

#include "mt_device.cuh"
#include "mt_kernels.h"
#include "mt_scan.cuh"
#include "mt_shade.cuh"

namespace mt {

using namespace dv;
using namespace scan;

namespace {

// Benchmark semantics: a warp appends its survivors to the next queue and its
// shadow rays to the shadow queue, one atomic per queue (ranks by ballot).
__device__ __forceinline__ void append_warp(Ctrl* ctrl, int b, const FrameBufs& fb, const PathState& P,
                                            const ShadeOut& R) {
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  const int nq = b & 1;  // queue written for bounce b + 1
  const unsigned am = __ballot_sync(0xffffffffu, P.alive), sm = __ballot_sync(0xffffffffu, R.has_shadow);
  int qa = 0, qs = 0;
  if (lane == 0) {
    if (am) qa = atomicAdd(&ctrl->count[b + 1], __popc(am));
    if (sm) qs = atomicAdd(&ctrl->shadow[b], __popc(sm));
  }
  qa = __shfl_sync(0xffffffffu, qa, 0);
  qs = __shfl_sync(0xffffffffu, qs, 0);
  if (P.alive) {
    const int slot = qa + __popc(am & lt);
    fb.q_o[nq][slot] = mk(P.H.p.x, P.H.p.y, P.H.p.z, __int_as_float(P.pixel));
    fb.q_d[nq][slot] = mk(R.ndir.x, R.ndir.y, R.ndir.z, P.ps.w);
    fb.q_t[nq][slot] = P.thr;
  }
  if (R.has_shadow) {
    const int sslot = qs + __popc(sm & lt);
    fb.s_o[sslot] = R.sho;
    fb.s_d[sslot] = R.shd;
    fb.s_c[sslot] = R.shc;
  }
}

// Reference semantics (mode 0), one 256-path tile per block: survivors are
// compacted in order (block scan + decoupled look-back) between the two phases,
// and the light and BSDF samples of a survivor are keyed on its compacted slot
// as DirectLight and SampleBSDFRayDirection key them on get_global_id; the
// shadow ray of survivor j' sits at shadow slot j' (pixel -1: none).
// TEX: the scene has textures (a separate instance keeps the untextured one lean).
template <int MINB, bool TEX = false, int L = kAnyLights>
__global__ void __launch_bounds__(kShadeThreads, MINB) k_shade_ref(DevScene S, DevEnv E, const PassParams* __restrict__ pp,
                                                             Ctrl* ctrl, int b, FrameBufs fb,
                                                             unsigned long long* status) {
  __shared__ unsigned long long sh[kShadeThreads / 32 + 1];
  __shared__ int s_tile;
  __shared__ unsigned long long s_base;
  const int count = ctrl->count[b];
  const int ntiles = (count + kShadeThreads - 1) / kShadeThreads;
  if (threadIdx.x == 0) s_tile = atomicAdd(&ctrl->tiles[b], 1);
  __syncthreads();
  const int tile = s_tile;
  if (tile >= ntiles) return;
  const int j = tile * kShadeThreads + threadIdx.x;
  PathState P;
  shade_hit<0, L>(S, E, OneFrame{pp}, b, fb, j, count, P);
  unsigned long long tot = 0;
  unsigned long long excl = block_rank2<kShadeThreads>(P.alive, false, &tot, sh);
  if (threadIdx.x < 32) {
    const unsigned long long base = lookback(status, tile, tot, &ctrl->error);
    if (threadIdx.x == 0) s_base = base;
  }
  __syncthreads();
  const int slot = (int)(s_base + excl);
  if (tile == ntiles - 1 && threadIdx.x == 0) {
    ctrl->count[b + 1] = (int)(s_base + tot);
    ctrl->shadow[b] = (int)(s_base + tot);
  }
  if (!P.alive) return;
  ShadeOut R;
  shade_continue<0, TEX, L>(S, E, b, fb, slot, P, R);
  const int nq = b & 1;  // queue written for bounce b + 1
  fb.q_o[nq][slot] = mk(P.H.p.x, P.H.p.y, P.H.p.z, __int_as_float(P.pixel));
  fb.q_d[nq][slot] = mk(R.ndir.x, R.ndir.y, R.ndir.z, P.ps.w);
  fb.q_t[nq][slot] = P.thr;
  if (R.has_shadow) {
    fb.s_o[slot] = R.sho;
    fb.s_d[slot] = R.shd;
    fb.s_c[slot] = R.shc;
  } else {
    fb.s_o[slot] = mk(0.f, 0.f, 0.f, __int_as_float(-1));
  }
}

// Benchmark semantics (mode 1): samples are keyed on the pixel, so the order of
// the queues carries no meaning and no block ever waits for another. Warps run
// persistently over 32-path chunks (a chunk counter per bounce); each warp
// appends its survivors and its shadow rays to the next queues with one atomic
// per queue per chunk (ballot ranks inside the warp). Russian roulette runs after
// the BSDF sample.
// Res: OneFrame (pp = the frame's parameters) or BatchFrames (a merged batch pass).
template <int MINB, bool TEX = false, int L = kAnyLights, class Res = OneFrame>
__global__ void __launch_bounds__(kShadeThreads, MINB) k_shade(DevScene S, DevEnv E, Res res, Ctrl* ctrl, int b,
                                                         FrameBufs fb) {
  const int count = ctrl->count[b];
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  const int nq = b & 1;  // queue written for bounce b + 1
  for (;;) {
    int chunk = 0;
    if (lane == 0) chunk = atomicAdd(&ctrl->tiles[b], 1);
    chunk = __shfl_sync(0xffffffffu, chunk, 0);
    if (chunk * 32 >= count) break;
    const int j = chunk * 32 + lane;
    PathState P;
    shade_hit<1, L>(S, E, res, b, fb, j, count, P);
    ShadeOut R;
    R.has_shadow = false;
    if (P.alive) shade_continue<1, TEX, L>(S, E, b, fb, pixel_gid(P.local), P, R);
    const unsigned am = __ballot_sync(0xffffffffu, P.alive), sm = __ballot_sync(0xffffffffu, R.has_shadow);
    int qa = 0, qs = 0;
    if (lane == 0) {
      if (am) qa = atomicAdd(&ctrl->count[b + 1], __popc(am));
      if (sm) qs = atomicAdd(&ctrl->shadow[b], __popc(sm));
    }
    qa = __shfl_sync(0xffffffffu, qa, 0);
    qs = __shfl_sync(0xffffffffu, qs, 0);
    if (P.alive) {
      const int slot = qa + __popc(am & lt);
      fb.q_o[nq][slot] = mk(P.H.p.x, P.H.p.y, P.H.p.z, __int_as_float(P.pixel));
      fb.q_d[nq][slot] = mk(R.ndir.x, R.ndir.y, R.ndir.z, P.ps.w);
      fb.q_t[nq][slot] = P.thr;
    }
    if (R.has_shadow) {
      const int sslot = qs + __popc(sm & lt);
      fb.s_o[sslot] = R.sho;
      fb.s_d[sslot] = R.shd;
      fb.s_c[sslot] = R.shc;
    }
  }
}

// Benchmark semantics in two launches (shade_split, by the pass's size). k_shade_hit runs the hit record, the BSDF set-up and
// LightHitPass over the whole queue and lists the slots of the paths that go
// on; k_shade_cont runs the texture pass, DirectLight, SampleBSDFRayDirection
// and Russian roulette over that list alone. Each is half the code (less
// instruction fetch), and the second runs on full warps instead of warps whose
// terminated paths idle through the light and BSDF samples. Samples are keyed on
// the pixel, so the list's order carries no meaning.
template <int MINB, int L = kAnyLights, class Res = OneFrame>
__global__ void __launch_bounds__(kShadeThreads, MINB) k_shade_hit(DevScene S, DevEnv E, Res res, Ctrl* ctrl, int b,
                                                             FrameBufs fb) {
  const int count = ctrl->count[b];
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  for (;;) {
    int chunk = 0;
    if (lane == 0) chunk = atomicAdd(&ctrl->tiles[b], 1);
    chunk = __shfl_sync(0xffffffffu, chunk, 0);
    if (chunk * 32 >= count) break;
    const int j = chunk * 32 + lane;
    PathState P;
    shade_hit<1, L>(S, E, res, b, fb, j, count, P);
    const unsigned am = __ballot_sync(0xffffffffu, P.alive);
    int base = 0;
    if (lane == 0 && am) base = atomicAdd(&ctrl->live[b], __popc(am));
    base = __shfl_sync(0xffffffffu, base, 0);
    if (P.alive) fb.live[base + __popc(am & lt)] = j;
  }
}

template <int MINB, bool TEX = false, int L = kAnyLights, class Res = OneFrame>
__global__ void __launch_bounds__(kShadeThreads, MINB) k_shade_cont(DevScene S, DevEnv E, Res res, Ctrl* ctrl, int b,
                                                              FrameBufs fb) {
  const int count = ctrl->live[b];
  const int lane = threadIdx.x & 31;
  for (;;) {
    int chunk = 0;
    if (lane == 0) chunk = atomicAdd(&ctrl->tiles2[b], 1);
    chunk = __shfl_sync(0xffffffffu, chunk, 0);
    if (chunk * 32 >= count) break;
    const int k = chunk * 32 + lane;
    PathState P;
    P.alive = false;
    ShadeOut R;
    R.has_shadow = false;
    if (k < count) {
      shade_load(S, res, b, fb, __ldg(fb.live + k), P);
      shade_continue<1, TEX, L>(S, E, b, fb, pixel_gid(P.local), P, R);
    }
    append_warp(ctrl, b, fb, P, R);
  }
}

// Resident blocks per SM of the benchmark-semantics shading kernels (their grids are
// one resident wave of persistent warps).
int blocks_per_sm(int minb) {
  static int bps[6] = {};
  if (bps[minb] == 0) {
    int n = 0;
    if (minb == 4) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_shade<4>, kShadeThreads, 0);
    else if (minb == 5) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_shade<5>, kShadeThreads, 0);
    else cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_shade<3>, kShadeThreads, 0);
    bps[minb] = n > 0 ? n : 1;
  }
  return bps[minb];
}

// MT_LIGHT_KINDS=0 in the environment (read once per process): the general instance of every
// shading kernel, whatever lights the scene.
Lights lights_of(const DevScene& S, const DevEnv& E) {
  static const bool kinds = [] {
    const char* e = std::getenv("MT_LIGHT_KINDS");
    return !(e && std::atoi(e) == 0);
  }();
  if (!kinds) return kAnyLights;
  if (S.nlights > 0) return E.present ? kAnyLights : kMeshLights;
  if (!E.present) return kAnyLights;
  if (E.grid_on) return E.cell_marg && E.tile_marg ? kGridLights : kAnyLights;
  return E.env_marg ? kMapLights : kAnyLights;
}

// The instances: with textures, for mesh lights and for any; the bounds of 3 and 5
// blocks per SM (Tuning::shade_minb) for any lights.
template <int L, class Res>
void hit_kernel(cudaStream_t st, int grid, const DevScene& S, const DevEnv& E, Res R, Ctrl* ctrl, int b, FrameBufs fb) {
  k_shade_hit<4, L><<<grid, kShadeThreads, 0, st>>>(S, E, R, ctrl, b, fb);
}
template <int L, class Res>
void cont_kernel(cudaStream_t st, int grid, const DevScene& S, const DevEnv& E, Res R, Ctrl* ctrl, int b, FrameBufs fb) {
  k_shade_cont<4, false, L><<<grid, kShadeThreads, 0, st>>>(S, E, R, ctrl, b, fb);
}
template <class Res>
void launch_two(cudaStream_t st, int grid, const DevScene& S, const DevEnv& E, Res R, int minb, Ctrl* ctrl, int b,
                FrameBufs fb) {
  const Lights l = lights_of(S, E);
  constexpr bool one = std::is_same<Res, OneFrame>::value;  // merged batches have no light grid
  if (l == kMeshLights) hit_kernel<kMeshLights>(st, grid, S, E, R, ctrl, b, fb);
  else if (l == kMapLights) hit_kernel<kMapLights>(st, grid, S, E, R, ctrl, b, fb);
  else if (one && l == kGridLights) hit_kernel<one ? kGridLights : kAnyLights>(st, grid, S, E, R, ctrl, b, fb);
  else hit_kernel<kAnyLights>(st, grid, S, E, R, ctrl, b, fb);
  if (S.tex_on && l == kMeshLights)
    k_shade_cont<4, true, kMeshLights><<<grid, kShadeThreads, 0, st>>>(S, E, R, ctrl, b, fb);
  else if (S.tex_on)
    k_shade_cont<4, true><<<grid, kShadeThreads, 0, st>>>(S, E, R, ctrl, b, fb);
  else if (one && minb == 5)
    k_shade_cont<one ? 5 : 4><<<grid, kShadeThreads, 0, st>>>(S, E, R, ctrl, b, fb);
  else if (one && minb == 3)
    k_shade_cont<one ? 3 : 4><<<grid, kShadeThreads, 0, st>>>(S, E, R, ctrl, b, fb);
  else if (l == kMeshLights)
    cont_kernel<kMeshLights>(st, grid, S, E, R, ctrl, b, fb);
  else if (l == kMapLights)
    cont_kernel<kMapLights>(st, grid, S, E, R, ctrl, b, fb);
  else if (one && l == kGridLights)
    cont_kernel<one ? kGridLights : kAnyLights>(st, grid, S, E, R, ctrl, b, fb);
  else
    cont_kernel<kAnyLights>(st, grid, S, E, R, ctrl, b, fb);
}

}  // namespace

void launch_shade_ref(cudaStream_t st, const DevScene& S, const DevEnv& E, const PassParams* pp, int N, Ctrl* ctrl, int b,
                      FrameBufs fb, unsigned long long* status) {
  const int tiles = (N + kShadeThreads - 1) / kShadeThreads;
  const Lights l = lights_of(S, E);
  if (S.tex_on && l == kMeshLights)
    k_shade_ref<3, true, kMeshLights><<<tiles, kShadeThreads, 0, st>>>(S, E, pp, ctrl, b, fb, status);
  else if (S.tex_on)
    k_shade_ref<3, true><<<tiles, kShadeThreads, 0, st>>>(S, E, pp, ctrl, b, fb, status);
  else if (l == kMeshLights)
    k_shade_ref<4, false, kMeshLights><<<tiles, kShadeThreads, 0, st>>>(S, E, pp, ctrl, b, fb, status);
  else if (l == kMapLights)
    k_shade_ref<3, false, kMapLights><<<tiles, kShadeThreads, 0, st>>>(S, E, pp, ctrl, b, fb, status);
  else
    k_shade_ref<3><<<tiles, kShadeThreads, 0, st>>>(S, E, pp, ctrl, b, fb, status);
}

void launch_shade(cudaStream_t st, const DevScene& S, const DevEnv& E, const PassParams* pp, bool two, int minb,
                  int num_sms, int N, Ctrl* ctrl, int b, FrameBufs fb) {
  const int grid = std::max(1, std::min(num_sms * blocks_per_sm(minb), (N + kShadeThreads - 1) / kShadeThreads));
  const OneFrame R{pp};
  if (two) {
    launch_two(st, grid, S, E, R, minb, ctrl, b, fb);
    return;
  }
  const Lights l = lights_of(S, E);
  if (S.tex_on && l == kMeshLights)
    k_shade<4, true, kMeshLights><<<grid, kShadeThreads, 0, st>>>(S, E, R, ctrl, b, fb);
  else if (S.tex_on)
    k_shade<4, true><<<grid, kShadeThreads, 0, st>>>(S, E, R, ctrl, b, fb);
  else if (minb == 5)
    k_shade<5><<<grid, kShadeThreads, 0, st>>>(S, E, R, ctrl, b, fb);
  else if (minb == 3)
    k_shade<3><<<grid, kShadeThreads, 0, st>>>(S, E, R, ctrl, b, fb);
  else if (l == kMeshLights)
    k_shade<4, false, kMeshLights><<<grid, kShadeThreads, 0, st>>>(S, E, R, ctrl, b, fb);
  else if (l == kMapLights)
    k_shade<4, false, kMapLights><<<grid, kShadeThreads, 0, st>>>(S, E, R, ctrl, b, fb);
  else if (l == kGridLights)
    k_shade<4, false, kGridLights><<<grid, kShadeThreads, 0, st>>>(S, E, R, ctrl, b, fb);
  else
    k_shade<4><<<grid, kShadeThreads, 0, st>>>(S, E, R, ctrl, b, fb);
}

void launch_shade_batch(cudaStream_t st, const DevScene& S, const DevEnv& E, const int* d_start, const int* d_film,
                        const PassParams* d_pp, int nframes, bool two, int num_sms, int total, Ctrl* ctrl, int b,
                        FrameBufs fb) {
  const int grid = std::max(1, std::min(num_sms * blocks_per_sm(4), (total + kShadeThreads - 1) / kShadeThreads));
  const BatchFrames B{d_start, d_film, d_pp, nframes};
  if (two) launch_two(st, grid, S, E, B, 4, ctrl, b, fb);
  else if (S.tex_on) k_shade<4, true, kAnyLights><<<grid, kShadeThreads, 0, st>>>(S, E, B, ctrl, b, fb);
  else k_shade<4, false, kAnyLights><<<grid, kShadeThreads, 0, st>>>(S, E, B, ctrl, b, fb);
}

}  // namespace mt

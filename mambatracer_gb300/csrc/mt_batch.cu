// Merged batches: frames of uneven size (cameras, resolutions, spp) rendered
// through one set of wavefront queues. Pass p of the batch holds every frame
// with more than p passes; its paths are the frames' pixels back to back, so
// each bounce is one launch per kernel for the whole batch instead of one per
// frame. A path keys its samples on its frame's pixel and frame number, as a
// frame rendered alone does (benchmark semantics, full-map environment
// sampling, as served requests): every frame's film equals that frame rendered
// alone, bit for bit. The reference renders one frame at a time; this is the
// batched configuration of the benchmark (jobs of uneven resolution sharing
// global work queues).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <vector>

#include "mt_internal.h"

extern "C" int mt_batch_render(mt_context* ctx, mt_scene* s, const mt_batch_frame* frames, int nframes, int max_depth,
                               int rr_depth, int film_kahan, float* films_out, int64_t* rays_out) {
  if (!ctx || !s || !frames || !films_out || nframes <= 0) return fail(MT_ERR_INVALID, "bad argument");
  if (s->ctx != ctx) return fail(MT_ERR_INVALID, "scene belongs to another context");
  if (!s->has_bvh) return fail(MT_ERR_INVALID, "scene has no BVH");
  if (max_depth < 1 || max_depth > kMaxDepth) return fail(MT_ERR_INVALID, "max_depth %d (1..%d)", max_depth, kMaxDepth);
  size_t total = 0;
  int max_spp = 0;
  for (int k = 0; k < nframes; ++k) {
    const mt_batch_frame& f = frames[k];
    if (f.width <= 0 || f.height <= 0 || f.spp <= 0 || f.spp > 4096)
      return fail(MT_ERR_INVALID, "frame %d: %d x %d, %d spp", k, f.width, f.height, f.spp);
    total += (size_t)f.width * f.height;
    max_spp = std::max(max_spp, f.spp);
  }
  if (total > (size_t)INT32_MAX / 2) return fail(MT_ERR_INVALID, "batch of %zu pixels", total);
  std::lock_guard<std::recursive_mutex> lk(ctx->mu);
  CU(cudaSetDevice(ctx->device));
  cudaStream_t st = ctx->stream;

  // per pass: the frames still rendering, their first path, film offset and parameters
  std::vector<int> h_start((size_t)max_spp * (nframes + 1)), h_film((size_t)max_spp * nframes);
  std::vector<PassParams> h_pp((size_t)max_spp * nframes);
  std::vector<int> nact(max_spp), tot(max_spp);
  std::vector<size_t> film_off(nframes);
  for (int k = 0, off = 0; k < nframes; ++k) {
    film_off[k] = (size_t)off;
    off += frames[k].width * frames[k].height;
  }
  for (int p = 0; p < max_spp; ++p) {
    int n = 0, g = 0;
    for (int k = 0; k < nframes; ++k) {
      const mt_batch_frame& f = frames[k];
      if (f.spp <= p) continue;
      PassParams& pp = h_pp[(size_t)p * nframes + n];
      std::memset(&pp, 0, sizeof(pp));
      camera_constants(f.camera, f.width, f.height, pp);
      pp.frame_count = f.frame_count + (float)p;
      pp.width = f.width;
      pp.height = f.height;
      pp.max_depth = max_depth;
      pp.mode = 1;
      pp.rr_depth = rr_depth;
      pp.kahan = film_kahan;
      pp.grid_accum = 0;
      h_start[(size_t)p * (nframes + 1) + n] = g;
      h_film[(size_t)p * nframes + n] = (int)film_off[k];
      g += f.width * f.height;
      ++n;
    }
    h_start[(size_t)p * (nframes + 1) + n] = g;
    nact[p] = n;
    tot[p] = g;
  }

  // Passes overlap as a job's do (mt_job.cu), as far as the kept scratch holds them.
  auto R = [](size_t b) { return Workspace::round(b); };
  const size_t fixed = 2 * R(total * 16) + R(sizeof(Ctrl) * (size_t)max_spp) + R(h_start.size() * 4) +
                       R(h_film.size() * 4) + R(h_pp.size() * sizeof(PassParams)) + R(32);
  const size_t queues = 9 * R(total * 16) + 3 * R(total * 4),
               log = R(total * 16 * 2 * (size_t)max_depth) + R(total * 4);
  const size_t room = kWorkspaceMax > fixed ? (kWorkspaceMax - fixed) / (queues + log) : 0;
  int nbuf = (int)std::max<size_t>(1, std::min<size_t>({room, (size_t)max_spp, 4}));
  while ((int)ctx->pass_streams.size() < nbuf) {
    mt_context::PassStream p;
    cudaError_t e = cudaStreamCreateWithFlags(&p.stream, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&p.side, cudaStreamNonBlocking);
    for (cudaEvent_t* v : {&p.fork, &p.join, &p.done})
      if (e == cudaSuccess) e = cudaEventCreateWithFlags(v, cudaEventDisableTiming);
    ctx->pass_streams.push_back(p);  // also a half-made one: the context frees it
    if (e != cudaSuccess) return fail(MT_ERR_CUDA, "batch streams: %s", cudaGetErrorString(e));
  }
  Workspace ws;
  int r = ws.get(ctx, fixed + nbuf * (queues + (nbuf > 1 ? log : 0)));
  if (r && nbuf > 1) r = ws.get(ctx, fixed + (nbuf = 1) * queues);  // memory is short: one pass after the other
  if (r) return r;
  const bool logged = nbuf > 1;
  float4* film = ws.take<float4>(total);
  float4* film_c = ws.take<float4>(total);
  std::vector<FrameBufs> fbs(nbuf);
  for (FrameBufs& fb : fbs) {
    for (auto* p : {&fb.q_o[0], &fb.q_o[1], &fb.q_d[0], &fb.q_d[1], &fb.q_t[0], &fb.q_t[1], &fb.s_o, &fb.s_d, &fb.s_c})
      *p = ws.take<float4>(total);
    fb.hit_t = ws.take<float>(total);
    fb.hit_prim = ws.take<int>(total);
    fb.live = ws.take<int>(total);
    fb.film = film;
    fb.film_c = film_c;
    if (logged) {
      fb.log = ws.take<float4>(total * 2 * (size_t)max_depth);
      fb.log_n = ws.take<int>(total);
      fb.log_stride = (int)total;
    }
  }
  Ctrl* d_ctrl = ws.take<Ctrl>((size_t)max_spp);
  int* d_start = ws.take<int>(h_start.size());
  int* d_film = ws.take<int>(h_film.size());
  PassParams* d_pp = ws.take<PassParams>(h_pp.size());
  unsigned long long* d_totals = ws.take<unsigned long long>(4);
  auto done = [&](int code) {
    for (int k = 0; k < nbuf; ++k) {
      cudaStreamSynchronize(ctx->pass_streams[k].stream);
      cudaStreamSynchronize(ctx->pass_streams[k].side);
    }
    cudaStreamSynchronize(st);
    ws.release();
    return code;
  };
  cudaError_t e = cudaMemsetAsync(film, 0, total * 16, st);
  if (e == cudaSuccess) e = cudaMemsetAsync(film_c, 0, total * 16, st);
  if (e == cudaSuccess) e = cudaMemsetAsync(d_ctrl, 0, sizeof(Ctrl) * (size_t)max_spp, st);
  if (e == cudaSuccess) e = cudaMemsetAsync(d_totals, 0, 32, st);
  if (e == cudaSuccess) e = cudaMemcpyAsync(d_start, h_start.data(), h_start.size() * 4, cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess) e = cudaMemcpyAsync(d_film, h_film.data(), h_film.size() * 4, cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(d_pp, h_pp.data(), h_pp.size() * sizeof(PassParams), cudaMemcpyHostToDevice, st);
  if (e != cudaSuccess) return done(fail(MT_ERR_CUDA, "batch set-up: %s", cudaGetErrorString(e)));
  const DevScene S = s->view();
  const DevEnv E = s->env_view();  // full-map environment sampling
  e = cudaEventRecord(ctx->ready, st);  // the set-up
  for (int k = 0; k < nbuf && e == cudaSuccess; ++k) e = cudaStreamWaitEvent(ctx->pass_streams[k].stream, ctx->ready, 0);
  if (e != cudaSuccess) return done(fail(MT_ERR_CUDA, "batch set-up: %s", cudaGetErrorString(e)));
  for (int p = 0; p < max_spp; ++p) {
    const int k = p % nbuf;
    mt_context::PassStream& P = ctx->pass_streams[k];
    const int* start = d_start + (size_t)p * (nframes + 1);
    const int* fmap = d_film + (size_t)p * nframes;
    if (launch_batch_pass(P.stream, S, E, start, fmap, d_pp + (size_t)p * nframes, nact[p], tot[p], max_depth, film_kahan,
                          d_ctrl + p, fbs[k], ctx->num_sms, logged ? nullptr : d_totals, P.side, P.fork, P.join, nbuf))
      return done(fail(MT_ERR_CUDA, "batch pass: %s", cudaGetErrorString(cudaGetLastError())));
    if (logged) {
      Replay Rp{};
      Rp.log[0] = fbs[k].log;
      Rp.count[0] = fbs[k].log_n;
      Rp.ctrl[0] = d_ctrl + p;
      Rp.passes = 1;
      Rp.stride = (int)total;
      Rp.n = tot[p];
      Rp.max_depth = max_depth;
      Rp.kahan = film_kahan;
      Rp.start = start;
      Rp.film = fmap;
      Rp.frames = nact[p];
      if (p > 0) e = cudaStreamWaitEvent(P.stream, ctx->pass_streams[(p - 1) % nbuf].done, 0);
      if (e != cudaSuccess || launch_replay(P.stream, Rp, film, film_c, d_totals))
        return done(fail(MT_ERR_CUDA, "batch film: %s", cudaGetErrorString(cudaGetLastError())));
    }
    e = cudaEventRecord(P.done, P.stream);
    if (e != cudaSuccess) return done(fail(MT_ERR_CUDA, "batch: %s", cudaGetErrorString(e)));
  }
  for (int k = 0; k < std::min(nbuf, max_spp) && e == cudaSuccess; ++k)
    e = cudaStreamWaitEvent(st, ctx->pass_streams[k].done, 0);
  if (e != cudaSuccess) return done(fail(MT_ERR_CUDA, "batch: %s", cudaGetErrorString(e)));
  e = cudaEventRecord(ctx->ready, st);
  if (e != cudaSuccess) return done(fail(MT_ERR_CUDA, "batch: %s", cudaGetErrorString(e)));
  prefault(films_out, total * 16, ctx->ready);
  unsigned long long h_tot[4] = {0, 0, 0, 0};
  e = cudaMemcpyAsync(films_out, film, total * 16, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaMemcpyAsync(h_tot, d_totals, 32, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return done(fail(MT_ERR_CUDA, "batch: %s", cudaGetErrorString(e)));
  if (h_tot[3]) return done(fail(MT_ERR_DEVICE, "batch: device error %llu", h_tot[3]));
  if (rays_out)
    for (int i = 0; i < 3; ++i) rays_out[i] = (int64_t)h_tot[i];
  return done(MT_OK);
}

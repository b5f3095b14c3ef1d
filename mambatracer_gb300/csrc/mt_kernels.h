// Host-visible declarations of the device launchers.
#pragma once
#include <cuda_runtime.h>

#include "mt_common.h"

namespace mt {

// Per-job frame buffers (structure of arrays).
struct FrameBufs {
  float4* q_o[2];   // ray queue: origin.xyz, bits(pixel)  (ping-pong by bounce parity)
  float4* q_d[2];   // ray queue: direction.xyz, lastPdfW
  float4* q_t[2];   // ray queue: throughput (4 lanes as the reference); bounce 1 has none
  float* hit_t;     // closest-hit distance per queue slot
  int* hit_prim;    // closest-hit face id per queue slot (-1 = miss)
  float4* s_o;      // shadow queue: origin.xyz, bits(pixel or -1)
  float4* s_d;      // shadow queue: direction.xyz, tMax
  float4* s_c;      // shadow queue: contribution.xyz
  float4* film;     // accumulated radiance per pixel
  float4* film_c;   // Kahan compensation per pixel
  int* live;        // queue slots of the paths that go on after the hit phase (two-launch shading)
  // Contributions kept for later (passes that overlap): path g's k-th one at
  // log[k * log_stride + g], log_n[g] of them; log NULL: added to the film at once.
  float4* log;
  int* log_n;
  int log_stride;
};

// Up to kReplayPasses finished passes' contributions, added to the film pass by
// pass in the order they were made (what film_add does as they come), and the
// passes' ray counts to the totals.
constexpr int kReplayPasses = 4;
struct Replay {
  const float4* log[kReplayPasses];
  const int* count[kReplayPasses];
  const Ctrl* ctrl[kReplayPasses];
  int passes, stride, max_depth, kahan;
  int n;  // paths of a pass
  // merged batch passes: path to pixel as in launch_batch_pass; frames 0: pixel = path
  const int *start, *film;
  int frames;
};
int launch_replay(cudaStream_t st, const Replay& R, float4* film, float4* film_c, unsigned long long* totals);

// Rays of a short queue kept together in a warp, by `beside`: the passes or frames that run
// side by side over a job (the larger of its slots and a slot's buffers) or a batch, a
// server's lanes or merge streams (the rounds of one stream that overlap, up to three, are
// not counted: with them, one stream of 1 to 4 requests is 4 to 7 % slower, four streams with 2
// requests 12 %, with 16 5 % faster, FP32 records). Alone, one ray to a warp is fastest (1, 2, 4, 8, 16, 32: the 200k soup at 800 x
// 600, passes one by one, 12.2, 12.3, 12.5, 12.7, 13.3, 14.2 ms); with six 1080p frames of
// the 1M soup in flight the GPU's issue slots are taken and the spread rays'
// instructions cost (46.8, 46.6, 46.4, 46.1, 45.5, 45.2 ms for eight frames); a served
// mix on four streams lies between (12.5, 12.7, 12.8, 13.1, 13.5, 14.3 ms), and so do
// four passes at once (200k soup 6.70 ms with 8, 6.94 with 32). A tree of a few hundred
// nodes is in L1 and its rays are short, so there is no latency to spread for beside
// others (room 500 x 500, four frames at once, 2.32 ms with 8, 2.16 with 32).
inline int tail_lanes(const DevScene& S, int beside) {
  return beside <= 1 ? 1 : beside <= 4 && S.nrec > kTinyRecords ? 8 : 32;
}

// Launch shapes of the hot kernels, process-wide (one GPU per process):
// closest_minb / shadow_minb: the traversal build, by the resident blocks per
// SM its registers are bounded for (8, 12, 16); closest_grid / shadow_grid:
// blocks per SM of a traversal launch that shares the GPU with other frames (0:
// half of what fits); shade_minb: the benchmark-semantics shading build (3, 4,
// 5); refill_steps: traversal steps between refills of finished lanes (4..1024);
// shadow_stream: a frame's shadow rays of bounce b run on a second stream beside
// its extension rays of bounce b + 1 (1) or after them on one stream (0).
// Every choice gives the same results; only the speed differs.
struct Tuning {
  int closest_minb, shadow_minb, closest_grid, shadow_grid, shade_minb, refill_steps, shadow_stream;
};
Tuning get_tuning();
bool set_tuning(const Tuning& t);  // false when a field is out of range
unsigned tuning_version();         // bumped by every set_tuning (jobs recapture their graphs)

// events: optional array of 2 + 3 * max_depth events recorded around each launch.
// totals: optional running ray counts [primary, extension, shadow, error] of the job.
// shared: other frames or requests run beside this pass on the GPU (frames in
// flight, served lanes): each persistent traversal launch then takes half the
// blocks an SM can hold, leaving room for their kernels.
// side, fork, join: a second stream and two events of the caller's; with the
// tuning's shadow_stream on, the shadow rays run there.
// min_lanes: rays of a short queue that a traversal warp takes at least
// (tail_lanes; tr::trace_persistent).
// A merged batch pass (benchmark semantics, full-map environment sampling):
// frames 0 .. nframes-1 share the queues; path g belongs to the frame k with
// d_start[k] <= g < d_start[k+1] (pixel g - d_start[k]), its film slots start at
// d_film[k], its parameters are d_pp[k]. total = d_start[nframes].
int launch_batch_pass(cudaStream_t st, const DevScene& S, const DevEnv& E, const int* d_start, const int* d_film,
                      const PassParams* d_pp, int nframes, int total, int max_depth, int kahan, Ctrl* ctrl,
                      FrameBufs fb, int num_sms, unsigned long long* totals, cudaStream_t side, cudaEvent_t fork,
                      cudaEvent_t join, int beside);
int launch_pass(cudaStream_t st, const DevScene& S, const DevEnv& E, const PassParams* d_pp, int mode,
                int max_depth, int kahan, int width, int height, Ctrl* ctrl, FrameBufs fb,
                unsigned long long* status, size_t status_stride, int num_sms, cudaEvent_t* events,
                unsigned long long* totals, bool shared = false, cudaStream_t side = nullptr,
                cudaEvent_t fork = nullptr, cudaEvent_t join = nullptr, bool two_launches = false, int min_lanes = 1);
// Shading of one bounce (mt_shade.cu): reference semantics; benchmark semantics of
// one frame (in one launch or two) and of a merged batch pass. N, total: paths a
// queue holds at most.
void launch_shade_ref(cudaStream_t st, const DevScene& S, const DevEnv& E, const PassParams* pp, int N, Ctrl* ctrl, int b,
                      FrameBufs fb, unsigned long long* status);
void launch_shade(cudaStream_t st, const DevScene& S, const DevEnv& E, const PassParams* pp, bool two, int minb,
                  int num_sms, int N, Ctrl* ctrl, int b, FrameBufs fb);
void launch_shade_batch(cudaStream_t st, const DevScene& S, const DevEnv& E, const int* d_start, const int* d_film,
                        const PassParams* d_pp, int nframes, bool two, int num_sms, int total, Ctrl* ctrl, int b,
                        FrameBufs fb);
// Whether a pass of n paths shades in two launches (MT_SHADE_SPLIT in the environment:
// 0 never, 1 always): beside, other passes or frames run beside it (on a server: other
// lanes or merge streams). The second
// launch's full warps and smaller code gain with the paths; its fixed cost of a few
// us a bounce matters below a million paths alone and, hidden behind the others,
// below 2^18 beside others. One launch against two, alone: room 256 x 256, 4 passes,
// 944 and 1061 us; 200k soup 800 x 600, 3.02 and 3.05 ms; textured room 1920 x 1080, 4
// passes, 5.84 and 5.71 ms; overlapping: 200k soup 800 x 600, 4 passes, 6.89 and 6.70;
// stadium 1080p, 4 passes, 8.17 and 7.55; eight frames of the stadium in flight 16.8 and
// 15.2, of the 1M soup 44.2 and 40.7.
bool shade_split(int n, bool beside);

// Closest or any hit of reference-layout rays with the traversal work per ray
// (interior-node visits, triangle tests), one ray per thread.
int launch_count(cudaStream_t st, const DevScene& S, const float4* rays, int n, int any, float* t_out, int* prim_out,
                 int* counts, int* err);
int launch_query(cudaStream_t st, const DevScene& S, const float4* rays, int n, int any, float* t_out,
                 int* prim_out, int* work, int* err, int num_sms);

// Environment: luminance (FP32, RGBSpace.cl:28-32) and the inclusive SAT built
// in FP64, with an FP32 copy for sampling.
int launch_env_build(cudaStream_t st, const float4* rgb, int w, int h, float* lum, double* sat64, float* sat32);

// Light-grid per-cell SAT (row passes of rx, column passes of ry), FP32 in the
// reference's Kogge-Stone order or FP64.
int launch_grid_sat(cudaStream_t st, const float* func, float* sat32, double* sat64, int nu, int nv, int rx, int ry,
                    int fp64);
// Initial light-grid func: each cell's tiles get the map's luminance summed over
// the tile (from sat64 when not NULL, else sat32).
int launch_grid_init(cudaStream_t st, const double* sat64, const float* sat32, int w, int h, int nu, int nv, int rx,
                     int ry, float* func);
// CDF tables of the grid-guided environment sampling (dv::RegionTab): for the
// rx x ry tiles of the map (from its FP32 SAT) and for the grid's cells (from
// the per-cell SATs). *_floats return the cond table's size and the marg table's
// through *marg_floats.
size_t tile_table_floats(int w, int h, int rx, int ry, size_t* marg_floats);
size_t map_table_floats(int w, int h, size_t* marg_floats);
int launch_map_tables(cudaStream_t st, const float* sat, int w, int h, float* marg, float* cond);
size_t cell_table_floats(int nu, int nv, int rx, int ry, size_t* marg_floats);
int launch_tile_tables(cudaStream_t st, const float* sat, int w, int h, int rx, int ry, float* marg, float* cond);
int launch_cell_tables(cudaStream_t st, const float* grid_sat, int nu, int nv, int rx, int ry, float* marg,
                       float* cond);

}  // namespace mt

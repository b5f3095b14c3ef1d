// Internal definitions shared by the C-ABI translation units.
#pragma once
#include <cuda_runtime.h>

#include <cstdarg>
#include <cstdint>
#include <cstdio>
#include <atomic>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/mambatracer.h"
#include "mt_common.h"
#include "mt_kernels.h"

using namespace mt;

struct mt_context;
struct mt_job;
struct mt_server;

// ------------------------------------------------------------------ errors
namespace mt {
// Records the message mt_last_error() returns on this thread; returns code.
__attribute__((visibility("hidden"))) int fail(int code, const char* fmt, ...);
// cudaMalloc and cudaFree of the library's arrays. MT_DEVICE_ROOM in the environment, where
// it is set when the process allocates its first array, makes the device look nearly
// full: the arrays may grow by that many bytes beyond what they held when the value was
// first seen (empty: no limit; the value may change while the process runs).
__attribute__((visibility("hidden"))) cudaError_t device_malloc(void** p, size_t bytes);
__attribute__((visibility("hidden"))) void device_free(void* p);
__attribute__((visibility("hidden"))) size_t device_left();  // bytes that further arrays can take
}  // namespace mt
using mt::fail;

// Gives the scratch kept between calls back, where an allocation has failed (the context
// lock held); false when there is none or a call is using it.
bool drop_workspace(mt_context* c);

namespace {
#define CU(call)                                                                         \
  do {                                                                                   \
    cudaError_t e_ = (call);                                                             \
    if (e_ != cudaSuccess) return fail(MT_ERR_CUDA, "%s: %s", #call, cudaGetErrorString(e_)); \
  } while (0)

template <class T>
int dalloc(T** p, size_t count) {
  *p = nullptr;
  if (count == 0) count = 1;
  cudaError_t e = mt::device_malloc((void**)p, count * sizeof(T));
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(MT_ERR_NOMEM, "cudaMalloc(%zu B): %s", count * sizeof(T), cudaGetErrorString(e));
  }
  return MT_OK;
}
// As above, and once more without the scratch kept between the context's calls: what fits
// the device without it is not refused because of an earlier call (the context lock held).
template <class T>
int dalloc(mt_context* c, T** p, size_t count) {
  const int r = dalloc(p, count);
  return r == MT_ERR_NOMEM && drop_workspace(c) ? dalloc(p, count) : r;
}
template <class T>
void dfree(T*& p) {
  if (p) mt::device_free((void*)p);
  p = nullptr;
}
}  // namespace

// ----------------------------------------------------------------- structs
struct mt_context {
  int device = 0;
  int num_sms = 0;
  cudaStream_t stream = nullptr;
  std::recursive_mutex mu;
  int* d_scratch = nullptr;  // [0] work counter, [1] error for ray queries
  cudaEvent_t ev[8] = {};
  cudaEvent_t ready = nullptr;  // the call's results are on the device
  // compaction scratch, grown on demand
  unsigned long long* cs_status = nullptr;
  int* cs_words = nullptr;
  size_t cs_tiles = 0;
  // Scratch of the calls that use device memory only until they return (ray queries,
  // previews, batches, builds), kept between them: allocating and freeing it cost 80-280 us a
  // call. Used on `stream` under `mu`, so one call at a time; at most kWorkspaceMax
  // bytes are kept (a larger call allocates its own), given back when an allocation of
  // the context fails (drop_workspace) and with the context.
  char* ws = nullptr;
  size_t ws_bytes = 0;
  bool ws_used = false;  // a call is using it
  // streams of a batch's overlapping passes, created by the first batch
  struct PassStream {
    cudaStream_t stream = nullptr, side = nullptr;
    cudaEvent_t fork = nullptr, join = nullptr, done = nullptr;
  };
  std::vector<PassStream> pass_streams;
  std::vector<mt_job*> jobs;  // jobs whose streams join into `stream`
  std::vector<mt_server*> servers;  // served-mode schedulers on this context
  int* d_plain_err = nullptr;       // error latched by kernels launched by name
};

struct mt_buffer {
  mt_context* ctx;
  void* ptr;
  size_t bytes;
};

// MT_TRAVERSAL=bitstack (read once per process): the binary formats traverse
// without a deferred-node stack, as the reference does (bitstack_steps).
bool traversal_bitstack();

struct mt_scene {
  mt_context* ctx;
  int npoints = 0, nuvs = 0, nnormals = 0, ntri = 0, nmat = 0;
  std::vector<uint8_t> h_materials;
  char* d_mesh = nullptr;  // points, uvs, normals and faces, one allocation
  float4* d_points = nullptr;
  float2* d_uvs = nullptr;
  float4* d_normals = nullptr;
  Face* d_faces = nullptr;
  Material* d_materials = nullptr;
  int* d_light_faces = nullptr;
  int nlights = 0;
  // traversal layout
  float4* d_nodes = nullptr;
  float4* d_tris = nullptr;
  uint4* d_qnodes = nullptr;  // FP16 records (precision 1)
  uint4* d_wnodes = nullptr;  // wide BVH with 8-bit child boxes (precision 2)
  uint4* d_quad = nullptr;    // 4-wide FP16 nodes (precision 3): the surface-area tree's, the reference's
  int quad_again = 0;         // the first node of the latter
  int2* d_up = nullptr;       // parent links of the records (the stackless traversal)
  float4* d_wtris = nullptr;
  int nwide = 0, wdepth = 0;
  int nrec = 0, root_ref = 0, depth = 0, has_bvh = 0, precision = 0;
  // environment: the arrays below, one allocation
  char* d_env = nullptr;
  size_t env_bytes = 0;
  float4* d_env_rgb = nullptr;
  float* d_env_lum = nullptr;
  float* d_env_sat = nullptr;
  double* d_env_sat64 = nullptr;
  float* d_env_marg = nullptr;  // CDF tables of the whole map (dv::RegionTab)
  float* d_env_cond = nullptr;
  int env_w = 0, env_h = 0, env_present = 0;
  int grid_nu = 1600, grid_nv = 1600, grid_rx = 16, grid_ry = 32, grid_on = 0;  // grid_on: 0, 1 FP32, 2 FP64 SAT
  // textures: host images per (material, kind), the device pool and table
  struct HostTex {
    std::vector<int32_t> argb;
    int w = 0, h = 0;
  };
  std::vector<HostTex> h_tex;  // 4 per material: diffuse, glossy, roughness, mirror
  int* d_texels = nullptr;
  int4* d_tex_ref = nullptr;
  int tex_on = 0;
  unsigned version = 0;  // bumped when device arrays or the grid configuration change
  std::atomic<int> refs{0};  // served requests queued or running on this scene

  DevScene view() const {
    DevScene s{};
    s.nodes = d_nodes;
    s.qnodes = reinterpret_cast<const float4*>(d_qnodes);
    s.tris = d_tris;
    s.root_ref = root_ref;
    s.ntri = ntri;
    s.nrec = nrec;
    s.wnodes = d_wnodes;
    s.wtris = d_wtris;
    s.quad = d_quad;
    s.quad_again = quad_again;
    s.up = d_up;
    s.bitstack = d_up && traversal_bitstack();
    s.precision = (precision == 1 && d_qnodes) ? 1
                  : (precision == 2 && d_wnodes) ? 2
                  : (precision == 3 && d_quad)   ? 3
                                                 : 0;
    s.points = d_points;
    s.uvs = d_uvs;
    s.normals = d_normals;
    s.faces = d_faces;
    s.materials = d_materials;
    s.light_faces = d_light_faces;
    s.nlights = nlights;
    s.texels = d_texels;
    s.tex_ref = d_tex_ref;
    s.tex_on = tex_on;
    return s;
  }
  DevEnv env_view() const {
    DevEnv e{};
    e.rgb = d_env_rgb;
    e.lum = d_env_lum;
    e.sat = d_env_sat;
    e.w = env_w;
    e.h = env_h;
    e.present = env_present;
    e.grid_on = 0;
    e.env_marg = d_env_marg;
    e.env_cond = d_env_cond;
    return e;
  }
};

// What one pass in flight needs: path state and queues, its stream and the stream of
// its shadow rays.
struct PassBuf {
  FrameBufs fb{};
  cudaStream_t stream = nullptr;  // the slot's own for its first buffer
  cudaStream_t side = nullptr;    // shadow rays beside the next bounce's extension rays
  cudaEvent_t sfork = nullptr, sjoin = nullptr, done = nullptr;
};
// One in-flight frame's resources: pass buffers, film, parameters, control blocks (device
// arrays in the job's slab), and the stream its frames run on.
struct JobSlot {
  std::vector<PassBuf> bufs;               // passes of a frame that overlap
  float4 *film = nullptr, *film_c = nullptr;  // the slot's own film (not when passes go to the job's)
  Ctrl* d_ctrl = nullptr;                  // one per pass
  unsigned long long* d_status = nullptr;  // mode 0: compaction tile status, per pass and bounce
  PassParams* h_pp = nullptr;              // pinned, one per pass
  PassParams* d_pp = nullptr;
  cudaStream_t stream = nullptr;
  cudaEvent_t pfork = nullptr;  // the other buffers' streams start after the frame's set-up
  cudaEvent_t fork = nullptr, ev0 = nullptr, ev1 = nullptr, done = nullptr;
  cudaGraphExec_t graphs[2] = {nullptr, nullptr};  // of a frame among others, and of one alone (logged jobs)
};

struct mt_job {
  mt_context* ctx;
  mt_scene* scene;
  mt_render_config cfg;
  // Passes of one frame, and frames rendered one after the other, run side by side
  // in `logged` jobs: each logs its contributions, and they are added to the film in
  // pass order. merge: the caller's own frames in flight (cfg.inflight > 1).
  int nslots = 1;
  bool logged = false, merge = false;
  std::vector<JobSlot> slots;
  char* slab = nullptr;         // the slots' device arrays, the film and the totals, one allocation
  PassParams* h_pp = nullptr;   // the slots' pinned parameters, one allocation
  int next = 0;   // slot of the next frame
  int last = -1;  // slot of the last frame
  size_t status_stride = 0;
  unsigned char camera[64];
  int has_camera = 0;
  double frames = 0;                       // passes accumulated in the film
  // merge: each frame renders into its slot's film from zero, and a merge on the
  // slot's stream adds it into this film in frame order; logged without merge: the
  // film itself
  float4* d_film = nullptr;
  float4* d_film_c = nullptr;
  std::vector<cudaEvent_t> kev;            // profile: 2 + 3 * max_depth per pass
  unsigned long long* d_totals = nullptr;  // running [primary, extension, shadow, error]
  std::vector<Ctrl> h_ctrl;
  // asynchronous film reads
  static constexpr int kMaxReads = 8;
  struct Read {
    float* host = nullptr;
    cudaEvent_t ev = nullptr;
  };
  cudaStream_t rstream = nullptr;
  cudaEvent_t rfork = nullptr;
  cudaEvent_t rdone = nullptr;  // the latest read's event: one of reads[].ev
  Read reads[kMaxReads];        // pending reads, oldest at r_head
  int r_head = 0, r_count = 0;
  float4* d_resolved = nullptr;  // the film divided by its frames, for resolved reads (first one on)
  const float4* film() const { return d_film ? d_film : slots[0].film; }
  // adaptive light grid (mode 1, scene grid on, environment present)
  unsigned scene_version = 0;
  unsigned tune_version = 0;  // launch-shape version the graphs were captured with
  int64_t launches = 0;  // kernels of the render passes and film merges issued (mt_job_launches)
  int grid_on = 0, grid_fp64 = 0;
  int nu = 0, nv = 0, rx = 0, ry = 0;
  float* d_grid_func = nullptr;
  float* d_grid_sat = nullptr;
  float* d_grid_accum = nullptr;
  double* d_grid_sat64 = nullptr;
  // CDF tables of the grid-guided sampling: per cell (rebuilt with the cells'
  // SATs) and per tile of the map
  float *d_cell_marg = nullptr, *d_cell_cond = nullptr, *d_tile_marg = nullptr, *d_tile_cond = nullptr;
  int grid_tables = 1;
  int grid_frames = 0;           // frames that have accumulated into the grid since it was set up
  cudaEvent_t grid_ev = nullptr;  // recorded after the last grid update
  // displayed image (mt_image_argb), allocated on first use
  int32_t* d_argb = nullptr;
  float4* d_fb = nullptr;
  double* d_tone_part = nullptr;
  int* d_tone_cnt = nullptr;
  float* d_tone_tot = nullptr;
};

// Scratch of at least `bytes` for a call on the context's stream, the context lock
// held; release() when the call's work has finished. Arrays are taken from it in turn.
constexpr size_t kWorkspaceMax = 2ull << 30;
struct Workspace {
  mt_context* ctx = nullptr;
  char* base = nullptr;
  size_t at = 0;
  bool own = false;  // larger than what is kept
  int get(mt_context* c, size_t bytes);
  void release();
  template <class T>
  T* take(size_t count) {
    T* p = reinterpret_cast<T*>(base + at);
    at += round(count * sizeof(T));
    return p;
  }
  static size_t round(size_t b) { return (b + 255) / 256 * 256; }
};
// Touches the pages of a host buffer that the caller is about to fill from the device,
// until `ready` has happened: a fresh buffer's pages are then mapped while the GPU
// still works, not one fault after the other during the copy (33 MB: 2 ms).
void prefault(void* p, size_t bytes, cudaEvent_t ready);

// What the path state of passes that run side by side may take of the device: `most`
// bytes, and a quarter of what is left (the scratch kept between calls, which is given back
// where it is needed, counts as left), so that what a program makes next still fits
// where it did without them. The context lock held.
size_t overlap_bytes(mt_context* c, size_t most);

constexpr int kOpaqueBlack = (int)0xFF000000u;  // getIntARGB((0, 0, 0, 1))

// Per-pass camera constants of InitCameraRayDataJitter from a 64-byte
// CameraStruct, for a width x height frame.
void camera_constants(const void* cam64, int W, int H, PassParams& pp);

// Makes the context stream wait for every job stream's submitted work.
void join_jobs(mt_context* ctx);
// Waits for all work on the context and its jobs' streams, before device arrays
// that frames read are freed or rewritten.
int quiesce(mt_context* ctx);
// Waits for the requests running on the context's servers' lanes.
void servers_sync(mt_context* ctx);
// Mesh arrays on the device (mt_mesh.cu), on the context's stream and waited for. The
// first face with an index out of range, or (mat_only) with a material of nmat or
// more: INT_MAX when there is none.
int first_bad_face(mt_scene* s, int nmat, bool mat_only, int* bad);
// The faces whose material (emits[m] != 0) emits, in face order.
int list_light_faces(mt_scene* s, const std::vector<unsigned char>& emits);
// Triangle slots in the given order of faces.
int order_triangles(mt_scene* s, const std::vector<int>& order, float4* tris);
// Rebuild or drop the scene's derived traversal formats from its FP32 records:
// FP16 records (precision 1), 4-wide FP16 nodes (precision 3), and the wide BVH
// (precision 2, refresh_wide).
int refresh_qnodes(mt_scene* s);
// FP32 records of a surface-area-heuristic tree over the scene's triangle slots
// (mt_sah.cu), in ws, which the caller releases; NULL where that tree would be
// deeper than the traversal stack holds. Two triangles or more.
struct Workspace;
int build_sah_records(mt_scene* s, Workspace& ws, float4** recs_out);
int refresh_wide(mt_scene* s);
// MT_CDF_TABLES=0 turns the CDF tables of environment sampling off (the samplers
// then search the SATs directly; the tables hold the same values).
bool cdf_tables_enabled();

// Internal host-side types of libpiko_b200.so shared by runtime.cu and
// reyes_kernels.cu (not part of the C ABI).
#pragma once
#include <cstdio>
#include <algorithm>
#include <cstring>
#include <vector>

#include "piko_device.cuh"
#include "../../include/piko_b200.h"

using namespace piko;

struct ReyesState;

struct piko_ctx {
  int device = 0;
  int sms = 0;
  bool time_kernels = false;
  cudaStream_t stream = nullptr;
  char err[512] = {0};
};

struct piko_pipe {
  piko_ctx* ctx = nullptr;
  int kind = 0;  // 1 raster, 2 reyes
  int tile = 16;
  int ctas_per_sm = 0;
  uint32_t chunk = 0;
  float split_threshold = 4.0f;
  int max_splits = 20;
  int dice_grid = 0;
  int samples_per_pixel = 1;
  uint32_t sample_seed = 0;
  int phong = 0;
};

enum { kPipeRaster = 1, kPipeReyes = 2 };

// Tile grid of a W x H framebuffer cut into T x T tiles; returns the tile count.
inline int tiles_for(int W, int H, int T, int* tx, int* ty)
{
  *tx = (W + T - 1) / T;
  *ty = (H + T - 1) / T;
  return *tx * *ty;
}

// The fields of a RasterSceneDev that follow from the framebuffer size, the
// triangle count and the tile edge T: the reference's 8x8 and 32x32 bin grids,
// the submission-order constants, the tile grid and the viewport halves.
// Every path that fills a RasterSceneDev starts from this (the rest is zero).
inline void scene_dev_geometry(RasterSceneDev& d, int W, int H, int N, int T)
{
  memset(&d, 0, sizeof(d));
  d.W = W; d.H = H;
  d.nBx = W / kRefBin; d.nBy = H / kRefBin;
  d.nVS = (W / kVsBin) * (H / kVsBin);
  d.N = N;
  scene_vs_consts(d);
  tiles_for(W, H, T, &d.tiles_x, &d.tiles_y);
  d.tiles_x_m = divmod_magic((uint32_t)d.tiles_x);
  d.halfW = 0.5f * (float)W;
  d.halfH = 0.5f * (float)H;
}

inline piko_status set_err(piko_ctx* ctx, piko_status st, const char* fmt, const char* detail = "")
{
  if (ctx) snprintf(ctx->err, sizeof(ctx->err), fmt, detail);
  return st;
}

#define CU(ctx, call)                                                                 \
  do {                                                                                \
    cudaError_t e_ = (call);                                                          \
    if (e_ != cudaSuccess) {                                                          \
      return set_err((ctx), e_ == cudaErrorMemoryAllocation ? PIKO_ERR_OOM : PIKO_ERR_CUDA, \
                     "%s", cudaGetErrorString(e_));                                   \
    }                                                                                 \
  } while (0)

// Allocations of device and of pinned memory.  A failed one leaves null and no
// error behind: cudaGetLastError after a later launch is to tell of that launch.
template <class T>
inline cudaError_t dalloc(T** p, size_t count)
{
  *p = nullptr;
  if (count == 0) count = 1;
  const cudaError_t e = cudaMalloc((void**)p, count * sizeof(T));
  if (e) { *p = nullptr; cudaGetLastError(); }
  return e;
}
template <class T>
inline cudaError_t halloc(T** p, size_t count)
{
  *p = nullptr;
  const cudaError_t e = cudaMallocHost((void**)p, count * sizeof(T));
  if (e) { *p = nullptr; cudaGetLastError(); return e; }
  memset((void*)*p, 0, count * sizeof(T));
  return cudaSuccess;
}
template <class T>
inline void dfree(T*& p)
{
  if (p) cudaFree(p);
  p = nullptr;
}

// Is st recording a graph?  (What it is given then runs later, or never.)
inline cudaError_t stream_capturing(cudaStream_t st, bool* capturing)
{
  cudaStreamCaptureStatus c = cudaStreamCaptureStatusNone;
  const cudaError_t e = cudaStreamIsCapturing(st, &c);
  *capturing = c != cudaStreamCaptureStatusNone;
  return e;
}

// The frames of one scene or batch follow one another whichever streams they are
// given: a frame leaves the working counters as the next one needs them, so two at
// once would spoil them for every later frame too.  before() makes a frame's stream
// wait for the frame before, after() marks where the frame ends.  The object's own
// stream is marked only once another one is used (it lives as long as the object);
// a caller's stream may be destroyed behind the frame, and its handle given to
// another, so it is marked at once and told by its id.  Frames that a stream capture
// records are left out: their order is the caller's.
struct FrameOrder {
  cudaEvent_t ev = nullptr;
  unsigned long long id = 0;         // the last frame's stream
  bool any = false;
  cudaStream_t unmarked = nullptr;   // the object's own stream, if the last frame ran there

  cudaError_t mark(cudaStream_t st)
  {
    cudaError_t e = ev ? cudaSuccess : cudaEventCreateWithFlags(&ev, cudaEventDisableTiming);
    if (!e) e = cudaEventRecord(ev, st);
    return e;
  }
  cudaError_t before(cudaStream_t st)
  {
    if (!any || st == unmarked) return cudaSuccess;
    bool capturing = false;
    unsigned long long now = 0;
    cudaError_t e = stream_capturing(st, &capturing);
    if (e || capturing) return e;
    if ((e = cudaStreamGetId(st, &now)) || now == id) return e;
    if (unmarked) {
      if ((e = mark(unmarked))) return e;
      unmarked = nullptr;
    }
    return cudaStreamWaitEvent(st, ev, 0);
  }
  cudaError_t after(cudaStream_t st, cudaStream_t own)
  {
    if (any && st == unmarked) return cudaSuccess;
    bool capturing = false;
    cudaError_t e = stream_capturing(st, &capturing);
    if (e || capturing) return e;
    if ((e = cudaStreamGetId(st, &id))) return e;
    any = true;
    unmarked = st == own ? st : nullptr;
    return unmarked ? cudaSuccess : mark(st);
  }
  void release()
  {
    if (ev) cudaEventDestroy(ev);
    *this = FrameOrder();
  }
};

// A launch sequence's counters, and a scene record: the table of a captured frame of
// one scene.
struct CounterBlock {
  FrameCounters ctr;
  RasterSceneDev one;
};

// Frame scratch shared by every scene drawn in one launch sequence.
struct RasterScratch {
  TriSetup* setup = nullptr;
  uint32_t* tile_cnt = nullptr;
  uint2* tile_span = nullptr;
  uint32_t* tile_list = nullptr;
  unsigned long long* pair_tl = nullptr;  // count-pass pair records, [list_cap] each
  uint32_t* pair_g = nullptr;
  uint2* large_seg = nullptr;   // large-triangle segment items
  uint32_t seg_cap = 0;
  WalkTri* large_walk = nullptr;  // walk records of the large triangles, [seg_cap]: each has a segment
  uint32_t* hdone = nullptr;                // finished chunks, per key slot and bin of the tile
  unsigned long long* chunk_keys = nullptr; // tile * tile keys per key slot
  ChunkDesc* chunk_desc = nullptr;
  uint32_t chunk_cap = 0, key_cap = 0;
  uint32_t key_stride = 0;                  // keys per key slot (tile * tile)
  BinWork* work = nullptr;
  FrameCounters* ctr = nullptr;
  FrameCounters* h_ctr = nullptr;  // pinned; the fragment kernel writes its bin part
  bool clean = false;              // tile_cnt and work are all zero (every frame leaves them so)
  bool captured = false;           // a caller's capture holds a frame on them: cleared before every frame
  RasterSceneDev* d_scenes = nullptr;      // scene table of launch sequences over several scenes
  RasterSceneDev* one_scene = nullptr;     // that of a caller's captured frame of one scene (beside ctr)
  std::vector<RasterSceneDev> h_scenes;    // the last frame's records; pageable: a copy from it has read it when the call returns
  RasterSceneDev* cap_scenes = nullptr;    // pinned: the source of a copy that a stream capture records
  RasterSceneDev* cap_one = nullptr;       // the same for one scene (beside h_ctr)
  uint32_t tris_cap = 0, tiles_cap = 0, list_cap = 0;
  int scenes_cap = 0;
  uint32_t cov_cap = 0;
  uint32_t* cov_tri = nullptr;
  uint32_t* cov_pix = nullptr;
  cudaEvent_t ev[5] = {};
  bool ev_made = false;

  void release()
  {
    dfree(setup); dfree(tile_cnt); dfree(tile_span); dfree(tile_list); dfree(pair_tl); dfree(pair_g);
    dfree(large_seg); dfree(large_walk); dfree(hdone); dfree(chunk_keys);
    dfree(chunk_desc);
    dfree(work); dfree(ctr); dfree(d_scenes); dfree(cov_tri); dfree(cov_pix);   // (ctr begins its CounterBlock)
    if (h_ctr) cudaFreeHost(h_ctr);
    if (cap_scenes) cudaFreeHost(cap_scenes);
    h_ctr = nullptr; cap_scenes = nullptr; one_scene = nullptr; cap_one = nullptr;
    clean = false;
    if (ev_made) for (auto& e : ev) cudaEventDestroy(e);
    ev_made = false;
    tris_cap = tiles_cap = list_cap = chunk_cap = key_cap = seg_cap = key_stride = 0;
    scenes_cap = 0;
    cov_cap = 0;
  }

  // Heavy-tile queue.  A heavy tile has more than `queue_min` list entries, so
  // at most list_cap / (queue_min + 1) of them exist, and their lists make at
  // most list_cap / chunk further chunks: descriptors for all of these.  Key
  // slots, T * T keys each, are for lists in several chunks only; they start at
  // an estimate and grow after a frame reports that it needed more (regrow).
  cudaError_t ensure_heavy(uint32_t n_tiles, int T, uint32_t chunk, uint32_t queue_min)
  {
    cudaError_t e = cudaSuccess;
    const uint32_t need = std::min<uint32_t>(n_tiles, list_cap / (queue_min + 1)) + list_cap / chunk + 1;
    if (need > chunk_cap) {
      dfree(chunk_desc);
      chunk_cap = 0;
      if ((e = dalloc(&chunk_desc, need))) return e;
      chunk_cap = need;
    }
    const uint32_t stride = (uint32_t)(T * T), want = list_cap / (8 * chunk) + 64;
    if (want > key_cap || stride != key_stride) return grow_keys(std::max(want, stride == key_stride ? key_cap : 0u), stride);
    return cudaSuccess;
  }

  // The tile lists and the count passes' pair records (the same number of
  // entries) grow together.
  cudaError_t grow_list(uint32_t n)
  {
    dfree(tile_list); dfree(pair_tl); dfree(pair_g);
    list_cap = 0;
    cudaError_t e = dalloc(&tile_list, n);
    if (!e) e = dalloc(&pair_tl, n);
    if (!e) e = dalloc(&pair_g, n);
    if (!e) list_cap = n;
    return e;
  }

  cudaError_t grow_segs(uint32_t n)
  {
    dfree(large_seg);
    dfree(large_walk);
    seg_cap = 0;
    cudaError_t e = dalloc(&large_seg, n);
    if (!e) e = dalloc(&large_walk, n);
    if (!e) seg_cap = n;
    return e;
  }

  // n key slots of `stride` keys each, with a counter for each 8x8 bin
  cudaError_t grow_keys(uint32_t n, uint32_t stride)
  {
    dfree(chunk_keys);
    dfree(hdone);
    key_cap = 0;
    cudaError_t e = dalloc(&chunk_keys, (size_t)n * stride);
    if (!e) e = dalloc(&hdone, (size_t)n * (stride / (kRefBin * kRefBin)));
    if (!e) { key_cap = n; key_stride = stride; }
    return e;
  }

  // After a frame whose counters report a queue overflow: grows what
  // overflowed (the tile lists and / or the key slots) so that the
  // frame can be drawn again.
  cudaError_t regrow(const BinCounts& c)
  {
    cudaError_t e = cudaSuccess;
    // the lists hold every pair, and each pair partition its share
    const uint32_t need = std::max<uint32_t>(c.list_total, (uint32_t)std::min<unsigned long long>(
                                                               (unsigned long long)c.pair_part_max * kPairParts,
                                                               0xffffffffull));
    if (need > list_cap || c.pair_part_max > list_cap / kPairParts) {
      if ((e = grow_list(need + need / 4 + 1024))) return e;
    }
    const uint32_t keys = (uint32_t)(c.heavy_acc >> 32);
    if (key_stride && keys > key_cap) {
      if ((e = grow_keys(keys + keys / 4 + 64, key_stride))) return e;
    }
    // every large triangle has at least one segment: seg_cap bounds both
    const uint32_t segs = std::max((uint32_t)c.large_acc, (uint32_t)(c.large_acc >> 32));
    if (segs > seg_cap) {
      if ((e = grow_segs(segs + segs / 4 + 1024))) return e;
    }
    return cudaSuccess;
  }

  // Buffers for a frame.  A capacity stands only while all of its buffers do: one
  // whose allocation failed part way is 0 until the next frame allocates again.
  cudaError_t ensure(uint32_t n_tris, uint32_t n_tiles, uint32_t list_need, int n_scenes)
  {
    cudaError_t e = cudaSuccess;
    if (n_tris > tris_cap || !setup) {
      dfree(setup);
      tris_cap = 0;
      if ((e = dalloc(&setup, n_tris))) return e;
      tris_cap = n_tris;
    }
    // segment items of large triangles: an estimate, grown after an overflow
    if (tris_cap / 8 + 1024 > seg_cap && (e = grow_segs(tris_cap / 8 + 1024))) return e;
    if (n_tiles > tiles_cap) {
      clean = false;
      dfree(tile_cnt); dfree(tile_span);
      tiles_cap = 0;
      if ((e = dalloc(&tile_cnt, n_tiles))) return e;
      if ((e = dalloc(&tile_span, n_tiles))) return e;
      tiles_cap = n_tiles;
    }
    if (list_need > list_cap) {
      if ((e = grow_list(list_need))) return e;
    }
    if (!work) {
      clean = false;
      if ((e = dalloc(&work, 1))) return e;
    }
    if (!ctr) {
      CounterBlock* p;
      if ((e = dalloc(&p, 1))) return e;
      ctr = &p->ctr;
      one_scene = &p->one;
    }
    if (!h_ctr) {
      CounterBlock* p;
      if ((e = halloc(&p, 1))) return e;
      h_ctr = &p->ctr;
      cap_one = &p->one;
    }
    if (n_scenes > 1 && n_scenes > scenes_cap) {
      dfree(d_scenes);
      if (cap_scenes) cudaFreeHost(cap_scenes);
      cap_scenes = nullptr;
      scenes_cap = 0;
      if ((e = dalloc(&d_scenes, n_scenes))) return e;
      if ((e = halloc(&cap_scenes, n_scenes))) return e;
      scenes_cap = n_scenes;
    }
    if (!ev_made) {
      for (auto& ev_ : ev) if ((e = cudaEventCreate(&ev_))) return e;
      ev_made = true;
    }
    return cudaSuccess;
  }
};

struct piko_scene {
  piko_pipe* pipe = nullptr;
  int kind = 0;
  int W = 0, H = 0, N = 0;
  float4* pos = nullptr;
  float4* nrm = nullptr;
  float* pos3 = nullptr;   // packed scenes: float3 positions and normals instead
  float* nrm3 = nullptr;
  int packed = 0;
  float4* col = nullptr;
  float2* uv = nullptr;
  uchar4* tex = nullptr;
  int tex_w = 0, tex_h = 0;
  float* wtri_xyz = nullptr;
  uint32_t* wtri_icol = nullptr;
  float4* patches = nullptr;
  uint32_t* fb = nullptr;
  float* depth = nullptr;
  piko_const_state state{};
  RasterScratch scr;
  cudaStream_t own_stream = nullptr;
  cudaStream_t last_stream = nullptr;
  bool pending = false;
  bool timed = false;
  FrameOrder order;
  ReyesState* reyes = nullptr;
};

// Launch configuration of a raster launch sequence: tile edge, persistent
// CTAs per SM (0 = the kernel's occupancy) and list entries per chunk of the
// tile queue (0 = default_chunk).
struct TuneCfg {
  int tile = 8;
  int ctas_per_sm = 0;
  uint32_t chunk = 0;
  bool operator==(const TuneCfg& o) const { return tile == o.tile && ctas_per_sm == o.ctas_per_sm && chunk == o.chunk; }
};
inline TuneCfg pipe_cfg(const piko_pipe* p) { return TuneCfg{p->tile, p->ctas_per_sm, p->chunk}; }

// Scene-size buckets of the tuner: 4 resolution classes x 4 triangle classes.
constexpr int kTuneBuckets = 16;
int tune_bucket(int W, int H, int N);

struct piko_tuner {
  TuneCfg cfg[kTuneBuckets];
  float ms[kTuneBuckets] = {};
  bool tuned[kTuneBuckets] = {};
};

// Scenes of a batch that share one launch configuration: one launch sequence
// over all of them, on its own branch of the batch's stream fork.
struct BatchGroup {
  TuneCfg cfg;
  std::vector<piko_scene*> scenes;
  RasterScratch scr;
  RasterSceneDev recorded;        // a single scene's record in the batch's graph
  bool recorded_clears = false;   // that graph clears the counters (scr.captured)
  cudaStream_t stream = nullptr;  // the branch (group 0 runs on the caller's stream)
  cudaEvent_t done = nullptr;
};

struct piko_batch {
  piko_ctx* ctx = nullptr;
  std::vector<piko_scene*> scenes;
  std::vector<BatchGroup*> groups;
  cudaEvent_t fork = nullptr;
  cudaStream_t last_stream = nullptr;
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t graph_exec = nullptr;
  bool pending = false;
  bool counted = true;   // the groups' h_ctr hold all counts of the last finished frame
  FrameOrder order;
};
piko_status batch_make(piko_ctx* ctx, piko_scene* const* scenes, int n, const TuneCfg* cfgs, piko_batch** out);

// Reyes device path (reyes_kernels.cu)
piko_status piko_reyes_run(piko_scene* s, cudaStream_t st, bool timed);
piko_status piko_reyes_finish(piko_scene* s);
piko_status piko_reyes_stats(piko_scene* s, piko_frame_stats* out);
void piko_reyes_release(piko_scene* s);
// Shared Reyes work buffers: frames on one stream may use one set.
ReyesState* reyes_buffers_new();
void reyes_buffers_free(ReyesState* b);
void reyes_borrow_buffers(piko_scene* s, ReyesState* b);

// One draw of a launch sequence: a resident mesh seen with one camera state,
// rendered into one framebuffer / depth buffer.
struct RasterDraw {
  const piko_scene* mesh;
  const piko_const_state* state;
  uint32_t* fb;
  float* depth;
};
// chunk: list entries per chunk of the tile queue (default_chunk when 0); lists
// longer than kQueueMin entries are queued as chunks
// (the parts of a 32-px list that one bin takes fill a pass better from longer
// chunks: 200K triangles at 1080p 206 -> 186 us, 24-scene batch 494 -> 457)
inline uint32_t default_chunk(int tile) { return tile == 32 ? 128u : 64u; }
constexpr uint32_t kQueueMin = 8;
// The scene records that a launch sequence draws with: the scenes' present state; the
// last frame's (scr.h_scenes); or those in the batch's own graph.
enum class Records { now, kept, graph };
piko_status enqueue_raster_draws(piko_ctx* ctx, const RasterDraw* draws, int n, RasterScratch& scr, int T, int ctas,
                                 cudaStream_t st, bool timed, bool coverage, uint32_t chunk = 0,
                                 Records records = Records::now);
// One launch sequence over resident scenes drawn with their own camera states.
piko_status enqueue_raster(piko_ctx* ctx, piko_scene* const* scenes, int n, RasterScratch& scr, const TuneCfg& cfg,
                           cudaStream_t st, bool timed, bool coverage, Records records = Records::now);
int raster_ctas(piko_ctx* ctx, int tile, int ctas_per_sm);

// Device-side data layout and scalar helpers shared by the raster and Reyes
// kernels of piko-public_b200.
//
// Arithmetic pinning.  Every kernel file is compiled with --fmad=false and the
// default IEEE division and square root, so each float expression below is the
// sequence of individually rounded operations the reference's CPU backend
// performs (g++ on x86-64, SSE, no contraction).  The conversions the
// reference gets from x86 instructions are spelled out explicitly:
//   (int)f       -> cvt_i32_x86  (cvttss2si: INT_MIN for NaN / out of range)
//   (unsigned)f  -> cvt_u32_x86  (64-bit cvttss2si, low 32 bits kept)
// and the 28.4 fixed-point edge functions use wrapping int32 arithmetic, as the
// reference's int expressions do on the CPU.
#pragma once
#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

namespace piko {

// --------------------------------------------------------------- constants
constexpr int kVsBin = 32;          // VertexShaderStage bin size (vertexShader.pikostage:18)
constexpr int kVsChunk = 512;       // ids per VS-bin chunk, assignBin (vertexShader.pikostage:27)
constexpr int kRefBinLg2 = 3;       // RasterStage bin size 8 (raster.pikostage:14)
constexpr int kRefBin = 1 << kRefBinLg2;
constexpr int kGuard = 225 << 4;    // guard band (rasterMacros.h:37)
constexpr uint32_t kClearColor = 0xff663313u;  // PikoScreen initial colour (stage.h:83-85)

// tile scan: threads per block and tile counts per thread (scan_tiles)
constexpr int kScanThreads = 256;
constexpr int kScanItems = 2;
constexpr int kScanTile = kScanThreads * kScanItems;

// 8x8 raster queue: short lists (at most kQueueMax entries, one per lane) are
// drawn in groups of up to kLightGroup consecutive tiles
constexpr int kLightGroup = 8;
constexpr uint32_t kQueueMax = 32;

// 16/32-px tiles: a heavy tile's list is cut into at most kMaxTileChunks
// chunks of at least `chunk` entries (different warps rasterize them; the last
// one merges their per-pixel keys, so the merge reads a bounded number of
// chunk key buffers).  8x8 tiles use chunks of exactly `chunk` entries.
constexpr uint32_t kMaxTileChunks = 32;
__host__ __device__ __forceinline__ uint32_t tile_chunk_entries(uint32_t cnt, uint32_t chunk, bool t8)
{
  if (t8) return chunk;
  const uint32_t c = (cnt + kMaxTileChunks - 1) / kMaxTileChunks;
  return c > chunk ? c : chunk;
}
__host__ __device__ __forceinline__ uint32_t tile_chunks(uint32_t cnt, uint32_t chunk, bool t8)
{
  const uint32_t c = tile_chunk_entries(cnt, chunk, t8);
  return (cnt + c - 1) / c;
}

// frame status bits (the C ABI maps them to piko_status)
constexpr uint32_t kStatusListOverflow = 1u << 0;
constexpr uint32_t kStatusUpolyOverflow = 1u << 2;
constexpr uint32_t kStatusPatchOverflow = 1u << 3;
constexpr uint32_t kStatusDepthNeverSettles = 1u << 4;
constexpr uint32_t kStatusBarrierTimeout = 1u << 5;

// ------------------------------------------------- programmatic dependent launch
// A kernel launched with programmatic stream serialisation may start while the
// previous kernel of its stream still runs; pdl_wait() blocks until that
// kernel has completed and its memory is visible, so a kernel that calls it
// before touching global memory behaves exactly as if launched normally (the
// instruction does nothing for a normal launch).  pdl_trigger() lets the next
// such kernel be scheduled once every CTA of this one has started.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// --------------------------------------------------------------- scalar helpers
__device__ __forceinline__ int32_t cvt_i32_x86(float f)
{
  return (f >= -2147483648.0f && f < 2147483648.0f) ? __float2int_rz(f) : INT32_MIN;
}
__device__ __forceinline__ uint32_t cvt_u32_x86(float f)
{
  // |f| < 2^31: the 32-bit truncation has the same low 32 bits as the 64-bit one
  if (fabsf(f) < 2147483648.0f) return (uint32_t)__float2int_rz(f);
  return (f > -9223372036854775808.0f && f < 9223372036854775808.0f) ? (uint32_t)__float2ll_rz(f) : 0u;
}
__device__ __forceinline__ int32_t wadd(int32_t a, int32_t b) { return (int32_t)((uint32_t)a + (uint32_t)b); }
__device__ __forceinline__ int32_t wsub(int32_t a, int32_t b) { return (int32_t)((uint32_t)a - (uint32_t)b); }
__device__ __forceinline__ int32_t wmul(int32_t a, int32_t b) { return (int32_t)((uint32_t)a * (uint32_t)b); }
__device__ __forceinline__ int32_t wshl(int32_t a, int s) { return (int32_t)((uint32_t)a << s); }
// n / d and n % d for any 32-bit n and d >= 1, given m = 0xffffffff / d: the
// high product is the quotient or one less, fixed by one comparison.
__host__ __device__ __forceinline__ uint32_t divmod_magic(uint32_t d) { return 0xffffffffu / d; }
__device__ __forceinline__ uint32_t fast_divmod(uint32_t n, uint32_t d, uint32_t m, uint32_t& r)
{
  uint32_t q = __umulhi(n, m);
  r = n - q * d;
  if (r >= d) { ++q; r -= d; }
  return q;
}
// std::min / std::max on the CPU (piko/math.h:24-52): NaN handling differs from fminf
__device__ __forceinline__ float std_minf(float a, float b) { return (b < a) ? b : a; }
__device__ __forceinline__ float std_maxf(float a, float b) { return (a < b) ? b : a; }

// --------------------------------------------------------------- scenes
// kInputWtriWorld: the raster_wtri payload of the pipe built without
// VTX_PRETRANSFORM (world positions the vertex stage transforms; no colours)
enum : int { kInputSoA = 0, kInputWtri = 1, kInputWtriWorld = 2 };

// One raster scene as the kernels see it.  All device pointers are owned by the
// scene object of the runtime.
struct RasterSceneDev {
  // geometry
  int W, H;
  int nBx, nBy;          // reference 8x8 bin grid (W/8, H/8; floor)
  int nVS;               // VertexShaderStage bins ((W/32)*(H/32))
  int N;                 // triangles
  // submission order constants: C = ceil(N / 512) chunks over nVS bins,
  // C / nVS and C % nVS, the bin of the last chunk, the empty ids of the last chunk
  uint32_t vs_m;         // divmod_magic(nVS)
  uint32_t vs_q, vs_rem, vs_last, vs_deficit, vs_chunks;
  int input_kind;
  int light_mode;
  int tiles_x, tiles_y;  // tile grid of this scene (tile size from RasterFrameArgs)
  uint32_t tiles_x_m;    // divmod_magic(tiles_x)
  uint32_t tile_base;    // first global tile id
  uint32_t tri_base;     // first global triangle-setup slot
  float halfW, halfH;
  float vp[16];
  float light[3];
  float eye[3];
  // inputs (SoA float4 [3][N] per attribute; or the pre-transformed payload)
  const float4* pos;
  const float4* nrm;
  const float* pos3;     // non-null: positions and normals are float3 [3][N] (pos / nrm unused)
  const float* nrm3;
  const float4* col;
  const float2* uv;      // textured variant only ([3][N])
  const float* wtri_xyz; // [N][9] (screen, or world for kInputWtriWorld)
  const uint32_t* wtri_icol;  // [N][3]
  const uchar4* tex;     // [TH][TW], power-of-two sizes
  int tex_w, tex_h;
  // outputs
  uint32_t* fb;          // [H][W] RGBA8 (R in the low byte), row 0 = bottom
  float* depth;          // [H][W]
};

// The submission-order constants of a scene of N triangles and nVS bins.
__host__ __device__ inline void scene_vs_consts(RasterSceneDev& d)
{
  const uint32_t nvs = (uint32_t)d.nVS, n = (uint32_t)d.N;
  const uint32_t C = (n + kVsChunk - 1) / kVsChunk;
  d.vs_m = divmod_magic(nvs);
  d.vs_chunks = C;
  d.vs_q = C / nvs;
  d.vs_rem = C % nvs;
  d.vs_last = C ? (C - 1) % nvs : 0u;
  d.vs_deficit = C * kVsChunk - n;
}

// Per-triangle setup record written by the setup kernel, read by the binning,
// raster and resolve phases.  80 bytes, 16-byte aligned.
struct __align__(16) TriSetup {
  int32_t x[3], y[3];   // 28.4 fixed point
  float z[3];
  uint32_t c[3];        // ABGR vertex colours
  float inv;            // 1.0f / (float)barydenom
  uint32_t bxr, byr;    // clamped reference-bin range: lo | hi << 16
  int32_t hix, hiy;     // pixel bounding box high corner (28.4, rounded up to 16 px)
  uint32_t rank1;       // submission rank + 1 (0 = culled)
  uint32_t flags;       // kTriRisk (no tile-level reject), kTriAreaRisk
  uint32_t id;          // triangle index within its scene
};
static_assert(sizeof(TriSetup) == 80, "TriSetup layout");

constexpr uint32_t kTriRisk = 1u;      // an edge value may wrap inside the bin range
constexpr uint32_t kTriAreaRisk = 2u;  // the area may wrap: its reciprocal says nothing of the depth's range

// What the binning passes (setup, large count, scan) count.  The heavy-tile
// queue and the large-triangle queue each reserve two ranges with one 64-bit
// atomic.
constexpr uint32_t kPairParts = 128;
struct BinCounts {
  uint32_t status;
  uint32_t list_total;           // list entries
  uint32_t kept;
  uint32_t pair_part_max;        // largest partition fill asked for (past its capacity: overflow)
  // (triangle, tile) pairs that pass the tile-level reject but cannot hold a
  // covered pixel: part of the bin queues of the reference, not listed here
  unsigned long long skipped;
  unsigned long long risk;
  unsigned long long heavy_acc;  // key slots << 32 | items (chunks, or without chunk buffers heavy tiles)
  unsigned long long large_acc;  // large triangles << 32 | their box-tile segments
};

// A frame's result: the binning counts as the scatter pass found them, and what
// the fragment kernel counts (started at 0 by the scatter pass).
struct FrameCounters {
  BinCounts bin;
  unsigned long long covered;
  uint32_t work_next;
  uint32_t cov_count;
};

// Per-frame working counters.  No launch clears them before a frame (the
// scene-record copy and three memsets that used to precede the setup kernel
// took 15 us of a frame, a fifth of the 1080p forest's): they are zero between
// frames because a later kernel of the frame sets back what an earlier one
// used -- raster_scatter the counts, the fragment kernels the pair partitions,
// scan_tiles the tile counters it has read.  The host
// clears them when they are allocated and after a launch that failed.
struct BinWork {
  BinCounts bin;
  // The count passes record their (triangle, tile) pairs in kPairParts
  // partitions of list_cap / kPairParts slots each (chosen by block and warp),
  // so that slot reservations spread over kPairParts counters instead of
  // queueing on one address.
  uint32_t pair_part[kPairParts];
};

// A triangle's box-tile walk: its reference bin range, first tile and tiles per
// row (with the divide-by-tw magic), global setup slot and scene tile base, the
// part of the box that is listed, and for 8x8 tiles the reference's
// trivial-reject value of each edge at the first bin with its change per bin in
// x and y (wrapping int32, so equal to evaluating each bin directly), for larger
// tiles the 28.4 vertices.  Large triangles keep theirs in memory for the
// segment walk (96 bytes, 16-byte aligned).
struct __align__(16) WalkTri {
  int32_t bx1, bx2, by1, by2;
  int32_t tx1, ty1, tw;
  uint32_t tw_m;          // divmod_magic(tw)
  uint32_t gidx;
  uint32_t tile_base;
  int32_t tiles_x;
  uint32_t flags;
  uint32_t ltx, lty;      // columns and rows of the box that are listed: lo | hi << 16 (lty 1: none)
  union {
    struct { int32_t tr0[3], trx[3], try_[3]; };
    struct { int32_t x[3], y[3]; };
  };
};
static_assert(sizeof(WalkTri) == 96, "WalkTri layout");

// A chunk of a heavy tile's list, written by the scan: all that the warp that
// takes it needs, in one 32-byte read.
struct __align__(16) ChunkDesc {
  uint32_t tile;
  uint32_t off, n;     // list entries [off, off + n)
  uint32_t ks;         // the tile's first key slot (lists in several chunks)
  uint32_t j, nch;     // chunk j of the tile's nch
  uint32_t pad[2];
};
static_assert(sizeof(ChunkDesc) == 32, "ChunkDesc layout");

// raster_setup's launch for n triangles, given a full wave of CTAs: one wave at
// most; every CTA takes the same number of equal batches, and a small scene is
// spread over the whole device, at least 8 triangles a batch.  No triangles: no
// CTAs.
struct SetupShape {
  uint32_t batch;    // triangles a CTA takes at a time
  uint32_t blocks;
};
inline SetupShape setup_shape(uint32_t n, uint32_t wave, uint32_t threads)
{
  if (n == 0) return {8u, 0u};
  const uint64_t n64 = n, full = (uint64_t)wave * threads;
  const uint64_t slots = (n64 + full - 1) / full * wave;
  uint64_t batch = (n64 + slots - 1) / slots;
  batch = batch > 32 ? (batch + 31) & ~31ull : batch < 8 ? 8 : batch;
  const uint64_t blocks = (n64 + batch - 1) / batch;
  return {(uint32_t)batch, (uint32_t)(blocks < wave ? blocks : wave)};
}

struct RasterFrameArgs {
  RasterSceneDev one;       // the scene of a one-scene frame: it travels with the launch, no copy precedes the frame
  const RasterSceneDev* scenes;  // [n_scenes] when there are several (or a capture holds one); else null
  int n_scenes;
  int tile;                 // tile edge in pixels: 8, 16 or 32
  uint32_t n_tris_total;    // sum of N
  uint32_t n_tiles_total;
  uint32_t batch;           // triangles a raster_setup CTA takes at a time (set by the launch)
  TriSetup* setup;          // [n_tris_total]; written only for triangles that reach a bin (rank1 != 0)
  uint32_t* tile_cnt;       // [n_tiles_total]
  uint2* tile_span;         // [n_tiles_total] first list entry, entries
  uint32_t* tile_list;      // [list_cap]
  uint32_t list_cap;
  uint32_t spill;           // a full pair partition spills into the next ones (lists of a fixed size)
  uint32_t* heavy;          // [heavy_cap] heavy tiles, when there are no chunk buffers
  uint32_t heavy_cap;
  // one record per (triangle, tile) pair, written by the count passes: the
  // tile | the pair's index in the tile's list << 32 (the old value of the
  // tile's counter), and the triangle's setup slot; [list_cap] each (pairs
  // and list entries are the same set, so one capacity bounds both)
  unsigned long long* pair_tl;
  uint32_t* pair_g;
  uint2* large_seg;         // [seg_cap] (large triangle, segment index) of every box-tile segment of a large triangle
  uint32_t seg_cap;
  WalkTri* large_walk;      // [big_cap] walk record of each large triangle, written by raster_setup
  uint32_t big_cap;
  // Heavy tiles (lists longer than queue_min) are split into chunks
  // (tile_chunk_entries) that different warps rasterize.  Of a tile in several
  // chunks each leaves its per-pixel keys (tile * tile of them) in its key slot;
  // the warp that completes the last chunk takes the per-pixel minimum over the
  // tile's chunks and resolves the tile.  Without chunk buffers (chunk_desc
  // null) heavy tiles are rasterized whole.
  uint32_t chunk;
  uint32_t queue_min;       // tiles with more entries than this are queued as chunks
  uint32_t group;           // 8x8 tiles per short-list group (at most kLightGroup); 16/32-px tiles: 8x8 bins
                            // of a quad that a work item draws (1 or 4)
  ChunkDesc* chunk_desc;    // [chunk_cap]; the chunks of a tile are consecutive
  uint32_t chunk_cap;
  uint32_t* hdone;          // [key_cap][bins per tile] finished chunks, at a tile's first key slot
  unsigned long long* chunk_keys;  // [key_cap][tile * tile]
  uint32_t key_cap;
  BinWork* work;
  FrameCounters* ctr;
  BinCounts* host_bin;      // pinned host memory (or null): the fragment kernel leaves ctr->bin there, so that
                            // checking a frame takes no copy
  // coverage dump (parity tests): one (triangle id, pixel index) record per
  // covered sample, appended in any order; counted in ctr->cov_count
  uint32_t* cov_tri;
  uint32_t* cov_pix;
  uint32_t cov_cap;
};

}  // namespace piko

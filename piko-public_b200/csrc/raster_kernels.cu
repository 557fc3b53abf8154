// Binned raster pipeline for sm_100a: the reference's RasterPipe
// (VertexShaderStage -> RasterStage -> PikoScreen, pikoc/samples/rasterPipelineFixPt)
// as five kernels per frame, over one scene or a batch of scenes:
//
//   raster_setup    one thread per triangle.  Vertex shading + triangle setup
//                   (R1: main.cpp:299-400 moved on device; R3: vertexShader.pikostage:36-109)
//                   from coalesced SoA loads, then AssignBin (R4,
//                   raster.pikostage:40-117) as a block-cooperative tile walk: one
//                   counter atomic per (triangle, tile) pair (shared by the
//                   warp's lanes with the same tile at 16/32-px tiles), whose old
//                   value is the pair's index in the tile's list, and a pair
//                   record.  Triangles with more than 256 box tiles are queued
//                   as 128-tile segments for
//   raster_large_count, which walks them the same way over the whole grid.
//   scan_tiles      tile counts -> each tile's place in the lists.  Tiles with
//                   long lists are queued as chunks of list entries.
//   raster_scatter  a streaming pass over the pair records: each becomes its
//                   list entry at its tile's offset plus its index (no walk, no
//                   atomics): the compaction.
//   raster_frag8 /  persistent CTAs.  A warp takes up to 32 list entries of an
//   raster_bins     8x8 reference bin, or of several with short lists: each lane
//                   builds one entry's coverage as a 64-bit mask, the masks are
//                   transposed over the warp, and each lane resolves the depth
//                   of two pixels from registers, nearest entries first.
//                   Coverage is the reference's 28.4 edge test with its 8x8-bin
//                   trivial reject/accept (R6, raster.pikostage:124-242); the z
//                   test, the shading of each pixel's winner and the composite
//                   are fused in (R7/R8), and every pixel is written once.
//
// Order independence.  The reference's depth test is an atomicMin on the float
// bits compared as signed ints, with ties passing (raster.pikostage:274-285).
// Run sequentially that leaves, per pixel, the minimum depth bits and the
// colour of the LAST fragment, in submission order, that has those bits.  So
// each fragment carries its triangle's submission rank and a pixel keeps the
// fragment with the smallest (depth bits, -rank): the result equals the
// sequential one whatever order the tile lists come in, and no list is sorted.
#include <atomic>

#include "piko_device.cuh"

namespace piko {

constexpr unsigned kFull = 0xffffffffu;
// Threads of a raster_setup CTA, for one scene and for several.  Smaller CTAs wait
// less at the barriers between their steps, but leave fewer kept triangles to fill
// each step.  Several scenes, 256 -> 128 threads: faster whatever share is kept (six
// of 200,000 triangles, 10% kept 217 -> 215 us, half 745 -> 741, all 648 -> 637; six
// forests, 23% kept, 181.1 -> 180.6).  One scene: 200,000 triangles, half kept, at
// 1080p 134.0 -> 132.4 and the others within 0.5%, but the packed 1277x715 forest
// with a wait for every frame 60.7 -> 61.5, which keeps it at 256.
template <bool ONE>
constexpr int kSetupThreads = ONE ? 256 : 128;
constexpr uint32_t kLargeTiles = 256; // box tiles above which a triangle's walk is spread over the grid
constexpr uint32_t kWalkQueue = 256;  // tiles a warp of the walk can have queued
constexpr uint32_t kItemMap = 4096;   // row items of a block's walk whose triangle is looked up
static_assert(kLargeTiles <= 256 && kSetupThreads<true> <= 256, "the walk's queue holds 8-bit tiles and triangles");
constexpr uint32_t kLargeSeg = 128;   // box tiles per work item of the large-triangle walk

// ------------------------------------------------------------------ helpers
// Scene s of the frame.  The kernels that read scene records exist for one
// scene (ONE: its record is a kernel argument, read as constants; reading it
// through a pointer that could be either cost raster_setup 6 us of 21 on the
// 1080p forest) and for several (a table in global memory).
template <bool ONE>
__device__ __forceinline__ const RasterSceneDev& scene_at(const RasterFrameArgs& a, int s)
{
  if constexpr (ONE) return a.one;
  else return a.scenes[s];
}

template <class S>
__device__ __forceinline__ int find_base(const S* sc, int n, uint32_t g, bool by_tile)
{
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    uint32_t b = by_tile ? sc[mid].tile_base : sc[mid].tri_base;
    if (b <= g) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// The scenes' first triangles or tiles in shared memory (batches of up to
// CAP scenes; larger ones search the scene records), so that finding a
// triangle's or a tile's scene is a shared-memory search.
constexpr int kSceneTable = 1024;
template <bool ONE, int CAP>
__device__ __forceinline__ void load_scene_table(const RasterFrameArgs& a, uint32_t* tb, bool by_tile)
{
  if constexpr (!ONE) {
    if (a.n_scenes > CAP) return;
    for (int i = threadIdx.x; i < a.n_scenes; i += blockDim.x)
      tb[i] = by_tile ? a.scenes[i].tile_base : a.scenes[i].tri_base;
  }
}
template <bool ONE, int CAP>
__device__ __forceinline__ int scene_of(const RasterFrameArgs& a, const uint32_t* tb, uint32_t x, bool by_tile)
{
  if constexpr (ONE) {
    return 0;
  } else {
    if (a.n_scenes > CAP) return find_base(a.scenes, a.n_scenes, x, by_tile);
    int lo = 0, hi = a.n_scenes - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (tb[mid] <= x) lo = mid; else hi = mid - 1;
    }
    return lo;
  }
}
template <bool ONE>
__device__ __forceinline__ int scene_of_tile(const RasterFrameArgs& a, const uint32_t* tb, uint32_t tile)
{
  return scene_of<ONE, kSceneTable>(a, tb, tile, true);
}

// Rank of triangle `id` in the order the one-thread CPU backend submits
// triangles to the raster bins: VS bins in index order (kernel1 blocks), and in
// VS bin b the ids with (id/512) % nVS == b ascending (vertexShader.pikostage:25-29).
__device__ __forceinline__ uint32_t submission_rank(uint32_t id, const RasterSceneDev& S)
{
  const uint32_t c = id / kVsChunk;
  uint32_t b;
  const uint32_t cq = fast_divmod(c, (uint32_t)S.nVS, S.vs_m, b);
  const uint32_t start = kVsChunk * (b * S.vs_q + min(b, S.vs_rem)) - (S.vs_last < b ? S.vs_deficit : 0u);
  return start + cq * kVsChunk + (id % kVsChunk);
}

// (depth bits as signed ints ascending, submission rank descending) as one
// unsigned 64-bit key: the smallest key is the sequential depth test's winner.
__device__ __forceinline__ unsigned long long frag_key(float z, uint32_t rank1)
{
  return ((unsigned long long)((uint32_t)__float_as_int(z) ^ 0x80000000u) << 32) | (uint32_t)(~rank1);
}
constexpr unsigned long long kInitKey = ((unsigned long long)(0x3f800000u ^ 0x80000000u) << 32) | 0xffffffffull;

__device__ __forceinline__ TriSetup load_setup(const TriSetup* p)
{
  TriSetup r;
  const uint4* src = reinterpret_cast<const uint4*>(p);
  uint4* dst = reinterpret_cast<uint4*>(&r);
#pragma unroll
  for (int k = 0; k < 5; ++k) dst[k] = __ldg(src + k);
  return r;
}

struct F3 { float x, y, z; };

__device__ __forceinline__ float sat1(float v) { return v > 1.0f ? 1.0f : (v < 0.0f ? 0.0f : v); }

// toABGR by truncation (piko/math.h:279-289).  One range test for the three
// channels: only a triangle whose edge values wrapped can leave it (and a NaN
// channel converts to 0 either way).
__device__ __forceinline__ uint32_t pack_abgr(float r, float g, float b)
{
  const float fr = r * 255.0f, fg = g * 255.0f, fb = b * 255.0f;
  if (fmaxf(fmaxf(fabsf(fr), fabsf(fg)), fabsf(fb)) < 2147483648.0f)
    return 0xff000000u | ((uint32_t)__float2int_rz(fb) << 16) | ((uint32_t)__float2int_rz(fg) << 8) |
           (uint32_t)__float2int_rz(fr);
  return 0xff000000u | (cvt_u32_x86(fb) << 16) | (cvt_u32_x86(fg) << 8) | cvt_u32_x86(fr);
}

// computeLightingHost + toABGRHost (main.cpp:317-334)
__device__ __forceinline__ uint32_t light_abgr(F3 n, F3 l, F3 m)
{
  float d = n.x * l.x + n.y * l.y + n.z * l.z;
  d = d < 0.0f ? 0.0f : d;
  float r = sat1(d * m.x + 0.15f);
  float g = sat1(d * m.y + 0.15f);
  float b = sat1(d * m.z + 0.30f);
  return pack_abgr(r, g, b);
}

// E_i(X, Y) = (Y - y_i) * dx_i - (X - x_i) * dy_i  (wrapping int32)
__device__ __forceinline__ int32_t edge_at(int32_t X, int32_t Y, int32_t xi, int32_t yi, int32_t dx, int32_t dy)
{
  return wsub(wmul(wsub(Y, yi), dx), wmul(wsub(X, xi), dy));
}

// Conservative trivial reject of a 16/32-px tile (exact int64 arithmetic): the
// tile, clipped to the triangle's bin range, can hold an assigned reference bin
// only if every edge function is >= 0 at the tile corner that maximises it.
// Only used for triangles whose edge values cannot wrap inside the bin range.
__device__ __forceinline__ bool tile_may_cover(const WalkTri& w, int tx, int ty, int T)
{
  if (w.flags & kTriRisk) return true;
  long long X0 = (long long)max(tx * T, w.bx1 * kRefBin) * 16;
  long long X1 = (long long)min((tx + 1) * T, (w.bx2 + 1) * kRefBin) * 16;
  long long Y0 = (long long)max(ty * T, w.by1 * kRefBin) * 16;
  long long Y1 = (long long)min((ty + 1) * T, (w.by2 + 1) * kRefBin) * 16;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    int j = i == 2 ? 0 : i + 1;
    long long dx = (long long)w.x[j] - w.x[i], dy = (long long)w.y[j] - w.y[i];
    long long X = dy < 0 ? X1 : X0;
    long long Y = dx > 0 ? Y1 : Y0;
    long long e = (Y - w.y[i]) * dx - (X - w.x[i]) * dy;
    if (e < 0) return false;
  }
  return true;
}

// Writes the records of the warp's pairs (bits m) to slots from `slot` on of a
// partition, those that lie in [base, part_cap) of it.
template <int R>
__device__ __forceinline__ void put_pairs(const RasterFrameArgs& a, const uint32_t (&key)[R], const uint32_t (&gidx)[R],
                                          const uint32_t (&local)[R], const unsigned (&m)[R], uint32_t part,
                                          uint32_t part_cap, uint32_t base, uint32_t slot, int lane)
{
  const unsigned lt = (1u << lane) - 1u;
  const size_t at = (size_t)part * part_cap;
#pragma unroll
  for (int q = 0; q < R; ++q) {
    const uint32_t mine = slot + (uint32_t)__popc(m[q] & lt);
    if (key[q] != 0xffffffffu && mine >= base && mine < part_cap) {
      a.pair_tl[at + mine] = (unsigned long long)key[q] | ((unsigned long long)local[q] << 32);
      a.pair_g[at + mine] = gidx[q];
    }
    slot += (uint32_t)__popc(m[q]);
  }
}

// Counts the pairs of R rounds held by the warp's lanes (key = global tile, or
// ~0 for none): one atomicAdd per pair on its tile's counter (per group of
// lanes with the same tile at 16/32-px tiles), whose old value gives the
// pair's index in the tile's list, and one reservation per warp for the
// pair records, which the scatter pass turns into list entries without
// walking again.  Every lane of the warp calls this (ballots).  Records past
// the list capacity are dropped; the scan reports the overflow (the pair
// total equals the list total) and the frame is drawn again.
template <int R>
__device__ __forceinline__ void count_pairs(const RasterFrameArgs& a, const uint32_t (&key)[R],
                                            const uint32_t (&gidx)[R], int lane)
{
  uint32_t local[R];
  if (a.tile == kRefBin) {
#pragma unroll
    for (int q = 0; q < R; ++q) local[q] = key[q] != 0xffffffffu ? atomicAdd(&a.tile_cnt[key[q]], 1u) : 0u;
  } else {
    // 16/32-px tiles: lanes of a round with the same tile share one counter
    // atomic (the group's lowest lane adds the group's size; a lane's index is
    // the old count plus its rank in the group).  (At 8x8 tiles, where fewer
    // of a warp's pairs share a tile, the match costs more than it saves.)
    const unsigned lt0 = (1u << lane) - 1u;
    unsigned grp[R];
#pragma unroll
    for (int q = 0; q < R; ++q) {
      grp[q] = __match_any_sync(kFull, key[q]);
      local[q] = 0u;
      if (key[q] != 0xffffffffu && (grp[q] & lt0) == 0u)
        local[q] = atomicAdd(&a.tile_cnt[key[q]], (uint32_t)__popc(grp[q]));
    }
#pragma unroll
    for (int q = 0; q < R; ++q)
      local[q] = __shfl_sync(kFull, local[q], __ffs(grp[q]) - 1) + (uint32_t)__popc(grp[q] & lt0);
  }
  unsigned m[R];
  uint32_t n = 0;
#pragma unroll
  for (int q = 0; q < R; ++q) {
    m[q] = __ballot_sync(kFull, key[q] != 0xffffffffu);
    n += (uint32_t)__popc(m[q]);
  }
  if (n == 0) return;
  // (by block first: a block's first warps record the most)
  const uint32_t part = (blockIdx.x + (threadIdx.x >> 5) * (kPairParts / 8)) & (kPairParts - 1u);
  const uint32_t part_cap = a.list_cap / kPairParts;
  uint32_t base = 0;
  if (lane == 0) base = atomicAdd(&a.work->pair_part[part], n);
  base = __shfl_sync(kFull, base, 0);
  put_pairs<R>(a, key, gidx, local, m, part, part_cap, base, base, lane);
  if (base + n <= part_cap) return;
  // The partition is full.  Lists that grow: the host grows them so that every
  // partition fits, and draws again.  Fixed ones: the rest goes to the next
  // partitions, which fills all of them before a pair is dropped.
  uint32_t done = part_cap - min(base, part_cap), p = part;   // pairs that have their records
  if (a.spill) {
#pragma unroll 1
    for (uint32_t k = 1; k < kPairParts && done < n; ++k) {
      p = (p + 1u) & (kPairParts - 1u);
      if (lane == 0) base = atomicAdd(&a.work->pair_part[p], n - done);
      base = __shfl_sync(kFull, base, 0);
      put_pairs<R>(a, key, gidx, local, m, p, part_cap, base, base - done, lane);
      done += min(part_cap - min(base, part_cap), n - done);
    }
  }
  if (lane == 0 && done < n) {
    atomicMax(&a.work->bin.pair_part_max, base + n);
    atomicOr(&a.work->bin.status, kStatusListOverflow);
  }
}

// A frame whose pairs overran the list buffers is drawn again with larger
// ones; its tile lists have entries that no pair filled (a pair counted in
// tile_cnt but past list_cap has no record), so the fragment kernels must not
// read them.  The status is final once the scan has run; the scatter pass
// copies it to the frame's result.
__device__ __forceinline__ bool list_overflowed(const RasterFrameArgs& a)
{
  return (a.ctr->bin.status & kStatusListOverflow) != 0;
}

// First thing a fragment kernel does: the pair partitions, which the scatter
// pass has read, go back to 0, and the binning counts go to the host.
__device__ __forceinline__ void frame_begin(const RasterFrameArgs& a)
{
  if (blockIdx.x != 0) return;
  if (threadIdx.x < kPairParts) a.work->pair_part[threadIdx.x] = 0u;
  if (threadIdx.x == 0 && a.host_bin) *a.host_bin = a.ctr->bin;
}

// Which of columns [c0, c0 + n) (n <= 32) of row `row` of triangle w's box tiles
// pass the tile-level reject, as bits.  At 8x8 tiles that is the reference's
// own trivial reject at the bin corner (raster.pikostage:77-105), stepped from
// bin (tx1, ty1).
__device__ __forceinline__ uint32_t row_mask(const WalkTri& w, uint32_t row, uint32_t c0, uint32_t n, int T)
{
  uint32_t m = 0;
  if (T == kRefBin) {
    // last column first, so that column c0 ends in bit 0: bits of rejected tiles
    int32_t t[3], dx[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      dx[i] = w.trx[i];
      t[i] = wadd(wadd(w.tr0[i], wmul((int32_t)row, w.try_[i])), wmul((int32_t)(c0 + n - 1), dx[i]));
    }
#pragma unroll 4
    for (uint32_t k = 0; k < n; ++k) {
      m = __funnelshift_l((uint32_t)(t[0] | t[1] | t[2]), m, 1);
#pragma unroll
      for (int i = 0; i < 3; ++i) t[i] = wsub(t[i], dx[i]);
    }
    return ~m & (n < 32u ? (1u << n) - 1u : 0xffffffffu);
  }
  for (uint32_t k = 0; k < n; ++k)
    m |= (uint32_t)tile_may_cover(w, w.tx1 + (int)(c0 + k), w.ty1 + (int)row, T) << k;
  return m;
}

// The tiles of row_mask's range that can hold a covered pixel centre (the box
// that holds the triangle's tiles is rounded up to 16 px and one bin beyond).
__device__ __forceinline__ uint32_t listed_mask(const WalkTri& w, uint32_t row, uint32_t c0, uint32_t n)
{
  const uint32_t x0 = w.ltx & 0xffffu, x1 = w.ltx >> 16, y0 = w.lty & 0xffffu, y1 = w.lty >> 16;
  if (row < y0 || row > y1 || x0 >= c0 + n || x1 < c0) return 0u;   // (no tile: y0 > y1)
  const uint32_t lo = x0 > c0 ? x0 - c0 : 0u, hi = min(x1 - c0, n - 1);
  return (0xffffffffu >> (31u - hi)) & (0xffffffffu << lo);
}

// Counts and records queue entries [first, first + n), n <= 128, one per lane at
// a time; key_of(entry, gidx) turns an entry into its global tile.
template <class F>
__device__ __forceinline__ void record_queue(const RasterFrameArgs& a, const uint16_t* queue, uint32_t first, uint32_t n,
                                             int lane, F key_of)
{
  uint32_t key[4], gidx[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const uint32_t p = (uint32_t)(q * 32 + lane);
    key[q] = 0xffffffffu;
    gidx[q] = 0;
    if (p < n) key[q] = key_of(queue[first + p], gidx[q]);
  }
  count_pairs<4>(a, key, gidx, lane);
}

// Appends the tiles of the warp's masks to its queue of qn entries (a mask per
// lane: bit k of m is tile at + k of the lane's triangle, tagged tag) and
// records them 128 at a time, so that all of count_pairs' rounds are full; fewer
// than 128 stay queued.
template <class F>
__device__ __forceinline__ void queue_masks(const RasterFrameArgs& a, uint16_t* queue, uint32_t& qn, uint32_t m,
                                            uint32_t tag, uint32_t at, int lane, F key_of)
{
  uint32_t incl = (uint32_t)__popc(m);
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t v = __shfl_up_sync(kFull, incl, o);
    if (lane >= o) incl += v;
  }
  uint32_t pos = qn + incl - (uint32_t)__popc(m), end = qn + __shfl_sync(kFull, incl, 31);
  for (;;) {
    for (; m && pos < kWalkQueue; m &= m - 1u, ++pos)
      queue[pos] = (uint16_t)((tag << 8) | (at + (uint32_t)__ffs(m) - 1u));
    __syncwarp();
    const uint32_t had = min(end, kWalkQueue);
    for (qn = had; qn >= 128u; qn -= 128u) record_queue(a, queue, qn - 128u, 128u, lane, key_of);
    if (end <= kWalkQueue) return;
    __syncwarp();   // the queue is refilled behind its first qn entries
    pos -= had - qn;
    end -= had - qn;
  }
}

__device__ __forceinline__ uint32_t tile_key(const WalkTri& w, uint32_t j)
{
  uint32_t lx;
  const uint32_t ly = fast_divmod(j, (uint32_t)w.tw, w.tw_m, lx);
  return w.tile_base + (uint32_t)((w.ty1 + (int)ly) * w.tiles_x + w.tx1 + (int)lx);
}

// Walks the box tiles of the block's triangles wt[0, n) (at most kLargeTiles
// each) with all of its threads: a thread tests a row of a triangle's box (up to
// 32 columns of it), stepping the edge values (row item i belongs to triangle
// item_tri[i], the first whose inclusive item-count prefix pre[] exceeds i; past
// kItemMap items it is searched).  The tiles that
// can hold a covered pixel are counted and recorded, one per lane; the others
// that pass the reject are returned as a number, the warp's in each lane.  (A
// thread per tile, each with its own search and divide, took about 110
// instructions a box tile where this takes some 25.)
__device__ __forceinline__ uint32_t walk_tiles(const RasterFrameArgs& a, const WalkTri* wt, const uint32_t* pre,
                                               const uint8_t* item_tri, int n, uint16_t* queue)
{
  const int lane = threadIdx.x & 31;
  const uint32_t total = n ? pre[n - 1] : 0u;
  const auto key_of = [&](uint32_t e, uint32_t& gidx) {
    const WalkTri& w = wt[e >> 8];
    gidx = w.gidx;
    return tile_key(w, e & 255u);
  };
  uint32_t skipped = 0, qn = 0;
  for (uint32_t base = threadIdx.x & ~31u; base < total; base += blockDim.x) {
    const uint32_t i = base + (uint32_t)lane;
    uint32_t m = 0, tri = 0, at = 0;
    if (i < total) {
      if (i < kItemMap) {
        tri = item_tri[i];
      } else {
        int lo = 0, hi = n - 1;
        while (lo < hi) {
          const int mid = (lo + hi) >> 1;
          if (pre[mid] > i) hi = mid; else lo = mid + 1;
        }
        tri = (uint32_t)lo;
      }
      const WalkTri& w = wt[tri];
      const uint32_t tw = (uint32_t)w.tw, parts = (tw + 31u) >> 5;
      uint32_t row = i - (tri ? pre[tri - 1] : 0u), c0 = 0;
      if (parts > 1) {
        c0 = (row % parts) * 32u;
        row /= parts;
      }
      const uint32_t cols = min(tw - c0, 32u);
      m = row_mask(w, row, c0, cols, a.tile);
      skipped += (uint32_t)__popc(m);
      m &= listed_mask(w, row, c0, cols);
      skipped -= (uint32_t)__popc(m);
      at = row * tw + c0;
    }
    queue_masks(a, queue, qn, m, tri, at, lane, key_of);
  }
  if (qn) record_queue(a, queue, 0u, qn, lane, key_of);
  return __reduce_add_sync(kFull, skipped);
}

// The walk record of triangle g, and the number of tiles in its box.
__device__ __forceinline__ void fill_walk(const RasterFrameArgs& a, const RasterSceneDev& S, const TriSetup& r,
                                          uint32_t g, WalkTri& w, uint32_t& ntiles)
{
  const int tsh = __ffs(a.tile) - 1 - kRefBinLg2;   // tile edge = 8 << tsh
  w.bx1 = (int)(r.bxr & 0xffff); w.bx2 = (int)(r.bxr >> 16);
  w.by1 = (int)(r.byr & 0xffff); w.by2 = (int)(r.byr >> 16);
  w.tx1 = w.bx1 >> tsh;
  w.ty1 = w.by1 >> tsh;
  const int tx2 = w.bx2 >> tsh, ty2 = w.by2 >> tsh;
  w.tw = tx2 - w.tx1 + 1;
  w.tw_m = divmod_magic((uint32_t)w.tw);
  w.gidx = g;
  w.tile_base = S.tile_base;
  w.tiles_x = S.tiles_x;
  w.flags = r.flags;
  ntiles = (uint32_t)w.tw * (uint32_t)(ty2 - w.ty1 + 1);
  // The tiles to list: those that hold a pixel centre of the triangle's own
  // bounds (a covered centre lies inside the triangle unless an edge value may
  // wrap; then all).
  int lx0 = w.tx1, lx1 = tx2, ly0 = w.ty1, ly1 = ty2;
  if (!(r.flags & kTriRisk)) {
    const int px0 = (min(min(r.x[0], r.x[1]), r.x[2]) + 7) >> 4, px1 = (max(max(r.x[0], r.x[1]), r.x[2]) - 8) >> 4;
    const int py0 = (min(min(r.y[0], r.y[1]), r.y[2]) + 7) >> 4, py1 = (max(max(r.y[0], r.y[1]), r.y[2]) - 8) >> 4;
    lx0 = max(lx0, px0 >> (kRefBinLg2 + tsh)); lx1 = min(lx1, px1 >> (kRefBinLg2 + tsh));
    ly0 = max(ly0, py0 >> (kRefBinLg2 + tsh)); ly1 = min(ly1, py1 >> (kRefBinLg2 + tsh));
    if (px0 > px1 || py0 > py1 || lx0 > lx1) ly1 = ly0 - 1;
  }
  w.ltx = (uint32_t)(lx0 - w.tx1) | ((uint32_t)(lx1 - w.tx1) << 16);
  w.lty = ly0 <= ly1 ? (uint32_t)(ly0 - w.ty1) | ((uint32_t)(ly1 - w.ty1) << 16) : 1u;   // (rows [1, 0]: none)
  if (tsh == 0) {
    const int32_t BX = w.tx1 * 128, BY = w.ty1 * 128;   // bin corner, 28.4
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const int j = i == 2 ? 0 : i + 1;
      const int32_t dx = wsub(r.x[j], r.x[i]), dy = wsub(r.y[j], r.y[i]);
      int32_t off = dy < 0 ? -wshl(dy, 7) : 0;
      off = wadd(off, dx >= 0 ? wshl(dx, 7) : 0);
      w.tr0[i] = wadd(off, wsub(wmul(wsub(BY, r.y[i]), dx), wmul(wsub(BX, r.x[i]), dy)));
      w.trx[i] = -wshl(dy, 7);
      w.try_[i] = wshl(dx, 7);
    }
  } else {
    for (int k = 0; k < 3; ++k) { w.x[k] = r.x[k]; w.y[k] = r.y[k]; }
  }
}

// Vertex attribute i (slot-major index k * N + id): float4, or float3 with w
// 0 in a packed scene (w is never read).
__device__ __forceinline__ float4 load_attr3(const float4* a4, const float* a3, size_t i)
{
  if (a3) return make_float4(__ldg(&a3[3 * i]), __ldg(&a3[3 * i + 1]), __ldg(&a3[3 * i + 2]), 0.0f);
  return __ldg(&a4[i]);
}

// ------------------------------------------------------------------ kernel 1
// A block takes a.batch triangles at a time (at most its threads), in steps
// that each spread what is left of them over all threads:
//   1. a thread per triangle: transform, 28.4 quantisation and the culls;
//   2. the kept triangles' vertices, one per thread, are lit (a culled
//      triangle's colours are never read: only kept ones load normals);
//   3. a thread per kept triangle: bin range, setup record, walk record;
//   4. a thread per row of a kept triangle's box tiles: the tile walk.
// (One thread taking its triangle through all of it had half of its lanes culled
// on the batched mix, three quarters on the forest.  Setup and large count of
// one frame together, before and now: 1,000 triangles 13 -> 8 us, 1080p forest
// 33 -> 24, 200K triangles 47 -> 34, 24-scene batch 111 -> 98.)  The walk counts every
// pair that passes the reject, as the reference's queues do, but lists only
// tiles that can hold a covered pixel centre: a third fewer list entries, which
// the later kernels do not touch (200K triangles: fragment pass 100 -> 92 us).
template <int T>   // threads of the CTA
struct SetupSmem {
  WalkTri walk[T];
  union {
    struct {   // the kept triangles, in order (steps 1 to 3)
      int32_t x[3][T], y[3][T];
      float z[3][T];
      uint32_t c[3][T];
      uint32_t g[T];
    };
    struct {   // step 4
      uint32_t pre[T];
      uint8_t item_tri[kItemMap];
      uint16_t queue[T / 32][kWalkQueue];
    };
  };
  uint32_t warp[T / 32];
  unsigned nk, nr;
  unsigned skipped;   // pairs that pass the reject and are not listed (of one CTA: below 2^32)
};

// Inclusive scan of v over the block of T threads.
template <int T>
__device__ __forceinline__ uint32_t block_scan_incl(uint32_t v, uint32_t* s_warp)
{
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(kFull, v, o);
    if (lane >= o) v += t;
  }
  if (lane == 31) s_warp[warp] = v;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < T / 32; ++w)
    if (w < warp) v += s_warp[w];
  return v;
}

// (1024 threads an SM: 64 registers)
template <bool ONE>
__global__ void __launch_bounds__(kSetupThreads<ONE>, 1024 / kSetupThreads<ONE>)
raster_setup(const __grid_constant__ RasterFrameArgs a)
{
  pdl_trigger();
  extern __shared__ __align__(16) unsigned char setup_smem[];
  constexpr int T = kSetupThreads<ONE>;
  SetupSmem<T>& B = *reinterpret_cast<SetupSmem<T>*>(setup_smem);
  uint32_t* s_tb = reinterpret_cast<uint32_t*>(&B + 1);   // the scene table, several scenes only
  load_scene_table<ONE, kSceneTable>(a, s_tb, false);
  if (threadIdx.x == 0) B.nk = B.nr = B.skipped = 0u;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  for (uint32_t base = blockIdx.x * a.batch; base < a.n_tris_total; base += gridDim.x * a.batch) {
    // 1
    const uint32_t g = base + threadIdx.x;
    int32_t x[3], y[3];
    float z[3];
    bool keep = false;
    if (threadIdx.x < a.batch && g < a.n_tris_total) {
      const int s = scene_of<ONE, kSceneTable>(a, s_tb, g, false);
      const RasterSceneDev& S = scene_at<ONE>(a, s);
      const uint32_t id = g - S.tri_base;
      float sx[3], sy[3];
      const bool soa = S.input_kind == kInputSoA;
      if (soa || S.input_kind == kInputWtriWorld) {
        // R1, main.cpp:299-308: vtransform, perspective divide, viewport.  World
        // raster_wtri input: the vertex stage's vtxTransform (rasterMacros.h:14-21,
        // matmultfloat4 and rcp_approx = 1.0f / w on the CPU) is the same float
        // sequence; that mode has no colours (left 0).
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          float4 p;
          if (soa) {
            p = load_attr3(S.pos, S.pos3, (size_t)k * S.N + id);
          } else {
            p.x = __ldg(&S.wtri_xyz[(size_t)id * 9 + 3 * k + 0]);
            p.y = __ldg(&S.wtri_xyz[(size_t)id * 9 + 3 * k + 1]);
            p.z = __ldg(&S.wtri_xyz[(size_t)id * 9 + 3 * k + 2]);
            p.w = 1.0f;
          }
          const float* m = S.vp;
          float tx = p.x * m[0] + p.y * m[4] + p.z * m[8] + m[12];
          float ty = p.x * m[1] + p.y * m[5] + p.z * m[9] + m[13];
          float tz = p.x * m[2] + p.y * m[6] + p.z * m[10] + m[14];
          float tw = p.x * m[3] + p.y * m[7] + p.z * m[11] + m[15];
          float onebyw = 1.0f / tw;
          sx[k] = (tx * onebyw + 1.0f) * S.halfW;
          sy[k] = (ty * onebyw + 1.0f) * S.halfH;
          z[k] = (tz * onebyw);
        }
      } else {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          sx[k] = S.wtri_xyz[(size_t)id * 9 + 3 * k + 0];
          sy[k] = S.wtri_xyz[(size_t)id * 9 + 3 * k + 1];
          z[k] = S.wtri_xyz[(size_t)id * 9 + 3 * k + 2];
        }
      }
      // R3: 28.4 quantisation by truncation and the three culls
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        x[k] = cvt_i32_x86(sx[k] * 16.0f);
        y[k] = cvt_i32_x86(sy[k] * 16.0f);
      }
      keep = wsub(wmul(wsub(y[2], y[0]), wsub(x[1], x[0])), wmul(wsub(x[2], x[0]), wsub(y[1], y[0]))) > 0;
      const int32_t Wf = cvt_i32_x86((float)S.W * 16.0f), Hf = cvt_i32_x86((float)S.H * 16.0f);
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        keep = keep && !(x[k] < -kGuard || x[k] >= wadd(Wf, kGuard));
        keep = keep && !(y[k] < -kGuard || y[k] >= wadd(Hf, kGuard));
      }
      const int32_t loy = min(min(y[0], y[1]), y[2]), hiy = max(max(y[0], y[1]), y[2]);
      keep = keep && !((wsub(loy, 8) >> 4) == (wsub(hiy, 8) >> 4));
    }
    {
      const unsigned m = __ballot_sync(kFull, keep);
      if (lane == 0) B.warp[threadIdx.x >> 5] = (uint32_t)__popc(m);
      __syncthreads();
      uint32_t at = (uint32_t)__popc(m & ((1u << lane) - 1u));
#pragma unroll
      for (int w = 0; w < T / 32; ++w)
        if (w < (int)(threadIdx.x >> 5)) at += B.warp[w];
      if (keep) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          B.x[k][at] = x[k];
          B.y[k][at] = y[k];
          B.z[k][at] = z[k];
        }
        B.g[at] = g;
      }
    }
    uint32_t n = 0;
#pragma unroll
    for (int w = 0; w < T / 32; ++w) n += B.warp[w];
    __syncthreads();
    // 2.  R1, main.cpp:310-400: per-vertex Gouraud lighting with the normal
    // normalised by HOST::normalize; no colour array: the reference's fixed
    // material colour (main.cpp:380)
    for (uint32_t v = threadIdx.x; v < 3 * n; v += T) {
      const uint32_t t = v / 3u, k = v - 3u * t, vg = B.g[t];
      const int s = scene_of<ONE, kSceneTable>(a, s_tb, vg, false);
      const RasterSceneDev& S = scene_at<ONE>(a, s);
      const uint32_t id = vg - S.tri_base;
      uint32_t col = 0u;
      if (S.input_kind == kInputSoA) {
        const size_t i = (size_t)k * S.N + id;
        const float4 n4 = load_attr3(S.nrm, S.nrm3, i);
        const float4 c4 = S.col ? __ldg(&S.col[i]) : make_float4(0.9f, 0.9f, 0.6f, 1.0f);
        float mag = sqrtf(n4.x * n4.x + n4.y * n4.y + n4.z * n4.z);
        F3 nn = {n4.x / mag, n4.y / mag, n4.z / mag};
        F3 l;
        if (S.light_mode == 1) {
          const float4 p = load_attr3(S.pos, S.pos3, i);
          l.x = S.eye[0] - p.x; l.y = S.eye[1] - p.y; l.z = S.eye[2] - p.z;
          float mm = sqrtf(l.x * l.x + l.y * l.y + l.z * l.z);
          if (mm != 0.0f) { float rr = 1.0f / mm; l.x = l.x * rr; l.y = l.y * rr; l.z = l.z * rr; }
        } else {
          l.x = S.light[0]; l.y = S.light[1]; l.z = S.light[2];
        }
        col = light_abgr(nn, l, F3{c4.x, c4.y, c4.z});
      } else if (S.input_kind == kInputWtri) {
        col = S.wtri_icol[(size_t)id * 3 + k];
      }
      B.c[k][t] = col;
    }
    __syncthreads();
    // 3
    uint32_t ntiles = 0;
    bool risk_flag = false;
    if (threadIdx.x < n) {
      const uint32_t t = threadIdx.x, kg = B.g[t];
      const int s = scene_of<ONE, kSceneTable>(a, s_tb, kg, false);
      const RasterSceneDev& S = scene_at<ONE>(a, s);
      TriSetup r;
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        r.x[k] = B.x[k][t];
        r.y[k] = B.y[k][t];
        r.z[k] = B.z[k][t];
        r.c[k] = B.c[k][t];
      }
      r.id = kg - S.tri_base;
      r.flags = 0;
      // R4: pixel bounding box rounded to 16 px, reference bin range (8x8)
      const int32_t lox = min(min(r.x[0], r.x[1]), r.x[2]) & (int32_t)0xffffff00;
      const int32_t loy = min(min(r.y[0], r.y[1]), r.y[2]) & (int32_t)0xffffff00;
      const int32_t hix = wadd(max(max(r.x[0], r.x[1]), r.x[2]), 0xff) & (int32_t)0xffffff00;
      const int32_t hiy = wadd(max(max(r.y[0], r.y[1]), r.y[2]), 0xff) & (int32_t)0xffffff00;
      const int bits = 4 + kRefBinLg2;
      const int bx1 = max(0, lox >> bits), bx2 = min(hix >> bits, S.nBx - 1);
      const int by1 = max(0, loy >> bits), by2 = min(hiy >> bits, S.nBy - 1);
      r.hix = hix; r.hiy = hiy;
      const int32_t x1mx0 = wsub(r.x[1], r.x[0]), y1my0 = wsub(r.y[1], r.y[0]);
      const int32_t x0mx2 = wsub(r.x[0], r.x[2]), y0my2 = wsub(r.y[0], r.y[2]);
      const int32_t barydenom = wadd(wmul(-y0my2, x1mx0), wmul(x0mx2, y1my0));
      r.inv = 1.0f / (float)barydenom;
      // 80-byte record as five 16-byte stores, for the triangles that reach a
      // tile list: only lists (and the winners they give) lead to a record
      if (bx1 <= bx2 && by1 <= by2) {
        r.rank1 = submission_rank(r.id, S) + 1u;
        r.bxr = (uint32_t)bx1 | ((uint32_t)bx2 << 16);
        r.byr = (uint32_t)by1 | ((uint32_t)by2 << 16);
        // can any edge value the reference compares wrap inside the bin range?
        const long long X0 = (long long)bx1 * 128, X1 = (long long)(bx2 + 1) * 128;
        const long long Y0 = (long long)by1 * 128, Y1 = (long long)(by2 + 1) * 128;
        // |e(X, Y)| <= max|Y - y_i| * |dx| + max|X - x_i| * |dy| over the range
        // (a bound at least the largest corner value), plus the trivial-accept
        // offsets
        long long worst = 0;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          const int j = i == 2 ? 0 : i + 1;
          const long long dx = llabs((long long)r.x[j] - r.x[i]), dy = llabs((long long)r.y[j] - r.y[i]);
          const long long ax = max(llabs(X0 - r.x[i]), llabs(X1 - r.x[i]));
          const long long ay = max(llabs(Y0 - r.y[i]), llabs(Y1 - r.y[i]));
          worst = max(worst, ay * dx + ax * dy + 512 * (dx + dy));
        }
        if (worst >= 2147483647LL) r.flags |= kTriRisk;
        const long long area = (long long)(r.y[2] - r.y[0]) * (r.x[1] - r.x[0]) -
                               (long long)(r.x[2] - r.x[0]) * (r.y[1] - r.y[0]);
        if (area >= 2147483647LL) r.flags |= kTriAreaRisk;
        risk_flag = (r.flags & kTriRisk) != 0;
        fill_walk(a, S, r, kg, B.walk[t], ntiles);
        if (B.walk[t].lty != 1u) {
          const uint4* src = reinterpret_cast<const uint4*>(&r);
          uint4* dst = reinterpret_cast<uint4*>(&a.setup[kg]);
#pragma unroll
          for (int k = 0; k < 5; ++k) dst[k] = src[k];
        }
      }
    }
    // Triangles with many tiles in their box go to raster_large_count, which
    // walks their box tiles in segments of kLargeSeg: one atomic per warp
    // reserves the warp's segment items.
    const bool is_big = ntiles > kLargeTiles;
    const unsigned big = __ballot_sync(kFull, is_big);
    if (big) {
      const uint32_t nseg = is_big ? (ntiles + kLargeSeg - 1) / kLargeSeg : 0u;
      uint32_t incl = nseg;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(kFull, incl, o);
        if (lane >= o) incl += t;
      }
      unsigned long long old = 0;
      if (lane == 31) old = atomicAdd(&a.work->bin.large_acc, ((unsigned long long)__popc(big) << 32) | incl);
      old = __shfl_sync(kFull, old, 31);
      if (is_big) {
        // the triangle's walk record, then one (large triangle, segment) item
        // per segment; records or items past the capacities are reported (the
        // host grows the buffers and draws the frame again)
        const uint32_t bi = (uint32_t)(old >> 32) + (uint32_t)__popc(big & ((1u << lane) - 1u));
        const uint32_t first = (uint32_t)old + incl - nseg;
        if (bi < a.big_cap) {
          a.large_walk[bi] = B.walk[threadIdx.x];
          for (uint32_t k = 0; k < nseg; ++k) {
            if (first + k < a.seg_cap) a.large_seg[first + k] = make_uint2(bi, k);
            else { atomicOr(&a.work->bin.status, kStatusListOverflow); break; }
          }
        } else {
          atomicOr(&a.work->bin.status, kStatusListOverflow);
        }
        ntiles = 0;
      }
    }
    const unsigned risks = (unsigned)__popc(__ballot_sync(kFull, risk_flag));
    if (lane == 0 && risks) atomicAdd(&B.nr, risks);
    if (threadIdx.x == 0) B.nk += n;
    uint32_t items = 0;
    if (ntiles) {
      const uint32_t tw = (uint32_t)B.walk[threadIdx.x].tw;
      items = (ntiles / tw) * ((tw + 31u) >> 5);
    }
    // (the scan's barrier lies between the last read of x .. g and this write)
    const uint32_t incl = block_scan_incl<T>(items, B.warp);
    B.pre[threadIdx.x] = incl;
    for (uint32_t i = incl - items; i < min(incl, kItemMap); ++i) B.item_tri[i] = (uint8_t)threadIdx.x;
    __syncthreads();
    // 4
    const uint32_t skipped = walk_tiles(a, B.walk, B.pre, B.item_tri, (int)n, B.queue[threadIdx.x >> 5]);
    if (lane == 0 && skipped) atomicAdd(&B.skipped, skipped);
    __syncthreads();  // the shared arrays are rewritten by the next batch
  }
  // frame counters: one atomic per CTA
  if (threadIdx.x == 0) {
    if (B.nk) atomicAdd(&a.work->bin.kept, B.nk);
    if (B.nr) atomicAdd(&a.work->bin.risk, (unsigned long long)B.nr);
    if (B.skipped) atomicAdd(&a.work->bin.skipped, (unsigned long long)B.skipped);
  }
}

// ------------------------------------------------------------------ kernel 2
// Gives every tile its place in the tile lists: a scan within the block, and one
// atomic for the block's share of the lists.  The lists' order means nothing, so
// the blocks need not wait for one another (a decoupled look-back took 1 to 2 us
// of the frame).  The tile counters are set back to 0 as they are read.
__global__ void __launch_bounds__(kScanThreads) scan_tiles(const __grid_constant__ RasterFrameArgs a)
{
  pdl_wait();
  pdl_trigger();
  __shared__ uint32_t s_warp[kScanThreads / 32];
  __shared__ uint32_t s_first;
  __shared__ unsigned long long s_heavy[kScanThreads / 32];   // per warp: (key slots << 32) | items
  const uint32_t n = a.n_tiles_total;
  const uint32_t base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
  uint32_t v[kScanItems];
  uint32_t sum = 0;
#pragma unroll
  for (int i = 0; i < kScanItems; ++i) {
    v[i] = (base + i < n) ? a.tile_cnt[base + i] : 0u;
    if (v[i]) a.tile_cnt[base + i] = 0u;
    sum += v[i];
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t incl = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    uint32_t t = __shfl_up_sync(kFull, incl, o);
    if (lane >= o) incl += t;
  }
  // Heavy tiles (lists longer than queue_min) become items of the fragment
  // kernel's queue -- their chunks, or without chunk buffers the tiles -- and
  // the chunks of lists in several chunks need key slots: counted now, reserved
  // below with one atomic per block
  const bool t8 = a.tile == kRefBin;
  const bool chunked = a.chunk_desc != nullptr;
  const uint32_t thr = a.queue_min, bins = (uint32_t)(a.tile / kRefBin) * (uint32_t)(a.tile / kRefBin);
  uint32_t nk = 0, nc = 0;
#pragma unroll
  for (int i = 0; i < kScanItems; ++i) {
    if (base + i < n && v[i] > thr) {
      const uint32_t nch = chunked ? tile_chunks(v[i], a.chunk, t8) : 1u;
      nc += nch;
      if (nch > 1) nk += nch;
    }
  }
  uint32_t ki = nk, ci = nc;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t tk = __shfl_up_sync(kFull, ki, o), tc = __shfl_up_sync(kFull, ci, o);
    if (lane >= o) { ki += tk; ci += tc; }
  }
  if (lane == 31) {
    s_warp[warp] = incl;
    s_heavy[warp] = ((unsigned long long)ki << 32) | ci;
  }
  __syncthreads();
  if (warp == 1 && lane == 0) {
    // the block's reservation; each warp's base replaces its count
    unsigned long long tot = 0;
#pragma unroll
    for (int w = 0; w < kScanThreads / 32; ++w) tot += s_heavy[w];
    unsigned long long run_h = tot ? atomicAdd(&a.work->bin.heavy_acc, tot) : 0ull;
#pragma unroll
    for (int w = 0; w < kScanThreads / 32; ++w) {
      const unsigned long long cnt = s_heavy[w];
      s_heavy[w] = run_h;
      run_h += cnt;
    }
  }
  uint32_t warp_excl = 0, agg = 0;
#pragma unroll
  for (int w = 0; w < kScanThreads / 32; ++w) {
    if (w < warp) warp_excl += s_warp[w];
    agg += s_warp[w];
  }
  if (threadIdx.x == 0) {
    const uint32_t first = agg ? atomicAdd(&a.work->bin.list_total, agg) : 0u;
    // (a total past 32 bits is past the capacity before it wraps)
    if (first + agg > a.list_cap || first + agg < first) atomicOr(&a.work->bin.status, kStatusListOverflow);
    s_first = first;
  }
  __syncthreads();
  uint32_t run = s_first + warp_excl + (incl - sum);
  const unsigned long long old = s_heavy[warp];
  uint32_t ks = (uint32_t)(old >> 32) + ki - nk;
  uint32_t c = (uint32_t)old + ci - nc;
#pragma unroll
  for (int i = 0; i < kScanItems; ++i) {
    if (base + i < n) {
      a.tile_span[base + i] = make_uint2(run, v[i]);
      if (v[i] > thr) {
        if (chunked) {
          const uint32_t ce = tile_chunk_entries(v[i], a.chunk, t8), nch = (v[i] + ce - 1) / ce;
          for (uint32_t j = 0; j < nch && c + j < a.chunk_cap; ++j) {
            uint4* d = reinterpret_cast<uint4*>(&a.chunk_desc[c + j]);
            d[0] = make_uint4(base + i, run + j * ce, min(ce, v[i] - j * ce), ks);
            d[1] = make_uint4(j, nch, 0u, 0u);
          }
          if (nch > 1 && ks + nch <= a.key_cap)
            for (uint32_t k = 0; k < bins; ++k) a.hdone[(size_t)ks * bins + k] = 0;
          c += nch;
          if (nch > 1) ks += nch;
          // chunks past the buffers are not rasterized: report it
          if (c > a.chunk_cap || ks > a.key_cap) atomicOr(&a.work->bin.status, kStatusListOverflow);
        } else {
          if (c < a.heavy_cap) a.heavy[c] = base + i;
          else atomicOr(&a.work->bin.status, kStatusListOverflow);
          ++c;
        }
      }
    }
    run += v[i];
  }
}

// ------------------------------------------------------------------ kernel 3
// Large triangles (more than kLargeTiles tiles in their box): their box tiles,
// numbered row by row, are cut into segments of kLargeSeg, and a warp takes one
// segment at a time, a run of consecutive tiles per lane, so a huge triangle
// spreads over many warps.  The tiles are counted and recorded like the small
// triangles'; returns the lane's number of tiles that pass and are not listed.
__device__ __forceinline__ uint32_t large_segment(const RasterFrameArgs& a, uint32_t it, uint16_t* queue, int lane)
{
  constexpr uint32_t kLaneRun = kLargeSeg / 32;
  const uint2 sg = a.large_seg[it];
  const WalkTri& w = a.large_walk[sg.x];
  const uint32_t j0 = sg.y * kLargeSeg, tw = (uint32_t)w.tw;
  const int tsh = __ffs(a.tile) - 1 - kRefBinLg2;   // tile edge = 8 << tsh
  const uint32_t ntiles = tw * (uint32_t)((w.by2 >> tsh) - w.ty1 + 1);
  uint32_t m = 0, skipped = 0;
  for (uint32_t k = 0; k < kLaneRun;) {   // the parts of the run that lie in one row
    const uint32_t j = j0 + (uint32_t)lane * kLaneRun + k;
    if (j >= ntiles) break;
    uint32_t col;
    const uint32_t row = fast_divmod(j, tw, w.tw_m, col);
    const uint32_t n = min(kLaneRun - k, tw - col);
    const uint32_t pass = row_mask(w, row, col, n, a.tile), list = pass & listed_mask(w, row, col, n);
    skipped += (uint32_t)(__popc(pass) - __popc(list));
    m |= list << k;
    k += n;
  }
  const auto key_of = [&](uint32_t e, uint32_t& gidx) {
    gidx = w.gidx;
    return tile_key(w, j0 + e);
  };
  uint32_t qn = 0;
  __syncwarp();
  queue_masks(a, queue, qn, m, 0u, (uint32_t)lane * kLaneRun, lane, key_of);
  if (qn) record_queue(a, queue, 0u, qn, lane, key_of);
  return skipped;
}

// The count pass of the large triangles' segments.
__global__ void __launch_bounds__(256, 4) raster_large_count(const __grid_constant__ RasterFrameArgs a)
{
  pdl_wait();
  pdl_trigger();
  __shared__ uint16_t s_queue[8][kWalkQueue];
  const uint32_t items = min((uint32_t)a.work->bin.large_acc, a.seg_cap);
  const uint32_t warps = gridDim.x * (blockDim.x >> 5);
  const int lane = threadIdx.x & 31;
  unsigned long long skipped = 0;
  for (uint32_t it = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); it < items; it += warps)
    skipped += __reduce_add_sync(kFull, large_segment(a, it, s_queue[threadIdx.x >> 5], lane));
  if (lane == 0 && skipped) atomicAdd(&a.work->bin.skipped, skipped);
}

// The scatter pass (the compaction): every recorded pair becomes its list
// entry at its tile's first entry + its index in the tile, a streaming pass with no
// atomics; four pairs per thread per trip, loads first.
__global__ void __launch_bounds__(256) raster_scatter(const __grid_constant__ RasterFrameArgs a)
{
  pdl_wait();
  pdl_trigger();
  // the counts are final: they become the frame's result, and the next frame
  // finds the working counters at 0
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    a.ctr->bin = a.work->bin;
    a.ctr->covered = 0ull;
    a.ctr->work_next = 0u;
    a.ctr->cov_count = 0u;
    a.work->bin = BinCounts{};
  }
  // gridDim.x is a multiple of kPairParts: every partition gets
  // gridDim.x / kPairParts CTAs
  const uint32_t p = blockIdx.x % kPairParts, sub = blockIdx.x / kPairParts;
  const uint32_t part_cap = a.list_cap / kPairParts;
  const uint32_t n = min(a.work->pair_part[p], part_cap);
  const unsigned long long* ptl = a.pair_tl + (size_t)p * part_cap;
  const uint32_t* pg = a.pair_g + (size_t)p * part_cap;
  const uint32_t stride = (gridDim.x / kPairParts) * blockDim.x;
  for (uint32_t i0 = sub * blockDim.x + threadIdx.x; i0 < n; i0 += 4 * stride) {
    unsigned long long tl[4];
    uint32_t gi[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const uint32_t i = i0 + (uint32_t)q * stride;
      tl[q] = i < n ? __ldcs(&ptl[i]) : ~0ull;
      gi[q] = i < n ? __ldcs(&pg[i]) : 0u;
    }
    uint32_t off[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) off[q] = tl[q] != ~0ull ? a.tile_span[(uint32_t)tl[q]].x : 0u;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      if (tl[q] == ~0ull) continue;
      const uint32_t dst = off[q] + (uint32_t)(tl[q] >> 32);
      if (dst < a.list_cap) a.tile_list[dst] = gi[q];
    }
  }
}

// ------------------------------------------------------------------ kernel 4
// Inverse of submission_rank: the triangle id with the given rank.
__device__ __forceinline__ uint32_t rank_to_id(uint32_t r, const RasterSceneDev& S)
{
  const uint32_t nVS = (uint32_t)S.nVS;
  if (S.vs_chunks <= nVS) return r;  // at most one chunk per VS bin: ids are submitted in order
  uint32_t lo = 0, hi = nVS - 1;
  while (lo < hi) {
    const uint32_t b = (lo + hi + 1) >> 1;
    const uint32_t start = kVsChunk * (b * S.vs_q + min(b, S.vs_rem)) - (S.vs_last < b ? S.vs_deficit : 0u);
    if (start <= r) lo = b; else hi = b - 1;
  }
  const uint32_t start = kVsChunk * (lo * S.vs_q + min(lo, S.vs_rem)) - (S.vs_last < lo ? S.vs_deficit : 0u);
  const uint32_t pos = r - start;
  return (lo + (pos / kVsChunk) * nVS) * kVsChunk + pos % kVsChunk;
}


// colour of the winning fragment (raster.pikostage:244-309), triangle `id` of
// scene S whose setup records start at `setup`: barycentrics from
// the same edge values, Gouraud interpolation, optional texel, toABGR by
// truncation.  inv255[k] holds (float)k / 255.0f, the exact quotient fromABGR
// computes (piko/math.h:323-330), so no division is repeated per pixel.
__device__ __forceinline__ uint32_t shade_winner(const RasterSceneDev& S, const TriSetup* setup, uint32_t id, int px,
                                                 int py, const float* inv255)
{
  // the texture coordinates are fetched by triangle id, alongside the setup record
  float2 q0 = make_float2(0.0f, 0.0f), q1 = q0, q2 = q0;
  if (S.uv) {
    q0 = __ldg(&S.uv[id]);
    q1 = __ldg(&S.uv[(size_t)S.N + id]);
    q2 = __ldg(&S.uv[2 * (size_t)S.N + id]);
  }
  const TriSetup r = load_setup(&setup[id]);
  const int32_t Xc = px * 16 + 8, Yc = py * 16 + 8;
  const int32_t e1 = edge_at(Xc, Yc, r.x[1], r.y[1], wsub(r.x[2], r.x[1]), wsub(r.y[2], r.y[1]));
  const int32_t e2 = edge_at(Xc, Yc, r.x[2], r.y[2], wsub(r.x[0], r.x[2]), wsub(r.y[0], r.y[2]));
  const float alpha = (float)e1 * r.inv;
  const float beta = (float)e2 * r.inv;
  float vc[3][3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    vc[k][0] = inv255[(r.c[k] >> 0) & 255u];
    vc[k][1] = inv255[(r.c[k] >> 8) & 255u];
    vc[k][2] = inv255[(r.c[k] >> 16) & 255u];
  }
  float col[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const float d0 = vc[0][c] - vc[2][c], d1 = vc[1][c] - vc[2][c];
    col[c] = vc[2][c] + alpha * d0 + beta * d1;
  }
  if (S.uv) {
    const float u = q2.x + alpha * (q0.x - q2.x) + beta * (q1.x - q2.x);
    const float v = q2.y + alpha * (q0.y - q2.y) + beta * (q1.y - q2.y);
    const int tx = cvt_i32_x86(floorf(u * (float)S.tex_w)) & (S.tex_w - 1);
    const int ty = cvt_i32_x86(floorf(v * (float)S.tex_h)) & (S.tex_h - 1);
    const uchar4 t = __ldg(&S.tex[(size_t)ty * S.tex_w + tx]);
    col[0] = col[0] * inv255[t.x];
    col[1] = col[1] * inv255[t.y];
    col[2] = col[2] * inv255[t.z];
  }
  return pack_abgr(col[0], col[1], col[2]);
}

// 8x8 tiles (one reference bin each): a warp takes up to 32 list entries at a
// time, one per lane, of one tile or of several with short lists.  Lists hold
// exactly the reference's (triangle, bin) pairs.
//
//   1. Each lane builds its entry's coverage of the tile as a 64-bit mask:
//      the edge functions are stepped over the pixels, and the sign of their
//      OR is shifted into the mask (5 instructions a pixel for 32 entries at
//      once; testing every entry by the whole warp, two pixels a lane, took
//      about 34 warp instructions an entry, this takes about 14).
//   2. The entries are put in the order of a lower bound of their depth in the
//      tile, and the masks transposed (five shuffle stages), so that lane p
//      holds one bit per entry for pixels p and p + 32.
//   3. Each lane evaluates the depth of its covered entries, nearest bound
//      first, and stops at the first whose bound lies behind its pixel's
//      current depth: with the mix's overdraw most entries are never evaluated.
struct __align__(16) BinTri {
  int32_t e1, e2, sx1, sx2;     // edge values at the centre of the tile's pixel (0, 0); per-pixel x steps
  int32_t sy1, sy2;             // per-pixel y steps
  float inv, z2;
  float z0mz2, z1mz2;
  uint32_t rank1;
  uint32_t bound;               // the high 24 bits of the depth key no fragment of the entry in this tile is below
};
static_assert(sizeof(BinTri) == 48, "BinTri layout");

// Scene and pixel origin of an 8x8 tile.
struct Tile8 {
  const RasterSceneDev* S;
  int X0, Y0;
};

template <bool ONE>
__device__ __forceinline__ Tile8 tile8_geom(const RasterFrameArgs& a, const uint32_t* tb, uint32_t tile)
{
  Tile8 t;
  const int s = scene_of_tile<ONE>(a, tb, tile);
  t.S = &scene_at<ONE>(a, s);
  uint32_t tx;
  const uint32_t ty = fast_divmod(tile - t.S->tile_base, (uint32_t)t.S->tiles_x, t.S->tiles_x_m, tx);
  t.X0 = (int)tx * kRefBin;
  t.Y0 = (int)ty * kRefBin;
  return t;
}

// One stage of a 32x32 bit transpose over the warp's lanes.
__device__ __forceinline__ uint32_t transpose_stage(uint32_t x, int s, uint32_t m, int lane)
{
  const uint32_t y = __shfl_xor_sync(kFull, x, s);
  return (lane & s) ? ((x & ~m) | ((y >> s) & m)) : ((x & m) | ((y << s) & ~m));
}
// Word `lane` becomes the bits `lane` of the 32 lanes' words.
__device__ __forceinline__ uint32_t transpose32(uint32_t x, int lane)
{
  x = transpose_stage(x, 16, 0x0000ffffu, lane);
  x = transpose_stage(x, 8, 0x00ff00ffu, lane);
  x = transpose_stage(x, 4, 0x0f0f0f0fu, lane);
  x = transpose_stage(x, 2, 0x33333333u, lane);
  return transpose_stage(x, 1, 0x55555555u, lane);
}

// A lower bound of the depth that the fragments of entry t (least vertex depth
// zmin, greatest magnitude zmax) can have in its tile: the larger of the least
// vertex depth and the least corner value of the depth plane over the
// tile's pixel centres, less the rounding that the reference's float sequence
// (and this one) can add.  With u = 2^-24 every factor below is exact to 4u and
// every sum to a few u of the magnitudes added, so a margin of 2^-18 of those
// magnitudes (64 u) covers both.  Returned as the high 24 bits of a fragment
// key's depth half (frag_key), rounded down; 0 (no bound) where the bound is
// not positive -- negative depths order the other way round -- or not a
// number.  Not for triangles whose edge values or area may wrap.
__device__ __forceinline__ uint32_t depth_bound(const BinTri& t, float zmin, float zmax)
{
  constexpr float kMargin = 3.814697265625e-6f;   // 2^-18
  const float vertex = zmin - kMargin * zmax;
  const float d0 = t.inv * t.z0mz2, d1 = t.inv * t.z1mz2;
  const float t0 = (float)t.e1 * d0, t1 = (float)t.e2 * d1;
  const float x0 = 7.0f * ((float)t.sx1 * d0), x1 = 7.0f * ((float)t.sx2 * d1);
  const float y0 = 7.0f * ((float)t.sy1 * d0), y1 = 7.0f * ((float)t.sy2 * d1);
  const float mag = fabsf(t.z2) + fabsf(t0) + fabsf(t1) + fabsf(x0) + fabsf(x1) + fabsf(y0) + fabsf(y1) + zmax;
  const float plane = t.z2 + t0 + t1 + fminf(x0 + x1, 0.0f) + fminf(y0 + y1, 0.0f) - kMargin * mag;
  const float lb = plane > vertex ? plane : vertex;
  return lb > 0.0f ? (__float_as_uint(lb) | 0x80000000u) >> 8 : 0u;
}

// What the resolve of a tile needs of an entry besides its BinTri, staged in
// shared memory when the entry is built, so a pixel's winner is shaded from
// shared memory: the vertex colours as floats (byte / 255) and the texture
// coordinates, each as vertex 2's value and vertex 0's and 1's minus it -- the
// differences shade_winner forms for every pixel, formed once.
struct __align__(16) BinShade {
  float c2[3], dc0[3], dc1[3];   // per channel
  float u2, du0, du1;
  float v2, dv0, dv1, pad;
};
static_assert(sizeof(BinShade) == 64, "BinShade layout");

// A warp's entries.
struct WarpEntries {
  BinTri tri[32];
  BinShade shade[32];
  uint32_t mlo[32], mhi[32];   // coverage of pixel rows 0-3 and 4-7
};

// Depth bounds and their order are worth their cost (some 130 warp
// instructions for 32 entries) only where the entries cover the tile's pixels
// several times over: with at most this many covered samples (2.5 a pixel of
// one tile) the entries stay in list order and every one is evaluated.
constexpr unsigned kSparseSamples = 160;

// Builds n <= 32 entries, entry l by lane l -- and lane l + 16 when n <= 16:
// the two lanes then take four pixel rows each.  The lane's entry is list entry
// gi (nothing drawn when ok is false) in the tile of scene S at (X0, Y0); seq
// numbers the tiles of the entries, ascending with l.  Entries land in w
// ordered by (seq, depth bound); m0 / m1 get bit i set where entry i covers the
// lane's pixel (lane & 7, lane >> 3) / the pixel 4 rows above.  stage: w.shade
// too.
__device__ __forceinline__ void frag8_build(const RasterFrameArgs& a, const RasterSceneDev& S, int n, bool ok,
                                            uint32_t gi, uint32_t seq, int X0, int Y0, bool stage, WarpEntries& w,
                                            int lane, const float* inv255, unsigned& covered, uint32_t& m0,
                                            uint32_t& m1)
{
  const bool pair = n <= 16;
  const int ent = pair ? lane & 15 : lane;
  BinTri t;
  uint32_t lo = 0u, hi = 0u, vc[3] = {0u, 0u, 0u};
  float2 q0 = make_float2(0.0f, 0.0f), q1 = q0, q2 = q0;
  bool bounded = false;
  float zmin = 0.0f, zmax = 0.0f;
  if (ok) {
    // the uv arrays are indexed by triangle id = setup slot - the scene's base
    if (stage && S.uv) {
      const uint32_t id = gi - S.tri_base;
      q0 = __ldg(&S.uv[id]);
      q1 = __ldg(&S.uv[(size_t)S.N + id]);
      q2 = __ldg(&S.uv[2 * (size_t)S.N + id]);
    }
    const TriSetup r = load_setup(&a.setup[gi]);
    const int32_t Xc = X0 * 16 + 8, Yc = Y0 * 16 + 8;
    int32_t e[3], sx[3], sy[3], ta = 0;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const int j = i == 2 ? 0 : i + 1;
      const int32_t dx = wsub(r.x[j], r.x[i]), dy = wsub(r.y[j], r.y[i]);
      e[i] = edge_at(Xc, Yc, r.x[i], r.y[i], dx, dy);
      sx[i] = -wshl(dy, 4);
      sy[i] = wshl(dx, 4);
      // trivial accept at the first pixel centre (raster.pikostage:201-211)
      int32_t off = dy >= 0 ? sx[i] : 0;
      off = wadd(off, dx < 0 ? sy[i] : 0);
      ta |= wadd(e[i], wshl(off, kRefBinLg2));
    }
    // the bin is the triangle's: only its pixels remain to be tested
    if (ta >= 0) {
      lo = hi = 0xffffffffu;
    } else if (r.hix > X0 * 16 && r.hiy > Y0 * 16) {
      // (the box's high corner is rounded up to 16 px: it cuts no tile)
      int ya = 0, yb = kRefBin - 1;
      if (!(r.flags & kTriRisk)) {   // covered centres lie inside the triangle when no edge value can wrap
        ya = max((min(min(r.y[0], r.y[1]), r.y[2]) >> 4) - 1 - Y0, 0);
        yb = min((max(max(r.y[0], r.y[1]), r.y[2]) >> 4) - Y0, kRefBin - 1);
      }
      if (pair) {   // (the other lane of the pair takes the other rows)
        if (lane < 16) yb = min(yb, 3); else ya = max(ya, 4);
      }
      int32_t r0 = wadd(e[0], wmul(ya, sy[0])), r1 = wadd(e[1], wmul(ya, sy[1])), r2 = wadd(e[2], wmul(ya, sy[2]));
      unsigned long long m = 0ull;
#pragma unroll 1
      for (int y = ya; y <= yb; ++y) {
        // pixel 7 first, so that pixel 0 ends in bit 0: bits of outside pixels
        int32_t f0 = wadd(r0, wmul(7, sx[0])), f1 = wadd(r1, wmul(7, sx[1])), f2 = wadd(r2, wmul(7, sx[2]));
        uint32_t out = 0u;
#pragma unroll
        for (int x = 0; x < kRefBin; ++x) {
          out = __funnelshift_l((uint32_t)(f0 | f1 | f2), out, 1);
          f0 = wsub(f0, sx[0]); f1 = wsub(f1, sx[1]); f2 = wsub(f2, sx[2]);
        }
        m |= (unsigned long long)(~out & 0xffu) << (8 * y);
        r0 = wadd(r0, sy[0]); r1 = wadd(r1, sy[1]); r2 = wadd(r2, sy[2]);
      }
      lo = (uint32_t)m;
      hi = (uint32_t)(m >> 32);
    }
    if (pair) {
      if (lane < 16) hi = 0u; else lo = 0u;
    }
    t.e1 = e[1]; t.e2 = e[2];
    t.sx1 = sx[1]; t.sx2 = sx[2];
    t.sy1 = sy[1]; t.sy2 = sy[2];
    t.inv = r.inv; t.z2 = r.z[2];
    t.z0mz2 = r.z[0] - r.z[2];
    t.z1mz2 = r.z[1] - r.z[2];
    t.rank1 = r.rank1;
    vc[0] = r.c[0]; vc[1] = r.c[1]; vc[2] = r.c[2];
    bounded = !(r.flags & (kTriRisk | kTriAreaRisk));
    zmin = fminf(fminf(r.z[0], r.z[1]), r.z[2]);
    zmax = fmaxf(fmaxf(fabsf(r.z[0]), fabsf(r.z[1])), fabsf(r.z[2]));
    if (a.cov_cap) {   // coverage dump
      for (unsigned long long m = ((unsigned long long)hi << 32) | lo; m; m &= m - 1) {
        const int p = __ffsll(m) - 1;
        const uint32_t slot = atomicAdd(&a.ctr->cov_count, 1u);
        if (slot < a.cov_cap) {
          a.cov_tri[slot] = gi - S.tri_base;
          a.cov_pix[slot] = (uint32_t)((Y0 + (p >> 3)) * S.W + X0 + (p & 7));
        }
      }
    }
  }
  const unsigned mine = __popc(lo) + __popc(hi);
  covered += mine;
  // place by (tile, depth bound, lane)
  int at = ent;
  t.bound = 0u;
  if (__reduce_add_sync(kFull, mine) > kSparseSamples) {
    if (bounded) t.bound = depth_bound(t, zmin, zmax);
    const uint32_t key = (seq << 29) | (t.bound << 5) | (uint32_t)ent;
    at = 0;
    for (int i = 0; i < n; ++i) at += __shfl_sync(kFull, key, i) < key ? 1 : 0;
  }
  __syncwarp();   // every lane is done with the entries that w held
  if (lane < n) {
    w.tri[at] = t;
    if (stage) {
      BinShade h;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const float v0 = inv255[(vc[0] >> (8 * c)) & 255u], v1 = inv255[(vc[1] >> (8 * c)) & 255u];
        const float v2 = inv255[(vc[2] >> (8 * c)) & 255u];
        h.c2[c] = v2;
        h.dc0[c] = v0 - v2;
        h.dc1[c] = v1 - v2;
      }
      h.u2 = q2.x; h.du0 = q0.x - q2.x; h.du1 = q1.x - q2.x;
      h.v2 = q2.y; h.dv0 = q0.y - q2.y; h.dv1 = q1.y - q2.y;
      h.pad = 0.0f;
      w.shade[at] = h;
    }
  }
  if (ent >= n) at = ent;   // no entry: an empty mask
  if (!pair || lane < 16) w.mlo[at] = lo;
  if (!pair) w.mhi[at] = hi;
  else if (lane >= 16) w.mhi[at] = hi;
  if (pair && lane >= 16) { w.mlo[lane] = 0u; }
  if (pair && lane < 16) { w.mhi[lane + 16] = 0u; }
  __syncwarp();
  m0 = transpose32(w.mlo[lane], lane);
  m1 = transpose32(w.mhi[lane], lane);
}

// Entry t's fragment at tile pixel (ox, ly): barycentrics from the edge values,
// z in the reference's operation order, as a key of the order-independent depth
// test.
__device__ __forceinline__ unsigned long long frag8_key(const BinTri& t, int ox, int ly)
{
  const int32_t g1 = wadd(wadd(t.e1, wmul(ox, t.sx1)), wmul(ly, t.sy1));
  const int32_t g2 = wadd(wadd(t.e2, wmul(ox, t.sx2)), wmul(ly, t.sy2));
  const float alpha = (float)g1 * t.inv;
  const float beta = (float)g2 * t.inv;
  const float z = t.z2 + alpha * t.z0mz2 + beta * t.z1mz2;
  return frag_key(z, t.rank1);
}

// Folds the fragments of entries m0 / m1 (bits: the lane's two pixels) into the
// lane's keys; w0 / w1 follow the entry of each pixel's current winner.  A trip
// takes the next covered entry of each pixel: two independent evaluations
// without a branch (a pixel that is done evaluates entry 31 or 0 and drops the
// result).  A pixel is done when its bits are, or at the first entry whose
// bound lies behind its depth: later ones of the tile lie behind it too.
__device__ __forceinline__ void frag8_test(const BinTri* st, uint32_t m0, uint32_t m1, int lane,
                                           unsigned long long& k0, unsigned long long& k1, int& w0, int& w1)
{
  const int ox = lane & 7, oy = lane >> 3;   // first pixel; the second is (ox, oy + 4)
  while (m0 | m1) {
    const int i0 = (__ffs(m0) - 1) & 31, i1 = (__ffs(m1) - 1) & 31;
    const BinTri a = st[i0], b = st[i1];
    const unsigned long long ka = frag8_key(a, ox, oy), kb = frag8_key(b, ox, oy + 4);
    const bool pa = m0 != 0u && a.bound <= (uint32_t)(k0 >> 40), pb = m1 != 0u && b.bound <= (uint32_t)(k1 >> 40);
    if (pa && ka < k0) { k0 = ka; w0 = i0; }
    if (pb && kb < k1) { k1 = kb; w1 = i1; }
    m0 = pa ? m0 & (m0 - 1u) : 0u;
    m1 = pb ? m1 & (m1 - 1u) : 0u;
  }
}

// Writes the lane's two pixels: the winner's colour (shaded once per pixel)
// and depth, or the clear colour and 1.0.
__device__ __forceinline__ void resolve8(const RasterFrameArgs& a, const Tile8& tl, int lane, unsigned long long k0,
                                         unsigned long long k1, const float* inv255)
{
  const RasterSceneDev& S = *tl.S;
  const int px = tl.X0 + (lane & 7);
  if (px >= S.W) return;
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const int py = tl.Y0 + (lane >> 3) + 4 * k;
    if (py >= S.H) continue;
    const unsigned long long key = k ? k1 : k0;
    uint32_t c = kClearColor;
    float z = 1.0f;
    if (key != kInitKey) {
      const uint32_t rank = ~(uint32_t)key - 1u;
      z = __uint_as_float((uint32_t)(key >> 32) ^ 0x80000000u);
      const uint32_t id = rank_to_id(rank, S);
      c = shade_winner(S, a.setup + S.tri_base, id, px, py, inv255);
    }
    const size_t idx = (size_t)py * S.W + px;
    S.fb[idx] = c;
    S.depth[idx] = z;
  }
}

// The colour of entry t / sh at tile pixel (ox, ly): shade_winner's arithmetic
// (raster.pikostage:244-309) from the tile-local edge values, which equal the
// pixel-centre edge values bit for bit (both are the same wrapping int32
// linear function).
__device__ __forceinline__ uint32_t shade_entry(const RasterSceneDev& S, const BinTri& t, const BinShade& sh, int ox,
                                                int ly, const float* inv255)
{
  const int32_t g1 = wadd(wadd(t.e1, wmul(ox, t.sx1)), wmul(ly, t.sy1));
  const int32_t g2 = wadd(wadd(t.e2, wmul(ox, t.sx2)), wmul(ly, t.sy2));
  const float alpha = (float)g1 * t.inv;
  const float beta = (float)g2 * t.inv;
  float col[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) col[c] = sh.c2[c] + alpha * sh.dc0[c] + beta * sh.dc1[c];
  if (S.uv) {
    const float u = sh.u2 + alpha * sh.du0 + beta * sh.du1;
    const float v = sh.v2 + alpha * sh.dv0 + beta * sh.dv1;
    const int tx = cvt_i32_x86(floorf(u * (float)S.tex_w)) & (S.tex_w - 1);
    const int ty = cvt_i32_x86(floorf(v * (float)S.tex_h)) & (S.tex_h - 1);
    const uchar4 tt = __ldg(&S.tex[(size_t)ty * S.tex_w + tx]);
    col[0] = col[0] * inv255[tt.x];
    col[1] = col[1] * inv255[tt.y];
    col[2] = col[2] * inv255[tt.z];
  }
  return pack_abgr(col[0], col[1], col[2]);
}

// Writes the lane's two pixels of a light tile from its winners' staged data
// (st / sh indexed by w0 / w1), or the clear colour and 1.0.
__device__ __forceinline__ void resolve8_staged(const Tile8& tl, int lane, unsigned long long k0, unsigned long long k1,
                                                int w0, int w1, const BinTri* st, const BinShade* sh,
                                                const float* inv255)
{
  const RasterSceneDev& S = *tl.S;
  const int ox = lane & 7;
  const int px = tl.X0 + ox;
  if (px >= S.W) return;
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const int ly = (lane >> 3) + 4 * k;
    const int py = tl.Y0 + ly;
    if (py >= S.H) continue;
    const unsigned long long key = k ? k1 : k0;
    const int w = k ? w1 : w0;
    uint32_t c = kClearColor;
    float z = 1.0f;
    if (key != kInitKey) {
      z = __uint_as_float((uint32_t)(key >> 32) ^ 0x80000000u);
      c = shade_entry(S, st[w], sh[w], ox, ly, inv255);
    }
    const size_t idx = (size_t)py * S.W + px;
    S.fb[idx] = c;
    S.depth[idx] = z;
  }
}

// Chunk j of nch of a tile (key slots from ks on) is done with bin `bin` of the
// tile's `bins`: leaves its keys; true for the last chunk to arrive, whose
// k0 / k1 are then the least keys over the tile's chunks.
__device__ __forceinline__ bool merge_chunks(const RasterFrameArgs& a, uint32_t bins, uint32_t bin, uint32_t ks,
                                             uint32_t j, uint32_t nch, int lane, unsigned long long& k0,
                                             unsigned long long& k1)
{
  // pixel p of the bin is key p: the lane's pixels are lane and lane + 32
  unsigned long long* ck = a.chunk_keys + ((size_t)(ks + j) * bins + bin) * 64;
  ck[lane] = k0;
  ck[lane + 32] = k1;
  __threadfence();
  __syncwarp();
  uint32_t done = 0;
  if (lane == 0) done = atomicAdd(&a.hdone[(size_t)ks * bins + bin], 1u);
  done = __shfl_sync(kFull, done, 0);
  if (done + 1 != nch) return false;
  // the last chunk: every other chunk's keys are in chunk_keys
  __threadfence();
  for (uint32_t o = 0; o < nch; ++o) {
    if (o == j) continue;
    const unsigned long long* cj = a.chunk_keys + ((size_t)(ks + o) * bins + bin) * 64;
    k0 = min(k0, __ldcg(&cj[lane]));
    k1 = min(k1, __ldcg(&cj[lane + 32]));
  }
  return true;
}

// Persistent.  A warp works in passes of up to 32 list entries (one copy of the
// code for every kind of pass: the kernel's instruction footprint matters more
// than the branches between them).  Warp w of the grid first draws the
// short-list groups w, w + warps, ... (a.group consecutive tiles; of these
// the ones with at most a.queue_min entries, as many tiles at a time as have 32
// entries together); then it takes chunks of the longer lists (scan_tiles
// queued them) from a counter, which also evens out the warps' finishing times.
// A tile whose list fits one pass is resolved from shared memory.  Of a list
// in several chunks each leaves its keys, and the warp that completes the last
// one takes the per-pixel minimum over the tile's chunks and resolves the tile.
// The key order makes the result independent of which warp merges when.
// (Taking most chunks by warp index instead, with the next one's list read
// ahead, measured 5-20% slower: the short-list phase leaves the warps too
// uneven.  So did asking for the next chunk before the current one is done.)
template <bool ONE>
__global__ void __launch_bounds__(256, 4) raster_frag8(const __grid_constant__ RasterFrameArgs a)
{
  pdl_wait();
  frame_begin(a);
  if (list_overflowed(a)) return;
  __shared__ WarpEntries s_ent[8];
  __shared__ float s_inv255[256];
  __shared__ unsigned s_cov[8];
  __shared__ uint32_t s_tb[kSceneTable];
  s_inv255[threadIdx.x] = (float)threadIdx.x / 255.0f;
  load_scene_table<ONE, kSceneTable>(a, s_tb, true);
  __syncthreads();
  const int wid = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  WarpEntries& w = s_ent[wid];
  unsigned covered = 0;
  const uint32_t n_chunks = min((uint32_t)a.ctr->bin.heavy_acc, a.chunk_cap);
  const uint32_t n_groups = (a.n_tiles_total + a.group - 1) / a.group;
  const uint32_t nwarps = gridDim.x * (blockDim.x >> 5);
  uint32_t g = blockIdx.x * (blockDim.x >> 5) + (uint32_t)wid;   // the next group
  // The group being drawn: tiles t0 + ja .. t0 + nt remain; lane j < nt holds
  // the offset, the entries (0 when it is served as chunks) and the inclusive
  // prefix of tile t0 + j.
  uint32_t t0 = 0, off_j = 0, cnt_j = 0, incl_j = 0;
  unsigned served = 0;
  int ja = 0, nt = 0;
  // The chunk being drawn: entries [b0, len) at off remain; lane l < 8 holds
  // word l of its descriptor.
  uint32_t ci = 0, desc = 0, b0 = 0, len = 0;
  unsigned long long k0 = kInitKey, k1 = kInitKey;
  int w0 = 0, w1 = 0;
  for (;;) {
    const bool light = ja < nt || g < n_groups;
    bool ok, stage = true;
    int n, jb;
    uint32_t base = 0, tile, idx, seq = 0;
    if (light) {
      if (ja >= nt) {
        t0 = g * a.group;
        nt = (int)min(a.group, a.n_tiles_total - t0);
        g += nwarps;
        ja = 0;
        const uint2 span = lane < nt ? a.tile_span[t0 + lane] : make_uint2(0u, 0u);
        off_j = span.x;
        cnt_j = span.y;
        const bool fits = lane < nt && cnt_j <= a.queue_min;
        if (!fits) cnt_j = 0;
        served = __ballot_sync(kFull, fits);
        incl_j = cnt_j;
#pragma unroll
        for (int o = 1; o < kLightGroup; o <<= 1) {
          const uint32_t v = __shfl_up_sync(kFull, incl_j, o);
          if (lane >= o) incl_j += v;
        }
      }
      // tiles [ja, jb): as many as have at most 32 entries together
      if (ja) base = __shfl_sync(kFull, incl_j, ja - 1);
      jb = ja + __popc(__ballot_sync(kFull, lane >= ja && lane < nt && incl_j - base <= 32u));
      n = (int)(__shfl_sync(kFull, incl_j, jb - 1) - base);
      // entry l is of tile j = the first with an inclusive prefix above l
      const uint32_t l = (uint32_t)(n <= 16 ? lane & 15 : lane);
      int j = ja;
      for (int q = ja; q < jb - 1; ++q) j += __shfl_sync(kFull, incl_j, q) - base <= l ? 1 : 0;
      idx = __shfl_sync(kFull, off_j, j) + (l + base - __shfl_sync(kFull, incl_j - cnt_j, j));
      ok = l < (uint32_t)n;
      tile = t0 + (uint32_t)j;
      seq = (uint32_t)(j - ja);
    } else {
      if (b0 >= len) {
        if (lane == 0) ci = atomicAdd(&a.ctr->work_next, 1u);
        ci = __shfl_sync(kFull, ci, 0);
        if (ci >= n_chunks) break;
        if (lane < 8) desc = reinterpret_cast<const uint32_t*>(&a.chunk_desc[ci])[lane];
        len = __shfl_sync(kFull, desc, 2);
        b0 = 0;
        k0 = k1 = kInitKey;
      }
      ja = nt = 0;
      jb = 1;
      n = (int)min(32u, len - b0);
      const uint32_t l = (uint32_t)(n <= 16 ? lane & 15 : lane);
      tile = __shfl_sync(kFull, desc, 0);
      idx = __shfl_sync(kFull, desc, 1) + b0 + l;
      ok = l < (uint32_t)n;
      stage = len <= 32u && __shfl_sync(kFull, desc, 5) == 1u;
      b0 += 32;
    }
    uint32_t m0 = 0u, m1 = 0u;
    if (n) {
      const Tile8 tl = tile8_geom<ONE>(a, s_tb, tile);
      ok = ok && idx < a.list_cap;   // (past the list capacity: the frame reports the overflow)
      frag8_build(a, *tl.S, n, ok, ok ? a.tile_list[idx] : 0u, seq, tl.X0, tl.Y0, stage, w, lane, s_inv255, covered, m0,
                  m1);
    }
#pragma unroll 1
    for (int q = ja; q < jb; ++q) {
      uint32_t bits = 0xffffffffu;
      Tile8 tl;
      if (light) {
        if (!((served >> q) & 1u)) continue;   // (longer lists are drawn as chunks)
        const uint32_t last = __shfl_sync(kFull, incl_j, q) - base, cnt = __shfl_sync(kFull, cnt_j, q);
        if (cnt < 32u) bits = ((1u << cnt) - 1u) << ((last - cnt) & 31u);
        tl = tile8_geom<ONE>(a, s_tb, t0 + (uint32_t)q);
        k0 = k1 = kInitKey;
      } else {
        tl = tile8_geom<ONE>(a, s_tb, tile);
      }
      frag8_test(w.tri, m0 & bits, m1 & bits, lane, k0, k1, w0, w1);
      if (stage) {
        resolve8_staged(tl, lane, k0, k1, w0, w1, w.tri, w.shade, s_inv255);
      } else if (b0 >= len) {
        const uint32_t nch = __shfl_sync(kFull, desc, 5);
        if (nch > 1 && !merge_chunks(a, 1, 0, __shfl_sync(kFull, desc, 3), __shfl_sync(kFull, desc, 4), nch, lane, k0, k1))
          continue;
        resolve8(a, tl, lane, k0, k1, s_inv255);
      }
    }
    ja = light ? jb : 0;
  }

  // fragment count: one atomic per CTA
  covered = __reduce_add_sync(kFull, covered);
  if (lane == 0) s_cov[wid] = covered;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long t = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) t += s_cov[w];
    if (t) atomicAdd(&a.ctr->covered, t);
  }
}

// The bins of the 2 x 2 quad at pixel (X0, Y0) that triangle gi is assigned to
// (bit 2 * dy + dx): its bin range and the trivial reject at each bin's corner
// (raster.pikostage:77-105, 128 = 8 px in 28.4).
__device__ __forceinline__ uint32_t quad_assigned(const RasterFrameArgs& a, uint32_t gi, int X0, int Y0)
{
  const TriSetup r = load_setup(&a.setup[gi]);
  int32_t t00 = 0, t10 = 0, t01 = 0, t11 = 0;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const int j = i == 2 ? 0 : i + 1;
    const int32_t dx = wsub(r.x[j], r.x[i]), dy = wsub(r.y[j], r.y[i]);
    const int32_t sx = -wshl(dy, 7), sy = wshl(dx, 7);
    int32_t t = wadd(dy < 0 ? sx : 0, dx >= 0 ? sy : 0);
    t = wadd(t, edge_at(X0 * 16, Y0 * 16, r.x[i], r.y[i], dx, dy));
    t00 |= t;
    t10 |= wadd(t, sx);
    t01 |= wadd(t, sy);
    t11 |= wadd(wadd(t, sx), sy);
  }
  const int bx = X0 / kRefBin, by = Y0 / kRefBin;
  const int bx1 = (int)(r.bxr & 0xffff), bx2 = (int)(r.bxr >> 16), by1 = (int)(r.byr & 0xffff), by2 = (int)(r.byr >> 16);
  const uint32_t cols = (bx >= bx1 && bx <= bx2 ? 5u : 0u) | (bx + 1 >= bx1 && bx + 1 <= bx2 ? 10u : 0u);
  const uint32_t rows = (by >= by1 && by <= by2 ? 3u : 0u) | (by + 1 >= by1 && by + 1 <= by2 ? 12u : 0u);
  return cols & rows & ((t00 >= 0 ? 1u : 0u) | (t10 >= 0 ? 2u : 0u) | (t01 >= 0 ? 4u : 0u) | (t11 >= 0 ? 8u : 0u));
}

// 16/32-px tiles: raster_frag8's passes over the reference bins of a tile.  An
// item is a list (a short one by warp index, a chunk of a longer one from the
// counter, or without chunk buffers a heavy tile's whole list) and a quad of
// the tile's bins, or one bin of it (a.group).  The list's entries are tested against the quad's four bins
// at once, 32 at a time, and queued per bin; a bin with 32 queued entries gets a
// pass of its own, and the remainders share passes at the end.  A bin drawn by
// one pass is resolved from shared memory, one drawn by several keeps its keys
// there in between.  (Spreading the warp's lanes over one entry's pixels after
// the other, with the tile's keys in shared memory, left most lanes idle on
// small triangles: a 61,200-triangle forest at 800x600 in 16-px tiles, lists of
// up to 400 entries, took 83 us.)
struct BinsSmem {
  WarpEntries ent[8];
  unsigned long long keys[8][4][64];
  uint16_t queue[8][4][64];
  float inv255[256];
  unsigned cov[8];
  uint32_t tb[512];
};

template <int T, bool ONE>
__global__ void __launch_bounds__(256, 4) raster_bins(const __grid_constant__ RasterFrameArgs a)
{
  pdl_wait();
  frame_begin(a);
  if (list_overflowed(a)) return;
  constexpr uint32_t QPT = T / (2 * kRefBin), QUADS = QPT * QPT, NB = 4 * QUADS;
  extern __shared__ __align__(16) unsigned char bins_smem[];
  BinsSmem& B = *reinterpret_cast<BinsSmem*>(bins_smem);
  B.inv255[threadIdx.x] = (float)threadIdx.x / 255.0f;
  load_scene_table<ONE, 512>(a, B.tb, true);
  __syncthreads();
  const int wid = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  WarpEntries& w = B.ent[wid];
  unsigned covered = 0;
  const bool chunked = a.chunk_desc != nullptr;
  // parts of a tile: its quads, or the single bins of its quads
  const uint32_t split = 4u / a.group, parts = QUADS * split;
  const uint32_t n_items = min((uint32_t)a.ctr->bin.heavy_acc, chunked ? a.chunk_cap : a.heavy_cap) * parts;
  const uint32_t n_light = a.n_tiles_total * parts;
  const uint32_t nwarps = gridDim.x * (blockDim.x >> 5);
  uint32_t g = blockIdx.x * (blockDim.x >> 5) + (uint32_t)wid;
  for (;;) {
    uint32_t tile, quad, off, len, ks = 0, j = 0, nch = 1;   // (quad: the part, then its quad)
    if (g < n_light) {
      tile = g / parts;
      quad = g % parts;
      g += nwarps;
      const uint2 span = a.tile_span[tile];
      off = span.x;
      len = span.y;
      if (len > a.queue_min) continue;   // drawn from the queue
    } else {
      uint32_t it = 0;
      if (lane == 0) it = atomicAdd(&a.ctr->work_next, 1u);
      it = __shfl_sync(kFull, it, 0);
      if (it >= n_items) break;
      quad = it % parts;
      if (chunked) {
        const uint4* d = reinterpret_cast<const uint4*>(&a.chunk_desc[it / parts]);
        const uint4 d0 = d[0], d1 = d[1];
        tile = d0.x; off = d0.y; len = d0.z; ks = d0.w;
        j = d1.x; nch = d1.y;
      } else {
        tile = a.heavy[it / parts];
        const uint2 span = a.tile_span[tile];
        off = span.x;
        len = span.y;
      }
    }
    // entries past the list capacity are never read (the frame reports the overflow)
    len = min(len, a.list_cap - min(off, a.list_cap));
    int done = 0, bins_end = 4;    // bins [done, bins_end) of the quad are to be resolved
    if (split > 1) {
      done = (int)(quad & 3u);
      bins_end = done + 1;
      quad >>= 2;
    }
    const uint32_t mine = ((1u << bins_end) - 1u) & ~((1u << done) - 1u);
    Tile8 tl;   // the quad's scene and first pixel
    {
      const int s = scene_of<ONE, 512>(a, B.tb, tile, true);
      tl.S = &scene_at<ONE>(a, s);
      uint32_t tx;
      const uint32_t ty = fast_divmod(tile - tl.S->tile_base, (uint32_t)tl.S->tiles_x, tl.S->tiles_x_m, tx);
      tl.X0 = (int)(tx * T + 2 * (quad % QPT) * kRefBin);
      tl.Y0 = (int)(ty * T + 2 * (quad / QPT) * kRefBin);
    }
    uint32_t b0 = 0, q_base = 0;   // entries [b0, len) remain; queued entries are numbered from q_base
    uint32_t queued = 0;           // lane q < 4: entries queued for bin q
    unsigned touched = 0;          // bins with keys in shared memory
    while (done < bins_end) {
      unsigned full = __ballot_sync(kFull, queued >= 32u);
      while (!full && b0 < len) {
        if (!__any_sync(kFull, queued != 0u)) q_base = b0;
        if (b0 - q_base >= 65504u) break;   // (queue entries are 16-bit: drain first)
        uint32_t in = 0;
        if (b0 + lane < len) in = quad_assigned(a, a.tile_list[off + b0 + lane], tl.X0, tl.Y0) & mine;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const unsigned m = __ballot_sync(kFull, (in >> q) & 1u);
          const uint32_t at = __shfl_sync(kFull, queued, q);
          if ((in >> q) & 1u) B.queue[wid][q][at + __popc(m & lt)] = (uint16_t)(b0 - q_base + lane);
          if (lane == q) queued += __popc(m);
        }
        b0 += 32;
        full = __ballot_sync(kFull, queued >= 32u);
      }
      __syncwarp();
      // the pass: 32 entries of a bin that has as many, or what remains of bins [ja, jb)
      const bool last = !full && b0 >= len;
      int ja, jb;
      uint32_t cnt;   // lane q: entries of bin q in this pass
      if (last) {
        ja = done;
        uint32_t incl = lane >= ja && lane < 4 ? queued : 0u;
        const uint32_t up1 = __shfl_up_sync(kFull, incl, 1);
        if (lane >= 1) incl += up1;
        const uint32_t up2 = __shfl_up_sync(kFull, incl, 2);
        if (lane >= 2) incl += up2;
        jb = ja + __popc(__ballot_sync(kFull, lane >= ja && lane < bins_end && incl <= 32u));
        cnt = lane >= ja && lane < jb ? queued : 0u;
      } else {
        if (!full) full = __ballot_sync(kFull, queued != 0u);
        ja = __ffs(full) - 1;
        jb = ja + 1;
        cnt = lane == ja ? min(queued, 32u) : 0u;
      }
      uint32_t incl = cnt;
#pragma unroll
      for (int o = 1; o < 4; o <<= 1) {
        const uint32_t v = __shfl_up_sync(kFull, incl, o);
        if (lane >= o) incl += v;
      }
      const int n = (int)__shfl_sync(kFull, incl, 3);
      const bool stage = last && nch == 1;   // (for the bins that have no keys yet)
      uint32_t m0 = 0u, m1 = 0u;
      if (n) {
        const uint32_t l = (uint32_t)(n <= 16 ? lane & 15 : lane);
        uint32_t bin = 0;
#pragma unroll
        for (int q = 0; q < 3; ++q) bin += __shfl_sync(kFull, incl, q) <= l ? 1u : 0u;
        const uint32_t top = __shfl_sync(kFull, queued, bin), end = __shfl_sync(kFull, incl, bin);
        const bool ok = l < (uint32_t)n;
        const uint32_t gi = ok ? a.tile_list[off + q_base + B.queue[wid][bin][top - (end - l)]] : 0u;
        frag8_build(a, *tl.S, n, ok, gi, bin, tl.X0 + (int)(bin & 1u) * kRefBin, tl.Y0 + (int)(bin >> 1) * kRefBin, stage, w,
                    lane, B.inv255, covered, m0, m1);
        queued -= cnt;
      }
#pragma unroll 1
      for (int q = ja; q < jb; ++q) {
        const uint32_t cq = __shfl_sync(kFull, cnt, q), eq = __shfl_sync(kFull, incl, q);
        const uint32_t bits = cq >= 32u ? 0xffffffffu : ((1u << cq) - 1u) << ((eq - cq) & 31u);
        unsigned long long* keys = B.keys[wid][q];
        const bool had = (touched >> q) & 1u;
        unsigned long long k0 = kInitKey, k1 = kInitKey;
        int w0 = 0, w1 = 0;
        if (had) { k0 = keys[lane]; k1 = keys[lane + 32]; }
        frag8_test(w.tri, m0 & bits, m1 & bits, lane, k0, k1, w0, w1);
        if (!last) {
          keys[lane] = k0;
          keys[lane + 32] = k1;
          touched |= 1u << q;
          continue;
        }
        const Tile8 bt = {tl.S, tl.X0 + (q & 1) * kRefBin, tl.Y0 + (q >> 1) * kRefBin};
        if (stage && !had) {
          resolve8_staged(bt, lane, k0, k1, w0, w1, w.tri, w.shade, B.inv255);
          continue;
        }
        if (nch > 1 && !merge_chunks(a, NB, quad * 4 + q, ks, j, nch, lane, k0, k1)) continue;
        resolve8(a, bt, lane, k0, k1, B.inv255);
      }
      if (last) done = jb;
    }
  }

  // fragment count: one atomic per CTA
  covered = __reduce_add_sync(kFull, covered);
  if (lane == 0) B.cov[wid] = covered;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long t = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) t += B.cov[k];
    if (t) atomicAdd(&a.ctr->covered, t);
  }
}

// ------------------------------------------------------------------ launch
static int raster_scan_blocks(uint32_t n_tiles) { return (int)((n_tiles + kScanTile - 1) / kScanTile); }

// CTAs of one full wave of a kernel on the current device (cached; every
// launch of this library targets B200s of one kind).  Host threads may launch
// frames concurrently: the cache is an atomic, and two threads that both miss
// it compute and store the same value.
template <class K>
static int wave_ctas(K kernel, std::atomic<int>* cache, int threads = 256, size_t smem = 0)
{
  int v = cache->load(std::memory_order_relaxed);
  if (v <= 0) {
    int dev = 0, sms = 148, per_sm = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem);
    v = sms * (per_sm > 0 ? per_sm : 1);
    cache->store(v, std::memory_order_relaxed);
  }
  return v;
}

// A launch that may begin while the previous kernel of the stream finishes
// (the kernel's pdl_wait() holds it until that kernel's writes are visible).
template <typename K>
static cudaError_t launch_pdl(K kernel, int grid, int block, cudaStream_t st, const RasterFrameArgs& a, size_t smem = 0)
{
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3((unsigned)block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, a);
}

// raster_bins needs more shared memory than a static allocation may have; set
// once per device the library runs on.
static cudaError_t bins_setup()
{
  static std::atomic<unsigned long long> done{0};   // a bit per device ordinal
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  const unsigned long long bit = 1ull << (dev & 63);
  if (e || (done.load(std::memory_order_acquire) & bit)) return e;
  const auto set = [](const void* f) {
    return cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(BinsSmem));
  };
  e = set((const void*)raster_bins<16, true>);
  if (!e) e = set((const void*)raster_bins<16, false>);
  if (!e) e = set((const void*)raster_bins<32, true>);
  if (!e) e = set((const void*)raster_bins<32, false>);
  if (!e) done.fetch_or(bit, std::memory_order_release);
  return e;
}

cudaError_t launch_raster_frame(const RasterFrameArgs& args, int raster_ctas, cudaStream_t st, cudaEvent_t* ev)
{
  RasterFrameArgs a = args;
  static std::atomic<int> setup_wave[2] = {{0}, {0}}, scatter_wave{0}, large_wave{0};
  const bool one = !a.scenes;
  const auto setup = one ? raster_setup<true> : raster_setup<false>;
  const int threads = one ? kSetupThreads<true> : kSetupThreads<false>;
  const size_t setup_smem = one ? sizeof(SetupSmem<kSetupThreads<true>>)
                                : sizeof(SetupSmem<kSetupThreads<false>>) + kSceneTable * sizeof(uint32_t);
  const SetupShape shape =
      setup_shape(a.n_tris_total, (uint32_t)wave_ctas(setup, &setup_wave[one], threads, setup_smem), (uint32_t)threads);
  a.batch = shape.batch;
  // the scatter grid covers the list groups of every triangle plus the large
  // triangles' segments (a grid-stride loop takes any excess)
  const int scatter_blocks = std::max(1, wave_ctas(raster_scatter, &scatter_wave) / (int)kPairParts) * (int)kPairParts;
  if (ev) cudaEventRecord(ev[0], st);
  const int large_blocks = wave_ctas(raster_large_count, &large_wave);
  // every launch after the first may start while its predecessor drains
  // (programmatic dependent launch); each waits for it before touching memory
  cudaError_t e = cudaSuccess;
  if (shape.blocks) setup<<<(int)shape.blocks, threads, setup_smem, st>>>(a);
  if (shape.blocks && !e) e = launch_pdl(raster_large_count, large_blocks, 256, st, a);
  if (ev) cudaEventRecord(ev[1], st);
  if (!e) e = launch_pdl(scan_tiles, raster_scan_blocks(a.n_tiles_total), kScanThreads, st, a);
  if (ev) cudaEventRecord(ev[2], st);
  if (!e) e = launch_pdl(raster_scatter, scatter_blocks, 256, st, a);
  if (ev) cudaEventRecord(ev[3], st);
  if (!e && a.tile != kRefBin) e = bins_setup();
  if (!e) {
    switch (a.tile) {
      case 8: e = launch_pdl(one ? raster_frag8<true> : raster_frag8<false>, raster_ctas, 256, st, a); break;
      case 32: e = launch_pdl(one ? raster_bins<32, true> : raster_bins<32, false>, raster_ctas, 256, st, a, sizeof(BinsSmem)); break;
      default: e = launch_pdl(one ? raster_bins<16, true> : raster_bins<16, false>, raster_ctas, 256, st, a, sizeof(BinsSmem)); break;
    }
  }
  if (ev) cudaEventRecord(ev[4], st);
  if (e) return e;
  return cudaGetLastError();
}

cudaError_t raster_tiles_occupancy(int tile, int* blocks_per_sm)
{
  if (tile == kRefBin) return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, raster_frag8<false>, 256, 0);
  const cudaError_t e = bins_setup();
  if (e) return e;
  if (tile == 32)
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, raster_bins<32, false>, 256, sizeof(BinsSmem));
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, raster_bins<16, false>, 256, sizeof(BinsSmem));
}

}  // namespace piko

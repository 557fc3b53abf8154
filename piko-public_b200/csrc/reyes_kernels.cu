// Reyes pipeline for sm_100a: the reference's ReyesPipe (SplitStage with its
// self loop -> DiceStage -> ShadeStage -> PikoScreen, pikoc/samples/reyesPipe)
// off a device work queue:
//
//   reyes_split    one cooperative launch (one CTA per SM), sixteen lanes per
//       patch: project the 16 control points, measure the u/v screen extents,
//       split at the halves (de Casteljau) or emit a leaf with its dice grid
//       (R11, split.pikostage:240-343).  Each CTA expands its patches level
//       after level in shared memory, with a stack of its own behind it; a
//       global frontier evens the CTAs out after a grid barrier; leaves are
//       staged and written out in batches.  No host round
//       trip between levels (the reference copies the Split stage back to the
//       host every level).
//   reyes_dice     every CTA an equal range of dice rows; per group of rows,
//       the control rows at each u once, each grid point once into shared
//       memory: patch position and normal, projection, the corner-averaged
//       "Phong" colour and the mean depth (R12, dice.pikostage:159-312; R13
//       colour, shade.pikostage:64-109), the 64-pixel Shade-bin range of three
//       corners (shade.pikostage:51-56) cut with the four-corner bounds to one
//       pixel rectangle, then a sample-parallel coverage pass over that
//       rectangle; every covered sample is a 64-bit atomic minimum on the
//       sample's state (depth, micropolygon).
//   reyes_big      the same for micropolygons with more than kSmallPx candidate
//       pixels, a warp each.
//   reyes_ties     the samples at which two fragments met at one depth: the
//       reference's order decides between them.
//   reyes_pixels   writes every pixel from its samples' states (averages them
//       with 4 samples per pixel) and sets the reached ones back to empty for
//       the next frame.
//       Shade work is spread per micropolygon and per fragment, not per
//       screen tile, so silhouette tiles where thousands of micropolygons pile
//       up cost no more than anywhere else.  The per-sample test is the
//       reference's (both windings, shade.pikostage:161-235).
//
// Order independence.  The reference resolves depth with
//   while (remote > z) remote = atomicMin(bits, z);  pass iff zbuf == z
// in the order Dice bins, leaves and grid points are processed.  Run
// sequentially that keeps, per pixel, the minimum depth m, the depth bits of
// the FIRST fragment with depth == m and the colour of the LAST one.  Every
// micropolygon carries a 64-bit key that sorts like the reference's processing
// order -- (Dice bin, split level, position in the level, grid index) -- so
// the kernels may visit fragments in any order.
#include <mutex>
#include <type_traits>

#include "runtime_internal.h"

namespace piko {

constexpr unsigned kFullR = 0xffffffffu;

struct __align__(16) PatchRec {
  float4 cp[16];
  uint32_t i0;          // input patch index
  uint32_t level;       // split level = numSplits
  unsigned long long s; // position key inside the level: children of s are 2s, 2s+1
  uint32_t nu, nv;      // dice grid (leaves)
  uint32_t rowbase;     // first dice row (leaves): leaf rows are numbered in slot order
  uint32_t pad;
};
static_assert(sizeof(PatchRec) == 288, "PatchRec layout");

struct __align__(16) UpolyRec {
  float sx[4], sy[4];   // screen x, y of the 4 corners
  float z;              // mean corner depth
  uint32_t color;       // ABGR
  unsigned long long key;  // processing-order key + 1
  int32_t x0, x1, y0, y1;  // shaded pixel rectangle [x0, x1) x [y0, y1), clipped to the screen
};
static_assert(sizeof(UpolyRec) == 64, "UpolyRec layout");

// The frame status and fragment count of a Reyes frame (status bits as the
// raster path's).
struct ReyesFrameCounters {
  uint32_t status;
  uint32_t pad;
  unsigned long long covered;
};

struct ReyesCounters {
  ReyesFrameCounters fc;
  uint32_t level_count[40];
  unsigned long long leaf_meta;   // (leaves << 40) | dice rows (nu + 1 per leaf)
  unsigned long long upolys;      // micropolygons of all leaves
  uint32_t levels_run;
  uint32_t negative_depth;
  uint32_t big_count;             // micropolygons queued for reyes_big
  uint32_t id_count;              // micropolygons with a covered sample
  uint32_t tie_count;
  uint32_t pad[1];
  unsigned long long bar_arrive;  // grid barrier of reyes_split: (arrivals << 40) | children
  unsigned long long bar_release; // (barriers passed << 32) | next level's patch count
};

struct ReyesArgs {
  int W, H, nBx, nBy, nDice;
  int P;
  float vp[16];
  float thr;
  int max_splits, grid;
  const float4* in_patches;
  PatchRec* lvl[2];
  uint32_t lvl_cap;
  PatchRec* stack;                // [CTAs of the split][kSplitStack]
  PatchRec* leaves;
  uint32_t leaf_cap;
  UpolyRec* up;                   // micropolygons with more than kSmallPx candidate pixels
  uint32_t up_cap;
  uint32_t* id_color;             // per micropolygon with a covered sample: colour (alpha: id_colour())
  unsigned long long* id_key;     // and processing-order key + 1
  uint32_t id_cap;
  uint4* ties;                    // (sample, depth code, micropolygon, the one it met)
  uint32_t tie_cap;
  ReyesCounters* ctr;             // zero between frames
  ReyesCounters* host_ctr;        // pinned: the last frame's
  uint32_t* fb;
  float* depth;
  unsigned long long* samp;       // per sample: depth code << 32 | micropolygon of the least fragment so far
  uint32_t* first0;               // per sample: the first micropolygon at a depth of +-0 (kNoId: none)
  // Multi-sample / Phong variant (no reference counterpart).  spp samples per
  // pixel (1: the reference's pixel centre; 4: one jittered sample per pixel
  // quadrant, seeded); phong = 1 lights the micropolygon's interpolated normal.
  // With spp > 1 reyes_pixels averages the samples into the pixel.
  int spp;
  uint32_t seed;
  int phong;
};

// Micropolygons whose shaded rectangle holds more pixels than this are shaded
// by a warp (one lane per pixel) instead of by the thread that owns them.
constexpr int kSmallPx = 16;

// Depth order as an unsigned integer: total over non-NaN floats, with -0 and +0
// equal (the CPU compares depths as floats).
__device__ __forceinline__ uint32_t zorder(float z)
{
  uint32_t b = __float_as_uint(z);
  if (b == 0x80000000u) b = 0u;
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float zorder_inv(uint32_t o)
{
  return __uint_as_float((o & 0x80000000u) ? (o & 0x7fffffffu) : ~o);
}
// The cleared sample state: above the state of every fragment of depth z <= 1
// (the only ones kept), so a sample stays empty exactly when no fragment
// reached it.
constexpr unsigned long long kSampEmpty = ~0ull;
constexpr uint32_t kNoId = 0xffffffffu;

// Sample s of pixel (x, y): the centre for one sample per pixel; otherwise
// quadrant (s & 1, s >> 1) of the pixel at a jitter from an integer hash of
// (seed, x, y, 2s + axis), 24 bits per axis.  The oracle's restatement uses the
// same function, operation for operation.
__device__ __forceinline__ uint32_t sample_hash(uint32_t seed, uint32_t x, uint32_t y, uint32_t k)
{
  uint32_t h = seed * 0x9E3779B1u;
  h ^= x * 0x85EBCA77u;
  h ^= y * 0xC2B2AE3Du;
  h ^= k * 0x27D4EB2Fu;
  h ^= h >> 16; h *= 0x7FEB352Du;
  h ^= h >> 15; h *= 0x846CA68Bu;
  h ^= h >> 16;
  return h;
}
__device__ __forceinline__ void sample_pos(int spp, uint32_t seed, int x, int y, int s, float& px, float& py)
{
  if (spp == 1) { px = (float)x + 0.5f; py = (float)y + 0.5f; return; }
  const float jx = (float)(sample_hash(seed, (uint32_t)x, (uint32_t)y, 2u * (uint32_t)s) >> 8) * 5.9604644775390625e-8f;
  const float jy = (float)(sample_hash(seed, (uint32_t)x, (uint32_t)y, 2u * (uint32_t)s + 1u) >> 8) * 5.9604644775390625e-8f;
  px = (float)x + ((float)(s & 1) + jx) * 0.5f;
  py = (float)y + ((float)(s >> 1) + jy) * 0.5f;
}

__device__ __forceinline__ float4 f4add(float4 a, float4 b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }
__device__ __forceinline__ float4 f4mul(float4 a, float k) { return make_float4(a.x * k, a.y * k, a.z * k, a.w * k); }

// piko::matmultfloat4 with a w component (piko/math.h:395-403)
__device__ __forceinline__ float4 matmul4(const float* m, float4 v)
{
  float4 o;
  o.x = m[0] * v.x + m[4] * v.y + m[8] * v.z + m[12] * v.w;
  o.y = m[1] * v.x + m[5] * v.y + m[9] * v.z + m[13] * v.w;
  o.z = m[2] * v.x + m[6] * v.y + m[10] * v.z + m[14] * v.w;
  o.w = m[3] * v.x + m[7] * v.y + m[11] * v.z + m[15] * v.w;
  return o;
}

__device__ __forceinline__ float dist2(float ax, float ay, float bx, float by)
{
  const float cx = ax - bx, cy = ay - by;
  return sqrtf(cx * cx + cy * cy);
}

__device__ __forceinline__ int pow2roundup(int x)
{
  if (x < 0) return 0;
  --x;
  x |= x >> 1; x |= x >> 2; x |= x >> 4; x |= x >> 8; x |= x >> 16;
  return x + 1;
}

// Grid-wide barrier between split levels that also carries the next level's
// patch count: every CTA arrives with the children it reserved; the last
// arrival sums them and releases barrier k with (k + 1) << 32 | count, so no
// CTA reads the count back afterwards.  It comes in two halves (arrive, wait).
// The wait is bounded: after 1 s without a release (the
// globaltimer; an iteration cap besides) the CTA records kStatusBarrierTimeout
// and goes on (the host reports PIKO_ERR_TIMEOUT).
constexpr unsigned long long kBarrierWaitNs = 1000000000ull;

__device__ __forceinline__ unsigned long long global_ns()
{
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ void barrier_arrive(ReyesCounters* c, uint32_t k, uint32_t* s_children)
{
  __syncthreads();
  if (threadIdx.x == 0) {
    const uint32_t children = *s_children;   // settled: every lane has passed the sync
    *s_children = 0;                         // next level's adds come after barrier_wait
    __threadfence();
    const unsigned long long old = atomicAdd(&c->bar_arrive, (1ull << 40) | children);
    if ((uint32_t)(old >> 40) == gridDim.x - 1) {
      const unsigned long long total = (old & ((1ull << 40) - 1)) + children;
      c->bar_arrive = 0;
      __threadfence();
      atomicExch(&c->bar_release, ((unsigned long long)(k + 1) << 32) | min(total, 0xffffffffull));
    }
  }
}

__device__ __forceinline__ uint32_t barrier_wait(ReyesCounters* c, uint32_t k, uint32_t* s_count)
{
  if (threadIdx.x == 0) {
    volatile unsigned long long* rel = &c->bar_release;
    volatile uint32_t* status = &c->fc.status;
    uint32_t spins = 0;
    unsigned long long v;
    const unsigned long long t0 = global_ns();
    while ((uint32_t)((v = *rel) >> 32) != k + 1) {
      // the time limit and another CTA's timeout are checked every 16 polls
      if ((++spins & 15u) != 0u) continue;
      __nanosleep(32);
      if (*status & kStatusBarrierTimeout) { v = 0; break; }
      if (global_ns() - t0 > kBarrierWaitNs || spins > (1u << 28)) {
        atomicOr(&c->fc.status, kStatusBarrierTimeout);
        v = 0;
        break;
      }
    }
    __threadfence();
    *s_count = (uint32_t)v;
  }
  __syncthreads();
  return *s_count;
}

// The patches of the split's next step, of `count` put on a frontier of `cap`.  A
// frontier that overflowed has slots that no patch was written to: what lies there is
// no patch, and splitting it might never end.  The split ends instead (every CTA has
// the same count), and the host grows the buffers and runs the frame again.
__host__ __device__ __forceinline__ uint32_t next_patches(uint32_t count, uint32_t cap)
{
  return count <= cap ? count : 0u;
}

// The per-sample state starts every frame empty: the buffers are set so when
// allocated, and reyes_pixels, which visits every sample last, sets a reached
// sample back.  The split clears nothing.

// One patch of one split level (R11, split.pikostage:240-343), sixteen lanes
// per patch: lane c holds control point c; the u and v polyline lengths are
// summed over shuffles in the reference's order.  split_measure decides split
// or leaf (and the leaf's dice grid); split_write then writes control point c
// of both children (split along u or v at the halves, de Casteljau) or copies
// it into the leaf.
struct SplitDecision {
  float ue, ve;
  bool split;
  int nu, nv;
};

__device__ __forceinline__ SplitDecision split_measure(const ReyesArgs& a, int L, float4 cp, int c, unsigned hmask)
{
  float4 q = matmul4(a.vp, cp);
  if (q.w == 0.0f) q.w = 1.0f;
  q.x = q.x / q.w;
  q.y = q.y / q.w;
  // (x + 1.0) * 0.5 * W in double, rounded to float, is one fma of floats:
  // the double sequence is exact wherever the value lies near a float
  // rounding boundary, so both round the exact value x * W/2 + W/2 once
  const float hw = 0.5f * (float)a.W, hh = 0.5f * (float)a.H;
  const float cx = __fmaf_rn(q.x, hw, hw);
  const float cy = __fmaf_rn(q.y, hh, hh);
  // distance to the next point along u (same row) and along v (same column)
  const float ux = __shfl_sync(hmask, cx, c + 1, 16), uy = __shfl_sync(hmask, cy, c + 1, 16);
  const float vx = __shfl_sync(hmask, cx, c + 4, 16), vy = __shfl_sync(hmask, cy, c + 4, 16);
  const float du = dist2(cx, cy, ux, uy);
  const float dv = dist2(cx, cy, vx, vy);
  // a row's (column's) length is ((d0 + d1) + d2), on its first lane; the largest
  // of 0 and the four lengths, which a NaN never is
  float su = du + __shfl_sync(hmask, du, c + 1, 16);
  float sv = dv + __shfl_sync(hmask, dv, c + 4, 16);
  su = fmaxf(0.0f, su + __shfl_sync(hmask, du, c + 2, 16));
  sv = fmaxf(0.0f, sv + __shfl_sync(hmask, dv, c + 8, 16));
  su = fmaxf(su, __shfl_xor_sync(hmask, su, 4, 16));
  sv = fmaxf(sv, __shfl_xor_sync(hmask, sv, 1, 16));
  su = fmaxf(su, __shfl_xor_sync(hmask, su, 8, 16));
  sv = fmaxf(sv, __shfl_xor_sync(hmask, sv, 2, 16));
  SplitDecision d;
  d.ue = __shfl_sync(hmask, su, 0, 16);
  d.ve = __shfl_sync(hmask, sv, 0, 16);
  d.split = (d.ue >= a.thr) || (d.ve >= a.thr);
  if (L >= a.max_splits) d.split = false;
  d.nu = d.nv = 0;
  if (!d.split) {
    if (a.grid > 0) {   // a fixed dice grid replaces the extent-derived one
      d.nu = d.nv = a.grid;
    } else {
      // (the reference rounds up in double: a float widened and rounded up is the float rounded up)
      int nu = pow2roundup(cvt_i32_x86(ceilf(d.ue / a.thr)) + 1);
      int nv = pow2roundup(cvt_i32_x86(ceilf(d.ve / a.thr)) + 1);
      d.nu = nu < 2 ? 2 : (nu > 32 ? 32 : nu);
      d.nv = nv < 2 ? 2 : (nv > 32 ? 32 : nv);
    }
  }
  return d;
}

// The split runs as one cooperative launch of kSplitThreads-thread CTAs, one
// per SM, sixteen lanes per patch.  A CTA expands its patches level after level:
// up to kSplitKeep children of a level stay in shared memory, further ones go to
// a stack of the CTA's own in global memory (and, once that holds kSplitStack, to
// the frontier), and leaves are staged and written out in batches.  A step ends
// with a grid barrier, after which the patches on the global frontier are dealt
// out to the CTAs, one each in turn, so that neighbours -- subtrees of similar
// size -- go to different CTAs; the split ends at the first step whose frontier
// is empty.  In the first step a CTA puts all patches of a level that has at
// least kSplitShare of them on the frontier: with few input patches the CTAs'
// subtrees differ in size, and dealt out at that width they even out (a split
// that put every patch past 64 per level on the frontier took 89 us of the
// default-constants sphere's 14 levels, in four steps; this takes 51 us).  The
// levels' passes are chains of latencies: 0.9 us a narrow level, and 37% issue
// active over the default-constants sphere's 50 us, whose last step takes some 700
// patches per CTA.  So a patch takes as few instructions as its arithmetic needs,
// and 64 of them are in flight (that sphere's frame 131.6 -> 127.0 us by the former,
// 124.3 by the latter; 32 in flight are 0.3 us faster where the split ends after a
// few narrow levels).  Nothing
// depends on which CTA or pass handles a patch: every leaf carries its input
// index, level and in-level position (children of s are 2s and 2s + 1), which
// give the order key.
constexpr int kSplitThreads = 1024;
constexpr int kSplitKeep = 128;         // patches a CTA takes per level
constexpr int kSplitStage = 192;
constexpr uint32_t kSplitStack = 1024;  // patches of a CTA's own stack
constexpr uint32_t kSplitShare = 96;
struct SplitSmem {
  PatchRec buf[2][2 * kSplitKeep];    // current level, children of the current level
  PatchRec stage[kSplitStage];        // leaves not yet written out
  uint32_t nnext, nleaf, ncur, maxlevel;
  uint32_t children;                  // patches this CTA put on the frontier in this step
  uint32_t word[4];
};
constexpr size_t kSplitSmem = sizeof(SplitSmem);

// Copies n patch records (18 float4 each) with the whole CTA.
__device__ __forceinline__ void copy_patches(PatchRec* dst, const PatchRec* src, uint32_t n, bool from_l2)
{
  constexpr uint32_t kQ = sizeof(PatchRec) / 16;
  const float4* s4 = reinterpret_cast<const float4*>(src);
  float4* d4 = reinterpret_cast<float4*>(dst);
  for (uint32_t i = threadIdx.x; i < n * kQ; i += blockDim.x) d4[i] = from_l2 ? __ldcg(&s4[i]) : s4[i];
}

// Input patches first, first + stride, ... (n of them) of a step: input patches
// at level 0 (i0 = s = i) or records of the global frontier.
__device__ __forceinline__ void load_inputs(const ReyesArgs& a, int step, uint32_t first, uint32_t stride, uint32_t n,
                                            PatchRec* dst)
{
  if (step == 0) {
    for (uint32_t q = threadIdx.x; q < n * 16u; q += blockDim.x) {
      const uint32_t i = q >> 4, c = q & 15u, in = first + i * stride;
      dst[i].cp[c] = __ldcg(&a.in_patches[(size_t)in * 16 + c]);
      if (c == 0) {
        dst[i].i0 = in;
        dst[i].level = 0;
        dst[i].s = in;
      }
    }
  } else {
    constexpr uint32_t kQ = sizeof(PatchRec) / 16;
    float4* d4 = reinterpret_cast<float4*>(dst);
    for (uint32_t q = threadIdx.x; q < n * kQ; q += blockDim.x) {
      const uint32_t i = q / kQ, c = q - i * kQ;
      d4[q] = __ldcg(reinterpret_cast<const float4*>(a.lvl[step & 1] + (first + i * stride)) + c);
    }
  }
}

// Writes the staged leaves out: one 64-bit atomic reserves their slots and
// dice rows together (so rows stay contiguous in slot order), and their
// micropolygon count is added.  Called by every thread of the CTA.
__device__ __forceinline__ void flush_leaves(const ReyesArgs& a, SplitSmem& S)
{
  __syncthreads();
  const uint32_t nl = S.nleaf;
  if (nl == 0) return;   // uniform
  if (threadIdx.x < 32) {
    const uint32_t lane = threadIdx.x;
    const uint32_t per = (nl + 31u) / 32u;
    const uint32_t b0 = min(lane * per, nl), b1 = min(b0 + per, nl);
    uint32_t rows = 0, ups = 0;
    for (uint32_t i = b0; i < b1; ++i) {
      rows += S.stage[i].nu + 1u;
      ups += (S.stage[i].nu + 1u) * (S.stage[i].nv + 1u);
    }
    uint32_t incl = rows;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(kFullR, incl, o);
      if (lane >= (uint32_t)o) incl += t;
    }
    const uint32_t total = __shfl_sync(kFullR, incl, 31);
    const uint32_t up_total = __reduce_add_sync(kFullR, ups);
    unsigned long long old = 0;
    if (lane == 0) {
      old = atomicAdd(&a.ctr->leaf_meta, ((unsigned long long)nl << 40) | total);
      atomicAdd(&a.ctr->upolys, (unsigned long long)up_total);
    }
    old = __shfl_sync(kFullR, old, 0);
    uint32_t r = (uint32_t)(old & ((1ull << 40) - 1)) + incl - rows;
    for (uint32_t i = b0; i < b1; ++i) {
      S.stage[i].rowbase = r;
      r += S.stage[i].nu + 1u;
    }
    if (lane == 0) S.word[3] = (uint32_t)(old >> 40);
  }
  __syncthreads();
  const uint32_t base = S.word[3];
  if (base + nl <= a.leaf_cap) {
    copy_patches(a.leaves + base, S.stage, nl, false);
  } else if (threadIdx.x == 0) {
    atomicOr(&a.ctr->fc.status, kStatusPatchOverflow);   // the host grows the buffer and runs again
  }
  __syncthreads();
  if (threadIdx.x == 0) S.nleaf = 0;
}

// One level of the CTA's current patches (at most kSplitKeep; 16-lane group
// q takes patches q, q + 64): split ones put their children in nxt, leaves
// go to the stage.
__device__ __forceinline__ void split_one(const ReyesArgs& a, SplitSmem& S, const PatchRec* cur, PatchRec* nxt,
                                          uint32_t p)
{
  const int c = threadIdx.x & 15;
  const unsigned hmask = 0xffffu << (threadIdx.x & 16);
  const float4 cp = cur[p].cp[c];
  const uint32_t i0 = cur[p].i0, L = cur[p].level;
  const unsigned long long s = cur[p].s;
  const SplitDecision d = split_measure(a, (int)L, cp, c, hmask);
  uint32_t slot = 0;
  if (c == 0) slot = d.split ? atomicAdd(&S.nnext, 2u) : atomicAdd(&S.nleaf, 1u);
  slot = __shfl_sync(hmask, slot, 0, 16);
  if (d.split) {
    const bool along_u = d.ue >= a.thr;
    // The lane's row (split along u) or column (along v), halved at t = 1/2 by de
    // Casteljau (splitU / splitV, split.pikostage:95-224): with points p0 .. p3 the
    // halves are p0, a1, a2, a3 and a3, b1, b2, p3.  Lane j writes point j of both;
    // lanes 2 and 3 take the points in reverse order (the sums commute), which
    // makes their points lane 1's and 0's with the halves exchanged.
    const int j = along_u ? (c & 3) : (c >> 2), st = along_u ? 1 : 4, at = c - j * st;
    const bool rev = j >= 2;
    const float4* q = cur[p].cp + (rev ? at + 3 * st : at);
    const int qs = rev ? -st : st;
    const float4 p0 = q[0], p1 = q[qs], p2 = q[2 * qs], p3 = q[3 * qs];
    const float4 a1 = f4mul(f4add(p0, p1), 0.5f), t = f4mul(f4add(p1, p2), 0.5f), b2 = f4mul(f4add(p2, p3), 0.5f);
    const float4 a2 = f4mul(f4add(a1, t), 0.5f), b1 = f4mul(f4add(b2, t), 0.5f);
    const bool end = j == 0 || j == 3;
    nxt[slot + (rev ? 1 : 0)].cp[c] = end ? p0 : a1;
    nxt[slot + (rev ? 0 : 1)].cp[c] = end ? f4mul(f4add(a2, b1), 0.5f) : b1;
    if (c < 2) {
      PatchRec& o = nxt[slot + c];
      o.i0 = i0;
      o.level = L + 1;
      o.s = 2 * s + (unsigned long long)c;
    }
    if (c == 0) atomicMax(&S.maxlevel, L + 1);
  } else {
    PatchRec& o = S.stage[slot];
    o.cp[c] = cp;
    if (c == 0) {
      o.i0 = i0;
      o.level = L;
      o.s = s;
      o.nu = (uint32_t)d.nu;
      o.nv = (uint32_t)d.nv;
    }
  }
}

__device__ __forceinline__ void split_pass(const ReyesArgs& a, SplitSmem& S, const PatchRec* cur, PatchRec* nxt,
                                           uint32_t ncur)
{
  for (uint32_t p = threadIdx.x >> 4; p < ncur; p += kSplitThreads / 16)   // whole 16-lane groups
    split_one(a, S, cur, nxt, p);
}

// The first levels of the step's patch `owner` (share 1; 0: none), by one warp:
// down the CTA's path of dr bits, then level by level until one has more than
// kNarrow patches.  Leaves S.ncur patches in S.buf[S.word[0]].
constexpr uint32_t kNarrow = 4;
__device__ __forceinline__ void narrow_levels(const ReyesArgs& a, SplitSmem& S, int step, uint32_t owner,
                                              uint32_t share, uint32_t path, uint32_t dr)
{
  const uint32_t lane = threadIdx.x;
  uint32_t ncur = share, cb = 0;
  if (share) {
    if (step == 0) {
      if (lane < 16) S.buf[0][0].cp[lane] = __ldcg(&a.in_patches[(size_t)owner * 16 + lane]);
      if (lane == 0) {
        S.buf[0][0].i0 = owner;
        S.buf[0][0].level = 0;
        S.buf[0][0].s = owner;
      }
    } else if (lane < sizeof(PatchRec) / 16) {
      reinterpret_cast<float4*>(&S.buf[0][0])[lane] = __ldcg(reinterpret_cast<const float4*>(a.lvl[step & 1] + owner) + lane);
    }
  }
  while (ncur > 0 && ncur <= kNarrow) {
    // (a level adds at most kNarrow leaves; the stage has room for far more levels)
    if (lane == 0) S.nnext = 0;
    __syncwarp();
    for (uint32_t p = lane >> 4; p < ncur; p += 2) split_one(a, S, S.buf[cb], S.buf[cb ^ 1], p);
    __syncwarp();
    uint32_t nn = S.nnext;
    if (dr > 0) {
      // one patch on the CTA's path: keep the child the path names, or drop a
      // leaf that another CTA of the group emits
      if (nn == 0) {
        if ((path & ((1u << dr) - 1u)) != 0u && lane == 0) S.nleaf -= 1;
      } else {
        if ((path >> (dr - 1)) & 1u) {
          float4* dst = reinterpret_cast<float4*>(&S.buf[cb ^ 1][0]);
          const float4* src = reinterpret_cast<const float4*>(&S.buf[cb ^ 1][1]);
          if (lane < sizeof(PatchRec) / 16) dst[lane] = src[lane];
        }
        nn = 1;
      }
      --dr;
    }
    ncur = nn;
    cb ^= 1;
    __syncwarp();
  }
  if (lane == 0) {
    S.ncur = ncur;
    S.word[0] = cb;
  }
}

__global__ void __launch_bounds__(kSplitThreads, 1) reyes_split(ReyesArgs a)
{
  pdl_trigger();
  extern __shared__ __align__(16) unsigned char split_smem[];
  SplitSmem& S = *reinterpret_cast<SplitSmem*>(split_smem);
  if (threadIdx.x == 0) {
    S.nleaf = 0;
    S.maxlevel = 0;
    S.children = 0;
  }
  uint32_t n_in = (uint32_t)a.P;
  for (int step = 0; n_in > 0; ++step) {   // n_in is uniform
    // This CTA's share of the step's frontier: patches blockIdx.x, blockIdx.x +
    // gridDim.x, ...  With fewer patches than CTAs, 2^d CTAs share a patch:
    // each takes the patch's descendants along its own d-bit path (the first d
    // levels of the patch are computed by all of them), so every CTA has a
    // subtree; a leaf met on the way is emitted by the group's CTA whose
    // remaining path bits are all 0.
    uint32_t d = 0;
    while (d < 16 && ((unsigned long long)n_in << (d + 1)) <= gridDim.x) ++d;
    const uint32_t path = blockIdx.x & ((1u << d) - 1u), owner = blockIdx.x >> d;
    const uint32_t share = d > 0 ? (owner < n_in ? 1u : 0u)
                                 : (blockIdx.x < n_in ? (n_in - blockIdx.x - 1) / gridDim.x + 1 : 0u);
    const bool deal = step == 0 && n_in < 8u * gridDim.x;   // too few patches to even out
    PatchRec* frontier = a.lvl[(step + 1) & 1];
    PatchRec* stack = a.stack + (size_t)blockIdx.x * kSplitStack;
    uint32_t taken = 0, ncur = 0, top = 0;
    int cb = 0;   // buf[cb] holds the current patches
    if (d > 0) {
      // One patch: its path and the first levels below it hold a few patches
      // each, which the first warp expands by itself (a pass of the CTA with its
      // barriers takes 1.2 us, one of a warp half of that)
      if (threadIdx.x < 32) narrow_levels(a, S, step, owner, share, path, d);
      __syncthreads();
      taken = share;
      ncur = S.ncur;
      cb = (int)S.word[0];
    }
    __syncthreads();
    while (ncur > 0 || top > 0 || taken < share) {   // uniform
      // top up the current patches from the stack, then from the share
      if (const uint32_t pop = min((uint32_t)kSplitKeep - ncur, top)) {
        top -= pop;
        copy_patches(&S.buf[cb][ncur], stack + top, pop, true);
        ncur += pop;
      }
      if (const uint32_t take = min((uint32_t)kSplitKeep - ncur, share - taken)) {
        load_inputs(a, step, blockIdx.x + taken * gridDim.x, gridDim.x, take, &S.buf[cb][ncur]);
        taken += take;
        ncur += take;
      }
      if (S.nleaf + (uint32_t)kSplitKeep > (uint32_t)kSplitStage) flush_leaves(a, S);
      if (threadIdx.x == 0) S.nnext = 0;
      __syncthreads();
      split_pass(a, S, S.buf[cb], S.buf[cb ^ 1], ncur);
      __syncthreads();
      uint32_t nn = S.nnext, keep = min(nn, (uint32_t)kSplitKeep);
      {
        if (deal && nn >= kSplitShare) keep = 0;   // the whole level to the frontier
        uint32_t own = nn - keep;                  // children for the CTA's stack
        if (deal && nn >= kSplitShare) own = 0;
        own = min(own, kSplitStack - top);
        if (own) {
          copy_patches(stack + top, &S.buf[cb ^ 1][keep], own, false);
          top += own;
        }
        if (const uint32_t extra = nn - keep - own) {
          if (threadIdx.x == 0) {
            S.word[3] = atomicAdd(&a.ctr->level_count[min(step + 1, 39)], extra);
            S.children += extra;
          }
          __syncthreads();
          const uint32_t at = S.word[3];
          if (at + extra <= a.lvl_cap) {
            copy_patches(frontier + at, &S.buf[cb ^ 1][keep + own], extra, false);
          } else if (threadIdx.x == 0) {
            atomicOr(&a.ctr->fc.status, kStatusPatchOverflow);
          }
        }
      }
      ncur = keep;
      cb ^= 1;
      __syncthreads();
    }
    // grid barrier: the frontier written by every CTA is read after it.  The
    // staged leaves go out between arriving and waiting: only later launches
    // read them, so the arrival need not wait for their stores.
    barrier_arrive(a.ctr, (uint32_t)step, &S.children);
    flush_leaves(a, S);
    n_in = next_patches(barrier_wait(a.ctr, (uint32_t)step, &S.word[1]), a.lvl_cap);
  }
  if (threadIdx.x == 0 && a.P > 0) atomicMax(&a.ctr->levels_run, S.maxlevel + 1u);
}

// ------------------------------------------------------------------ dice
__device__ __forceinline__ float B0(float u) { return ((1.0f - u) * (1.0f - u) * (1.0f - u)); }
__device__ __forceinline__ float B1(float u) { return ((3.0f * u) * (1.0f - u) * (1.0f - u)); }
__device__ __forceinline__ float B2(float u) { return ((3.0f * u) * (u - u * u)); }
__device__ __forceinline__ float B3(float u) { return ((u) * (u * u)); }
__device__ __forceinline__ float dB0(float u) { return (-3.0f * (1.0f - u) * (1.0f - u)); }
__device__ __forceinline__ float dB1(float u) { return (3.0f * (1.0f - u) * (1.0f - 3.0f * u)); }
__device__ __forceinline__ float dB2(float u) { return (3.0f * u * (2.0f - 3.0f * u)); }
__device__ __forceinline__ float dB3(float u) { return (3.0f * u * u); }

__device__ __forceinline__ float4 bez(float t, float4 a, float4 b, float4 c, float4 d)
{
  float4 o;
  o.x = B0(t) * a.x + B1(t) * b.x + B2(t) * c.x + B3(t) * d.x;
  o.y = B0(t) * a.y + B1(t) * b.y + B2(t) * c.y + B3(t) * d.y;
  o.z = B0(t) * a.z + B1(t) * b.z + B2(t) * c.z + B3(t) * d.z;
  o.w = B0(t) * a.w + B1(t) * b.w + B2(t) * c.w + B3(t) * d.w;
  return o;
}
__device__ __forceinline__ float4 dbez(float t, float4 a, float4 b, float4 c, float4 d)
{
  float4 o;
  o.x = dB0(t) * a.x + dB1(t) * b.x + dB2(t) * c.x + dB3(t) * d.x;
  o.y = dB0(t) * a.y + dB1(t) * b.y + dB2(t) * c.y + dB3(t) * d.y;
  o.z = dB0(t) * a.z + dB1(t) * b.z + dB2(t) * c.z + dB3(t) * d.z;
  o.w = dB0(t) * a.w + dB1(t) * b.w + dB2(t) * c.w + dB3(t) * d.w;
  return o;
}

// patchEval + normEval + projection of one corner (dice.pikostage:111-146,205-220),
// in two parts: dice_row evaluates the four control rows and their u
// derivatives at u, which every corner at that u shares; dice_corner finishes
// one corner at v.  Splitting changes no operation or its order.
struct DiceRow {
  float4 r[4], d[4];
};

__device__ __forceinline__ void dice_row(const float4* P, float u, DiceRow& R)
{
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    R.r[k] = bez(u, P[4 * k], P[4 * k + 1], P[4 * k + 2], P[4 * k + 3]);
    R.d[k] = dbez(u, P[4 * k], P[4 * k + 1], P[4 * k + 2], P[4 * k + 3]);
  }
}

__device__ __forceinline__ void dice_corner(const DiceRow& R, const ReyesArgs& a, float v, float& sx, float& sy,
                                            float& sz, float& nx, float& ny, float& nz)
{
  const float4 pt = bez(v, R.r[0], R.r[1], R.r[2], R.r[3]);
  const float4 v1 = bez(v, R.d[0], R.d[1], R.d[2], R.d[3]);
  const float4 v2 = dbez(v, R.r[0], R.r[1], R.r[2], R.r[3]);
  float cx = v1.y * v2.z - v1.z * v2.y;
  float cy = v1.z * v2.x - v1.x * v2.z;
  float cz = v1.x * v2.y - v1.y * v2.x;
  const float mag = sqrtf(cx * cx + cy * cy + cz * cz);
  nx = cx / mag; ny = cy / mag; nz = cz / mag;
  const float4 ss = matmul4(a.vp, pt);
  const float onebyw = 1.0f / ss.w;
  sx = (ss.x * onebyw + 1.0f) * (float)a.W * 0.5f;
  sy = (ss.y * onebyw + 1.0f) * (float)a.H * 0.5f;
  sz = (ss.z * onebyw);
}

// phongShadeReyes + computeLighting as called (shade.pikostage:22-30,64-85):
// negated normal; the dot product takes matcol, the scale takes lightvec
__device__ __forceinline__ float phong_channel(float nx, float ny, float nz, int ch)
{
  nx = -nx; ny = -ny; nz = -nz;
  float d = nx * 0.10f + ny * 0.35f + nz * 0.85f;
  d = d < 0.0f ? 0.0f : d;
  const float lv = ch == 0 ? 0.1773f : (ch == 1 ? 0.5773f : 0.973f);
  const float o = 0.2f + d * lv;
  return o > 1.0f ? 1.0f : (o < 0.0f ? 0.0f : o);
}


// ------------------------------------------------------------------ shade
// ShadeStage's per-pixel test (shade.pikostage:161-235): the sample is inside
// the micropolygon when all four edge functions are positive for either
// winding.  Every product and difference is rounded separately, as on the CPU.
// The reversed winding's edges are written with the forward deltas negated:
// b - a == -(a - b), x * -y == -(x * y) and -p - -q == -(p - q) hold exactly
// in round-to-nearest, so "reversed edge > 0" is "the same products with the
// forward delta, difference < 0", bit for bit.
__device__ __forceinline__ bool upoly_covers(float4 X4, float4 Y4, float px, float py)
{
  const float X[4] = {X4.x, X4.y, X4.z, X4.w}, Y[4] = {Y4.x, Y4.y, Y4.z, Y4.w};
  float dX[4], dY[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    dX[i] = X[(i + 1) & 3] - X[i];
    dY[i] = Y[(i + 1) & 3] - Y[i];
  }
  bool r1 = true, r2 = true;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float ay = py - Y[i], bx = px - X[i];
    if (!(ay * dX[i] - bx * dY[i] > 0.0f)) r1 = false;                   // edge i -> i+1
    if (!(ay * dX[(i + 3) & 3] - bx * dY[(i + 3) & 3] < 0.0f)) r2 = false; // edge i -> i-1
  }
  return r1 || r2;
}

// The first winding alone.  With the corners in reverse order (1 and 3 swapped)
// it is the second one, bit for bit.
__device__ __forceinline__ bool upoly_covers_one(float4 X4, float4 Y4, float px, float py)
{
  const float X[4] = {X4.x, X4.y, X4.z, X4.w}, Y[4] = {Y4.x, Y4.y, Y4.z, Y4.w};
  bool in = true;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float dX = X[(i + 1) & 3] - X[i], dY = Y[(i + 1) & 3] - Y[i];
    if (!((py - Y[i]) * dX - (px - X[i]) * dY > 0.0f)) in = false;
  }
  return in;
}

// Which samples can pass upoly_covers at all.  When every corner coordinate is
// at least 32 and the corners span less than 16 px per axis, each difference
// the test takes (sample minus corner, corner minus corner) is exact
// (Sterbenz), so a positive rounded edge value means a positive exact one;
// a sample inside all four edges of either winding has a non-zero winding
// number and lies strictly inside the corners' bounding box.  There the
// coverage pass tests only the cells (pixel quadrants, or pixel centres with
// one sample) whose sample range meets the open box; elsewhere it tests all.
// There, too, at most one winding can pass, known from the area: a product's
// rounding is monotone, so where all four rounded edge values are positive the
// exact ones are none of them negative, and the exact ones add up to twice the
// area wherever the sample is; the second winding needs them none positive.  The
// area's own sign is the comparison of two rounded products of exact differences
// (the diagonals), which orders the exact products unless they round equal.
__device__ __forceinline__ bool exact_box(float mnx, float mxx, float mny, float mxy)
{
  return mnx >= 32.0f && mny >= 32.0f && mxx - mnx < 16.0f && mxy - mny < 16.0f && mxx < 4194304.0f &&
         mxy < 4194304.0f;
}

// The depth resolve.  The CPU shades micropolygons in its processing order with
//   while (remote > z) remote = atomicMin(bits, z);  pass iff zbuf == z
// so, per sample, the surviving depth is the minimum m (the cleared 1.0
// included), its bits come from the FIRST fragment with depth m and the colour
// from the LAST one.  A micropolygon with a covered sample of depth z <= 1 gets
// a number (id), under which its colour and order key are kept, and each such
// sample is one atomicMin of zorder(z) << 32 | id on the sample's state: the
// least depth wins.  Two fragments of one depth at a sample see each other --
// the later atomic finds the earlier one's depth -- and leave a tie record;
// reyes_ties then gives the sample to the micropolygon with the greatest key of
// all that met there.  Only at depth +-0 can fragments of one depth differ in
// their bits: there every fragment leaves a record, and the one with the least
// key is kept in first0.
// (A list of all fragments, 32 bytes each, read again by a pass that took the
// greatest key at each sample's minimum and by one that wrote colour and depth,
// cost 35 us of the 4-sample 1280x720 sphere's 157.)

// A micropolygon's colour with the sign of a zero depth in the alpha's low bit
// (set for everything but -0; a colour's alpha is 255).
__device__ __forceinline__ uint32_t id_colour(const UpolyRec& u)
{
  return u.color ^ (__float_as_uint(u.z) == 0x80000000u ? 0x01000000u : 0u);
}

__device__ __forceinline__ void add_covered(const ReyesArgs& a, unsigned covered)
{
  covered = __reduce_add_sync(kFullR, covered);
  if ((threadIdx.x & 31) == 0 && covered) atomicAdd(&a.ctr->fc.covered, (unsigned long long)covered);
}

__device__ __forceinline__ void put_id(const ReyesArgs& a, uint32_t id, const UpolyRec& u)
{
  if (id < a.id_cap) {
    a.id_color[id] = id_colour(u);
    a.id_key[id] = u.key;
  } else {
    atomicOr(&a.ctr->fc.status, kStatusListOverflow);   // the host grows the tables and runs again
  }
}

__device__ __forceinline__ uint32_t sample_index(const ReyesArgs& a, int x, int y, int smp)
{
  return ((uint32_t)y * (uint32_t)a.W + (uint32_t)x) * (uint32_t)a.spp + (uint32_t)smp;
}

// Tie records of a CTA not yet in the list (a global append each, a tenth to a
// quarter of the fragments, took 16 us of the default-constants sphere's dice).
constexpr uint32_t kTieStage = 192;
struct TieStage {
  uint4 rec[kTieStage];
  uint32_t n, base;
};

__device__ __forceinline__ void put_tie(const ReyesArgs& a, uint32_t slot, uint4 t)
{
  if (slot < a.tie_cap) a.ties[slot] = t;
  else atomicOr(&a.ctr->fc.status, kStatusListOverflow);
}

// The fragment (zo, id) found `old` at sample p: leaves a record where the two
// share their depth, and at +-0 always.
__device__ __forceinline__ void check_tie(const ReyesArgs& a, TieStage* stage, uint32_t p, uint32_t zo, uint32_t id,
                                          unsigned long long old)
{
  const bool met = (uint32_t)(old >> 32) == zo;
  if (!met && zo != 0x80000000u) return;   // zorder(+-0)
  const uint4 t = make_uint4(p, zo, id, met ? (uint32_t)old : id);
  const uint32_t at = stage ? atomicAdd(&stage->n, 1u) : kTieStage;
  if (at < kTieStage) stage->rec[at] = t;
  else put_tie(a, atomicAdd(&a.ctr->tie_count, 1u), t);
}

// Writes the staged records out once there are more than `keep`; every thread
// of the CTA calls it, after a barrier behind the last check_tie.
__device__ __forceinline__ void flush_ties(const ReyesArgs& a, TieStage& stage, uint32_t keep)
{
  const uint32_t n = min(stage.n, kTieStage);
  if (n <= keep) return;   // uniform
  if (threadIdx.x == 0) stage.base = atomicAdd(&a.ctr->tie_count, n);
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) put_tie(a, stage.base + i, stage.rec[i]);
  __syncthreads();
  if (threadIdx.x == 0) stage.n = 0;
}

// Block-wide exclusive scan of n (all 256 threads call it) and one atomic on
// the id counter; returns this thread's first id.
__device__ __forceinline__ uint32_t block_append(const ReyesArgs& a, uint32_t n, uint32_t* s_warp, uint32_t* s_base)
{
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t inc = n;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(kFullR, inc, o);
    if (lane >= o) inc += t;
  }
  if (lane == 31) s_warp[warp] = inc;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t tot = 0;
    for (int w = 0; w < 8; ++w) { const uint32_t v = s_warp[w]; s_warp[w] = tot; tot += v; }
    *s_base = tot ? atomicAdd(&a.ctr->id_count, tot) : 0u;
  }
  __syncthreads();
  const uint32_t r = *s_base + s_warp[warp] + inc - n;
  __syncthreads();
  return r;
}

// ------------------------------------------------------------------ dice
// A dice grid point: screen position and depth, and the per-channel "Phong"
// term of its normal (the reference's corner lighting) or, in the Phong
// variant, the normal itself.
struct GridPt {
  float sx, sy, sz, ph[3];
};

__device__ __forceinline__ void grid_point_row(const DiceRow& R, const ReyesArgs& a, float v, GridPt& g)
{
  float nx, ny, nz;
  dice_corner(R, a, v, g.sx, g.sy, g.sz, nx, ny, nz);
  if (a.phong) {
    g.ph[0] = nx; g.ph[1] = ny; g.ph[2] = nz;
  } else {
#pragma unroll
    for (int ch = 0; ch < 3; ++ch) g.ph[ch] = phong_channel(nx, ny, nz, ch);
  }
}

__device__ __forceinline__ void grid_point(const float4* P, const ReyesArgs& a, float u, float v, GridPt& g)
{
  DiceRow R;
  dice_row(P, u, R);
  grid_point_row(R, a, v, g);
}

// The order key's leaf part: Dice bin of the leaf's id (dice.pikostage:18-43,
// ids (i0 + L(L+1)/2) / 128 mod the bin count), split level, position in the level.
__device__ __forceinline__ unsigned long long leaf_key(const ReyesArgs& a, uint32_t i0, uint32_t L,
                                                       unsigned long long s)
{
  const uint32_t id = i0 + L * (L + 1) / 2;
  const unsigned long long d = (unsigned long long)((id / 128u) % (uint32_t)a.nDice);
  return (d << 52) | ((unsigned long long)L << 47) | (s << 12);
}

// Micropolygon `local` of a leaf from its corners (k, j), (k+1, j), (k+1, j+1),
// (k, j+1): mean depth, averaged colour, order key (leaf part keyhi), and the
// pixel rectangle of its Shade bins (dice.pikostage:18-43,159-312;
// shade.pikostage:51-56,129-140).
__device__ __forceinline__ void make_upoly(const ReyesArgs& a, unsigned long long keyhi, uint32_t local,
                                           const GridPt& c0, const GridPt& c1, const GridPt& c2, const GridPt& c3,
                                           UpolyRec& o)
{
  o.sx[0] = c0.sx; o.sx[1] = c1.sx; o.sx[2] = c2.sx; o.sx[3] = c3.sx;
  o.sy[0] = c0.sy; o.sy[1] = c1.sy; o.sy[2] = c2.sy; o.sy[3] = c3.sy;
  o.z = ((c0.sz + c1.sz + c2.sz + c3.sz)) * 0.25f;
  float col[3];
  if (a.phong) {
    // Phong variant: the corner normals summed in corner order, renormalised,
    // and lit once (the reference lights the corners and averages)
    float nx = c0.ph[0] + c1.ph[0], ny = c0.ph[1] + c1.ph[1], nz = c0.ph[2] + c1.ph[2];
    nx = nx + c2.ph[0]; ny = ny + c2.ph[1]; nz = nz + c2.ph[2];
    nx = nx + c3.ph[0]; ny = ny + c3.ph[1]; nz = nz + c3.ph[2];
    const float mag = sqrtf(nx * nx + ny * ny + nz * nz);
    nx = nx / mag; ny = ny / mag; nz = nz / mag;
#pragma unroll
    for (int ch = 0; ch < 3; ++ch) col[ch] = phong_channel(nx, ny, nz, ch);
  } else {
#pragma unroll
    for (int ch = 0; ch < 3; ++ch) {
      float c = c0.ph[ch] + c1.ph[ch];
      c = c + c2.ph[ch];
      c = c + c3.ph[ch];
      col[ch] = std_minf(c, 4.0f) * 0.25f;
    }
  }
  o.color = (255u << 24) | (cvt_u32_x86(col[2] * 255.0f) << 16) | (cvt_u32_x86(col[1] * 255.0f) << 8) |
            cvt_u32_x86(col[0] * 255.0f);
  o.key = (keyhi | (unsigned long long)local) + 1ull;
  // Shade bins of corners 0..2 (computeBoundingBox + assignToBB)
  // (the reference takes these in double; widening a float is exact and the
  // comparisons are the same, so float std::min / std::max give the same values)
  const float lox = floorf(std_minf(o.sx[0], std_minf(o.sx[1], o.sx[2])));
  const float loy = floorf(std_minf(o.sy[0], std_minf(o.sy[1], o.sy[2])));
  const float hix = ceilf(std_maxf(o.sx[0], std_maxf(o.sx[1], o.sx[2])));
  const float hiy = ceilf(std_maxf(o.sy[0], std_maxf(o.sy[1], o.sy[2])));
  int bx1 = cvt_i32_x86(floorf(lox / 64.0f)), bx2 = cvt_i32_x86(floorf(hix / 64.0f));
  int by1 = cvt_i32_x86(floorf(loy / 64.0f)), by2 = cvt_i32_x86(floorf(hiy / 64.0f));
  if (bx1 < 0) bx1 = 0;
  if (by1 < 0) by1 = 0;
  if (bx2 >= a.nBx) bx2 = a.nBx - 1;
  if (by2 >= a.nBy) by2 = a.nBy - 1;
  // 4-corner bounds intersected with each Shade bin; the bins are adjacent,
  // so the union is one rectangle
  const float bminx = floorf(std_minf(std_minf(o.sx[0], o.sx[1]), std_minf(o.sx[2], o.sx[3])));
  const float bminy = floorf(std_minf(std_minf(o.sy[0], o.sy[1]), std_minf(o.sy[2], o.sy[3])));
  const float bmaxx = ceilf(std_maxf(std_maxf(o.sx[0], o.sx[1]), std_maxf(o.sx[2], o.sx[3])));
  const float bmaxy = ceilf(std_maxf(std_maxf(o.sy[0], o.sy[1]), std_maxf(o.sy[2], o.sy[3])));
  o.x0 = o.x1 = o.y0 = o.y1 = 0;
  if (bx1 <= bx2 && by1 <= by2) {
    const float fx0 = (float)(bx1 * 64), fx1 = (float)((bx2 + 1) * 64);
    const float fy0 = (float)(by1 * 64), fy1 = (float)((by2 + 1) * 64);
    int px0 = cvt_i32_x86((bminx > fx0) ? bminx : fx0);
    int px1 = cvt_i32_x86((bmaxx < fx1) ? bmaxx : fx1);
    int py0 = cvt_i32_x86((bminy > fy0) ? bminy : fy0);
    int py1 = cvt_i32_x86((bmaxy < fy1) ? bmaxy : fy1);
    px0 = max(px0, bx1 * 64); py0 = max(py0, by1 * 64);
    px1 = min(min(px1, (bx2 + 1) * 64), a.W);
    py1 = min(min(py1, (by2 + 1) * 64), a.H);
    if (px0 < px1 && py0 < py1) { o.x0 = px0; o.x1 = px1; o.y0 = py0; o.y1 = py1; }
  }
}

// Dice (R12, R13), then the fragments of micropolygons with at most kSmallPx
// candidate pixels (larger ones are queued for a warp each).
//
// The dice rows of all leaves (row k of a leaf: its micropolygons (k, 0..nv))
// are numbered in leaf-slot order and every CTA takes an equal range of them.
// It works through its range in groups of consecutive rows, possibly spanning
// leaves, of at most kUpBudget micropolygons whose grid points fit in shared
// memory.  For power-of-two grids (every extent-derived grid) k*du + du equals
// (k+1)*du exactly, so the grid points of a group's rows are evaluated once and
// shared by the four micropolygons around each (and the control rows at each
// u once per point row); other fixed grids evaluate the four corners of every
// micropolygon, as the CPU does.  Points and micropolygons of a group are
// spread over all threads whatever the leaves' sizes.
//
// Coverage is sample-parallel: each thread's micropolygon contributes a
// rectangle of cells (one per sample: a pixel quadrant with four samples, the
// pixel with one), cut to the cells exact_box allows; the CTA's cells go to a
// shared list and every thread tests one cell at a time, so lanes stay busy
// whatever the micropolygons' sizes.
// (shared memory for four CTAs per SM: three 18 x 18 grids of points, 30 rows of the widest)
constexpr int kMaxGridPts = 30 * 34;
constexpr int kLeafBatch = 32;     // leaf segments per group
constexpr int kDiceThreads = 256;
constexpr int kUpBudget = 1024;    // micropolygons per group
constexpr int kMaxPtRows = 128;    // grid point rows per group
constexpr int kCellCap = 2048;     // cells per pass of the shared list

constexpr uint32_t kNoDepth = 0xffffffffu;
constexpr uint32_t kBothWindings = 1u << 31;   // (else the corners' order makes the first winding the one to test)

struct DiceSmem {
  float4 cp[kLeafBatch][16];
  GridPt gp[kMaxGridPts];
  union {
    DiceRow rowdat[kMaxPtRows];                  // control rows at each point row's u (until the grid points stand)
    struct {
      float4 ux[kDiceThreads], uy[kDiceThreads];   // corners of each thread's micropolygon
      int2 org[kDiceThreads];                      // first cell of its cell rectangle
      uint32_t cwm[kDiceThreads];                  // rectangle width | (2^16 / width + 1) << 7 | kBothWindings
      unsigned long long mask[kDiceThreads];       // covered cells (!SPARSE)
      uint32_t zo[kDiceThreads];                   // depth code, kNoDepth: behind the cleared depth (SPARSE)
      uint16_t cell[kCellCap];                     // (thread << 6) | cell index
    };
  };
  // the group's segments: rows k0 .. of leaf[i]; gpre / upre / rpre = first
  // grid point / micropolygon / point row of each segment in the group
  uint32_t leaf[kLeafBatch], k0[kLeafBatch], nu[kLeafBatch], nv[kLeafBatch];
  unsigned long long keyhi[kLeafBatch];
  uint32_t gpre[kLeafBatch + 1], upre[kLeafBatch + 1], rpre[kLeafBatch + 1];
  uint32_t scan[8], append[8];
  uint32_t total, base;
  uint32_t nseg, next_leaf, next_row, found;
  uint32_t gid;         // the group's first id
  TieStage ties;
};
constexpr size_t kDiceSmem = sizeof(DiceSmem);

// q = n / d and r = n % d for the dice grid's row widths (d = nv + 1 or
// nv + 2 <= 34): a multiply by 0xffffffff / d and one correction
// (fast_divmod); wider rows divide.
struct DivMagic {
  uint32_t m[35];
  constexpr DivMagic() : m() { for (uint32_t d = 1; d < 35; ++d) m[d] = 0xffffffffu / d; }
};
__constant__ DivMagic kRowMagic = DivMagic();
__device__ __forceinline__ uint32_t row_divmod(uint32_t n, uint32_t d, uint32_t& r)
{
  if (d < 35u) return fast_divmod(n, d, kRowMagic.m[d], r);
  r = n % d;
  return n / d;
}

__device__ __forceinline__ int batch_find(const uint32_t* pre, int n, uint32_t f)
{
  int lo = 0, hi = n - 1;   // last i with pre[i] <= f
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (pre[mid] <= f) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// Exclusive block-wide scan of n; *total gets the sum (all threads call it).
__device__ __forceinline__ uint32_t block_scan(uint32_t n, uint32_t* s_warp, uint32_t* total)
{
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t inc = n;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(kFullR, inc, o);
    if (lane >= o) inc += t;
  }
  if (lane == 31) s_warp[warp] = inc;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t tot = 0;
    for (int w = 0; w < kDiceThreads / 32; ++w) { const uint32_t v = s_warp[w]; s_warp[w] = tot; tot += v; }
    *total = tot;
  }
  __syncthreads();
  return s_warp[warp] + inc - n;
}

// Cell index li of a rectangle cw cells wide: dy = li / cw by multiply-shift
// (exact for li < 64, cw <= 64).
__device__ __forceinline__ void cell_xy(uint32_t cwm, int2 org, int li, int& cx, int& cy)
{
  const int cw = (int)(cwm & 127u);
  const int dy = (int)(((uint32_t)li * ((cwm >> 7) & 0x1ffffu)) >> 16);
  cx = org.x + li - dy * cw;
  cy = org.y + dy;
}

// Tests cell q of the shared list: u = the thread whose micropolygon it is, li =
// its index in the rectangle, (x, y, smp) its sample.
__device__ __forceinline__ bool dice_cell(const ReyesArgs& a, const DiceSmem& S, uint32_t q, int& u, int& li, int& x,
                                          int& y, int& smp)
{
  const uint32_t e = S.cell[q];
  u = (int)(e >> 6);
  li = (int)(e & 63u);
  const uint32_t cwm = S.cwm[u];
  cell_xy(cwm, S.org[u], li, x, y);
  smp = 0;
  if (a.spp != 1) {
    smp = (x & 1) | ((y & 1) << 1);
    x >>= 1;
    y >>= 1;
  }
  float px, py;
  sample_pos(a.spp, a.seed, x, y, smp, px, py);
  return (cwm & kBothWindings) ? upoly_covers(S.ux[u], S.uy[u], px, py) : upoly_covers_one(S.ux[u], S.uy[u], px, py);
}

// Chooses the next group: rows from row0 (of leaf leaf0) on, whole leaves, a
// lane each, as many as the micropolygon budget, the shared grid points and the
// point rows allow (of a leaf too large for them, as many rows), and of those
// counts of leaves the one with the most micropolygons per step of the CTA: a
// batch of kDiceThreads micropolygons is a step, and so is what comes before
// them.  (One thread adding up to 16 leaves one after the other, 64 point rows
// per group, took half of the dice time of 2 x 2 grids.)
__device__ __forceinline__ void dice_group(const ReyesArgs& a, DiceSmem& S, uint32_t leaf0, uint32_t row0,
                                           uint32_t nleaf, uint32_t r_end)
{
  const uint32_t lane = threadIdx.x, L = leaf0 + lane;
  uint32_t nu = 0, nv = 0, first = r_end, k0 = 0, n = 0;
  if (L < nleaf) {
    nu = a.leaves[L].nu;
    nv = a.leaves[L].nv;
    const uint32_t rb = a.leaves[L].rowbase;
    first = lane == 0 ? row0 : rb;
    k0 = first - rb;
    if (first < r_end) n = min(nu + 1 - k0, r_end - first);
  }
  const bool pow2 = ((nu & (nu - 1)) == 0) && ((nv & (nv - 1)) == 0);
  uint32_t u = n * (nv + 1), g = pow2 && n ? (n + 1) * (nv + 2) : 0u, p = pow2 && n ? n + 1 : 0u;
  uint32_t iu = u, ig = g, ip = p;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t tu = __shfl_up_sync(kFullR, iu, o), tg = __shfl_up_sync(kFullR, ig, o);
    const uint32_t tp = __shfl_up_sync(kFullR, ip, o);
    if (lane >= (uint32_t)o) { iu += tu; ig += tg; ip += tp; }
  }
  const bool fits = n > 0 && iu <= (uint32_t)kUpBudget && ig <= (uint32_t)kMaxGridPts && ip <= (uint32_t)kMaxPtRows;
  const unsigned ok = __ballot_sync(kFullR, fits);
  uint32_t m = (uint32_t)__ffs(~ok) - 1u;   // leading leaves that fit together (0xffffffff: all 32)
  if (m > 32u) m = 32u;
  if (m > 0) {
    const uint32_t steps = (iu + kDiceThreads - 1) / kDiceThreads + 1;
    const uint32_t score = lane < m ? ((iu << 12) / steps) << 5 | lane : 0u;
    m = (__reduce_max_sync(kFullR, score) & 31u) + 1u;
  } else {
    // rows of the first leaf that fit
    if (lane == 0) {
      n = min(n, (uint32_t)kUpBudget / (nv + 1));
      if (pow2) {
        const uint32_t fit = min((uint32_t)kMaxGridPts / (nv + 2), (uint32_t)kMaxPtRows);
        n = min(n, fit > 0 ? fit - 1 : 0u);
      }
      iu = u = n * (nv + 1);
      ig = g = pow2 && n ? (n + 1) * (nv + 2) : 0u;
      ip = p = pow2 && n ? n + 1 : 0u;
    }
    m = __shfl_sync(kFullR, n, 0) ? 1u : 0u;
  }
  if (lane < m) {
    S.leaf[lane] = L;
    S.k0[lane] = k0;
    S.nu[lane] = nu;
    S.nv[lane] = nv;
    S.gpre[lane] = ig - g;
    S.upre[lane] = iu - u;
    S.rpre[lane] = ip - p;
    if (lane == m - 1) {
      S.gpre[m] = ig;
      S.upre[m] = iu;
      S.rpre[m] = ip;
      S.next_row = first + n;
      S.next_leaf = k0 + n == nu + 1 ? L + 1 : L;
    }
  }
  if (lane == 0) {
    S.nseg = m;
    if (m == 0) {   // rows and leaves disagree (cannot happen): stop, never spin
      S.gpre[0] = S.upre[0] = S.rpre[0] = 0;
      S.next_row = r_end;
    }
  }
}

// Four CTAs per SM (64 registers, 55 KB): bound by issue and latency together (at
// three CTAs the schedulers issued 53% of the time, a fifth of the stalls on
// memory and a sixth at barriers), so the extra warps hide more than a fourth
// more spilled values cost: 95 -> 89 us on the 4-sample 1280x720 sphere's 817,003
// micropolygons, 65 -> 60 us on the default constants' 451,467 of 50,163 leaves.
// (8 CTAs of 128 threads: 91 and 58 us; 5 of 192: 98 and 61; a warp per 32
// micropolygons with its own cell list instead of block-wide lists: 98 and 61,
// its lists end in half-empty trips.  Of the 89 us the cells take 46: the
// sample positions' hashes 13, the atomics 12, the edge tests the rest.)
//
// SPARSE: a group takes the ids of all of its micropolygons when it starts (the
// tables hold every micropolygon of the frame), and a covered cell is an atomic
// right where it was tested.  Otherwise only micropolygons with a covered sample
// get an id, by a block-wide scan, and their owners go over their covered cells
// afterwards: for frames of so many micropolygons that ids or tables for all of
// them would not fit.
template <bool SPARSE>
__global__ void __launch_bounds__(kDiceThreads, 4) reyes_dice(ReyesArgs a)
{
  pdl_wait();
  pdl_trigger();
  extern __shared__ __align__(16) unsigned char dice_smem[];
  DiceSmem& S = *reinterpret_cast<DiceSmem*>(dice_smem);
  const unsigned long long meta = a.ctr->leaf_meta;
  const uint32_t nleaf = (uint32_t)(meta >> 40);
  // after a leaf overflow the frame runs again: nothing to dice now
  const unsigned long long R = nleaf <= a.leaf_cap ? (meta & ((1ull << 40) - 1)) : 0ull;
  const uint32_t r_begin = (uint32_t)(R * blockIdx.x / gridDim.x);
  const uint32_t r_end = (uint32_t)(R * (blockIdx.x + 1) / gridDim.x);
  const int r = a.spp == 1 ? 1 : 2;   // cells per pixel edge
  unsigned covered = 0;
  {
    // the last leaf whose first row <= r_begin: kDiceThreads-way search rounds
    // (two for up to 65,536 leaves); leaf lo always qualifies
    uint32_t lo = 0, span = R ? nleaf : 0u;
    while (span > 1) {
      const uint32_t step = (span + kDiceThreads - 1) / kDiceThreads;
      if (threadIdx.x == 0) S.found = 0;
      __syncthreads();
      const uint32_t idx = lo + threadIdx.x * step;
      if (threadIdx.x > 0 && threadIdx.x * step < span && a.leaves[idx].rowbase <= r_begin)
        atomicMax(&S.found, (uint32_t)threadIdx.x);
      __syncthreads();
      const uint32_t t = S.found;
      lo += t * step;
      span = min(step, span - t * step);
      __syncthreads();
    }
    if (threadIdx.x == 0) {
      S.next_leaf = lo;
      S.next_row = r_begin;
      S.ties.n = 0;
    }
  }
  for (;;) {
    __syncthreads();
    const uint32_t row0 = S.next_row, leaf0 = S.next_leaf;
    if (row0 >= r_end) break;   // uniform
    __syncthreads();
    if (threadIdx.x < 32) {
      dice_group(a, S, leaf0, row0, nleaf, r_end);
      __syncwarp();
      if (SPARSE && threadIdx.x == 0) S.gid = atomicAdd(&a.ctr->id_count, S.upre[S.nseg]);
    }
    __syncthreads();
    const int m = (int)S.nseg;
    for (int q = threadIdx.x; q < m * 16; q += blockDim.x) S.cp[q >> 4][q & 15] = a.leaves[S.leaf[q >> 4]].cp[q & 15];
    if (threadIdx.x < m) {
      const PatchRec& p = a.leaves[S.leaf[threadIdx.x]];
      S.keyhi[threadIdx.x] = leaf_key(a, p.i0, p.level, p.s);
    }
    __syncthreads();
    const uint32_t gtot = S.gpre[m], utot = S.upre[m], rtot = S.rpre[m];
    // (a thread per control row of a point row)
    for (uint32_t q = threadIdx.x; q < 4 * rtot; q += blockDim.x) {
      const uint32_t t = q >> 2, c = q & 3u;
      const int i = batch_find(S.rpre, m, t);
      const uint32_t k = S.k0[i] + (t - S.rpre[i]);
      const float u = (float)k * (1.0f / ((float)S.nu[i]));
      const float4* P = &S.cp[i][4 * c];
      S.rowdat[t].r[c] = bez(u, P[0], P[1], P[2], P[3]);
      S.rowdat[t].d[c] = dbez(u, P[0], P[1], P[2], P[3]);
    }
    __syncthreads();
    for (uint32_t f = threadIdx.x; f < gtot; f += blockDim.x) {
      const int i = batch_find(S.gpre, m, f);
      const uint32_t nv = S.nv[i], g = f - S.gpre[i];
      uint32_t j;
      const uint32_t kk = row_divmod(g, nv + 2, j);
      grid_point_row(S.rowdat[S.rpre[i] + kk], a, (float)j * (1.0f / ((float)nv)), S.gp[f]);
    }
    __syncthreads();
    for (uint32_t f0 = 0; f0 < utot; f0 += blockDim.x) {
      const uint32_t f = f0 + threadIdx.x;
      UpolyRec o;
      int cnt = 0;          // cells to test
      uint32_t cwm = 0;
      bool swap = false;
      int2 org = make_int2(0, 0);
      if (f < utot) {
        const int i = batch_find(S.upre, m, f);
        const uint32_t nu = S.nu[i], nv = S.nv[i], tl = f - S.upre[i];
        const uint32_t nv1 = nv + 1;
        uint32_t j;
        const uint32_t kk = row_divmod(tl, nv1, j);                  // row kk of the segment
        const uint32_t k = S.k0[i] + kk, t = k * nv1 + j;             // micropolygon t of the leaf
        const bool pow2 = ((nu & (nu - 1)) == 0) && ((nv & (nv - 1)) == 0);
        if (pow2) {
          const GridPt* gp = S.gp + S.gpre[i];
          const uint32_t gw = nv + 2;
          make_upoly(a, S.keyhi[i], t, gp[kk * gw + j], gp[(kk + 1) * gw + j], gp[(kk + 1) * gw + j + 1],
                     gp[kk * gw + j + 1], o);
        } else {
          const float du = 1.0f / ((float)nu), dv = 1.0f / ((float)nv);
          const float myU = (float)k * du, myV = (float)j * dv;
          GridPt c0, c1, c2, c3;
          grid_point(S.cp[i], a, myU, myV, c0);
          grid_point(S.cp[i], a, myU + du, myV, c1);
          grid_point(S.cp[i], a, myU + du, myV + dv, c2);
          grid_point(S.cp[i], a, myU, myV + dv, c3);
          make_upoly(a, S.keyhi[i], t, c0, c1, c2, c3, o);
        }
        if (o.z < 0.0f) atomicAdd(&a.ctr->negative_depth, 1u);
        const int n = (o.x1 - o.x0) * (o.y1 - o.y0);
        if (n > kSmallPx) {
          const uint32_t b = atomicAdd(&a.ctr->big_count, 1u);
          if (b < a.up_cap) {
            const uint4* src = reinterpret_cast<const uint4*>(&o);
            uint4* dst = reinterpret_cast<uint4*>(&a.up[b]);
#pragma unroll
            for (int q = 0; q < 4; ++q) dst[q] = src[q];
          } else {
            atomicOr(&a.ctr->fc.status, kStatusUpolyOverflow);
          }
        } else if (n > 0) {
          int cx0 = o.x0 * r, cx1 = o.x1 * r - 1, cy0 = o.y0 * r, cy1 = o.y1 * r - 1;
          const float mnx = std_minf(std_minf(o.sx[0], o.sx[1]), std_minf(o.sx[2], o.sx[3]));
          const float mxx = std_maxf(std_maxf(o.sx[0], o.sx[1]), std_maxf(o.sx[2], o.sx[3]));
          const float mny = std_minf(std_minf(o.sy[0], o.sy[1]), std_minf(o.sy[2], o.sy[3]));
          const float mxy = std_maxf(std_maxf(o.sy[0], o.sy[1]), std_maxf(o.sy[2], o.sy[3]));
          cwm = kBothWindings;
          if (exact_box(mnx, mxx, mny, mxy)) {
            const float p = (o.sx[2] - o.sx[0]) * (o.sy[3] - o.sy[1]), q = (o.sx[3] - o.sx[1]) * (o.sy[2] - o.sy[0]);
            if (p != q) cwm = 0u;
            swap = p < q;
            if (r == 1) {   // centre x + 0.5 strictly inside (mnx, mxx)
              cx0 = max(cx0, (int)floorf(mnx - 0.5f) + 1); cx1 = min(cx1, (int)ceilf(mxx - 0.5f) - 1);
              cy0 = max(cy0, (int)floorf(mny - 0.5f) + 1); cy1 = min(cy1, (int)ceilf(mxy - 0.5f) - 1);
            } else {        // quadrant q spans [q / 2, q / 2 + 1/2]
              cx0 = max(cx0, (int)floorf(2.0f * mnx)); cx1 = min(cx1, (int)ceilf(2.0f * mxx) - 1);
              cy0 = max(cy0, (int)floorf(2.0f * mny)); cy1 = min(cy1, (int)ceilf(2.0f * mxy) - 1);
            }
          }
          const int cw = cx1 - cx0 + 1, ch = cy1 - cy0 + 1;
          if (cw > 0 && ch > 0) {
            cnt = cw * ch;
            cwm |= (uint32_t)cw | ((0x10000u / (uint32_t)cw + 1u) << 7);
            org = make_int2(cx0, cy0);
            // (the test of both windings takes the corners as they are)
            const bool rev = swap && !(cwm & kBothWindings);
            S.ux[threadIdx.x] = make_float4(o.sx[0], rev ? o.sx[3] : o.sx[1], o.sx[2], rev ? o.sx[1] : o.sx[3]);
            S.uy[threadIdx.x] = make_float4(o.sy[0], rev ? o.sy[3] : o.sy[1], o.sy[2], rev ? o.sy[1] : o.sy[3]);
            S.org[threadIdx.x] = org;
            S.cwm[threadIdx.x] = cwm;
            if (SPARSE) {
              S.zo[threadIdx.x] = o.z <= 1.0f ? zorder(o.z) : kNoDepth;   // (a NaN depth never survives)
              if (o.z <= 1.0f) put_id(a, S.gid + f, o);
            } else {
              S.mask[threadIdx.x] = 0ull;
            }
          }
        }
      }
      // (the scan's barriers lie between the last batch's records and the flush)
      const uint32_t pre = block_scan((uint32_t)cnt, S.scan, &S.total);
      flush_ties(a, S.ties, kTieStage / 2);
      const uint32_t total = S.total;
      for (uint32_t w0 = 0; w0 < total; w0 += kCellCap) {
        const int lo = max(0, (int)w0 - (int)pre), hi = min(cnt, (int)(w0 + kCellCap) - (int)pre);
        for (int c = lo; c < hi; ++c) S.cell[pre + (uint32_t)c - w0] = (uint16_t)((threadIdx.x << 6) | (uint32_t)c);
        __syncthreads();
        const uint32_t nw = min((uint32_t)kCellCap, total - w0);
        // an atomic's answer is looked at after the next one is on its way
        unsigned long long old = kSampEmpty;
        uint32_t o_at = 0, o_zo = 0, o_id = 0;   // (no depth code is 0)
        for (uint32_t q = threadIdx.x; q < nw; q += blockDim.x) {
          int u, li, x, y, smp;
          if (!dice_cell(a, S, q, u, li, x, y, smp)) continue;
          if (!SPARSE) {
            atomicOr(&S.mask[u], 1ull << li);
            continue;
          }
          ++covered;
          const uint32_t zo = S.zo[u];
          if (zo == kNoDepth) continue;
          const uint32_t id = S.gid + f0 + (uint32_t)u, at = sample_index(a, x, y, smp);
          const unsigned long long got = atomicMin(&a.samp[at], ((unsigned long long)zo << 32) | id);
          if (o_zo) check_tie(a, &S.ties, o_at, o_zo, o_id, old);
          old = got;
          o_at = at;
          o_zo = zo;
          o_id = id;
        }
        if (SPARSE && o_zo) check_tie(a, &S.ties, o_at, o_zo, o_id, old);
        __syncthreads();
      }
      if (SPARSE) continue;
      unsigned long long mask = cnt > 0 ? S.mask[threadIdx.x] : 0ull;
      covered += __popcll(mask);
      if (cnt > 0 && !(o.z <= 1.0f)) mask = 0;  // behind the cleared depth (or NaN): never survives
      const uint32_t id = block_append(a, mask ? 1u : 0u, S.append, &S.base);
      if (mask) {
        put_id(a, id, o);
        const uint32_t zo = zorder(o.z);
        while (mask) {
          const int c = __ffsll(mask) - 1;
          mask &= mask - 1;
          int cx, cy;
          cell_xy(cwm, org, c, cx, cy);
          const uint32_t at = r == 1 ? sample_index(a, cx, cy, 0)
                                     : sample_index(a, cx >> 1, cy >> 1, (cx & 1) | ((cy & 1) << 1));
          check_tie(a, &S.ties, at, zo, id, atomicMin(&a.samp[at], ((unsigned long long)zo << 32) | id));
        }
      }
    }
  }
  __syncthreads();
  flush_ties(a, S.ties, 0u);
  add_covered(a, covered);
}

// The fragments of the queued micropolygons: a warp each, a lane per sample.
__global__ void __launch_bounds__(256) reyes_big(ReyesArgs a)
{
  pdl_wait();
  pdl_trigger();
  const uint32_t nbig = min(a.ctr->big_count, a.up_cap);
  const int lane = threadIdx.x & 31;
  const uint32_t nwarps = gridDim.x * (blockDim.x / 32);
  unsigned covered = 0;
  for (uint32_t wi = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32; wi < nbig; wi += nwarps) {
    UpolyRec u;
    const uint4* src = reinterpret_cast<const uint4*>(&a.up[wi]);
    uint4* dst = reinterpret_cast<uint4*>(&u);
#pragma unroll
    for (int q = 0; q < 4; ++q) dst[q] = src[q];
    const int bw = u.x1 - u.x0;
    const int n = bw * (u.y1 - u.y0) * a.spp;   // candidate samples
    const uint32_t zo = zorder(u.z);
    uint32_t id = kNoId;
    for (int k0 = 0; k0 < n; k0 += 32) {
      const int k = k0 + lane;
      const int pk = k / a.spp, smp = k - pk * a.spp;
      const int x = u.x0 + (bw ? pk % bw : 0), y = u.y0 + (bw ? pk / bw : 0);
      float px = 0.0f, py = 0.0f;
      if (k < n) sample_pos(a.spp, a.seed, x, y, smp, px, py);
      const bool cov = k < n && upoly_covers(make_float4(u.sx[0], u.sx[1], u.sx[2], u.sx[3]),
                                              make_float4(u.sy[0], u.sy[1], u.sy[2], u.sy[3]), px, py);
      covered += cov ? 1u : 0u;
      const unsigned keep = __ballot_sync(kFullR, cov && u.z <= 1.0f);
      if (!keep) continue;
      if (id == kNoId) {
        if (lane == 0) {
          id = atomicAdd(&a.ctr->id_count, 1u);
          put_id(a, id, u);
        }
        id = __shfl_sync(kFullR, id, 0);
      }
      if ((keep >> lane) & 1u) {
        const uint32_t p = sample_index(a, x, y, smp);
        check_tie(a, nullptr, p, zo, id, atomicMin(&a.samp[p], ((unsigned long long)zo << 32) | id));
      }
    }
  }
  add_covered(a, covered);
}

// Samples at which fragments met at one depth: of all that did (each but the
// first has a record, which names one it met), the one with the greatest key
// takes the sample, if that depth is still the sample's.  At +-0 the one with
// the least key goes to first0.
__global__ void __launch_bounds__(256) reyes_ties(ReyesArgs a)
{
  pdl_wait();
  pdl_trigger();
  const uint32_t first = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
  // the first record is read along with the counters (tie_cap is at least the grid)
  uint4 t = a.ties[min(first, a.tie_cap - 1)];
  const uint32_t n = min(a.ctr->tie_count, a.tie_cap);
  // after an overflow of the tables the frame runs again: no key to look up
  if (a.ctr->fc.status & kStatusListOverflow) return;
  for (uint32_t i = first; i < n; i += stride, t = a.ties[min(i, a.tie_cap - 1)]) {
    unsigned long long cur = __ldcg(&a.samp[t.x]);
    const unsigned long long key_z = a.id_key[t.z], key_w = a.id_key[t.w];
    if ((uint32_t)(cur >> 32) != t.y) continue;   // (this pass changes no depth)
    const unsigned long long key = key_z > key_w ? key_z : key_w;
    const unsigned long long mine = ((unsigned long long)t.y << 32) | (key_z > key_w ? t.z : t.w);
    while (cur != mine && key > a.id_key[(uint32_t)cur]) {   // (the key kept only grows)
      const unsigned long long was = atomicCAS(&a.samp[t.x], cur, mine);
      if (was == cur) break;
      cur = was;
    }
    if (t.y != 0x80000000u) continue;   // zorder(+-0)
    const uint32_t low = key_z < key_w ? t.z : t.w;
    const unsigned long long low_key = key_z < key_w ? key_z : key_w;
    uint32_t f = __ldcg(&a.first0[t.x]);
    while (f == kNoId || low_key < a.id_key[f]) {   // (the key kept only falls)
      const uint32_t was = atomicCAS(&a.first0[t.x], f, low);
      if (was == f) break;
      f = was;
    }
  }
}

// Sample si's colour and depth from its state st; a reached one is set back.
__device__ __forceinline__ bool take_sample(const ReyesArgs& a, size_t si, unsigned long long st, uint32_t& c, float& z)
{
  c = kClearColor;
  z = 1.0f;
  if (st == kSampEmpty) return false;
  const uint32_t id = (uint32_t)st;
  if (id >= a.id_cap) return true;   // the tables overflowed: the frame runs again
  c = a.id_color[id] | 0xff000000u;
  z = zorder_inv((uint32_t)(st >> 32));
  if (z == 0.0f) {
    const uint32_t f = a.first0[si];
    a.first0[si] = kNoId;
    if (f < a.id_cap && !(a.id_color[f] & 0x01000000u)) z = -0.0f;
  }
  return true;
}

// The last pass, over every pixel.  One sample per pixel: the sample's colour
// and depth, the clear colour and depth 1 where no fragment reached it.  More
// samples: a pixel takes the rounded mean of its samples' colours per channel
// and the depth of its nearest sample (the first such sample on ties).  Every
// reached sample's state is set back to empty, so the next frame finds it so.
//
// The counters are final: block 0 hands them to the host and leaves them zero
// for the next frame, so that no memset precedes a frame and no copy follows it
// (together 7 us of a 320x240 sphere's 52).
__global__ void __launch_bounds__(256) reyes_pixels(ReyesArgs a, uint32_t npx)
{
  pdl_wait();
  static_assert(sizeof(ReyesCounters) % 4 == 0 && sizeof(ReyesCounters) / 4 <= 256, "a word per thread");
  if (blockIdx.x == 0 && threadIdx.x < sizeof(ReyesCounters) / 4) {
    uint32_t* c = reinterpret_cast<uint32_t*>(a.ctr) + threadIdx.x;
    reinterpret_cast<uint32_t*>(a.host_ctr)[threadIdx.x] = *c;
    *c = 0u;
  }
  const uint32_t stride = gridDim.x * blockDim.x;
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (a.spp == 1) {
    // (the next pixel's state is on its way while this one's colour is fetched)
    unsigned long long next = i < npx ? a.samp[i] : kSampEmpty;
    for (; i < npx; i += stride) {
      const unsigned long long st = next;
      if (i + stride < npx) next = a.samp[i + stride];
      uint32_t c;
      float z;
      if (take_sample(a, i, st, c, z)) a.samp[i] = kSampEmpty;
      a.fb[i] = c;
      a.depth[i] = z;
    }
    return;
  }
  // four samples: 32 contiguous, aligned bytes; a pixel with any reached sample
  // has all four set back
  ulonglong2 nlo = make_ulonglong2(kSampEmpty, kSampEmpty), nhi = nlo;
  if (i < npx) {
    const ulonglong2* sp = reinterpret_cast<const ulonglong2*>(&a.samp[4 * (size_t)i]);
    nlo = sp[0];
    nhi = sp[1];
  }
  for (; i < npx; i += stride) {
    ulonglong2* sp = reinterpret_cast<ulonglong2*>(&a.samp[4 * (size_t)i]);
    const unsigned long long st[4] = {nlo.x, nlo.y, nhi.x, nhi.y};
    if (i + stride < npx) {
      nlo = sp[2 * (size_t)stride];
      nhi = sp[2 * (size_t)stride + 1];
    }
    uint32_t c[4] = {kClearColor, kClearColor, kClearColor, kClearColor};
    float z[4] = {1.0f, 1.0f, 1.0f, 1.0f};
    if ((st[0] & st[1] & st[2] & st[3]) != kSampEmpty) {
      sp[0] = make_ulonglong2(kSampEmpty, kSampEmpty);
      sp[1] = make_ulonglong2(kSampEmpty, kSampEmpty);
#pragma unroll
      for (int k = 0; k < 4; ++k) take_sample(a, 4 * (size_t)i + k, st[k], c[k], z[k]);
    }
    uint32_t sum[3] = {0u, 0u, 0u};
    float best = 1.0f;
    uint32_t best_o = 0xffffffffu;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      sum[0] += c[k] & 255u;
      sum[1] += (c[k] >> 8) & 255u;
      sum[2] += (c[k] >> 16) & 255u;
      const uint32_t o = zorder(z[k]);
      if (k == 0 || o < best_o) { best_o = o; best = z[k]; }
    }
    a.fb[i] = 0xff000000u | (((sum[2] + 2u) / 4u) << 16) | (((sum[1] + 2u) / 4u) << 8) | ((sum[0] + 2u) / 4u);
    a.depth[i] = best;
  }
}

// A launch that may begin while the previous kernel of the stream finishes
// (the kernel's pdl_wait() holds it until that kernel's writes are visible).
template <typename... KArgs, typename... Args>
static cudaError_t launch_chained(void (*kernel)(KArgs...), int grid, int block, size_t smem, cudaStream_t st,
                                  Args... args)
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
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

cudaError_t launch_reyes_frame(const ReyesArgs& a, uint32_t npx, int sms, bool sparse, cudaStream_t st, cudaEvent_t* ev)
{
  // occupancies, found once per process (host threads may launch frames
  // concurrently; call_once makes the others wait for the first)
  static std::once_flag once;
  static int dice_per_sm = 1;
  static cudaError_t setup_err = cudaSuccess;
  std::call_once(once, [] {
    int sp = 0, dp = 1;
    cudaError_t e = cudaFuncSetAttribute(reyes_split, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSplitSmem);
    if (!e) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&sp, reyes_split, kSplitThreads, kSplitSmem);
    // the split's grid barriers need every CTA resident: one per SM
    if (!e && sp < 1) e = cudaErrorCooperativeLaunchTooLarge;
    if (!e) e = cudaFuncSetAttribute(reyes_dice<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDiceSmem);
    if (!e) e = cudaFuncSetAttribute(reyes_dice<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDiceSmem);
    if (!e) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&dp, reyes_dice<true>, kDiceThreads, kDiceSmem);
    setup_err = e;
    dice_per_sm = std::max(1, dp);
  });
  if (setup_err) return setup_err;
  if (ev) cudaEventRecord(ev[0], st);
  ReyesArgs args = a;
  void* params[] = {(void*)&args};
  cudaError_t e = cudaLaunchCooperativeKernel((const void*)reyes_split, dim3(sms), dim3(kSplitThreads), params,
                                              kSplitSmem, st);
  if (e != cudaSuccess) return e;
  if (ev) cudaEventRecord(ev[1], st);
  // the launches after the split may start while their predecessor drains
  // (programmatic dependent launch); each waits for it before touching memory
  const int grid = sms * 8;
  e = launch_chained(sparse ? reyes_dice<true> : reyes_dice<false>, sms * dice_per_sm, kDiceThreads, kDiceSmem, st, a);
  if (!e) e = launch_chained(reyes_big, grid, 256, 0, st, a);
  if (ev) cudaEventRecord(ev[2], st);
  if (!e) e = launch_chained(reyes_ties, sms * 4, 256, 0, st, a);
  if (ev) cudaEventRecord(ev[3], st);
  if (!e) e = launch_chained(reyes_pixels, grid, 256, 0, st, a, npx);
  if (ev) cudaEventRecord(ev[4], st);
  if (e) return e;
  return cudaGetLastError();
}

}  // namespace piko

using namespace piko;

// ------------------------------------------------------------------ host state
// Work buffers and counters of a Reyes scene.  A scene may borrow the work
// buffers of another state (`buffers`): frames run in stream order on one
// stream can share them (the served form gives each stream lane one set),
// while every scene keeps its own counters for its overflow checks.
struct ReyesState {
  ReyesState* buffers = nullptr;  // borrowed work buffers (not owned), or null
  unsigned char* block = nullptr; // the buffers as first allocated; one that grew has memory of its own
  size_t block_bytes = 0;
  PatchRec* lvl[2] = {nullptr, nullptr};
  PatchRec* stack = nullptr;
  PatchRec* leaves = nullptr;
  UpolyRec* up = nullptr;
  uint32_t* id_color = nullptr;
  unsigned long long* id_key = nullptr;
  uint4* ties = nullptr;
  uint32_t lvl_cap = 0, leaf_cap = 0, up_cap = 0, id_cap = 0, tie_cap = 0;
  unsigned long long* samp = nullptr;
  uint32_t* first0 = nullptr;
  size_t npx_cap = 0;   // samples
  bool sparse = true;   // an id for every micropolygon (reyes_dice); of a scene, not of borrowed buffers
  bool clean = false;   // per-sample state all empty (set when allocated; every frame leaves it so)
  ReyesCounters* ctr = nullptr;
  ReyesCounters* h_ctr = nullptr;   // pinned, written by reyes_pixels
  bool ctr_clean = false;
  bool captured = false;            // a caller's capture holds a frame: the counters are cleared before every frame
  cudaEvent_t ev[5] = {};
  bool ev_made = false;

  template <class T>
  void drop(T*& p)
  {
    const unsigned char* q = reinterpret_cast<const unsigned char*>(p);
    if (q >= block && q < block + block_bytes) p = nullptr;
    else dfree(p);
  }
};

static void reyes_state_free(ReyesState* r)
{
  r->drop(r->lvl[0]); r->drop(r->lvl[1]); r->drop(r->stack); r->drop(r->leaves); r->drop(r->up);
  r->drop(r->id_color); r->drop(r->id_key); r->drop(r->ties); r->drop(r->samp); r->drop(r->first0); r->drop(r->ctr);
  dfree(r->block);
  if (r->h_ctr) cudaFreeHost(r->h_ctr);
  if (r->ev_made) for (auto& e : r->ev) cudaEventDestroy(e);
  delete r;
}

void piko_reyes_release(piko_scene* s)
{
  if (!s->reyes) return;
  reyes_state_free(s->reyes);
  s->reyes = nullptr;
}

ReyesState* reyes_buffers_new() { return new ReyesState(); }
void reyes_buffers_free(ReyesState* b)
{
  if (b) reyes_state_free(b);
}
void reyes_borrow_buffers(piko_scene* s, ReyesState* b)
{
  if (!s->reyes) s->reyes = new ReyesState();
  s->reyes->buffers = b;
}

constexpr uint32_t kMaxSparse = 1u << 24;

// A state's first buffers, by one allocation: one takes 0.2 to 0.35 ms, whatever its
// size, a frame a tenth of a millisecond (fresh 320x240 sphere: first frame with
// fourteen allocations 5.1 ms, with one 3.0).  The split's stacks share their memory
// with the tables that only later kernels of a frame use (device memory of that
// sphere 122 -> 103 MB).
static cudaError_t reyes_block(ReyesState* r, int sms, uint32_t lvl_cap, uint32_t leaf_cap, uint32_t up_cap,
                               uint32_t id_cap, uint32_t tie_cap, size_t npx)
{
  size_t end = 0;
  const auto place = [&end](size_t bytes) {
    const size_t at = end;
    end += (bytes + 255) & ~(size_t)255;
    return at;
  };
  const size_t lvl0 = place(sizeof(PatchRec) * lvl_cap), lvl1 = place(sizeof(PatchRec) * lvl_cap);
  const size_t leaves = place(sizeof(PatchRec) * leaf_cap);
  const size_t samp = place(sizeof(*r->samp) * npx), first0 = place(sizeof(*r->first0) * npx);
  const size_t ctr = place(sizeof(ReyesCounters));
  const size_t shared = place(sizeof(PatchRec) * (size_t)sms * kSplitStack), stack_end = end;
  end = shared;
  const size_t up = place(sizeof(UpolyRec) * up_cap);
  const size_t id_color = place(sizeof(*r->id_color) * id_cap), id_key = place(sizeof(*r->id_key) * id_cap);
  const size_t ties = place(sizeof(uint4) * tie_cap);
  end = std::max(end, stack_end);
  unsigned char* p;
  if (const cudaError_t e = dalloc(&p, end)) return e;
  r->block = p;
  r->block_bytes = end;
  const auto cut = [p](auto*& q, size_t at) { q = reinterpret_cast<std::remove_reference_t<decltype(q)>>(p + at); };
  cut(r->lvl[0], lvl0); cut(r->lvl[1], lvl1); cut(r->leaves, leaves);
  cut(r->samp, samp); cut(r->first0, first0); cut(r->stack, shared);
  cut(r->up, up); cut(r->id_color, id_color); cut(r->id_key, id_key); cut(r->ties, ties);
  if (!r->ctr) cut(r->ctr, ctr);
  r->lvl_cap = lvl_cap; r->leaf_cap = leaf_cap; r->up_cap = up_cap;
  r->id_cap = id_cap; r->tie_cap = tie_cap; r->npx_cap = npx;
  r->clean = r->ctr_clean = false;
  return cudaSuccess;
}

static cudaError_t reyes_alloc(ReyesState* r, int sms, uint32_t lvl_cap, uint32_t leaf_cap, uint32_t up_cap,
                               uint32_t id_cap, uint32_t tie_cap, size_t npx)
{
  cudaError_t e = cudaSuccess;
  if (r->buffers) {
    if ((e = reyes_alloc(r->buffers, sms, lvl_cap, leaf_cap, up_cap, id_cap, tie_cap, npx))) return e;
    lvl_cap = leaf_cap = up_cap = id_cap = tie_cap = 0;
    npx = 0;
  }
  if (!r->block && lvl_cap && (e = reyes_block(r, sms, lvl_cap, leaf_cap, up_cap, id_cap, tie_cap, npx))) return e;
  // (a capacity stands only while all of its buffers do)
  if (lvl_cap > r->lvl_cap) {
    r->drop(r->lvl[0]); r->drop(r->lvl[1]);
    r->lvl_cap = 0;
    if ((e = dalloc(&r->lvl[0], lvl_cap)) || (e = dalloc(&r->lvl[1], lvl_cap))) return e;
    r->lvl_cap = lvl_cap;
  }
  if (leaf_cap > r->leaf_cap) {
    r->drop(r->leaves);
    r->leaf_cap = 0;
    if ((e = dalloc(&r->leaves, leaf_cap))) return e;
    r->leaf_cap = leaf_cap;
  }
  if (up_cap > r->up_cap) {
    r->drop(r->up);
    r->up_cap = 0;
    if ((e = dalloc(&r->up, up_cap))) return e;
    r->up_cap = up_cap;
  }
  if (id_cap > r->id_cap) {
    r->drop(r->id_color); r->drop(r->id_key);
    r->id_cap = 0;
    if ((e = dalloc(&r->id_color, id_cap)) || (e = dalloc(&r->id_key, id_cap))) return e;
    r->id_cap = id_cap;
  }
  if (tie_cap > r->tie_cap) {
    r->drop(r->ties);
    r->tie_cap = 0;
    if ((e = dalloc(&r->ties, tie_cap))) return e;
    r->tie_cap = tie_cap;
  }
  if (npx > r->npx_cap) {
    r->drop(r->samp); r->drop(r->first0);
    r->npx_cap = 0;
    r->clean = false;
    if ((e = dalloc(&r->samp, npx)) || (e = dalloc(&r->first0, npx))) return e;
    r->npx_cap = npx;
  }
  if (!r->ctr) {
    r->ctr_clean = false;
    if ((e = dalloc(&r->ctr, 1))) return e;
  }
  if (!r->h_ctr && (e = halloc(&r->h_ctr, 1))) return e;
  if (!r->ev_made) {
    for (auto& ev : r->ev)
      if ((e = cudaEventCreate(&ev))) return e;
    r->ev_made = true;
  }
  return cudaSuccess;
}

piko_status piko_reyes_run(piko_scene* s, cudaStream_t st, bool timed)
{
  piko_ctx* ctx = s->pipe->ctx;
  piko_pipe* p = s->pipe;
  if (!s->reyes) s->reyes = new ReyesState();
  ReyesState* r = s->reyes;
  ReyesState* b = r->buffers ? r->buffers : r;
  const uint32_t P = (uint32_t)s->N;
  const size_t npx = (size_t)s->W * (size_t)s->H;
  const size_t nsamp = npx * (size_t)p->samples_per_pixel;
  CU(ctx, reyes_alloc(r, ctx->sms, std::max<uint32_t>(1u << 16, 64u * P), std::max<uint32_t>(1u << 16, 64u * P),
                      b->up_cap ? b->up_cap : (1u << 16),
                      b->id_cap ? b->id_cap : (uint32_t)std::max<size_t>(1u << 20, npx),
                      b->tie_cap ? b->tie_cap : (uint32_t)std::max<size_t>(1u << 18, nsamp / 8), nsamp));
  bool capturing = false;
  CU(ctx, stream_capturing(st, &capturing));
  if (capturing) r->captured = true;
  const bool ran = !capturing;   // (what a capture records has not run yet)
  if (!r->ctr_clean || r->captured) {   // fresh, a frame whose launches failed part way, replays that nothing orders
    CU(ctx, cudaMemsetAsync(r->ctr, 0, sizeof(ReyesCounters), st));
    r->ctr_clean = ran;
  }
  ReyesArgs a;
  memset(&a, 0, sizeof(a));
  a.W = s->W; a.H = s->H; a.nBx = s->W / 64; a.nBy = s->H / 64;
  a.nDice = std::max(1, a.nBx * a.nBy);
  a.P = (int)P;
  memcpy(a.vp, s->state.view_proj, sizeof(a.vp));
  a.thr = p->split_threshold;
  a.max_splits = std::min(p->max_splits, 30);
  a.grid = p->dice_grid;
  a.in_patches = s->patches;
  a.lvl[0] = b->lvl[0]; a.lvl[1] = b->lvl[1]; a.lvl_cap = b->lvl_cap;
  a.stack = b->stack;
  a.leaves = b->leaves; a.leaf_cap = b->leaf_cap;
  a.up = b->up; a.up_cap = b->up_cap;
  a.id_color = b->id_color; a.id_key = b->id_key; a.id_cap = b->id_cap;
  a.ties = b->ties; a.tie_cap = b->tie_cap;
  a.ctr = r->ctr;
  a.host_ctr = r->h_ctr;
  a.fb = s->fb; a.depth = s->depth;
  a.samp = b->samp; a.first0 = b->first0;
  a.spp = p->samples_per_pixel;
  a.seed = p->sample_seed;
  a.phong = p->phong;
  if (!b->clean) {
    // fresh sample buffers, or a frame whose launches failed part way
    CU(ctx, cudaMemsetAsync(b->samp, 0xff, sizeof(unsigned long long) * b->npx_cap, st));
    CU(ctx, cudaMemsetAsync(b->first0, 0xff, sizeof(uint32_t) * b->npx_cap, st));
    b->clean = ran;
  }
  const cudaError_t le = launch_reyes_frame(a, (uint32_t)npx, ctx->sms, r->sparse, st, timed ? r->ev : nullptr);
  if (le != cudaSuccess) b->clean = r->ctr_clean = false;
  CU(ctx, le);
  return PIKO_OK;
}

piko_status piko_reyes_finish(piko_scene* s)
{
  piko_ctx* ctx = s->pipe->ctx;
  ReyesState* r = s->reyes;
  if (!r || !r->h_ctr) { s->pending = false; return PIKO_OK; }   // no frame was enqueued
  for (int attempt = 0; attempt < 6; ++attempt) {
    CU(ctx, cudaStreamSynchronize(s->last_stream));
    const ReyesCounters& c = *r->h_ctr;
    const uint32_t st = c.fc.status;
    if (st & kStatusBarrierTimeout) return set_err(ctx, PIKO_ERR_TIMEOUT, "%s", "split level barrier timed out");
    if (!(st & (kStatusPatchOverflow | kStatusUpolyOverflow | kStatusListOverflow))) {
      s->pending = false;
      return PIKO_OK;
    }
    uint32_t maxlvl = 0;
    for (int i = 0; i < 40; ++i) maxlvl = std::max(maxlvl, c.level_count[i]);
    const uint32_t leaves = (uint32_t)(c.leaf_meta >> 40);
    const ReyesState* b = r->buffers ? r->buffers : r;
    uint32_t lvl = b->lvl_cap, lf = b->leaf_cap, up = b->up_cap, ids = b->id_cap, ties = b->tie_cap;
    if (st & kStatusPatchOverflow) {
      // (the patches of a frontier that overflowed were not split: each has a leaf at least)
      const uint32_t unsplit = maxlvl > lvl ? maxlvl : 0u;
      lvl = std::max(lvl, maxlvl + maxlvl / 2 + 1024);
      lf = std::max(lf, 2 * (leaves + unsplit) + 1024);
    }
    if (st & kStatusUpolyOverflow) up = (uint32_t)std::min<unsigned long long>(c.big_count + c.big_count / 4ull + 4096, 0xffffffffull);
    const auto more = [](uint32_t n) {   // (an id of kNoId means none)
      return (uint32_t)std::min<unsigned long long>(n + n / 4ull + 4096, 0xfffffffeull);
    };
    // ids for all micropolygons while their tables stay below 200 MB
    // (the first frame without them then tells how many it needs)
    const bool was_sparse = r->sparse;
    if (c.upolys > kMaxSparse) r->sparse = false;
    const uint32_t need_ids = r->sparse ? (uint32_t)c.upolys + std::min(c.big_count, kMaxSparse)
                                        : was_sparse ? ids : c.id_count;
    if (need_ids > ids) ids = more(need_ids);
    if (c.tie_count > ties) ties = more(c.tie_count);
    CU(ctx, reyes_alloc(r, ctx->sms, lvl, lf, up, ids, ties, b->npx_cap));
    piko_status rr = piko_reyes_run(s, s->last_stream, s->timed);
    if (rr != PIKO_OK) return rr;
  }
  cudaStreamSynchronize(s->last_stream);   // (FrameOrder's mark lies before the last run)
  return set_err(ctx, PIKO_ERR_QUEUE_OVERFLOW, "%s", "Reyes queues kept overflowing");
}

namespace piko {
// One CTA waiting at level barrier 0 with no CTA to release it: the bounded
// wait must give up and record kStatusBarrierTimeout.
__global__ void __launch_bounds__(32) reyes_wait_selftest(ReyesCounters* c)
{
  __shared__ uint32_t s_count;
  barrier_wait(c, 0u, &s_count);
}
}  // namespace piko

extern "C" piko_status piko_selftest_wait_timeout(piko_ctx* ctx)
{
  if (!ctx) return PIKO_ERR_INVALID;
  cudaSetDevice(ctx->device);
  ReyesCounters* d = nullptr;
  CU(ctx, dalloc(&d, 1));
  ReyesCounters h;
  cudaError_t e = cudaMemset(d, 0, sizeof(ReyesCounters));
  if (!e) {
    reyes_wait_selftest<<<1, 32>>>(d);
    e = cudaGetLastError();
  }
  if (!e) e = cudaMemcpy(&h, d, sizeof(ReyesCounters), cudaMemcpyDeviceToHost);
  cudaFree(d);
  CU(ctx, e);
  if (h.fc.status & kStatusBarrierTimeout)
    return set_err(ctx, PIKO_ERR_TIMEOUT, "%s", "self-test: the bounded barrier wait gave up as designed");
  return PIKO_OK;
}

piko_status piko_reyes_stats(piko_scene* s, piko_frame_stats* o)
{
  ReyesState* r = s->reyes;
  if (!r || !r->h_ctr) return PIKO_OK;
  const ReyesCounters& c = *r->h_ctr;
  o->prims_in = (uint64_t)s->N;
  o->prims_kept = c.leaf_meta >> 40;
  o->upolys = c.upolys;
  o->bin_entries = c.big_count;   // micropolygons shaded a warp each
  o->covered = c.fc.covered;
  o->status = c.fc.status | (c.negative_depth ? kStatusDepthNeverSettles : 0u);
  o->split_levels = c.levels_run;
  o->n_kernels = 0;
  if (s->timed && r->ev_made) {
    o->n_kernels = 4;
    for (int i = 0; i < 4; ++i) {
      float ms = 0.0f;
      cudaEventElapsedTime(&ms, r->ev[i], r->ev[i + 1]);
      o->kernel_ms[i] = ms;
    }
  }
  return PIKO_OK;
}

// mh_raycast.cu -- trilinear raycast of the zero level set.
//
// CastKernel (visualization/ray_caster.cu:16-150): one thread per pixel
// marches the camera ray with a fixed step from min to max raycast depth,
// samples the SDF trilinearly (GetSpatialValue, geometry/spatial_query.h:23-66),
// and on a + to - sign change refines the hit with three regula-falsi steps
// (BisectionIntersection, geometry/isosurface_intersection.h:21-55).  The
// sample positions, the accumulation of t and every comparison follow the
// reference's single-precision order exactly, and so does every value the
// output depends on.
//
// GB300 structure.  A 640x480 frame of the 4 mm PSDF workload takes about 206
// samples per ray to the hit, of which about 3 lie near a voxel that is not
// non-negative; the rest cannot end a zero crossing.  So the march is split:
//  * k_ray_grid writes, before each raycast, a bit per 2^3-voxel cell of the
//    view's bounding box: set when a sample whose first corner lies in the cell
//    may read a voxel that is not non-negative (from the per-block masks `neg`
//    that every writer of sdf keeps);
//  * the march steps over clear cells with nothing but t += step, one
//    multiply-add per axis and one load, four samples in flight per step, and
//    evaluates only samples in set cells;
//  * the same pass writes the indices of the view's blocks into a dense array,
//    so a sample's eight blocks come from eight independent loads; without it
//    (a view of more than 2^26 blocks, or the footprint count) they come from
//    the hash table through a register cache;
//  * all state in registers: one sampler serves the march, the previous sample
//    and the regula falsi (a phase variable picks the next position);
//  * a warp covers 8x4 pixels, so its rays cross the same cells; in small
//    images, which leave the chip's lanes idle, 4 or 8 lanes share a ray.
// A 640x480 view of the 4 mm map (461 k blocks, grid included): 1.99 -> 0.39
// ms against hash lookups and block-wide skips; 161x119 at 8 mm: 0.46 -> 0.09
// ms.  What is left is latency: a ray's evaluations follow one another, two
// dependent loads and about 200 instructions each, and the rays with many of
// them (along surfaces, behind walls) end last.
#include "mh_internal.cuh"
#include "mh_kernels.h"
#include "mh_batch.cuh"

#include <algorithm>
#include <cmath>

// pixel tiles of a CTA: the raycast's, and the gradient's and normal equations'
#define RC_TX 8
#define RC_TY 8
#define GR_TX 16
#define GR_TY 8
// threads of a CTA where lanes share rays
#define RC_GROUP_THREADS 256
// Lanes with a sample to evaluate before a warp leaves the search for it.  All
// 32 is the fewest evaluations, but every lane waits for the longest search;
// 640x480 / 161x119 views, us: 32: 549 / 252, 16: 475 / 204, 8: 463 / 191,
// 4: 437 / 180, 2: 476 / 185, 1: 527 / 225.
#define RC_WAIT 4
// The same where lanes share a ray: lanes of half a warp's rays.
#define RC_GROUP_WAIT 16
// Largest images of which 8 lanes and 4 lanes share a ray, see launch_raycast.
#define RC_PIXELS8 65536
#define RC_PIXELS4 131072

// ------------------------------------------------------------------ forward
// The forward march keeps its whole state in registers: one sampler is
// inlined once, and a phase variable chooses where the next sample goes --
// the march itself, the sample before a negative one, the three regula-falsi
// steps, the six gradient samples of the normal.
//
// The skips are exact.  A march sample matters only when it is negative right
// after a positive one (the zero crossing), and then the previous valid
// sample's value matters too.  A sample in a clear cell is >= 0 or invalid (a
// corner block is missing), so it can never be the negative end.  Whether it
// was valid is asked only when a negative sample follows: the sample before
// is evaluated then (it is nearly always valid), and if it is invalid the
// samples since the last known one are looked through again for the last
// valid one (PH_SCAN).
namespace {

struct Nbhd {
  static constexpr int LANES = 1;
  int bx, by, bz;    // block of the first corner of the last sample
  unsigned looked;   // bit n: block n = (bx, by, bz) + (n & 1, n >> 1 & 1, n >> 2 & 1) looked up
  unsigned miss;     // bit n: block n is missing
  int p[8];          // block indices, indexed with constants only (registers)
  __device__ __forceinline__ void init() {
    bx = by = bz = 0x7fffffff;
    looked = miss = 0u;
#pragma unroll
    for (int j = 0; j < 8; ++j) p[j] = -1;
  }
};

// The blocks of a sample from the view's dense array; only the first corner's
// block is remembered.
struct DenseNbhd {
  static constexpr int LANES = 1;
  int bx, by, bz;
  __device__ __forceinline__ void init() { bx = by = bz = 0x7fffffff; }
};

// The same for G lanes that share a ray, lanes base .. base + G - 1 of the
// warp: lane j holds corners 8 / G j and up.
template <int G> struct GroupNbhd {
  static constexpr int LANES = G;
  int j;
  unsigned base;
  unsigned lanes;  // the warp's lanes that sample together, whole groups
  __device__ __forceinline__ void init() {
    j = threadIdx.x & (G - 1);
    base = threadIdx.x & 31 & ~(G - 1);
    lanes = 0xffffffffu;
  }
  // the group's bits of a warp ballot
  __device__ __forceinline__ unsigned of(unsigned ballot) const { return (ballot >> base) & ((1u << G) - 1u); }
};

// Block indices of the eight corners, corner i = 4 mx + 2 my + mz (m = 1: the
// upper voxel of that axis); false when one of the blocks is missing.
__device__ __forceinline__ bool blocks_at(const Dev &d, DenseNbhd &c, const Corners &k, int (&blk)[8]) {
  const RayGrid &g = d.grid;
  c.bx = k.v0x >> 3, c.by = k.v0y >> 3, c.bz = k.v0z >> 3;
  // every sample of a ray lies inside the box; the clamps keep the loads there
  const unsigned x0 = min((unsigned)(c.bx - g.bx), g.bnx - 1u), x1 = min((unsigned)((k.v1x >> 3) - g.bx), g.bnx - 1u);
  const unsigned y0 = min((unsigned)(c.by - g.by), g.bny - 1u), y1 = min((unsigned)((k.v1y >> 3) - g.by), g.bny - 1u);
  const unsigned z0 = min((unsigned)(c.bz - g.bz), g.bnz - 1u), z1 = min((unsigned)((k.v1z >> 3) - g.bz), g.bnz - 1u);
  const unsigned row[4] = {(z0 * g.bny + y0) * g.bnx, (z1 * g.bny + y0) * g.bnx, (z0 * g.bny + y1) * g.bnx,
                           (z1 * g.bny + y1) * g.bnx};
  unsigned any = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const unsigned e = __ldg(g.blocks + row[i & 3] + ((i & 4) ? x1 : x0)) ^ g.tag;
    any |= e;
    blk[i] = (int)(e & 0xffffffu);
  }
  return any < 0x1000000u;
}

__device__ __forceinline__ bool blocks_at(const Dev &d, Nbhd &c, const Corners &k, int (&blk)[8]) {
  // VoxelToBlock: floor division by 8 (geometry_helper.h:82-90)
  const int b0x = k.v0x >> 3, b0y = k.v0y >> 3, b0z = k.v0z >> 3;
  if (b0x != c.bx || b0y != c.by || b0z != c.bz) {
    c.bx = b0x, c.by = b0y, c.bz = b0z;
    c.looked = c.miss = 0u;
  }
  const int ex = (k.v1x >> 3) - b0x, ey = (k.v1y >> 3) - b0y, ez = (k.v1z >> 3) - b0z;
  unsigned need = 1u;
  if (ex) need |= need << 1;
  if (ey) need |= need << 2;
  if (ez) need |= need << 4;
  unsigned fresh = need & ~c.looked;
  if (fresh & 1u) {
    const int b0 = hash_find(d, b0x, b0y, b0z);
    c.p[0] = b0;
    if (b0 >= 0 && d.touch) d.touch[b0] = 1;
    if (b0 < 0) c.miss |= 1u;
    c.looked |= 1u;
    fresh &= ~1u;
  }
  if (c.miss & 1u) return false;
  while (fresh) {
    const int n = __ffs(fresh) - 1;
    fresh &= fresh - 1;
    const int bn = hash_find(d, b0x + (n & 1), b0y + ((n >> 1) & 1), b0z + ((n >> 2) & 1));
#pragma unroll
    for (int j = 1; j < 8; ++j)
      if (j == n) c.p[j] = bn;
    if (bn >= 0 && d.touch) d.touch[bn] = 1;
    if (bn < 0) c.miss |= 1u << n;
  }
  c.looked |= need;
  if (need & c.miss) return false;
  // block of each corner (mx, my, mz): p[(mx & ex) | (my & ey) << 1 | (mz & ez) << 2]
  blk[0] = c.p[0];
  blk[4] = ex ? c.p[1] : blk[0];
  blk[2] = ey ? c.p[2] : blk[0];
  blk[6] = ey ? (ex ? c.p[3] : c.p[2]) : blk[4];
  blk[1] = ez ? c.p[4] : blk[0];
  blk[5] = ez ? (ex ? c.p[5] : c.p[4]) : blk[4];
  blk[3] = ez ? (ey ? c.p[6] : c.p[4]) : blk[2];
  blk[7] = ez ? (ey ? (ex ? c.p[7] : c.p[6]) : (ex ? c.p[5] : c.p[4])) : blk[6];
  return true;
}

// GetSpatialValue (geometry/spatial_query.h:23-66) with the same corners,
// weights and summation order as spatial_sample: the value in s (untouched when
// want is false), or false for a sample that is invalid.
template <class N>
__device__ __forceinline__ bool nb_sample(const Dev &d, N &c, F3 pos, bool want, float &s) {
  const Corners k = corners_at(d.p, pos);
  int blk[8];
  if (!blocks_at(d, c, k, blk)) return false;
  if (!want) return true;
  // local voxel coordinates of the two corners of each axis
  const int l0x = k.v0x & 7, l1x = k.v1x & 7;
  const int yz[4] = {(k.v0y & 7) * 8 + (k.v0z & 7) * 64, (k.v0y & 7) * 8 + (k.v1z & 7) * 64,
                     (k.v1y & 7) * 8 + (k.v0z & 7) * 64, (k.v1y & 7) * 8 + (k.v1z & 7) * 64};
  const float w0x = 1.0f - k.rx, w0y = 1.0f - k.ry, w0z = 1.0f - k.rz;
  const float wxy[4] = {w0x * w0y, w0x * k.ry, k.rx * w0y, k.rx * k.ry};
  float v[8];
#pragma unroll
  for (int i = 0; i < 8; ++i)
    v[i] = __ldg(d.sdf + (size_t)blk[i] * MH_BLOCK_VOXELS + ((i & 4) ? l1x : l0x) + yz[i & 3]);
  float acc = 0.0f;
#pragma unroll
  for (int i = 0; i < 8; ++i) acc += wxy[i >> 1] * ((i & 1) ? k.rz : w0z) * v[i];
  s = acc;
  return true;
}

// 8 / G corners a lane; every lane of the group gets the result.
template <int G>
__device__ __forceinline__ bool nb_sample(const Dev &d, GroupNbhd<G> &c, F3 pos, bool, float &s) {
  const Corners k = corners_at(d.p, pos);
  const RayGrid &g = d.grid;
  float v[8 / G];
  bool there = true;
#pragma unroll
  for (int q = 0; q < 8 / G; ++q) {
    const int i = c.j * (8 / G) + q;
    const bool mx = i & 4, my = i & 2, mz = i & 1;
    const int vx = mx ? k.v1x : k.v0x, vy = my ? k.v1y : k.v0y, vz = mz ? k.v1z : k.v0z;
    const unsigned bx = min((unsigned)((vx >> 3) - g.bx), g.bnx - 1u), by = min((unsigned)((vy >> 3) - g.by), g.bny - 1u),
                   bz = min((unsigned)((vz >> 3) - g.bz), g.bnz - 1u);
    const unsigned b = __ldg(g.blocks + (bz * g.bny + by) * g.bnx + bx) ^ g.tag;
    float x = 0.0f;
    if (b < 0x1000000u) x = __ldg(d.sdf + (size_t)b * MH_BLOCK_VOXELS + (vx & 7) + (vy & 7) * 8 + (vz & 7) * 64);
    else there = false;
    v[q] = (mx ? k.rx : 1.0f - k.rx) * (my ? k.ry : 1.0f - k.ry) * (mz ? k.rz : 1.0f - k.rz) * x;
  }
  const bool ok = c.of(__ballot_sync(c.lanes, there)) == (1u << G) - 1u;
  float acc = 0.0f;
#pragma unroll
  for (int i = 0; i < 8; ++i) acc += __shfl_sync(c.lanes, v[i % (8 / G)], c.base + i / (8 / G));
  s = acc;
  return ok;
}

// One axis of a slab test with the direction's reciprocal: narrows [lo, hi]
// to the t for which the ray's coordinate lies inside (a, b).  The bounds
// carry a few ulp of rounding; the box margins below absorb them.
__device__ __forceinline__ void slab_r(float o, float dir, float idir, float a, float b, float &lo, float &hi) {
  if (dir != 0.0f) {
    const float t1 = (a - o) * idir, t2 = (b - o) * idir;
    lo = fmaxf(lo, fminf(t1, t2));
    hi = fminf(hi, fmaxf(t1, t2));
  } else if (!(o > a && o < b)) {
    lo = __int_as_float(0x7f800000);
    hi = -__int_as_float(0x7f800000);
  }
}

// t interval in which every sample of the ray cam + t * wd has its first
// corner voxel in block (bx, by, bz).  A coordinate at least 0.1 voxel inside
// the block's faces has floor(p / v) -- and, where p / v is within 0.01 of an
// integer, round-half-away(p / v - 1/2) -- in range; the margin adds 8 units
// in the last place of the coordinates for the rounding of the position and
// of the interval ends.
__device__ __forceinline__ void block_interval(const DevParams &p, int bx, int by, int bz, F3 cam, F3 wd, F3 iwd,
                                               float &lo, float &hi) {
  const float vs = p.voxel_size;
  const float side = (float)MH_BLOCK_SIDE * vs;
  lo = -__int_as_float(0x7f800000);
  hi = __int_as_float(0x7f800000);
  const float ax = (float)(bx * MH_BLOCK_SIDE) * vs, ay = (float)(by * MH_BLOCK_SIDE) * vs,
              az = (float)(bz * MH_BLOCK_SIDE) * vs;
  const float mx = 0.1f * vs + 5e-7f * (fabsf(ax) + side + fabsf(cam.x));
  const float my = 0.1f * vs + 5e-7f * (fabsf(ay) + side + fabsf(cam.y));
  const float mz = 0.1f * vs + 5e-7f * (fabsf(az) + side + fabsf(cam.z));
  slab_r(cam.x, wd.x, iwd.x, ax + mx, ax + side - mx, lo, hi);
  slab_r(cam.y, wd.y, iwd.y, ay + my, ay + side - my, lo, hi);
  slab_r(cam.z, wd.z, iwd.z, az + mz, az + side - mz, lo, hi);
}

// A ray in the cells of the view's grid: cell = MH_GRID_BIAS + cam' + t wd'
// in a float whose last bits are 1/256 cell, so one multiply-add gives a
// sample's cell and the low 22 bits of the result hold it with 8 bits of
// fraction.  Positions are shifted down by the grid's guard (ray_grid_of): a
// sample found in cell i has no corner below it, and k_ray_grid marks cell i for
// all voxels above that the sample may read.
struct GridRay {
  float ox, oy, oz, dx, dy, dz;
};
__device__ __forceinline__ GridRay grid_ray(const RayGrid &g, F3 cam, F3 wd) {
  GridRay r;
  r.ox = (cam.x - g.ox) * g.inv_cell - MH_GRID_GUARD + MH_GRID_BIAS;
  r.oy = (cam.y - g.oy) * g.inv_cell - MH_GRID_GUARD + MH_GRID_BIAS;
  r.oz = (cam.z - g.oz) * g.inv_cell - MH_GRID_GUARD + MH_GRID_BIAS;
  r.dx = wd.x * g.inv_cell, r.dy = wd.y * g.inv_cell, r.dz = wd.z * g.inv_cell;
  return r;
}
// A sample's cell on each axis, in the float's bits from bit 8 up.  Indices
// made from them are clamped to the grid, so samples past the end of a ray
// read some word of it.
struct GridCell {
  unsigned x, y, z;
};
__device__ __forceinline__ GridCell grid_cell(const GridRay &r, float t) {
  return GridCell{__float_as_uint(fmaf(t, r.dx, r.ox)), __float_as_uint(fmaf(t, r.dy, r.oy)),
                  __float_as_uint(fmaf(t, r.dz, r.oz))};
}
// The word that holds the cell's bit.  The words' coordinates still hold the
// float's upper bits: `base` takes them out.
__device__ __forceinline__ unsigned grid_word(const RayGrid &g, GridCell c, unsigned base) {
  return __ldg(g.bits + min((c.z >> 9) * (g.ny * g.nx) + (c.y >> 10) * g.nx + (c.x >> 10) - base, g.words - 1u));
}
__device__ __forceinline__ bool cell_bit(unsigned word, GridCell c) {
  return (word >> (((c.x >> 8) & 3u) | ((c.y >> 6) & 12u) | ((c.z >> 4) & 16u))) & 1u;
}
__device__ __forceinline__ unsigned grid_base(const RayGrid &g) {
  const unsigned u = __float_as_uint(MH_GRID_BIAS);
  return (u >> 9) * (g.ny * g.nx) + (u >> 10) * g.nx + (u >> 10);
}

// Four samples of the search for the next one that may be negative.  True: t
// is one, and tl the sample before it.  Most words are zero, so the cells'
// bits are looked at only when one of the four is not.
__device__ __forceinline__ bool search_step(const RayGrid &g, const GridRay &r, unsigned base, float step, float &t,
                                            float &tl) {
  const float t1 = t + step, t2 = t1 + step, t3 = t2 + step;
  const GridCell c0 = grid_cell(r, t), c1 = grid_cell(r, t1), c2 = grid_cell(r, t2), c3 = grid_cell(r, t3);
  const unsigned w0 = grid_word(g, c0, base), w1 = grid_word(g, c1, base), w2 = grid_word(g, c2, base),
                 w3 = grid_word(g, c3, base);
  if (w0 | w1 | w2 | w3) {
    if (cell_bit(w0, c0)) return true;
    if (cell_bit(w1, c1)) {
      tl = t, t = t1;
      return true;
    }
    if (cell_bit(w2, c2)) {
      tl = t1, t = t2;
      return true;
    }
    if (cell_bit(w3, c3)) {
      tl = t2, t = t3;
      return true;
    }
  }
  tl = t3;
  t = t3 + step;
  return false;
}

// 4 G samples of it at once, four a lane, for the group's ray (active:
// t is to move).  All 32 lanes call it.
//
// The march's t is t + step rounded, again and again.  While t keeps its
// exponent every step adds the same multiple d of its last place, unless step
// lies halfway between two multiples and they alternate; two equal steps rule
// that out.  Then t after n steps is t + n d, exactly, and a lane gets its
// samples with one multiply-add; else it takes the steps.
template <int G>
__device__ __forceinline__ bool search_step(const RayGrid &g, const GridRay &r, unsigned base, const GroupNbhd<G> &p,
                                            float step, bool active, float &t, float &tl) {
  float s0 = t, before = tl;  // this lane's first sample and the one before it
  const float t1 = t + step, d = t1 - t, end = fmaf((float)(4 * G), d, t);
  if (t1 + step - t1 == d && (__float_as_uint(t) ^ __float_as_uint(end)) < 0x800000u) {
    s0 = fmaf((float)(4 * p.j), d, t);
    if (p.j) before = fmaf((float)(4 * p.j - 1), d, t);
  } else {
    for (int i = 0; i < 4 * p.j; ++i) before = s0, s0 += step;
  }
  // where the ray goes on and the sample before, as far as this lane knows
  float next = s0, last = before;
  const bool mine = search_step(g, r, base, step, next, last);
  const unsigned hits = p.of(__ballot_sync(0xffffffffu, mine));
  const int from = p.base + (hits ? __ffs(hits) - 1 : G - 1);
  next = __shfl_sync(0xffffffffu, next, from);
  last = __shfl_sync(0xffffffffu, last, from);
  if (active) t = next, tl = last;
  return hits != 0u;
}

// The sample n steps before t of a march through `first`, or `first` if there
// are fewer between them.
__device__ __forceinline__ float step_back(float first, float t, float step, int n) {
  float a = first, b = first;
  while (a < t && n > 0) a += step, --n;
  while (a < t) a += step, b += step;
  return b;
}

// The first sample from x on, before `end`, whose first corner's block exists.
// The dense array is read four samples at a time.
__device__ __forceinline__ float skip_missing(const Dev &d, const DenseNbhd &, F3 cam, F3 wd, float step, float x,
                                              float end) {
  const RayGrid &g = d.grid;
  while (x < end) {
    float q = x;
    bool there[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const Corners k = corners_at(d.p, f3(cam.x + q * wd.x, cam.y + q * wd.y, cam.z + q * wd.z));
      const unsigned bx = min((unsigned)((k.v0x >> 3) - g.bx), g.bnx - 1u),
                     by = min((unsigned)((k.v0y >> 3) - g.by), g.bny - 1u),
                     bz = min((unsigned)((k.v0z >> 3) - g.bz), g.bnz - 1u);
      there[i] = (__ldg(g.blocks + (bz * g.bny + by) * g.bnx + bx) ^ g.tag) < 0x1000000u;
      q += step;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (there[i] || !(x < end)) return x;
      x += step;
    }
  }
  return x;
}
// Without it, a known missing block is left at one go.
__device__ __forceinline__ float skip_missing(const Dev &d, const Nbhd &c, F3 cam, F3 wd, float step, float x,
                                              float end) {
  if (!(c.miss & 1u)) return x;
  const F3 iwd = f3(wd.x != 0.0f ? 1.0f / wd.x : 0.0f, wd.y != 0.0f ? 1.0f / wd.y : 0.0f,
                    wd.z != 0.0f ? 1.0f / wd.z : 0.0f);
  float lo, hi;
  block_interval(d.p, c.bx, c.by, c.bz, cam, wd, iwd, lo, hi);
  while (x > lo && x < hi && x < end) x += step;
  return x;
}

// A sample a lane at a time; c.lanes scan together.
template <int G>
__device__ __forceinline__ float skip_missing(const Dev &d, const GroupNbhd<G> &c, F3 cam, F3 wd, float step, float x,
                                              float end) {
  const RayGrid &g = d.grid;
  while (true) {
    float q = x, next = x;
#pragma unroll
    for (int i = 0; i < G; ++i) {
      if (i == c.j) q = next;
      next += step;
    }
    const Corners k = corners_at(d.p, f3(cam.x + q * wd.x, cam.y + q * wd.y, cam.z + q * wd.z));
    const unsigned bx = min((unsigned)((k.v0x >> 3) - g.bx), g.bnx - 1u),
                   by = min((unsigned)((k.v0y >> 3) - g.by), g.bny - 1u),
                   bz = min((unsigned)((k.v0z >> 3) - g.bz), g.bnz - 1u);
    const bool stop = !(q < end) || (__ldg(g.blocks + (bz * g.bny + by) * g.bnx + bx) ^ g.tag) < 0x1000000u;
    const unsigned hits = c.of(__ballot_sync(c.lanes, stop));
    const float at = __shfl_sync(c.lanes, q, c.base + (hits ? __ffs(hits) - 1 : 0));
    if (__all_sync(c.lanes, hits != 0u)) return at;
    x = hits ? at : next;  // the groups go on together
  }
}

}  // namespace

// What one ray's march found: whether a hit was accepted, the two march
// samples around the zero crossing, which end each regula-falsi step
// replaced, the last regula-falsi point and, when asked, the spatial
// gradient at that point (g_ok false if a gradient sample was invalid).
struct March {
  bool hit, g_ok;
  float t0, t1, m;
  int side;  // bit k: regula-falsi step k replaced the left end
  F3 g;
};

// RayCaster::CastKernel's march (visualization/ray_caster.cu:62-150) for the
// ray cam + t * wd, t from t_min while t < t_max, with the exact skips
// described above; spacing > 0 also evaluates GetSpatialSDFGradient at the hit
// with central differences `spacing` voxels either side (spatial_query.h:68-97
// uses 0.5).  All 32 lanes of a warp call it, with their group's ray where lanes
// share one (active: there is a ray): it keeps them together, searching in one
// loop and evaluating, whatever their phases, in one inlined sampler, so that
// neither waits for lanes of the other kind that left the loop at another place.
template <class N>
__device__ __forceinline__ March ray_march(const Dev &d, bool active, F3 cam, F3 wd, float t_min, float t_max,
                                           float spacing) {
  const DevParams &p = d.p;
  const float vs = p.voxel_size;
  const float step = p.raycast_step;
  const float NI = -__int_as_float(0x7f800000);
  enum { PH_DONE, PH_SEARCH, PH_MARCH, PH_PREV, PH_SCAN, PH_REFINE };
  March out;
  out.hit = false, out.g_ok = false, out.t0 = out.t1 = out.m = 0.0f, out.side = 0;
  out.g = f3(0.0f, 0.0f, 0.0f);
  N c;
  c.init();
  const bool use_grid = d.grid.bits != nullptr;
  const GridRay gr = grid_ray(d.grid, cam, wd);
  const unsigned gbase = grid_base(d.grid);
  int phase = active ? PH_SEARCH : PH_DONE, k = 0, side = 0;
  // last evaluated valid sample (prev_t = -inf: none) and the sample before t
  // (tl = -inf: t is the first)
  float prev_t = NI, prev_sdf = 0.0f, tl = NI;
  float t = t_min, cur_s = 0.0f, m = 0.0f;
  // PH_PREV, PH_SCAN: the sample to look at (x) and the last valid one found (l);
  // PH_REFINE: the interval's ends and values
  float x = 0.0f, l = 0.0f, r = 0.0f, ls = 0.0f, rs = 0.0f;
#pragma unroll 1
  while (true) {
    unsigned searching;
#pragma unroll 1
    while ((searching = __ballot_sync(0xffffffffu, phase == PH_SEARCH)) != 0u &&
           __popc(__ballot_sync(0xffffffffu, phase > PH_SEARCH)) < (N::LANES > 1 ? RC_GROUP_WAIT : RC_WAIT)) {
      bool found = false;
      if constexpr (N::LANES > 1) {  // the warp's groups step together
        const bool mine = phase == PH_SEARCH && t < t_max;
        found = search_step(d.grid, gr, gbase, c, step, mine, t, tl) && mine;
      }
      if (phase == PH_SEARCH) {
        if constexpr (N::LANES == 1) found = t < t_max && (!use_grid || search_step(d.grid, gr, gbase, step, t, tl));
        if (!(t < t_max)) phase = PH_DONE;
        else if (found) phase = PH_MARCH;
      }
      __syncwarp();
    }
    if (!searching && !__any_sync(0xffffffffu, phase != PH_DONE)) break;
    if constexpr (N::LANES > 1) c.lanes = __ballot_sync(0xffffffffu, phase > PH_SEARCH);
    if (phase > PH_SEARCH) {
      float tp = phase == PH_MARCH ? t : x;
      if (phase == PH_REFINE) tp = m = l + (ls / (ls - rs)) * (r - l);
      const F3 pos = f3(cam.x + tp * wd.x, cam.y + tp * wd.y, cam.z + tp * wd.z);
      float s = 0.0f;
      const bool valid = nb_sample(d, c, pos, phase != PH_SCAN, s);
      if constexpr (N::LANES > 1) c.lanes = __ballot_sync(c.lanes, phase == PH_SCAN);
      bool refine = false, resume = false;  // start the regula falsi / go on after the negative sample at t
      if (phase == PH_MARCH) {
        if (valid && s < 0.0f && tl != NI && prev_t != tl) {
          // negative after a sample that was not evaluated or is invalid
          cur_s = s, x = tl;
          phase = PH_PREV;
        } else if (valid && s < 0.0f && prev_t == tl && prev_sdf > 0.0f) {
          cur_s = s, l = prev_t, ls = prev_sdf;
          refine = true;
        } else {
          if (valid) prev_sdf = s, prev_t = t;
          tl = t;
          t += step;
          phase = PH_SEARCH;
        }
      } else if (phase == PH_PREV) {
        if (valid) {
          // a crossing needs a positive sample before (ray_caster.cu:87-88)
          if (s > 0.0f) l = x, ls = s, refine = true;
          else resume = true;
        } else {
          // invalid: the last valid sample lies further back, after the last
          // evaluated one or the first of the ray.  It is looked for among
          // the last 8 samples, then the last 64, then all.
          const float first = prev_t != NI ? prev_t : t_min;
          l = NI, k = 0;
          x = step_back(first, tl, step, 8);
          if (x < tl) phase = PH_SCAN;
          else resume = true;
        }
      } else if (phase == PH_SCAN) {
        if (valid) l = x;
        x = skip_missing(d, c, cam, wd, step, x + step, tl);
        if (!(x < tl)) {
          const float first = prev_t != NI ? prev_t : t_min;
          if (l != NI) {
            x = l;  // valid, so PH_PREV gets its value
            phase = PH_PREV;
          } else if (k < 2 && step_back(first, tl, step, 8) > first) {
            x = k == 0 ? step_back(first, tl, step, 64) : first;
            ++k;
          } else {
            resume = true;
          }
        }
      } else {  // PH_REFINE
        bool last = true, hit = false;
        if (valid) {
          if (ls * s > 0.0f) l = m, ls = s, side |= 1 << k;
          else r = m, rs = s;
          last = ++k == 3;
          hit = last && fabsf(prev_sdf - cur_s) < p.sample_sdf_threshold && fabsf(cur_s) < p.sdf_threshold;
        }
        if (hit) {
          out.hit = true, out.t0 = prev_t, out.t1 = t, out.m = m, out.side = side;
          phase = PH_DONE;
        } else if (last) {
          // BisectionIntersection failed or the sample is not good enough: the
          // march goes on from this sample (ray_caster.cu:119-122)
          resume = true;
        }
      }
      if (refine) {
        prev_t = l, prev_sdf = ls;
        r = t, rs = cur_s, k = 0, side = 0;
        phase = PH_REFINE;
      }
      if (resume) {
        prev_sdf = cur_s, prev_t = t, tl = t;
        t += step;
        phase = PH_SEARCH;
      }
    }
    __syncwarp();
  }
  // the gradient's samples, axis by axis, minus side first
  if constexpr (N::LANES > 1) c.lanes = __ballot_sync(0xffffffffu, out.hit && spacing > 0.0f);
  if (out.hit && spacing > 0.0f) {
    const F3 iso = f3(cam.x + out.m * wd.x, cam.y + out.m * wd.y, cam.z + out.m * wd.z);
    const float h = spacing * vs;
    out.g_ok = true;
#pragma unroll 1
    for (k = 0; k < 6; ++k) {
      const float e = (k & 1) ? h : -h;
      const F3 pos = f3(k < 2 ? iso.x + e : iso.x, (k >> 1) == 1 ? iso.y + e : iso.y, k >= 4 ? iso.z + e : iso.z);
      float s = 0.0f;
      if (!nb_sample(d, c, pos, true, s)) out.g_ok = false;
      if (!(k & 1)) {
        ls = s;
      } else {
        const float gi = (s - ls) / (vs * (2.0f * spacing));
        if (k == 1) out.g.x = gi;
        else if (k == 3) out.g.y = gi;
        else out.g.z = gi;
      }
    }
  }
  return out;
}

template <class N, int TX, int TY>
__device__ __forceinline__ void raycast_body(const Dev &d, int tile_x, int tile_y, float *out_depth, float4 *out_vert, float4 *out_norm) {
  __shared__ float sm[32];
  const int tid = threadIdx.x + threadIdx.y * blockDim.x;
  if (tid < 16) sm[tid] = d.fc->rc_wTc[tid];
  else if (tid < 32) sm[tid] = d.fc->rc_cTw[tid - 16];
  __syncthreads();
  const float *wTc = sm, *cTw = sm + 16;
  const DevParams &p = d.p;
  // a warp covers 8x4 pixels; 2x2 or 4x2 where 8 or 4 lanes share one
  constexpr int WX = N::LANES == 8 ? 2 : N::LANES == 4 ? 4 : 8, WY = 32 / N::LANES / WX;
  const int warp = tid >> 5, ray = (tid & 31) / N::LANES, wx = TX / WX;
  const unsigned x = tile_x * TX + (warp % wx) * WX + ray % WX;
  const unsigned y = tile_y * TY + (warp / wx) * WY + ray / WX;
  const bool inside = x < p.rc_width && y < p.rc_height;
  const size_t pix = (size_t)y * p.rc_width + x;
  const float NI = -__int_as_float(0x7f800000);
  float o_depth = NI;
  float4 o_vert = make_float4(NI, NI, NI, NI), o_norm = make_float4(NI, NI, NI, NI);

  const float rx = ((float)x - p.rc_cx) / p.rc_fx, ry = ((float)y - p.rc_cy) / p.rc_fy;
  const F3 cd = normalize3(f3(1.0f * rx, 1.0f * ry, 1.0f));
  const float t_min = p.min_raycast_depth / cd.z;
  const float t_max = p.max_raycast_depth / cd.z;
  const F3 cam = mul_pt(wTc, f3(0.0f, 0.0f, 0.0f));
  const F3 wd = normalize3(mul_dir(wTc, cd));
  const bool want_normal = p.enable_gradients && out_norm;
  const March mr = ray_march<N>(d, inside, cam, wd, t_min, t_max, want_normal ? 0.5f : 0.0f);
  if (!inside) return;
  if (mr.hit) {
    const float dz = mr.m * cd.z;
    o_depth = dz;
    o_vert = make_float4(dz * rx, dz * ry, dz, 1.0f);
    if (want_normal) {
      const F3 g = mr.g;
      const float len = sqrtf(dot3(g, g));
      F3 nn = f3(0.0f, 0.0f, 0.0f);
      if (mr.g_ok && len > 0.0f) nn = f3(g.x / len, g.y / len, g.z / len);
      nn = f3(-nn.x, -nn.y, -nn.z);
      const F3 nc = mul_dir(cTw, nn);
      o_norm = make_float4(nc.x, nc.y, nc.z, 1.0f);
    }
  }
  // a group's lanes write an image each
  const int lane = tid & (N::LANES - 1);
  if (out_depth && (N::LANES == 1 || lane == 0)) out_depth[pix] = o_depth;
  if (out_vert && (N::LANES == 1 || lane == 1)) out_vert[pix] = o_vert;
  if (out_norm && (N::LANES == 1 || lane == 2)) out_norm[pix] = o_norm;
}
template <class N>
__global__ void __launch_bounds__(RC_TX *RC_TY, 12) k_raycast(Dev d, float *out_depth, float4 *out_vert, float4 *out_norm) {
  raycast_body<N, RC_TX, RC_TY>(d, blockIdx.x, blockIdx.y, out_depth, out_vert, out_norm);
}
template <int G>
__global__ void __launch_bounds__(RC_GROUP_THREADS, 4) k_raycast_group(Dev d, float *out_depth, float4 *out_vert,
                                                                       float4 *out_norm) {
  raycast_body<GroupNbhd<G>, 32 / G, RC_GROUP_THREADS / 32>(d, blockIdx.x, blockIdx.y, out_depth, out_vert, out_norm);
}
// batched raycast over the scenes' concatenated TX x TY tiles; the tile shape
// is an autotuned choice (the scene table's ray_tile0 follows it)
template <int TX, int TY>
__global__ void __launch_bounds__(TX *TY, 768 / (TX * TY)) k_raycast_b(const Scene *t, int n, int total) {
  each_tile(t, n, total, &Scene::ray_tile0, [&](const Scene &c, int lt) {
    const int tw = (c.d.p.rc_width + TX - 1) / TX;
    if (c.d.grid.blocks) raycast_body<DenseNbhd, TX, TY>(c.d, lt % tw, lt / tw, c.ray_depth, c.ray_vert, c.ray_norm);
    else raycast_body<Nbhd, TX, TY>(c.d, lt % tw, lt / tw, c.ray_depth, c.ray_vert, c.ray_norm);
  });
}

// tile shapes the batch autotuner chooses from
static const int kRayTiles[][2] = {{16, 8}, {8, 8}, {32, 4}};
int ray_tile_shapes() { return 3; }
void ray_tile_shape(int i, int &tx, int &ty) {
  tx = kRayTiles[i][0];
  ty = kRayTiles[i][1];
}

int launch_raycast_batch(const Scene *t, int n, int total, int shape, cudaStream_t s) {
  const int grid = std::max(1, std::min(total, mh_sm_count() * 16));
  switch (shape) {
    case 1: k_raycast_b<8, 8><<<grid, dim3(8, 8), 0, s>>>(t, n, total); break;
    case 2: k_raycast_b<32, 4><<<grid, dim3(32, 4), 0, s>>>(t, n, total); break;
    default: k_raycast_b<16, 8><<<grid, dim3(16, 8), 0, s>>>(t, n, total); break;
  }
  mh_count_launches(1);
  return cudaGetLastError() == cudaSuccess ? MH_OK : MH_ERR_CUDA;
}

// ------------------------------------------------------------------ the view's grid
// Cells are marked from the blocks' masks of 2^3 voxel groups.  With a reach of
// 1, a sample in cell i of U voxels reads voxels U i .. U i + U + 1 (the march's
// shift and rounding included, see ray_grid_of), so the group that starts at voxel
// 2 S marks the 2-voxel cells S and S - 1.  A block's 64 groups give the 64 bits
// of its own cells and of the last layers of the seven blocks below it on each
// axis; with U = 2 those are two words each, set with an atomic where not 0.
// Bound by the scattered writes and atomics; 640x480, 4 mm, 461 k blocks, half
// of them marked: 41 us (cold), of 390 us for the raycast with it.  Cells of 4
// voxels cost less here (14 us) and more in the march, which then evaluates 6.4
// samples a ray instead of 3.4 (507 us in all).  kFar: a reach above 1, marked cell
// by cell.
template <bool kFar> __device__ __forceinline__ void ray_grid_body(const Dev &d, Share sh) {
  const RayGrid &g = d.grid;
  if (!g.bits) return;
  const int n = *reinterpret_cast<volatile int *>(&d.ctr->high_water);
  const int nx = (int)g.nx, ny = (int)g.ny, nz = (int)g.nz;
  for (int i = sh.first * blockDim.x + threadIdx.x; i < n; i += sh.stride * blockDim.x) {
    const int4 b = d.block_pos[i];
    if (!b.w) continue;
    if (g.blocks) {
      const unsigned x = (unsigned)(b.x - g.bx), y = (unsigned)(b.y - g.by), z = (unsigned)(b.z - g.bz);
      if (x < g.bnx && y < g.bny && z < g.bnz) g.blocks[(z * g.bny + y) * g.bnx + x] = g.tag | (unsigned)i;
    }
    const unsigned long long m = __ldg(d.neg + i);
    if (!m) continue;
    if (kFar) {
      // large cells, or far from the origin: all cells from the reach below the
      // block's first marked group to its last, on each axis; at most 27 (U = 4)
      unsigned p = (unsigned)(m | m >> 32);
      p = (p | p >> 16) & 0xffffu;  // x and y
      const unsigned xs = (p | p >> 4 | p >> 8 | p >> 12) & 15u;
      unsigned ys = p | p >> 1;
      ys |= ys >> 2;
      ys = (ys & 1u) | (ys >> 3 & 2u) | (ys >> 6 & 4u) | (ys >> 9 & 8u);
      const unsigned zs = (m & 0xffffull ? 1u : 0u) | (m >> 16 & 0xffffull ? 2u : 0u) | (m >> 32 & 0xffffull ? 4u : 0u) |
                          (m >> 48 ? 8u : 0u);
      const int x0 = ((4 * b.x + __ffs(xs) - 1 - g.reach) >> g.shift) - g.cx, x1 = ((4 * b.x + 31 - __clz(xs)) >> g.shift) - g.cx;
      const int y0 = ((4 * b.y + __ffs(ys) - 1 - g.reach) >> g.shift) - g.cy, y1 = ((4 * b.y + 31 - __clz(ys)) >> g.shift) - g.cy;
      const int z0 = ((4 * b.z + __ffs(zs) - 1 - g.reach) >> g.shift) - g.cz, z1 = ((4 * b.z + 31 - __clz(zs)) >> g.shift) - g.cz;
      for (int z = max(z0, 0); z <= min(z1, 2 * nz - 1); ++z)
        for (int y = max(y0, 0); y <= min(y1, 4 * ny - 1); ++y)
          for (int x = max(x0, 0); x <= min(x1, 4 * nx - 1); ++x)
            atomicOr(g.bits + ((size_t)(z >> 1) * ny + (y >> 2)) * nx + (x >> 2), 1u << ((x & 3) | (y & 3) << 2 | (z & 1) << 4));
      continue;
    }
#pragma unroll 1
    for (int j = 0; j < 8; ++j) {
      // block b - j: along an axis of j, group 0 marks cell 3 of the block
      // below; along the others group S marks S and S - 1
      unsigned long long v = m;
      v = (j & 1) ? (v & 0x1111111111111111ull) << 3 : v | ((v >> 1) & 0x7777777777777777ull);
      v = (j & 2) ? (v & 0x000f000f000f000full) << 12 : v | ((v >> 4) & 0x0fff0fff0fff0fffull);
      v = (j & 4) ? v << 48 : v | (v >> 16);
      if (!v) continue;
      const int X = 4 * (b.x - (j & 1)), Y = 4 * (b.y - ((j >> 1) & 1)), Z = 4 * (b.z - (j >> 2));  // 2-voxel cells
      if (g.shift == 0) {
        const int x = (X - g.cx) >> 2, y = (Y - g.cy) >> 2, z = (Z - g.cz) >> 1;
        if ((unsigned)x >= (unsigned)nx || (unsigned)y >= (unsigned)ny) continue;
        unsigned *w = g.bits + ((size_t)z * ny + y) * nx + x;
        if ((unsigned)v && (unsigned)z < (unsigned)nz) atomicOr(w, (unsigned)v);
        if ((unsigned)(v >> 32) && (unsigned)(z + 1) < (unsigned)nz) atomicOr(w + (size_t)ny * nx, (unsigned)(v >> 32));
      } else {
        while (v) {
          const int k = __ffsll((long long)v) - 1;
          v &= v - 1;
          const int x = ((X + (k & 3)) >> g.shift) - g.cx, y = ((Y + ((k >> 2) & 3)) >> g.shift) - g.cy,
                    z = ((Z + (k >> 4)) >> g.shift) - g.cz;
          if ((unsigned)x >= 4u * nx || (unsigned)y >= 4u * ny || (unsigned)z >= 2u * nz) continue;
          atomicOr(g.bits + ((size_t)(z >> 1) * ny + (y >> 2)) * nx + (x >> 2),
                   1u << ((x & 3) | (y & 3) << 2 | (z & 1) << 4));
        }
      }
    }
  }
}
template <bool kFar> __global__ void __launch_bounds__(256) k_ray_grid(Dev d) { ray_grid_body<kFar>(d, whole_grid()); }
__global__ void __launch_bounds__(256, 5) k_ray_grid_b(const Scene *t, int n) {
  each_scene(t, n, 256, [&](const Scene &c) { return c.d.grid.bits ? count_of(c.d, &Counters::high_water) : 0; },
             [&](const Scene &c, Share sh) {
    if (c.d.grid.reach > 1) ray_grid_body<true>(c.d, sh);
    else ray_grid_body<false>(c.d, sh);
  });
}
__global__ void __launch_bounds__(256) k_ray_grid_clear_b(const Scene *t, int n) {
  each_scene(t, n, 256, [&](const Scene &c) { return c.d.grid.bits ? (int)max(c.d.grid.words, c.d.grid.clear) : 0; },
             [&](const Scene &c, Share sh) {
    for (unsigned i = sh.first * blockDim.x + threadIdx.x; i < c.d.grid.words; i += sh.stride * blockDim.x)
      c.d.grid.bits[i] = 0u;
    for (unsigned i = sh.first * blockDim.x + threadIdx.x; i < c.d.grid.clear; i += sh.stride * blockDim.x)
      c.d.grid.blocks[i] = 0u;
  });
}

static int fill_ray_grid(const Dev &d, cudaStream_t s) {
  if (!d.grid.bits || d.grid.filled) return MH_OK;
  MH_CUDA_TRY(cudaMemsetAsync(d.grid.bits, 0, sizeof(unsigned) * (size_t)d.grid.words, s));
  if (d.grid.clear)
    MH_CUDA_TRY(cudaMemsetAsync(d.grid.blocks, 0, sizeof(unsigned) * (size_t)d.grid.clear, s));
  if (d.grid.reach > 1) k_ray_grid<true><<<mh_sm_count() * 8, 256, 0, s>>>(d);
  else k_ray_grid<false><<<mh_sm_count() * 8, 256, 0, s>>>(d);
  mh_count_launches(1);
  return cudaGetLastError() == cudaSuccess ? MH_OK : MH_ERR_CUDA;
}
int launch_batch_ray_grid(const Scene *t, int n, cudaStream_t s) {
  k_ray_grid_clear_b<<<mh_sm_count() * 8, 256, 0, s>>>(t, n);
  k_ray_grid_b<<<mh_sm_count() * 8, 256, 0, s>>>(t, n);
  mh_count_launches(2);
  return cudaGetLastError() == cudaSuccess ? MH_OK : MH_ERR_CUDA;
}

// A raycast that a graph replays: the launches are recorded once, the pose and
// the map are those of each replay, so the grid has to be made on the device.  One
// thread writes it, with the scene, into a table of one entry, and the batch's
// kernels run over that table.
__global__ void k_ray_scene(Scene scene, mh_params P, RayGridBuf b, Scene *table) {
  scene.d.grid = ray_grid_replayed(P, scene.d.fc->rc_wTc, b);
  *table = scene;
}
int launch_raycast_replayed(const Dev &d, const mh_params &P, const RayGridBuf &b, Scene *table, float *depth,
                            float *vert4, float *norm4, cudaStream_t s) {
  Scene scene{};
  scene.d = d;
  scene.ray_depth = depth;
  scene.ray_vert = reinterpret_cast<float4 *>(vert4);
  scene.ray_norm = reinterpret_cast<float4 *>(norm4);
  scene.active = 1;
  k_ray_scene<<<1, 1, 0, s>>>(scene, P, b, table);
  mh_count_launches(1);
  const int r = launch_batch_ray_grid(table, 1, s);
  if (r != MH_OK) return r;
  int tx, ty;
  ray_tile_shape(0, tx, ty);
  return launch_raycast_batch(table, 1, ((P.rc_width + tx - 1) / tx) * ((P.rc_height + ty - 1) / ty), 0, s);
}

// number of nonzero bytes of flags[0, n) added to *out
__global__ void k_count_flags(const uint8_t *flags, int n, int *out) {
  int c = 0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) c += flags[i] != 0;
  c = __reduce_add_sync(0xffffffffu, c);
  if ((threadIdx.x & 31) == 0 && c) atomicAdd(out, c);
}
int launch_count_flags(const uint8_t *flags, int n, int *out, cudaStream_t s) {
  k_count_flags<<<std::max(1, std::min((n + 255) / 256, mh_sm_count() * 8)), 256, 0, s>>>(flags, n, out);
  mh_count_launches(1);
  return cudaGetLastError() == cudaSuccess ? MH_OK : MH_ERR_CUDA;
}

// A ray is a chain of dependent steps of about 1000 cycles each.  Lanes that
// share one search 4 G samples at once and evaluate with 8 / G corners each,
// which shortens the chain but takes more instructions in all (the position's
// and the state's on every lane), so it is for images that cannot fill the
// chip: 152 SMs x 768 lanes are 117 k.  Views of a 24-frame map, us, with
// 1 / 4 / 8 lanes a ray: 100x75, 8 mm: 190 / 146 / 110; 160x120, 4 mm: 356 /
// 230 / 188; 240x180, 6 mm: 202 / 156 / 129; 320x240, 4 mm: 475 / 350 / 332;
// 320x240, 8 mm: 161 / 135 / 146; 400x300, 6 mm: 205 / 200 / 226; 450x340, 5
// mm: 243 / 242 / 276; 640x480, 6 mm: 263 / 346 / 442.  Needs the dense array.
int launch_raycast(const Dev &d, float *depth, float *vert4, float *norm4, cudaStream_t s) {
  const int r = fill_ray_grid(d, s);
  if (r != MH_OK) return r;
  const size_t pixels = (size_t)d.p.rc_width * d.p.rc_height;
  const int lanes = !d.grid.bits || !d.grid.blocks || pixels > RC_PIXELS4 ? 1 : pixels > RC_PIXELS8 ? 4 : 8;
  const unsigned tx = lanes > 1 ? 32 / lanes : RC_TX, ty = lanes > 1 ? RC_GROUP_THREADS / 32 : RC_TY;
  const dim3 blk(RC_TX, RC_TY), grid((d.p.rc_width + tx - 1) / tx, (d.p.rc_height + ty - 1) / ty);
  float4 *v4 = reinterpret_cast<float4 *>(vert4), *n4 = reinterpret_cast<float4 *>(norm4);
  if (lanes == 8) k_raycast_group<8><<<grid, RC_GROUP_THREADS, 0, s>>>(d, depth, v4, n4);
  else if (lanes == 4) k_raycast_group<4><<<grid, RC_GROUP_THREADS, 0, s>>>(d, depth, v4, n4);
  else if (d.grid.blocks) k_raycast<DenseNbhd><<<grid, blk, 0, s>>>(d, depth, v4, n4);
  else k_raycast<Nbhd><<<grid, blk, 0, s>>>(d, depth, v4, n4);
  mh_count_launches(1);
  return cudaGetLastError() == cudaSuccess ? MH_OK : MH_ERR_CUDA;
}

// ------------------------------------------------------------------ backward
// Reverse-mode derivative of the raycast (no reference counterpart; the
// reference's raycaster is forward only).  For each pixel the march is run
// again with the forward's own code, so every discrete decision -- which
// samples are valid, where the sign changes, which end each regula-falsi step
// replaces -- is the forward's.  With those fixed, the rendered depth
// D = m * cd.z is a smooth function of
//   * the voxel sdf values (each sample is a trilinear sum, linear in them),
//   * the camera pose (every sample sits at cam + t * wd),
// through the two bracketing samples and the three regula-falsi steps
// m = l + ls / (ls - rs) * (r - l); the normal adds six gradient samples
// around the hit and a normalisation.  The kernel propagates adjoints back
// through exactly these steps, so its result is the derivative of what the
// forward computes (what central differences of the forward measure), not
// of an idealised surface.  Pose derivatives are for a left perturbation
// wTc <- exp(xi) wTc, xi = (translation v, rotation w), to first order:
// cam += w x cam + v, wd += w x wd, and the camera-frame normal R^T n
// changes by R^T (n x w).
namespace {

// a sample with what the backward needs: value (bit-identical to
// nb_sample's), spatial gradient, and the eight corners with their weights
struct SampleD {
  float s;
  F3 g;
  int ptr[8], li[8];
  float w[8];
};

template <class N> __device__ __noinline__ bool ray_sample_d(const Dev &d, N &c, F3 pos, SampleD &o) {
  const float vs = d.p.voxel_size;
  const Corners k = corners_at(d.p, pos);
  if (!blocks_at(d, c, k, o.ptr)) return false;
  const float rx = k.rx, ry = k.ry, rz = k.rz;
  const float w0x = 1.0f - rx, w0y = 1.0f - ry, w0z = 1.0f - rz;
  float s = 0.0f, gx = 0.0f, gy = 0.0f, gz = 0.0f;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int mx = (i & 4) > 0, my = (i & 2) > 0, mz = (i & 1) > 0;
    const float wx = mx ? rx : w0x, wy = my ? ry : w0y, wz = mz ? rz : w0z;
    const float w = wx * wy * wz;
    const int li = ((mx ? k.v1x : k.v0x) & 7) + ((my ? k.v1y : k.v0y) & 7) * 8 + ((mz ? k.v1z : k.v0z) & 7) * 64;
    const float v = __ldg(d.sdf + (size_t)o.ptr[i] * MH_BLOCK_VOXELS + li);
    s += w * v;
    // d(weight)/d(position): the fractions move at 1/voxel per metre
    gx += (mx ? 1.0f : -1.0f) * wy * wz * v;
    gy += (my ? 1.0f : -1.0f) * wx * wz * v;
    gz += (mz ? 1.0f : -1.0f) * wx * wy * v;
    o.li[i] = li;
    o.w[i] = w;
  }
  o.s = s;
  o.g = f3(gx / vs, gy / vs, gz / vs);
  return true;
}

struct RayTrace {
  bool hit;
  float t0, t1;  // the bracketing samples
  int side;      // bit k: regula-falsi step k replaced the left end
};

__device__ __forceinline__ F3 cross3(F3 a, F3 b) {
  return f3(a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x);
}
__device__ __forceinline__ void scatter(float *grad, const SampleD &o, float a) {
  if (!grad || a == 0.0f) return;
#pragma unroll
  for (int i = 0; i < 8; ++i) atomicAdd(grad + (size_t)o.ptr[i] * MH_BLOCK_VOXELS + o.li[i], a * o.w[i]);
}

// Adjoints of one pixel's depth (aD) and camera-frame normal (aN): voxel
// adjoints go to grad (may be null), pose adjoints to (av, aw).  Returns
// false when the hit cannot be re-evaluated.
template <class N>
__device__ bool pixel_backward(const Dev &d, N &c, const float *cTw, F3 cam, F3 wd, float cdz,
                               const RayTrace &tr, float aD, F3 aN, bool normals, float *grad, F3 &av, F3 &aw) {
  const float vs = d.p.voxel_size;
  F3 a_cam = f3(0.0f, 0.0f, 0.0f), a_wd = f3(0.0f, 0.0f, 0.0f), a_w_extra = f3(0.0f, 0.0f, 0.0f);
  // forward values of the regula falsi, in the forward's operation order
  SampleD S0, S1, Sm[3];
  if (!ray_sample_d(d, c, f3(cam.x + tr.t0 * wd.x, cam.y + tr.t0 * wd.y, cam.z + tr.t0 * wd.z), S0)) return false;
  if (!ray_sample_d(d, c, f3(cam.x + tr.t1 * wd.x, cam.y + tr.t1 * wd.y, cam.z + tr.t1 * wd.z), S1)) return false;
  float L[3], Rr[3], LS[3], RS[3], M[3];
  float l = tr.t0, r = tr.t1, ls = S0.s, rs = S1.s;
  for (int k = 0; k < 3; ++k) {
    L[k] = l, Rr[k] = r, LS[k] = ls, RS[k] = rs;
    const float m = l + (ls / (ls - rs)) * (r - l);
    M[k] = m;
    if (!ray_sample_d(d, c, f3(cam.x + m * wd.x, cam.y + m * wd.y, cam.z + m * wd.z), Sm[k])) return false;
    if ((tr.side >> k) & 1) l = m, ls = Sm[k].s;
    else r = m, rs = Sm[k].s;
  }
  const float m = M[2];
  float am = aD * cdz;
  if (normals && (aN.x != 0.0f || aN.y != 0.0f || aN.z != 0.0f)) {
    const F3 iso = f3(cam.x + m * wd.x, cam.y + m * wd.y, cam.z + m * wd.z);
    const float h = 0.5f * vs;
    SampleD up[3], dn[3];
    bool ok = true;
    for (int i = 0; i < 3 && ok; ++i) {
      F3 dm = f3(iso.x - (i == 0 ? h : 0.0f), iso.y - (i == 1 ? h : 0.0f), iso.z - (i == 2 ? h : 0.0f));
      F3 dp = f3(iso.x + (i == 0 ? h : 0.0f), iso.y + (i == 1 ? h : 0.0f), iso.z + (i == 2 ? h : 0.0f));
      ok = ray_sample_d(d, c, dm, dn[i]) && ray_sample_d(d, c, dp, up[i]);
    }
    const F3 g = f3((up[0].s - dn[0].s) / vs, (up[1].s - dn[1].s) / vs, (up[2].s - dn[2].s) / vs);
    const float len = sqrtf(dot3(g, g));
    if (ok && len > 0.0f) {
      const F3 u = f3(g.x / len, g.y / len, g.z / len);
      const F3 nn = f3(-u.x, -u.y, -u.z);
      // nc = Rc nn with Rc the rotation of cTw: a_nn = Rc^T aN
      const F3 a_nn = f3(cTw[0] * aN.x + cTw[4] * aN.y + cTw[8] * aN.z, cTw[1] * aN.x + cTw[5] * aN.y + cTw[9] * aN.z,
                         cTw[2] * aN.x + cTw[6] * aN.y + cTw[10] * aN.z);
      a_w_extra = cross3(a_nn, nn);
      const F3 a_u = f3(-a_nn.x, -a_nn.y, -a_nn.z);
      const float ua = dot3(u, a_u);
      const float ag[3] = {(a_u.x - u.x * ua) / len, (a_u.y - u.y * ua) / len, (a_u.z - u.z * ua) / len};
      F3 a_iso = f3(0.0f, 0.0f, 0.0f);
      for (int i = 0; i < 3; ++i) {
        const float ap = ag[i] / vs, an = -ag[i] / vs;
        scatter(grad, up[i], ap);
        scatter(grad, dn[i], an);
        a_iso = f3(a_iso.x + ap * up[i].g.x + an * dn[i].g.x, a_iso.y + ap * up[i].g.y + an * dn[i].g.y,
                   a_iso.z + ap * up[i].g.z + an * dn[i].g.z);
      }
      a_cam = f3(a_cam.x + a_iso.x, a_cam.y + a_iso.y, a_cam.z + a_iso.z);
      a_wd = f3(a_wd.x + m * a_iso.x, a_wd.y + m * a_iso.y, a_wd.z + m * a_iso.z);
      am += dot3(a_iso, wd);
    }
  }
  // regula falsi, last step first; (al, ar, als, ars) are the adjoints of
  // the state after step k
  float al = 0.0f, ar = 0.0f, als = 0.0f, ars = 0.0f;
  for (int k = 2; k >= 0; --k) {
    const bool left = (tr.side >> k) & 1;
    float a_mk = (k == 2 ? am : 0.0f) + (left ? al : ar);
    const float a_ms = left ? als : ars;
    if (left) al = 0.0f, als = 0.0f;
    else ar = 0.0f, ars = 0.0f;
    // ms_k = S(cam + m_k wd)
    scatter(grad, Sm[k], a_ms);
    const F3 ap = f3(a_ms * Sm[k].g.x, a_ms * Sm[k].g.y, a_ms * Sm[k].g.z);
    a_cam = f3(a_cam.x + ap.x, a_cam.y + ap.y, a_cam.z + ap.z);
    a_wd = f3(a_wd.x + M[k] * ap.x, a_wd.y + M[k] * ap.y, a_wd.z + M[k] * ap.z);
    a_mk += dot3(ap, wd);
    // m_k = l + q (r - l), q = ls / (ls - rs)
    const float den = LS[k] - RS[k], q = LS[k] / den, span = Rr[k] - L[k];
    al += a_mk * (1.0f - q);
    ar += a_mk * q;
    als += a_mk * span * (-RS[k]) / (den * den);
    ars += a_mk * span * LS[k] / (den * den);
  }
  // the bracketing samples sit at fixed t
  scatter(grad, S0, als);
  scatter(grad, S1, ars);
  const F3 p0 = f3(als * S0.g.x, als * S0.g.y, als * S0.g.z), p1 = f3(ars * S1.g.x, ars * S1.g.y, ars * S1.g.z);
  a_cam = f3(a_cam.x + p0.x + p1.x, a_cam.y + p0.y + p1.y, a_cam.z + p0.z + p1.z);
  a_wd = f3(a_wd.x + tr.t0 * p0.x + tr.t1 * p1.x, a_wd.y + tr.t0 * p0.y + tr.t1 * p1.y,
            a_wd.z + tr.t0 * p0.z + tr.t1 * p1.z);
  av = a_cam;
  const F3 c1 = cross3(cam, a_cam), c2 = cross3(wd, a_wd);
  aw = f3(c1.x + c2.x + a_w_extra.x, c1.y + c2.y + a_w_extra.y, c1.z + c2.z + a_w_extra.z);
  return true;
}

// Sum of NV values over the CTA into acc (doubles).  `slot` is the pixel's
// place in the tile, row by row: warps sum 32 consecutive places, so the
// float sums do not depend on which thread had which pixel.
template <int NV> __device__ __forceinline__ void cta_accumulate(float (&v)[NV], int slot, double *acc) {
  __shared__ float val[NV][GR_TX * GR_TY];
  __shared__ float red[NV][GR_TX * GR_TY / 32];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
#pragma unroll
  for (int k = 0; k < NV; ++k) val[k][slot] = v[k];
  __syncthreads();
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    float x = val[k][tid];
    for (int o = 16; o; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    if (lane == 0) red[k][wid] = x;
  }
  __syncthreads();
  if (tid < NV) {
    double s = 0.0;
    for (int w = 0; w < GR_TX * GR_TY / 32; ++w) s += red[tid][w];
    atomicAdd(acc + tid, s);
  }
}

}  // namespace

// mode 0: accumulate dL/dsdf into grad (if given) and dL/dxi into acc[0..5]
//         for L = sum dLdD * depth + dLdN . normal;
// mode 1: Gauss-Newton normal equations of frame-to-model alignment over
//         pixels with a hit, a valid observation and |depth - obs| < max_res:
//         the observed point on the pixel's ray against the tangent plane of
//         the model at the raycast hit (normal from the raycast's gradient),
//         r = n . (p_obs - p_hit), J = [n, p_obs x n] for the left increment;
//         acc = [J^T J upper triangle (21), J^T r (6), sum r^2, count].
template <class N>
__global__ void __launch_bounds__(GR_TX *GR_TY) k_raycast_grad(Dev d, int mode, const float *dLdD, const float4 *dLdN,
                                                              float *grad, const float *obs, float max_res,
                                                              double *acc) {
  __shared__ float sm[32];
  const int tid = threadIdx.x;
  if (tid < 16) sm[tid] = d.fc->rc_wTc[tid];
  else if (tid < 32) sm[tid] = d.fc->rc_cTw[tid - 16];
  __syncthreads();
  const float *wTc = sm, *cTw = sm + 16;
  const DevParams &p = d.p;
  // a warp covers 8x4 pixels
  const int lx = ((tid >> 5) & 1) * 8 + (tid & 7), ly = (tid >> 6) * 4 + ((tid >> 3) & 3), slot = lx + GR_TX * ly;
  const unsigned x = blockIdx.x * GR_TX + lx, y = blockIdx.y * GR_TY + ly;
  F3 av = f3(0.0f, 0.0f, 0.0f), aw = f3(0.0f, 0.0f, 0.0f);
  float res = 0.0f;
  bool used = false, want = false;
  const bool inside = x < p.rc_width && y < p.rc_height;
  const size_t pix = (size_t)y * p.rc_width + x;
  const float rx = ((float)x - p.rc_cx) / p.rc_fx, ry = ((float)y - p.rc_cy) / p.rc_fy;
  const F3 cd = normalize3(f3(1.0f * rx, 1.0f * ry, 1.0f));
  const float t_min = p.min_raycast_depth / cd.z;
  const float t_max = p.max_raycast_depth / cd.z;
  const F3 cam = mul_pt(wTc, f3(0.0f, 0.0f, 0.0f));
  const F3 wd = normalize3(mul_dir(wTc, cd));
  float aD = 0.0f, o = 0.0f;
  F3 aN = f3(0.0f, 0.0f, 0.0f);
  if (inside) {
    if (mode == 0) {
      aD = dLdD ? dLdD[pix] : 0.0f;
      if (dLdN) {
        const float4 q = dLdN[pix];
        aN = f3(q.x, q.y, q.z);
      }
      want = aD != 0.0f || aN.x != 0.0f || aN.y != 0.0f || aN.z != 0.0f;
    } else {
      o = obs[pix];
      want = o > 0.0f && o < 1e30f;
    }
  }
  // the forward's march: mode 1 takes its hit point and the alignment
  // normal, taken 2.5 voxels either side (inside the truncation band):
  // the half-voxel normal of the rendered image follows the noise of the
  // fused surface, and a noisy normal in J shrinks every Gauss-Newton
  // step (measured: from 2-8 cm / 1-2.5 degree starts, 8 iterations
  // reached 15-90 mm with the half-voxel normal and 1-3 mm on three of
  // four with this one)
  const float spacing = mode == 1 ? fminf(2.5f, 0.8f * p.truncation_distance / p.voxel_size) : 0.0f;
  const March mr = ray_march<N>(d, want, cam, wd, t_min, t_max, spacing);
  if (mr.hit) {
    if (mode == 1) {
      const float m = mr.m;
      const F3 pm = f3(cam.x + m * wd.x, cam.y + m * wd.y, cam.z + m * wd.z);
      const F3 g = mr.g;
      if (fabsf(m * cd.z - o) < max_res && mr.g_ok) {
        const float gl = sqrtf(dot3(g, g));
        if (gl > 0.0f) {
          // projective point-to-plane: the observed point on the same ray
          // against the tangent plane of the model at the hit
          const F3 n = f3(g.x / gl, g.y / gl, g.z / gl);
          const float to = o / cd.z;
          const F3 po = f3(cam.x + to * wd.x, cam.y + to * wd.y, cam.z + to * wd.z);
          res = dot3(n, f3(po.x - pm.x, po.y - pm.y, po.z - pm.z));
          av = n;
          aw = cross3(po, n);
          used = true;
        }
      }
    } else {
      // the adjoints re-evaluate the bracketing samples and the three
      // regula-falsi steps along the march's decisions
      N c;
      c.init();
      const RayTrace tr{true, mr.t0, mr.t1, mr.side};
      used = pixel_backward(d, c, cTw, cam, wd, cd.z, tr, aD, aN, dLdN != nullptr, grad, av, aw);
    }
  }
  if (!used) av = f3(0.0f, 0.0f, 0.0f), aw = f3(0.0f, 0.0f, 0.0f), res = 0.0f;
  if (mode == 0) {
    float v[6] = {av.x, av.y, av.z, aw.x, aw.y, aw.z};
    cta_accumulate<6>(v, slot, acc);
  } else {
    const float J[6] = {av.x, av.y, av.z, aw.x, aw.y, aw.z};
    float v[29];
    int k = 0;
#pragma unroll
    for (int i = 0; i < 6; ++i)
#pragma unroll
      for (int j = i; j < 6; ++j) v[k++] = J[i] * J[j];
#pragma unroll
    for (int i = 0; i < 6; ++i) v[21 + i] = J[i] * res;
    v[27] = res * res;
    v[28] = used ? 1.0f : 0.0f;
    cta_accumulate<29>(v, slot, acc);
  }
}

int launch_raycast_grad(const Dev &d, int mode, const float *dLdD, const float *dLdN4, float *grad, const float *obs,
                        float max_res, double *acc, cudaStream_t s) {
  const int r = fill_ray_grid(d, s);
  if (r != MH_OK) return r;
  const int blk = GR_TX * GR_TY;
  dim3 grid((d.p.rc_width + GR_TX - 1) / GR_TX, (d.p.rc_height + GR_TY - 1) / GR_TY);
  const float4 *n4 = reinterpret_cast<const float4 *>(dLdN4);
  if (d.grid.blocks) k_raycast_grad<DenseNbhd><<<grid, blk, 0, s>>>(d, mode, dLdD, n4, grad, obs, max_res, acc);
  else k_raycast_grad<Nbhd><<<grid, blk, 0, s>>>(d, mode, dLdD, n4, grad, obs, max_res, acc);
  mh_count_launches(1);
  return cudaGetLastError() == cudaSuccess ? MH_OK : MH_ERR_CUDA;
}

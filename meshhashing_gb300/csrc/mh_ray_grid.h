// mh_ray_grid.h -- the grid of a raycast's view: where its cells and blocks lie,
// and the buffers that hold them.  mh_raycast.cu fills and reads the grid.  The
// host makes it from the pose that it uploads; a raycast that a graph replays
// makes it on the device from the pose that it finds there.
#pragma once
#include <algorithm>
#include <cmath>

#include "../../include/meshhash.h"

#if defined(__CUDACC__)
#define MH_GRID_HD __host__ __device__
#else
#define MH_GRID_HD
#endif

// The cells of a raycast's view: a bit per cell of U = 2 << shift voxels in
// the view's bounding box.  A word holds 4 x 4 x 2 cells, so with U = 2 two
// words hold a block (mh_raycast.cu).
#define MH_GRID_BIAS 49152.0f        // 1.5 * 2^15: a float there has 8 bits of fraction
#define MH_GRID_GUARD 0.03125f       // cells that a sample is looked up below its position, at least
#define MH_GRID_MAX_WORDS (1u << 25) // 128 MB
#define MH_GRID_REPLAY_TAG 255u      // top byte of blocks written by replayed raycasts
struct RayGrid {
  unsigned *bits;            // null: no grid, every sample is evaluated
  int cx, cy, cz;            // first cell on each axis (a multiple of 4), in cells from the world's origin
  unsigned nx, ny, nz;       // words on each axis
  unsigned words;            // nx * ny * nz
  int shift;                 // U = 2 << shift
  float ox, oy, oz;          // world position of the first cell's lower corner, and the guard above MH_GRID_GUARD
  float inv_cell;            // 1 / (U voxel sizes)
  // The blocks of the same box: entry (z bny + y) bnx + x holds tag | block
  // index for a block that exists, anything with another top byte otherwise.
  unsigned *blocks;          // null: blocks are looked up in the hash table
  int bx, by, bz;            // first block on each axis
  unsigned bnx, bny, bnz;
  unsigned tag;              // this raycast's top byte, 1 .. 254, or MH_GRID_REPLAY_TAG
  unsigned clear;            // entries to clear first (all that the buffer has), 0 where old ones cannot be mistaken
  bool filled;               // the buffers hold this grid already
  short reach;               // a group of 2^3 voxels marks the cells down to that of the reach-th group below it
};

// A volume's buffers for its view's grid, of sizes for any view.  They come with
// the first raycast, since they are up to 384 MB that a volume without raycasts has
// no use for, but with the volume where they are a small part of it.
struct RayGridBuf {
  bool reserved = false;
  unsigned *bits = nullptr, *blocks = nullptr;
  unsigned words = 0, entries = 0;
  unsigned tag = 0;    // of the last grid handed out
  bool dirty = true;   // blocks may hold anything: new memory, or the tags have started over
};

// the view's corner rays at z = 1: x and y ranges, and the longest of them
struct ViewCone {
  double x[2], y[2], len;
  MH_GRID_HD explicit ViewCone(const mh_params &P) {
    x[0] = (0.0 - P.rc_cx) / P.rc_fx, x[1] = ((double)P.rc_width - 1.0 - P.rc_cx) / P.rc_fx;
    y[0] = (0.0 - P.rc_cy) / P.rc_fy, y[1] = ((double)P.rc_height - 1.0 - P.rc_cy) / P.rc_fy;
    const double mx = std::max(std::fabs(x[0]), std::fabs(x[1])), my = std::max(std::fabs(y[0]), std::fabs(y[1]));
    len = std::sqrt(mx * mx + my * my + 1.0);
  }
};

// Enough for the view in any direction: the cube around it.  No blocks at all if
// they would take more than 256 MB.  No more than 128 words of cells a pixel, since
// they are cleared before each raycast (larger cells then), but 256 where there
// are no blocks and a sample costs up to eight hash lookups: a 320x240 view at 1 mm
// takes 2.12 ms with 128 words a pixel and 1.98 ms with 256 (no more with 1024).
inline void ray_grid_sizes(const mh_params &P, RayGridBuf &b) {
  const ViewCone v(P);
  const double wx = v.x[1] - v.x[0], wy = v.y[1] - v.y[0], f = P.max_raycast_depth;
  const double diam = f * std::max(v.len, std::sqrt(wx * wx + wy * wy)) * 1.01;
  const double cells = diam / (2.0 * P.voxel_size) + 24.0, blocks = diam / (8.0 * P.voxel_size) + 8.0;
  const double entries = blocks * blocks * blocks;
  b.entries = entries <= 67108864.0 && P.value_capacity <= (1u << 24) ? (unsigned)entries : 0u;
  const double words = std::min(cells / 4.0 * (cells / 4.0) * (cells / 2.0),
                                (b.entries ? 128.0 : 256.0) * P.rc_width * P.rc_height);
  b.words = std::max((unsigned)std::min(words, (double)MH_GRID_MAX_WORDS), 4096u);
}

// Whether they take at most a sixteenth of what the voxels take.
inline bool ray_grid_small(const mh_params &P) {
  RayGridBuf b;
  ray_grid_sizes(P, b);
  return 4.0 * ((double)b.words + b.entries) <= P.value_capacity * 8192.0 / 16.0;
}

// The buffers' memory, from alloc(words) (null: there is none), asked for once.
// Without the blocks they are looked up in the hash table, without the cells every
// sample is evaluated: the same images, later.
template <class Alloc> inline void ray_grid_reserve(const mh_params &P, RayGridBuf &b, Alloc &&alloc) {
  if (b.reserved) return;
  b.reserved = true;
  ray_grid_sizes(P, b);
  b.bits = alloc(b.words);
  if (b.bits && b.entries) b.blocks = alloc(b.entries);
}

// The box around a view, false for a pose that is not finite or far out.  The
// samples of a pixel lie at wTc (z r), z in the raycast range and r the pixel's
// ray, so the box is the hull of the view's eight corners when wTc is rigid;
// any other matrix gets the ball that holds every ray (their directions are
// normalised).
MH_GRID_HD inline bool view_box(const mh_params &P, const float wTc[16], double lo[3], double hi[3]) {
  const ViewCone v(P);
  bool rigid = true;
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j) {
      const double dot = (double)wTc[i] * wTc[j] + (double)wTc[4 + i] * wTc[4 + j] + (double)wTc[8 + i] * wTc[8 + j];
      if (!(std::fabs(dot - (i == j ? 1.0 : 0.0)) < 1e-3)) rigid = false;
    }
  const double zs[2] = {P.min_raycast_depth, P.max_raycast_depth};
  for (int a = 0; a < 3; ++a) {
    const double o = wTc[4 * a + 3];
    if (rigid) {
      lo[a] = 1e300, hi[a] = -1e300;
      for (int c = 0; c < 8; ++c) {
        const double z = zs[c & 1];
        const double q = o + z * (wTc[4 * a] * v.x[(c >> 1) & 1] + wTc[4 * a + 1] * v.y[c >> 2] + wTc[4 * a + 2]);
        lo[a] = std::min(lo[a], q), hi[a] = std::max(hi[a], q);
      }
    } else {
      lo[a] = o - v.len * zs[1], hi[a] = o + v.len * zs[1];
    }
    // the directions' deviation from unit length, and the march's rounding
    const double pad = 2e-3 * v.len * zs[1];
    lo[a] -= pad, hi[a] += pad;
    if (!(lo[a] > -1e6 && hi[a] < 1e6)) return false;
  }
  return true;
}

// The smallest cells (U = 2, 4, ... voxels) for which a box fits the words.
//
// Roundings move a sample's cell coordinate by e at most: the positions' 4 units
// in the last place of the coordinates, and 1/128 cell in the grid's arithmetic.
// A sample is looked up `guard` >= e below its position, so that it is never found
// above the cell of its first corner; one that is found in cell i then has its
// first corner below voxel U (i + 1 + guard + e) and reads one voxel more.  The
// marks have to reach as far down: `reach` groups of two voxels, 1 near the origin
// with cells of up to 16 voxels.  More than a cell is too far; with U = 2 more
// than one group is, since the marks of those come from bit masks.
MH_GRID_HD inline RayGrid ray_grid_of(const mh_params &P, const double lo[3], const double hi[3], const RayGridBuf &b) {
  RayGrid g{};
  double far = 0.0;
  for (int a = 0; a < 3; ++a) far = std::max(far, std::max(std::fabs(lo[a]), std::fabs(hi[a])));
  for (int shift = 0; shift < 12; ++shift) {
    const int U = 2 << shift;
    const double cell = (double)U * (double)P.voxel_size;
    const double e = far / (cell * 2097152.0) + 0.0078125;
    const double guard = std::max(e, (double)MH_GRID_GUARD);
    if (!(guard + e < 1.0)) continue;
    const int reach = 1 + ((int)(U * (guard + e)) + 1) / 2;
    if (reach > (1 << shift)) continue;
    int c[3];
    double n[3];  // words
    for (int a = 0; a < 3; ++a) {
      c[a] = (int)std::floor((lo[a] / cell - 2.0) / 4.0) * 4;
      n[a] = std::ceil((std::floor(hi[a] / cell) + 3.0 - c[a]) / (a == 2 ? 2.0 : 4.0));
    }
    if (n[0] > 2000.0 || n[1] > 2000.0 || n[2] > 4000.0 || n[0] * n[1] * n[2] > (double)b.words) continue;
    g.bits = b.bits;
    g.cx = c[0], g.cy = c[1], g.cz = c[2];
    g.nx = (unsigned)n[0], g.ny = (unsigned)n[1], g.nz = (unsigned)n[2];
    g.words = g.nx * g.ny * g.nz;
    g.shift = shift;
    const double more = guard - MH_GRID_GUARD;
    g.ox = (float)((c[0] + more) * cell), g.oy = (float)((c[1] + more) * cell), g.oz = (float)((c[2] + more) * cell);
    g.inv_cell = (float)(1.0 / cell);
    g.reach = (short)reach;
    break;
  }
  // a block around the box: corners and gradient samples reach past a ray
  const double side = 8.0 * (double)P.voxel_size;
  int c[3];
  double n[3];
  for (int a = 0; a < 3; ++a) {
    c[a] = (int)std::floor(lo[a] / side) - 1;
    n[a] = std::floor(hi[a] / side) + 2.0 - c[a];
  }
  if (g.bits && b.blocks && n[0] * n[1] * n[2] <= (double)b.entries) {
    g.blocks = b.blocks;
    g.bx = c[0], g.by = c[1], g.bz = c[2];
    g.bnx = (unsigned)n[0], g.bny = (unsigned)n[1], g.bnz = (unsigned)n[2];
  }
  return g;
}

// The grid of the view from wTc, with the buffers' next tag.  No grid (null bits)
// for a pose that is not finite or far out.  `margin` widens the box on each side
// where that does not make the cells larger.  A grid may be dropped before
// anything of it is enqueued, so the clear that it asks for stays due until
// ray_grid_enqueued says that it is on its way.
inline RayGrid ray_grid_for(const mh_params &P, const float wTc[16], RayGridBuf &b, double margin = 0.0) {
  double lo[3], hi[3];
  if (!b.bits || !view_box(P, wTc, lo, hi)) return RayGrid{};
  RayGrid g = ray_grid_of(P, lo, hi, b);
  if (margin > 0.0 && g.bits) {
    for (int a = 0; a < 3; ++a) lo[a] -= margin, hi[a] += margin;
    const RayGrid wide = ray_grid_of(P, lo, hi, b);
    if (wide.bits && wide.shift == g.shift && !wide.blocks == !g.blocks) g = wide;
  }
  if (g.blocks) {
    if (b.tag + 1u == MH_GRID_REPLAY_TAG) b.tag = 0u, b.dirty = true;
    b.tag += 1u;
    g.tag = b.tag << 24;
    g.clear = b.dirty ? b.entries : 0u;
  }
  return g;
}

// The same for a raycast whose launches a graph replays.  Its tag is that of all
// replays, so each replay clears the entries of its own box first, and no other
// raycast uses that tag.
MH_GRID_HD inline RayGrid ray_grid_replayed(const mh_params &P, const float wTc[16], const RayGridBuf &b) {
  double lo[3], hi[3];
  if (!b.bits || !view_box(P, wTc, lo, hi)) return RayGrid{};
  RayGrid g = ray_grid_of(P, lo, hi, b);
  if (g.blocks) {
    g.tag = MH_GRID_REPLAY_TAG << 24;
    g.clear = g.bnx * g.bny * g.bnz;
  }
  return g;
}

// The clear and the blocks of g, the last grid handed out, are enqueued.
inline void ray_grid_enqueued(RayGridBuf &b, const RayGrid &g) {
  if (g.blocks) b.dirty = false;
}

// Whether g, made for another pose, holds this pose's view.
inline bool ray_grid_covers(const mh_params &P, const float wTc[16], const RayGrid &g) {
  double lo[3], hi[3];
  if (!g.bits || !view_box(P, wTc, lo, hi)) return false;
  const double cell = (double)(2 << g.shift) * (double)P.voxel_size, side = 8.0 * (double)P.voxel_size;
  const int c[3] = {g.cx, g.cy, g.cz}, bl[3] = {g.bx, g.by, g.bz};
  const unsigned n[3] = {4 * g.nx, 4 * g.ny, 2 * g.nz}, bn[3] = {g.bnx, g.bny, g.bnz};
  for (int a = 0; a < 3; ++a) {
    if (!(lo[a] / cell - 2.0 >= c[a] && std::floor(hi[a] / cell) + 3.0 <= c[a] + (double)n[a])) return false;
    if (g.blocks && !(std::floor(lo[a] / side) - 1.0 >= bl[a] && std::floor(hi[a] / side) + 2.0 <= bl[a] + (double)bn[a]))
      return false;
  }
  return true;
}

// mh_mesh.cu -- per-block marching cubes with shared, ref-counted vertices.
//
// Follows MarchingCubes (meshing/marching_cubes.cu:326-382) and its
// shared-vertex layout: the vertex on the edge (v, v + axis) lives in slot
// `axis` of voxel v's mesh unit (kEdgeOwnerCubeOffset, mc_tables.h:360-376);
// each cube keeps up to five triangle slots that are reused across frames;
// vertices carry reference counts and are freed when no triangle uses them.
//
// GB300 structure, per mesh call:
//   k_mc_cubes     one 512-thread CTA per candidate block (persistent grid);
//                  a block with no mesh page whose weight bound is below the
//                  MC gate (inv_sigma2 >= 1/voxel^2) has no valid cube, and one
//                  with only non-negative voxels in it and above no cut cube:
//                  k_mc_select leaves them out;
//                  the 9x9x9 corner tile (block + x/y/z halo) is staged in
//                  shared memory as valid/negative bits, after 7 neighbour
//                  lookups per block instead of 8 per cube; each cube gets its
//                  index and marks the vertices of its cut edges; those on the
//                  block's border are claimed for this epoch (one atomicCAS on
//                  the owner's claim word); the CTA that marked or first
//                  claimed one appends (owner, slot) to a compact work list.
//   k_mc_vertices  eight lanes per vertex: warp-aggregated pool pops,
//                  position (VertexIntersection, marching_cubes.cu:16-28)
//                  from the owner cube's view of the edge, radius and SDF
//                  gradient normal (marching_cubes.cu:49-71).  Each vertex is
//                  computed exactly once, so the result does not depend on
//                  which of the up to four sharing cubes ran last.
//   k_mc_triangles surfel counts and triangle slot reuse/allocation with
//                  warp-aggregated pops (TriangleExtractionKernel, :180-275).
//   k_mc_recycle_* surplus triangle slots and unreferenced vertices return to
//                  their pools (RecycleTrianglesKernel / RecycleVerticesKernel,
//                  :278-321); a page left with no vertex and no triangle is
//                  returned as well.
// Mesh units live in mesh pages: a block receives one when a cube in it has
// triangles or a cube claims a vertex it owns.  The triangle and recycle
// passes walk only the candidates that hold a page.
#include "mh_internal.cuh"
#include "mh_kernels.h"
#include "mh_batch.cuh"

#define MH_MC_TABLE_QUALIFIER __constant__
#include "mc_cases.inc"

#define MC_RECYCLE_THREADS 128

// Corner i of the cube at voxel v sits at v + kCorner[i] (mc_tables.h:335-344).
__constant__ int kCorner[8][3] = {{0, 1, 1}, {1, 1, 1}, {1, 1, 0}, {0, 1, 0},
                                  {0, 0, 1}, {1, 0, 1}, {1, 0, 0}, {0, 0, 0}};
// Owner of edge e: its lower endpoint's offset and the edge axis (= slot);
// equal to kEdgeOwnerCubeOffset (mc_tables.h:360-374).
#define MC_OWNERS                                                                                   \
  {{0, 1, 1, 0}, {1, 1, 0, 2}, {0, 1, 0, 0}, {0, 1, 0, 2}, {0, 0, 1, 0}, {1, 0, 0, 2},              \
   {0, 0, 0, 0}, {0, 0, 0, 2}, {0, 0, 1, 1}, {1, 0, 1, 1}, {1, 0, 0, 1}, {0, 0, 0, 1}}
__constant__ int kOwner[12][4] = MC_OWNERS;

__device__ __forceinline__ int case_tris(int c) { return (int)(kMcCases[c] & 0xF); }
__device__ __forceinline__ int case_edge(int c, int k) { return (int)((kMcCases[c] >> (4 + 4 * k)) & 0xF); }

// Claim the vertices `want` (a bit a slot) of claim word `cw` for `epoch`;
// returns those that nobody had claimed.
__device__ __forceinline__ unsigned claim_slots(const Dev &d, uint32_t *cw, unsigned want, unsigned epoch) {
  const uint32_t tag = epoch << 3;
  uint32_t old = *reinterpret_cast<volatile uint32_t *>(cw);
  for (int it = 0; it < 4096; ++it) {
    const uint32_t had = (old & ~7u) == tag ? old & 7u : 0u;
    if (!(want & ~had)) return 0u;
    const uint32_t prev = atomicCAS(cw, old, tag | had | want);
    if (prev == old) return want & ~had;
    old = prev;
  }
  set_error(d, MH_ERR_TIMEOUT);
  return 0u;
}

// Candidates the cube pass must tile: a block holding a mesh page, or one
// whose weight bound reaches the MC gate (otherwise no cube in it is valid)
// and that has a voxel which is not non-negative in it or in a block above
// (otherwise no cube in it is cut).  One thread per candidate, warp-ballot
// compaction; the blocks above are looked up by eight lanes a candidate.  The
// mesh pass of a 322x238 PSDF frame at 8 mm takes 119 us with this test and 137
// us without: most blocks past the gate are observed free space.
__device__ __forceinline__ void mc_select_body(const Dev &d, Share sh) {
  const int n = *reinterpret_cast<volatile int *>(&d.ctr->cand_count);
  const float lim = 1.0f / d.p.voxel_size;
  const float lim2 = lim * lim;
  const int stride = sh.stride * blockDim.x;
  const int lane = lane_id(), j = lane & 7;
  for (int base = sh.first * blockDim.x; base < n; base += stride) {
    const int i = base + threadIdx.x;
    int4 cb = make_int4(0, 0, 0, -1);
    bool keep = false, page = false;
    if (i < n) {
      cb = d.cand[i];
      if (cb.w >= 0) {
        page = d.page_of[cb.w] >= 0;
        keep = page || !(d.wmax[cb.w] < lim2);
      }
    }
    unsigned m = __ballot_sync(0xffffffffu, keep), ask = __ballot_sync(0xffffffffu, keep && !page);
    while (ask) {
      // four candidates at a time; no more: -1
      int of[4];
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        of[g] = __ffs(ask) - 1;
        ask &= ask - 1;
      }
      const int mine = lane < 8 ? of[0] : lane < 16 ? of[1] : lane < 24 ? of[2] : of[3], from = max(mine, 0);
      const int x = __shfl_sync(0xffffffffu, cb.x, from), y = __shfl_sync(0xffffffffu, cb.y, from),
                z = __shfl_sync(0xffffffffu, cb.z, from), w = __shfl_sync(0xffffffffu, cb.w, from);
      bool cut = false;
      if (mine >= 0) {
        const int q = j == 0 ? w : hash_find(d, x + (j & 1), y + ((j >> 1) & 1), z + (j >> 2));
        cut = q >= 0 && d.neg[q] != 0ull;
      }
      const unsigned cuts = __ballot_sync(0xffffffffu, cut);
#pragma unroll
      for (int g = 0; g < 4; ++g)
        if (of[g] >= 0 && !(cuts >> (8 * g) & 0xffu)) m &= ~(1u << of[g]);
    }
    int slot = 0;
    if (lane == 0 && m) slot = atomicAdd(&d.ctr->cube_list_count, __popc(m));
    slot = __shfl_sync(0xffffffffu, slot, 0);
    if (m >> lane & 1u) d.cube_list[slot + __popc(m & lanemask_lt())] = cb;
  }
}
__global__ void __launch_bounds__(256) k_mc_select(Dev d) { mc_select_body(d, whole_grid()); }
__global__ void __launch_bounds__(256) k_mc_select_b(const Scene *t, int n) {
  each_scene(t, n, 256, [&](const Scene &c) { return count_of(c.d, &Counters::cand_count); },
             [&](const Scene &c, Share sh) { mc_select_body(c.d, sh); });
}
// Counts of the finished pass, and the next pass's start.  Run by one thread of
// the last kernel, which reads only mesh_list_count (k_mc_cubes clears that).
__device__ __forceinline__ void mc_end_body(const Dev &d) {
  d.ctr->mesh_passes += 1;
  d.ctr->cand_sum += (unsigned long long)d.ctr->cand_count;
  d.ctr->vwork_sum += (unsigned long long)min(d.ctr->vwork_count, d.vwork_capacity);
  d.ctr->mesh_list_sum += (unsigned long long)d.ctr->mesh_list_count;
  d.ctr->epoch += 1;
  d.ctr->vwork_count = 0;
  d.ctr->cube_list_count = 0;
}

// ------------------------------------------------------------------ pass 1
// A vertex is shared by the four cubes around its edge.  The CTA gathers the
// vertices of its cubes as bits of their owners in shared memory, over the
// block and the layer above it on each axis; only those that a cube of another
// block may share too go through the owner's claim word, all slots of an owner
// with one atomic, and each warp takes its places in the work list at once.  An
// atomicCAS a cube and edge and an atomicAdd a vertex, one after the other, took
// 141 us against 55 us for a 322x238 PSDF frame at 8 mm (cold).  What is left is
// the latency of a block's chain: candidate, hash, tile, pages, claims.
__device__ __forceinline__ void mc_cubes_body(const Dev &d, Share sh) {
  __shared__ uint8_t tile[729];
  __shared__ unsigned own[729];
  __shared__ int nb[8], page[8];
  __shared__ unsigned owners_in;
  const int tid = threadIdx.x;
  const int n = *reinterpret_cast<volatile int *>(&d.ctr->cube_list_count);
  const unsigned epoch = *reinterpret_cast<volatile unsigned *>(&d.ctr->epoch);
  const float lim = 1.0f / d.p.voxel_size;
  const float lim2 = lim * lim;
  const int x = tid & 7, y = (tid >> 3) & 7, z = tid >> 6;
  if (sh.first == 0 && tid == 0) {
    d.ctr->mesh_list_count = 0;
    d.ctr->cube_blocks_sum += (unsigned long long)n;
  }
  for (int c = sh.first; c < n; c += sh.stride) {
    const int4 cb = d.cube_list[c];
    if (tid < 8) {
      const int dx = tid & 1, dy = (tid >> 1) & 1, dz = tid >> 2;
      nb[tid] = tid == 0 ? cb.w : hash_find(d, cb.x + dx, cb.y + dy, cb.z + dz);
      if (tid == 0) owners_in = 0u;
    }
    __syncthreads();
    for (int e = tid; e < 729; e += 512) {
      const int tx = e % 9, ty = (e / 9) % 9, tz = e / 81;
      const int ptr = nb[(tx >> 3) + 2 * (ty >> 3) + 4 * (tz >> 3)];
      uint8_t f = 0;
      if (ptr >= 0) {
        const size_t gi = (size_t)ptr * MH_BLOCK_VOXELS + (tx & 7) + 8 * (ty & 7) + 64 * (tz & 7);
        const float s = d.sdf[gi], w = d.w[gi], a = d.a[gi], b = d.b[gi];
        const float rho = a / (a + b);
        const bool ok = !(fabsf(s) > 0.20f) && !(rho < 0.1f || w < lim2);
        f = (ok ? 1 : 0) | (s < 0.0f ? 2 : 0);
      }
      tile[e] = f;
      own[e] = 0u;
    }
    __syncthreads();
    int cube = 0;
    bool valid = true;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const uint8_t f = tile[(x + kCorner[k][0]) + 9 * (y + kCorner[k][1]) + 81 * (z + kCorner[k][2])];
      valid &= (f & 1) != 0;
      cube |= ((f >> 1) & 1) << k;
    }
    if (!valid) cube = 0;
    const bool surf = cube != 0 && cube != 255;
    if (surf) {
      // corners joined by edge e (mc_tables.h:376-390), and its owner
      constexpr int ends[12][2] = {{0, 1}, {1, 2}, {2, 3}, {3, 0}, {4, 5}, {5, 6},
                                   {6, 7}, {7, 4}, {4, 0}, {5, 1}, {6, 2}, {7, 3}};
      constexpr int owner[12][4] = MC_OWNERS;
      unsigned in = 0u;
#pragma unroll
      for (int e = 0; e < 12; ++e) {
        if (((cube >> ends[e][0]) & 1) == ((cube >> ends[e][1]) & 1)) continue;
        const int ox = x + owner[e][0], oy = y + owner[e][1], oz = z + owner[e][2];
        atomicOr(own + ox + 9 * oy + 81 * oz, 1u << owner[e][3]);
        in |= 1u << ((ox >> 3) + 2 * (oy >> 3) + 4 * (oz >> 3));
      }
      atomicOr(&owners_in, in);
    }
    const int any_surf = __syncthreads_or(surf);
    if (tid < 8) {
      // the block's own page first: without one nothing is claimed
      int pg = -1;
      if (tid == 0) pg = any_surf ? ensure_page(d, cb.w) : d.page_of[cb.w];
      const int first = __shfl_sync(0xffu, pg, 0);
      if (tid > 0 && first >= 0 && nb[tid] >= 0 && (owners_in >> tid & 1u)) pg = ensure_page(d, nb[tid]);
      page[tid] = pg;
    }
    __syncthreads();
    if (page[0] >= 0) {
      d.cube[(size_t)page[0] * MH_BLOCK_VOXELS + tid] = (uint8_t)cube;
      if (any_surf) {
        for (int base = 0; base < 729; base += 512) {
          const int e = base + tid;
          unsigned got = e < 729 ? own[e] : 0u;
          int opg = -1, oli = 0, optr = -1;
          if (got) {
            const int ox = e % 9, oy = (e / 9) % 9, oz = e / 81;
            const int q = (ox >> 3) + 2 * (oy >> 3) + 4 * (oz >> 3);
            opg = page[q], optr = nb[q];
            oli = (ox & 7) + 8 * (oy & 7) + 64 * (oz & 7);
            // cubes share the vertex of slot a over the two other axes
            unsigned inside = 0u;
            if (q == 0) inside = (oy && oz ? 1u : 0u) | (ox && oz ? 2u : 0u) | (ox && oy ? 4u : 0u);
            const unsigned shared = got & ~inside;
            if (opg < 0) got = 0u;
            else if (shared) got = (got & inside) | claim_slots(d, d.claim + (size_t)opg * MH_BLOCK_VOXELS + oli, shared, epoch);
          }
          const unsigned g0 = __ballot_sync(0xffffffffu, got & 1u), g1 = __ballot_sync(0xffffffffu, got & 2u),
                         g2 = __ballot_sync(0xffffffffu, got & 4u);
          const int n0 = __popc(g0), n1 = __popc(g1), total = n0 + n1 + __popc(g2);
          if (!total) continue;
          int at = 0;
          if (lane_id() == 0) at = atomicAdd(&d.ctr->vwork_count, total);
          at = __shfl_sync(0xffffffffu, at, 0);
          if (at + total > d.vwork_capacity && lane_id() == 0) set_error(d, MH_ERR_CAPACITY);
          const unsigned lt = lanemask_lt();
          const int w0 = at + __popc(g0 & lt), w1 = at + n0 + __popc(g1 & lt), w2 = at + n0 + n1 + __popc(g2 & lt);
          if ((got & 1u) && w0 < d.vwork_capacity) d.vwork[w0] = make_int4(opg, oli, 0, optr);
          if ((got & 2u) && w1 < d.vwork_capacity) d.vwork[w1] = make_int4(opg, oli, 1, optr);
          if ((got & 4u) && w2 < d.vwork_capacity) d.vwork[w2] = make_int4(opg, oli, 2, optr);
        }
      }
    }
    __syncthreads();
  }
}
__global__ void __launch_bounds__(512, 3) k_mc_cubes(Dev d) { mc_cubes_body(d, whole_grid()); }
__global__ void __launch_bounds__(512, 2) k_mc_cubes_b(const Scene *t, int n) {
  each_scene(t, n, 1, [&](const Scene &c) { return max(1, count_of(c.d, &Counters::cube_list_count)); },
             [&](const Scene &c, Share sh) { mc_cubes_body(c.d, sh); });
}

// candidates holding a page after pass 1; the others get zero surfel counts
__device__ __forceinline__ void mc_list_body(const Dev &d, Share sh) {
  const int n = *reinterpret_cast<volatile int *>(&d.ctr->cand_count);
  const int stride = sh.stride * blockDim.x;
  for (int base = sh.first * blockDim.x; base < n; base += stride) {
    const int i = base + threadIdx.x;
    int ptr = -1;
    bool keep = false;
    if (i < n) {
      ptr = d.cand[i].w;
      if (ptr >= 0) {
        keep = d.page_of[ptr] >= 0;
        if (!keep) d.inner[ptr] = d.boundary[ptr] = 0;
      }
    }
    const unsigned m = __ballot_sync(0xffffffffu, keep);
    int slot = 0;
    if (lane_id() == 0 && m) slot = atomicAdd(&d.ctr->mesh_list_count, __popc(m));
    slot = __shfl_sync(0xffffffffu, slot, 0);
    if (keep) d.mesh_list[slot + __popc(m & lanemask_lt())] = ptr;
  }
}
__global__ void __launch_bounds__(256) k_mc_list(Dev d) { mc_list_body(d, whole_grid()); }
__global__ void __launch_bounds__(256) k_mc_list_b(const Scene *t, int n) {
  each_scene(t, n, 256, [&](const Scene &c) { return count_of(c.d, &Counters::cand_count); },
             [&](const Scene &c, Share sh) { mc_list_body(c.d, sh); });
}

// ------------------------------------------------------------------ vertices
// The blocks around a vertex for its eight lanes: lane j holds the block of
// offset (j & 1, j >> 1 & 1, j >> 2) from the one that holds voxel v - 1 on
// each axis, for voxels v - 1 .. v + 2.
struct VertexBlocks {
  int x, y, z, ex, ey, ez, block;
  unsigned base;
  __device__ __forceinline__ VertexBlocks(const Dev &d, bool live, int vx, int vy, int vz, int blk) {
    const int j = threadIdx.x & 7;
    base = threadIdx.x & 24;
    x = (vx - 1) >> 3, y = (vy - 1) >> 3, z = (vz - 1) >> 3;
    ex = ((vx + 2) >> 3) - x, ey = ((vy + 2) >> 3) - y, ez = ((vz + 2) >> 3) - z;
    const int dx = j & 1, dy = (j >> 1) & 1, dz = j >> 2;
    block = -1;
    if (live && dx <= ex && dy <= ey && dz <= ez) {
      const bool own = x + dx == vx >> 3 && y + dy == vy >> 3 && z + dz == vz >> 3;
      block = own ? blk : hash_find(d, x + dx, y + dy, z + dz);
    }
  }
  // Block of a voxel, any of them; all 32 lanes of the warp call it.
  __device__ __forceinline__ int get(const Dev &d, int vx, int vy, int vz) const {
    const int bx = vx >> 3, by = vy >> 3, bz = vz >> 3;
    const unsigned dx = bx - x, dy = by - y, dz = bz - z;
    const bool near = dx <= (unsigned)ex && dy <= (unsigned)ey && dz <= (unsigned)ez;
    const int b = __shfl_sync(0xffffffffu, block, base + (near ? dx + 2 * dy + 4 * dz : 0u));
    return near ? b : hash_find(d, bx, by, bz);
  }
};
__device__ __forceinline__ size_t voxel_index(int block, int x, int y, int z) {
  return (size_t)block * MH_BLOCK_VOXELS + (x & 7) + 8 * (y & 7) + 64 * (z & 7);
}

// Eight lanes a vertex.  They look up the eight blocks around it at once; then
// each of six evaluates one sample of the SDF gradient (GetSpatialSDFGradient,
// spatial_query.h:68-97) and each of eight one corner of the radius
// (GetSpatialValue, :23-66), summed in the reference's order.  Bound by the
// latency of dependent loads: a thread a vertex, with seven samples one after
// the other and a hash lookup for every corner in another block, took 78 us
// against 52 us for a 322x238 PSDF frame at 8 mm (cold).
__device__ __forceinline__ void mc_vertices_body(const Dev &d, Share sh) {
  const int n = min(*reinterpret_cast<volatile int *>(&d.ctr->vwork_count), d.vwork_capacity);
  const int per_cta = blockDim.x / 8, stride = sh.stride * per_cta;
  const int j = threadIdx.x & 7;
  const unsigned base8 = threadIdx.x & 24;
  const float vs = d.p.voxel_size;
#pragma unroll 1
  for (int base = sh.first * per_cta; base < n; base += stride) {
    const int i = base + threadIdx.x / 8;
    bool live = i < n;
    int4 wk = make_int4(0, 0, 0, 0);
    int *slotp = nullptr;
    int vp = -1;
    if (live) {
      wk = d.vwork[i];
      slotp = d.vtx_slot + ((size_t)wk.x * MH_BLOCK_VOXELS + wk.y) * 3 + wk.z;
      vp = *slotp;
    }
    __syncwarp();
    int fresh = warp_pop(d, &d.ctr->vtx_top, d.vtx_heap, live && vp < 0 && j == 0);
    fresh = __shfl_sync(0xffffffffu, fresh, base8);
    const int blk = wk.w;
    if (live && vp < 0) {
      vp = fresh;
      if (vp < 0) live = false;
      else if (j == 0) {
        *slotp = vp;
        atomicAdd(d.nvtx + blk, 1);
      }
    }
    const int4 bp = live ? d.block_pos[blk] : make_int4(0, 0, 0, 0);
    const int slot = wk.z;
    const int v0x = bp.x * MH_BLOCK_SIDE + (wk.y & 7), v0y = bp.y * MH_BLOCK_SIDE + ((wk.y >> 3) & 7),
              v0z = bp.z * MH_BLOCK_SIDE + (wk.y >> 6);
    const int v1x = v0x + (slot == 0), v1y = v0y + (slot == 1), v1z = v0z + (slot == 2);
    const VertexBlocks vb(d, live, v0x, v0y, v0z, blk);
    const float d0 = live ? d.sdf[(size_t)blk * MH_BLOCK_VOXELS + wk.y] : 0.0f;
    const int p1 = vb.get(d, v1x, v1y, v1z);
    const float d1 = p1 >= 0 ? d.sdf[voxel_index(p1, v1x, v1y, v1z)] : 0.0f;
    // owner cube's endpoint order: x edge (v+x, v), y edge (v, v+y), z edge (v, v+z)
    const F3 P = f3((float)v0x * vs, (float)v0y * vs, (float)v0z * vs);
    const F3 Q = f3(P.x + vs * (float)(slot == 0), P.y + vs * (float)(slot == 1), P.z + vs * (float)(slot == 2));
    F3 p1w, p2w;
    float e1, e2;
    if (slot == 0) {
      p1w = Q, p2w = P, e1 = d1, e2 = d0;
    } else {
      p1w = P, p2w = Q, e1 = d0, e2 = d1;
    }
    F3 pos;
    if ((double)fabsf(e1) < 0.008) {
      pos = p1w;
    } else if ((double)fabsf(e2) < 0.008) {
      pos = p2w;
    } else {
      const float mu = (0.0f - e1) / (e2 - e1);
      pos = f3(p1w.x + mu * (p2w.x - p1w.x), p1w.y + mu * (p2w.y - p1w.y), p1w.z + mu * (p2w.z - p1w.z));
    }
    // corner j of the sample at the vertex
    float rad = 0.0f;
    bool rad_ok;
    {
      const Corners k = corners_at(d.p, pos);
      const bool mx = j & 4, my = j & 2, mz = j & 1;
      const int vx = mx ? k.v1x : k.v0x, vy = my ? k.v1y : k.v0y, vz = mz ? k.v1z : k.v0z;
      const int b = vb.get(d, vx, vy, vz);
      float t = 0.0f;
      if (b >= 0) {
        const float w = (mx ? k.rx : 1.0f - k.rx) * (my ? k.ry : 1.0f - k.ry) * (mz ? k.rz : 1.0f - k.rz);
        t = w * sqrtf(1.0f / __ldg(d.w + voxel_index(b, vx, vy, vz)));
      }
      rad_ok = (__ballot_sync(0xffffffffu, b >= 0) >> base8 & 0xffu) == 0xffu;
#pragma unroll
      for (int q = 0; q < 8; ++q) rad += __shfl_sync(0xffffffffu, t, base8 + q);
    }
    // sample j of the gradient: axis j / 2, minus side first
    const float h = 0.5f * vs, off = j & 1 ? h : -h;
    const Corners k = corners_at(d.p, f3(pos.x + (j >> 1 == 0 ? off : 0.0f), pos.y + (j >> 1 == 1 ? off : 0.0f),
                                         pos.z + (j >> 1 == 2 ? off : 0.0f)));
    bool ok = true;
    float v[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int vx = q & 4 ? k.v1x : k.v0x, vy = q & 2 ? k.v1y : k.v0y, vz = q & 1 ? k.v1z : k.v0z;
      const int b = vb.get(d, vx, vy, vz);
      ok &= b >= 0;
      v[q] = b >= 0 ? __ldg(d.sdf + voxel_index(b, vx, vy, vz)) : 0.0f;
    }
    float s = 0.0f;
#pragma unroll
    for (int q = 0; q < 8; ++q)
      s += (q & 4 ? k.rx : 1.0f - k.rx) * (q & 2 ? k.ry : 1.0f - k.ry) * (q & 1 ? k.rz : 1.0f - k.rz) * v[q];
    const bool g_ok = (__ballot_sync(0xffffffffu, ok) >> base8 & 0x3fu) == 0x3fu;
    float g[3];
#pragma unroll
    for (int q = 0; q < 3; ++q)
      g[q] = (__shfl_sync(0xffffffffu, s, base8 + 2 * q + 1) - __shfl_sync(0xffffffffu, s, base8 + 2 * q)) / vs;
    if (live && j < 2) {
      float radius = 0.0f;
      if (rad_ok) {
        const float is2 = 1.0f / (rad * rad);
        radius = sqrtf(1.0f / is2);
      }
      F3 nrm = f3(0.0f, 0.0f, 0.0f);
      const F3 gv = f3(g[0], g[1], g[2]);
      const float l = sqrtf(dot3(gv, gv));
      if (g_ok && l > 0.0f) nrm = f3(gv.x / l, gv.y / l, gv.z / l);
      Vertex *vt = d.vtx + vp;
      float4 *v4 = reinterpret_cast<float4 *>(vt);
      if (j == 0) v4[0] = make_float4(pos.x, pos.y, pos.z, nrm.x);
      else v4[1] = make_float4(nrm.y, nrm.z, radius, __int_as_float(vt->ref_count));
    }
    __syncwarp();
  }
}
__global__ void __launch_bounds__(128) k_mc_vertices(Dev d) { mc_vertices_body(d, whole_grid()); }
__global__ void __launch_bounds__(128) k_mc_vertices_b(const Scene *t, int n) {
  each_scene(t, n, 16, [&](const Scene &c) { return count_of(c.d, &Counters::vwork_count); },
             [&](const Scene &c, Share sh) { mc_vertices_body(c.d, sh); });
}

// ------------------------------------------------------------------ pass 2
__device__ __forceinline__ void mc_triangles_body(const Dev &d, Share sh) {
  __shared__ int nbp[8];
  __shared__ int cnt[2];
  const int tid = threadIdx.x;
  const int n = *reinterpret_cast<volatile int *>(&d.ctr->mesh_list_count);
  const int x = tid & 7, y = (tid >> 3) & 7, z = tid >> 6;
  const bool inner = x >= 1 && y >= 1 && z >= 1 && x < 7 && y < 7 && z < 7;
  for (int c = sh.first; c < n; c += sh.stride) {
    const int blk = d.mesh_list[c];
    const int4 bp = d.block_pos[blk];
    if (tid < 8) {
      const int dx = tid & 1, dy = (tid >> 1) & 1, dz = tid >> 2;
      const int q = tid == 0 ? blk : hash_find(d, bp.x + dx, bp.y + dy, bp.z + dz);
      nbp[tid] = q >= 0 ? d.page_of[q] : -1;
    }
    if (tid < 2) cnt[tid] = 0;
    __syncthreads();
    const int pg = nbp[0];
    const size_t vi = (size_t)pg * MH_BLOCK_VOXELS + tid;
    // surfel counts (marching_cubes.cu:191-212)
    const int *vs = d.vtx_slot + vi * 3;
    const int here = (vs[0] >= 0) + (vs[1] >= 0) + (vs[2] >= 0);
    const int wsum = __reduce_add_sync(0xffffffffu, inner ? here : 0);
    const int bsum = __reduce_add_sync(0xffffffffu, inner ? 0 : here);
    if ((tid & 31) == 0) {
      if (wsum) atomicAdd(&cnt[0], wsum);
      if (bsum) atomicAdd(&cnt[1], bsum);
    }
    const int cube = d.cube[vi];
    const int ntri = (cube == 0 || cube == 255) ? 0 : case_tris(cube);
    int *ts = d.tri_slot + vi * 5;
#pragma unroll 1
    for (int t = 0; t < 5; ++t) {
      const bool need = t < ntri;
      const int old = need ? ts[t] : 0;
      const int fresh = warp_pop(d, &d.ctr->tri_top, d.tri_heap, need && old < 0);
      if (!need) continue;
      int vids[3];
      bool okv = true;
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        const int e = case_edge(cube, 3 * t + q);
        const int ox = x + kOwner[e][0], oy = y + kOwner[e][1], oz = z + kOwner[e][2];
        const int opg = nbp[(ox >> 3) + 2 * (oy >> 3) + 4 * (oz >> 3)];
        const int oli = (ox & 7) + 8 * (oy & 7) + 64 * (oz & 7);
        vids[q] = opg >= 0 ? d.vtx_slot[((size_t)opg * MH_BLOCK_VOXELS + oli) * 3 + kOwner[e][3]] : -1;
        okv &= vids[q] >= 0;
      }
      int tp = old;
      if (old >= 0) {
        const int4 ot = d.tri[old];
        atomicSub(&d.vtx[ot.x].ref_count, 1);
        atomicSub(&d.vtx[ot.y].ref_count, 1);
        atomicSub(&d.vtx[ot.z].ref_count, 1);
      } else {
        tp = fresh;
        if (tp < 0) continue;
        ts[t] = tp;
      }
      if (!okv) {
        // a pool ran dry earlier in this pass; keep the slot on the reserved vertex 0
        set_error(d, MH_ERR_CAPACITY);
        d.tri[tp] = make_int4(0, 0, 0, 0);
        atomicAdd(&d.vtx[0].ref_count, 3);
        continue;
      }
      d.tri[tp] = make_int4(vids[0], vids[1], vids[2], 0);
      atomicAdd(&d.vtx[vids[0]].ref_count, 1);
      atomicAdd(&d.vtx[vids[1]].ref_count, 1);
      atomicAdd(&d.vtx[vids[2]].ref_count, 1);
    }
    __syncthreads();
    if (tid == 0) {
      d.inner[blk] = cnt[0];
      d.boundary[blk] = cnt[1];
    }
    __syncthreads();
  }
}
__global__ void __launch_bounds__(512) k_mc_triangles(Dev d) { mc_triangles_body(d, whole_grid()); }
__global__ void __launch_bounds__(512) k_mc_triangles_b(const Scene *t, int n) {
  each_scene(t, n, 1, [&](const Scene &c) { return count_of(c.d, &Counters::mesh_list_count); },
             [&](const Scene &c, Share sh) { mc_triangles_body(c.d, sh); });
}

// ------------------------------------------------------------------ recycle
// Both passes read a page's slots as vectors, all of them before the first is
// looked at: what bounds them is the latency of one load after the other.  A
// slot at a time, and the triangle slots again for each page's end, took 17 and
// 20 us against 12 and 8 us for a 322x238 PSDF frame at 8 mm (cold).
__device__ __forceinline__ void mc_recycle_tri_body(const Dev &d, Share sh) {
  constexpr int N = MH_BLOCK_VOXELS * 5 / 4 / MC_RECYCLE_THREADS;
  const int n = *reinterpret_cast<volatile int *>(&d.ctr->mesh_list_count);
  for (int c = sh.first; c < n; c += sh.stride) {
    const int pg = d.page_of[d.mesh_list[c]];
    int *ts = d.tri_slot + (size_t)pg * MH_BLOCK_VOXELS * 5;
    int4 held[N];
#pragma unroll
    for (int k = 0; k < N; ++k) held[k] = reinterpret_cast<const int4 *>(ts)[threadIdx.x + k * MC_RECYCLE_THREADS];
#pragma unroll
    for (int k = 0; k < N; ++k) {
      const int4 q = held[k];
      if (q.x < 0 && q.y < 0 && q.z < 0 && q.w < 0) continue;
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        const int tp = m == 0 ? q.x : m == 1 ? q.y : m == 2 ? q.z : q.w;
        if (tp < 0) continue;
        const int i = 4 * (threadIdx.x + k * MC_RECYCLE_THREADS) + m;
        const int cube = d.cube[(size_t)pg * MH_BLOCK_VOXELS + i / 5];
        if (i % 5 < ((cube == 0 || cube == 255) ? 0 : case_tris(cube))) continue;
        const int4 ot = d.tri[tp];
        atomicSub(&d.vtx[ot.x].ref_count, 1);
        atomicSub(&d.vtx[ot.y].ref_count, 1);
        atomicSub(&d.vtx[ot.z].ref_count, 1);
        d.tri[tp] = make_int4(-1, -1, -1, 0);
        stack_push(&d.ctr->tri_top, d.tri_heap, tp);
        ts[i] = MH_FREE_PTR;
      }
    }
  }
}
__global__ void __launch_bounds__(MC_RECYCLE_THREADS) k_mc_recycle_tri(Dev d) { mc_recycle_tri_body(d, whole_grid()); }
__global__ void __launch_bounds__(MC_RECYCLE_THREADS) k_mc_recycle_tri_b(const Scene *t, int n) {
  each_scene(t, n, 1, [&](const Scene &c) { return count_of(c.d, &Counters::mesh_list_count); },
             [&](const Scene &c, Share sh) { mc_recycle_tri_body(c.d, sh); });
}

__device__ __forceinline__ void mc_recycle_vtx_body(const Dev &d, Share sh) {
  constexpr int N = MH_BLOCK_VOXELS * 3 / 4 / MC_RECYCLE_THREADS;
  const int n = *reinterpret_cast<volatile int *>(&d.ctr->mesh_list_count);
  if (sh.first == 0 && threadIdx.x == 0) mc_end_body(d);
  for (int c = sh.first; c < n; c += sh.stride) {
    const int blk = d.mesh_list[c];
    const int pg = d.page_of[blk];
    int *vs = d.vtx_slot + (size_t)pg * MH_BLOCK_VOXELS * 3;
    int4 held[N];
#pragma unroll
    for (int k = 0; k < N; ++k) held[k] = reinterpret_cast<const int4 *>(vs)[threadIdx.x + k * MC_RECYCLE_THREADS];
    int refs[4 * N];
#pragma unroll
    for (int k = 0; k < 4 * N; ++k) {
      const int4 q = held[k / 4];
      const int vp = k % 4 == 0 ? q.x : k % 4 == 1 ? q.y : k % 4 == 2 ? q.z : q.w;
      refs[k] = vp >= 0 ? d.vtx[vp].ref_count : 0;
    }
    int freed = 0;
    bool used = false;
#pragma unroll
    for (int k = 0; k < 4 * N; ++k) {
      const int4 q = held[k / 4];
      const int vp = k % 4 == 0 ? q.x : k % 4 == 1 ? q.y : k % 4 == 2 ? q.z : q.w;
      if (vp < 0) continue;
      if (refs[k] != 0) {
        used = true;
        continue;
      }
      float4 *v4 = reinterpret_cast<float4 *>(d.vtx + vp);
      v4[0] = make_float4(0.f, 0.f, 0.f, 0.f);
      v4[1] = make_float4(0.f, 0.f, 0.f, 0.f);
      stack_push(&d.ctr->vtx_top, d.vtx_heap, vp);
      vs[4 * (threadIdx.x + k / 4 * MC_RECYCLE_THREADS) + k % 4] = MH_FREE_PTR;
      ++freed;
    }
    if (freed) atomicSub(d.nvtx + blk, freed);
    if (__syncthreads_or(used)) continue;
    // no vertex is left: is there a triangle?
    bool tri = false;
    for (int v = threadIdx.x; v < MH_BLOCK_VOXELS * 5; v += MC_RECYCLE_THREADS)
      tri |= d.tri_slot[(size_t)pg * MH_BLOCK_VOXELS * 5 + v] >= 0;
    if (!__syncthreads_or(tri)) release_page_cta(d, blk, pg);
    __syncthreads();
  }
}
__global__ void __launch_bounds__(MC_RECYCLE_THREADS) k_mc_recycle_vtx(Dev d) { mc_recycle_vtx_body(d, whole_grid()); }
__global__ void __launch_bounds__(MC_RECYCLE_THREADS) k_mc_recycle_vtx_b(const Scene *t, int n) {
  each_scene(t, n, 1, [&](const Scene &c) { return max(1, count_of(c.d, &Counters::mesh_list_count)); },
             [&](const Scene &c, Share sh) { mc_recycle_vtx_body(c.d, sh); });
}

int launch_mesh(const Dev &d, cudaStream_t s) {
  const int sms = mh_sm_count();
  k_mc_select<<<sms * 4, 256, 0, s>>>(d);
  k_mc_cubes<<<sms * 3, 512, 0, s>>>(d);
  k_mc_list<<<sms * 4, 256, 0, s>>>(d);
  k_mc_vertices<<<sms * 8, 128, 0, s>>>(d);
  k_mc_triangles<<<sms * 2, 512, 0, s>>>(d);
  k_mc_recycle_tri<<<sms * 8, 128, 0, s>>>(d);
  k_mc_recycle_vtx<<<sms * 8, 128, 0, s>>>(d);
  mh_count_launches(7);
  return cudaGetLastError() == cudaSuccess ? MH_OK : MH_ERR_CUDA;
}

int launch_batch_mesh(const Scene *t, int n, cudaStream_t s) {
  const int sms = mh_sm_count();
  k_mc_select_b<<<sms * 4, 256, 0, s>>>(t, n);
  k_mc_cubes_b<<<sms * 2, 512, 0, s>>>(t, n);
  k_mc_list_b<<<sms * 4, 256, 0, s>>>(t, n);
  k_mc_vertices_b<<<sms * 8, 128, 0, s>>>(t, n);
  k_mc_triangles_b<<<sms * 2, 512, 0, s>>>(t, n);
  k_mc_recycle_tri_b<<<sms * 8, 128, 0, s>>>(t, n);
  k_mc_recycle_vtx_b<<<sms * 8, 128, 0, s>>>(t, n);
  mh_count_launches(7);
  return cudaGetLastError() == cudaSuccess ? MH_OK : MH_ERR_CUDA;
}

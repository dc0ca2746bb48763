// mh_batch.cuh -- the scene table of a batch and the loops that batched
// kernels run over it.
//
// A batch holds many independent volumes.  Each per-frame stage runs as ONE
// launch for all scenes: the batched twin of a kernel walks the device scene
// table and runs the same body as the single-scene kernel for every scene
// that takes a frame this step.  Persistent (grid-stride) bodies and
// pixel-tiled bodies both walk a virtual range that concatenates the scenes'
// items or tiles.  The scene descriptor is staged
// in shared memory, so the body's field reads are shared loads that the
// compiler knows do not alias the global stores of the body.
#pragma once
#include "mh_internal.cuh"

struct __align__(16) Scene {
  Dev d;
  const float *src;          // this step's depth frame (device, metres)
  float *tv;                 // TV scratch: 9 planes of W x H floats
  float *ray_depth;          // raycast outputs (device; null: not written)
  float4 *ray_vert, *ray_norm;
  int active;                // the scene takes a frame this step
  int recycle;               // run the periodic recycle pass this step
  int starve;                // simple update: starve + garbage + recycle this step
  int alloc_tile0;           // first virtual tile of the scene in the alloc grid
  int ray_tile0;             // first virtual tile of the scene in the raycast grid
  int pix0;                  // first pixel of the scene in the concatenated pixel range
  int tv_tile0;              // first virtual tile of the scene in the tiled-TV grid
  int pad;
};

__device__ __forceinline__ int flat_tid() { return threadIdx.x + blockDim.x * (threadIdx.y + blockDim.y * threadIdx.z); }
__device__ __forceinline__ int flat_nthreads() { return blockDim.x * blockDim.y * blockDim.z; }

__device__ __forceinline__ void stage_scene(Scene &cur, const Scene *t, int s) {
  const int4 *src = reinterpret_cast<const int4 *>(t + s);
  int4 *dst = reinterpret_cast<int4 *>(&cur);
  for (int i = flat_tid(); i < (int)(sizeof(Scene) / 16); i += flat_nthreads()) dst[i] = src[i];
}

// A counter of a scene that no launch changes while it is read.
__device__ __forceinline__ int count_of(const Dev &d, int Counters::*count) {
  return *reinterpret_cast<volatile int *>(&(d.ctr->*count));
}

// Runs f(scene, share) for the active scenes of which this CTA has a part.
// count(scene) gives a scene's items, of which a CTA takes `per` at a time;
// the scenes' tiles of `per` items are dealt to the CTAs in one round, so the
// CTAs that one scene leaves idle start with the next, and a CTA stages only
// the scenes that it works on.  With every CTA walking through every scene the
// staging alone was 1-2 us a scene and launch.  All warps read the same counts
// and take the same path; n <= 32 is one round of loads.
template <class C, class F>
__device__ __forceinline__ void each_scene(const Scene *t, int n, unsigned per, C &&count, F &&f) {
  __shared__ Scene cur;
  const int lane = flat_tid() & 31;
  const unsigned ctas = gridDim.x;
  unsigned dealt = 0;  // tiles of the scenes before, modulo the grid
  for (int s0 = 0; s0 < n; s0 += 32) {
    unsigned tiles = 0;
    if (s0 + lane < n && t[s0 + lane].active) tiles = ((unsigned)count(t[s0 + lane]) + per - 1) / per;
    const unsigned part = tiles % ctas;
    unsigned sum = part;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned v = __shfl_up_sync(0xffffffffu, sum, o);
      if (lane >= o) sum += v;
    }
    const unsigned first = (blockIdx.x + ctas - (dealt + sum - part) % ctas) % ctas;
    dealt = (dealt + __shfl_sync(0xffffffffu, sum, 31)) % ctas;
    unsigned mine = __ballot_sync(0xffffffffu, first < tiles);
    while (mine) {
      const int k = __ffs(mine) - 1;
      mine &= mine - 1;
      const Share sh{(int)__shfl_sync(0xffffffffu, first, k), (int)ctas};
      __syncthreads();
      stage_scene(cur, t, s0 + k);
      __syncthreads();
      f(cur, sh);
    }
  }
}

// Virtual tiles: tile vt belongs to the last scene whose first tile is <= vt.
// Runs f(scene, local tile) for every tile of an active scene; tile0 selects
// the prefix field (alloc or raycast tiling).
template <class F>
__device__ __forceinline__ void each_tile(const Scene *t, int n, int total, int Scene::*tile0, F &&f) {
  __shared__ Scene cur;
  __shared__ int cur_s;
  if (flat_tid() == 0) cur_s = -1;
  for (int vt = blockIdx.x; vt < total; vt += gridDim.x) {
    int s = 0;
    for (int s0 = 0; s0 < n; s0 += 32) {  // a lane a scene
      const int k = s0 + (flat_tid() & 31);
      const unsigned before = __ballot_sync(0xffffffffu, k < n && t[k].*tile0 <= vt);
      if (!before) break;
      s = s0 + 31 - __clz(before);
    }
    __syncthreads();
    if (s != cur_s) {
      stage_scene(cur, t, s);
      __syncthreads();
      if (flat_tid() == 0) cur_s = s;
    }
    __syncthreads();
    if (cur.active) f(cur, vt - cur.*tile0);
  }
}

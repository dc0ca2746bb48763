// mh_integrate.cu -- TSDF / PSDF voxel updates and inlier-ratio prediction.
//
// The reference launches one 512-thread CTA per candidate block with one
// thread per voxel and scalar loads of a 20-byte AoS Voxel
// (mapping/update_simple.cu:13-77, update_bayesian.cu:103-185).  Here a
// persistent grid walks the device-resident candidate list; each 128-thread
// CTA covers one block per iteration with 4 consecutive voxels per thread, so
// every voxel field moves as one aligned 128-bit load/store.  Voxel fields are
// only loaded when at least one of the thread's voxels projects onto a valid
// depth pixel inside the truncation band (sdf: of the warp's).
#include "mh_internal.cuh"
#include "mh_exp.h"
#include "mh_kernels.h"
#include "mh_batch.cuh"

#include <algorithm>
#include <cmath>

namespace {

// Pixel of a camera-frame point (update_simple.cu:26-46), or -1 outside the
// image: the integer part of c.x fx / c.z + cx + 1/2, and of y.  Seven
// roundings of 2^-24 (W + |cx|) at most lie between the value the divisions
// give and the one an approximate reciprocal (1 unit in the last place) gives,
// so the integer parts agree unless the latter comes that close to an integer
// (1 - 2 pix_half; 0.2 % of voxels at 640x480); only there, and for points
// that are not finite or far off, are the two divisions evaluated.
__device__ __forceinline__ int pixel_of(const DevParams &p, F3 c) {
  const float kMagic = 12582912.0f;  // 1.5 * 2^23: adding it rounds to an integer
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(c.z));
  const float ax = c.x * p.fx, ay = c.y * p.fy;
  const float wx = fmaf(ax, r, p.cx + 0.5f), wy = fmaf(ay, r, p.cy + 0.5f);
  const float mx = (wx - 0.5f) + kMagic, my = (wy - 0.5f) + kMagic;
  int px = __float_as_int(mx) - 0x4b400000, py = __float_as_int(my) - 0x4b400000;
  if (fabsf(wx - (mx - kMagic) - 0.5f) < p.pix_half && fabsf(wy - (my - kMagic) - 0.5f) < p.pix_half) {
    if (px == -1) px = 0;  // (-1, 0) truncates to 0
    if (py == -1) py = 0;
  } else {
    px = f2i(ax / c.z + p.cx + 0.5f);
    py = f2i(ay / c.z + p.cy + 0.5f);
  }
  return (unsigned)px < p.width && (unsigned)py < p.height ? (int)((unsigned)py * p.width + (unsigned)px) : -1;
}
// camera-frame position of voxel (x, y, z) given as floats
__device__ __forceinline__ F3 voxel_in_camera(const DevParams &p, const float *cTw, float x, float y, float z) {
  const float vs = p.voxel_size;
  return mul_pt(cTw, f3(x * vs, y * vs, z * vs));
}

__device__ __forceinline__ float get(const float4 &v, int k) { return k == 0 ? v.x : k == 1 ? v.y : k == 2 ? v.z : v.w; }
__device__ __forceinline__ void put(float4 &v, int k, float x) {
  if (k == 0) v.x = x;
  else if (k == 1) v.y = x;
  else if (k == 2) v.z = x;
  else v.w = x;
}

// Raise the block's weight bound (read by the mesh pass to skip blocks that
// cannot hold a valid cube).  Positive floats order like their bit patterns.
__device__ __forceinline__ void note_wmax(const Dev &d, int blk, float w) {
  const unsigned act = __activemask();
  const unsigned m = __reduce_max_sync(act, w > 0.0f ? __float_as_uint(w) : 0u);
  if ((int)lane_id() == __ffs(act) - 1 && m) atomicMax(reinterpret_cast<unsigned *>(d.wmax + blk), m);
}

// The block's mask (neg) for the two z layers that this warp of a 128-thread
// CTA holds: 16 bits of its own, so no other warp's bits are written.
__device__ __forceinline__ void note_neg(const Dev &d, int blk, const float4 &S) {
  const unsigned bits = neg_bits(S);
  if (lane_id() == 0) reinterpret_cast<uint16_t *>(d.neg + blk)[threadIdx.x >> 5] = (uint16_t)bits;
}

}  // namespace

// UpdateBlocksSimpleKernel + Voxel::Update (core/voxel.h:107-115)
__device__ __forceinline__ void integrate_simple_body(const Dev &d, Share sh) {
  __shared__ float cTw[16];
  if (threadIdx.x < 16) cTw[threadIdx.x] = d.fc->cTw[threadIdx.x];
  __syncthreads();
  const DevParams &p = d.p;
  const int n = *reinterpret_cast<volatile int *>(&d.ctr->cand_count);
  const int t = threadIdx.x;
  const int lx = (t & 1) * 4, ly = (t >> 1) & 7, lz = t >> 4;
  // the next candidate is fetched one iteration ahead
  int4 next = sh.first < n ? d.cand[sh.first] : make_int4(0, 0, 0, -1);
  for (int c = sh.first; c < n; c += sh.stride) {
    const int4 cb = next;
    if (c + sh.stride < n) next = d.cand[c + sh.stride];
    if (cb.w < 0) continue;
    const int vx0 = cb.x * MH_BLOCK_SIDE + lx, vy = cb.y * MH_BLOCK_SIDE + ly, vz = cb.z * MH_BLOCK_SIDE + lz;
    const float fx0 = (float)vx0, fy = (float)vy, fz = (float)vz;
    float sdf_new[4], w_new[4];
    bool act[4], any = false;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      act[k] = false;
      const F3 cam = voxel_in_camera(p, cTw, fx0 + (float)k, fy, fz);
      const int pix = pixel_of(p, cam);
      if (pix < 0) continue;
      const float depth = __ldg(d.depth + pix);
      if (depth_invalid(p, depth)) continue;
      float sdf = depth - cam.z;
      // 1 - normalized depth as (dmax - d) / (dmax - dmin): same value, no
      // cancellation near the far limit (update_simple.cu:49-55); the
      // compatibility mode keeps the reference's 1 - (d - dmin) / (dmax - dmin)
      const float far = p.compat ? 1.0f - normalize_depth(p, depth)
                                 : (p.max_depth_range - depth) / (p.max_depth_range - p.min_depth_range);
      const float w = fmaxf(10.0f * p.weight_sample * far, 1.0f);
      const float tr = truncate_dist(p, depth);
      if (sdf <= -tr) continue;
      sdf = sdf >= 0.0f ? fminf(tr, sdf) : fmaxf(-tr, sdf);
      sdf_new[k] = sdf;
      w_new[k] = w;
      act[k] = true;
      any = true;
    }
    // a warp that updates anything reads all its sdf: the block's mask of
    // voxels that are not non-negative is rewritten for its two layers
    if (!__any_sync(0xffffffffu, any)) continue;
    const size_t base = (size_t)cb.w * MH_BLOCK_VOXELS + t * 4;
    float4 S = *reinterpret_cast<const float4 *>(d.sdf + base);
    if (any) {
      float4 W = *reinterpret_cast<const float4 *>(d.w + base);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (!act[k]) continue;
        const float s0 = get(S, k), w0 = get(W, k);
        put(S, k, (s0 * w0 + sdf_new[k] * w_new[k]) / (w0 + w_new[k]));
        put(W, k, w0 + w_new[k]);
      }
      *reinterpret_cast<float4 *>(d.sdf + base) = S;
      *reinterpret_cast<float4 *>(d.w + base) = W;
      note_wmax(d, cb.w, fmaxf(fmaxf(W.x, W.y), fmaxf(W.z, W.w)));
    }
    __syncwarp();
    note_neg(d, cb.w, S);
  }
}
__global__ void __launch_bounds__(128) k_integrate_simple(Dev d) { integrate_simple_body(d, whole_grid()); }
__global__ void __launch_bounds__(128) k_integrate_simple_b(const Scene *t, int n) {
  each_scene(t, n, 1, [&](const Scene &c) { return c.d.p.enable_bayesian ? 0 : count_of(c.d, &Counters::cand_count); },
             [&](const Scene &c, Share sh) { integrate_simple_body(c.d, sh); });
}

// What the PSDF update needs of a pixel: depth (-inf if invalid), inlier ratio r,
// the measurement's variance and the outlier density (update_bayesian.cu:123-156).
__device__ __forceinline__ float4 pixel_record(const DevParams &p, float depth, float r) {
  const float tau = (depth - 0.4f) * 0.012f + 0.019f;
  const bool in_range = depth < p.max_depth_range && depth >= p.min_depth_range;
  const float out = p.compat ? (1.0f - r) * 1.0f / (5.0f - 0.1f) : (1.0f - r) * 0.204081632653061224f;
  return make_float4(depth_invalid(p, depth) ? -__int_as_float(0x7f800000) : depth, r, tau * tau, in_range ? out : 1.0f);
}

// The pixels' records, once per pixel instead of once per voxel that projects onto
// it.  Half a warp takes a tile of 4x4 pixels and keeps the depth up to which the
// tile updates voxels, as the bits of a float that is not negative.
__device__ __forceinline__ void pixels_body(const Dev &d, Share sh) {
  const DevParams &p = d.p;
  const int tw = far_tiles_x(p), n = tw * far_tiles_y(p), per_cta = blockDim.x / 16;
  if (sh.first == 0 && threadIdx.x == 0) d.ctr->upd_count = 0;
  for (int base = sh.first * per_cta; base < n; base += sh.stride * per_cta) {
    const int i = base + threadIdx.x / 16, j = threadIdx.x & 15;
    const unsigned x = i % tw * FAR_TILE + (j & 3), y = i / tw * FAR_TILE + (j >> 2);
    unsigned far = 0u;
    if (i < n && x < p.width && y < p.height) {
      const size_t pix = (size_t)y * p.width + x;
      const float dd = d.depth[pix];
      d.pixels[pix] = pixel_record(p, dd, d.inlier[pix]);
      const float f = dd + truncate_dist(p, dd);
      if (!depth_invalid(p, dd)) far = f <= 0.0f ? 0u : f < 1e30f ? __float_as_uint(f) : 0x7f800000u;  // NaN: no limit
    }
    far = __reduce_max_sync(lane_id() < 16 ? 0xffffu : 0xffff0000u, far);
    if (j == 0 && i < n) d.tile_far[i] = far;
  }
}
__global__ void __launch_bounds__(256) k_pixels(Dev d) { pixels_body(d, whole_grid()); }
__global__ void __launch_bounds__(256) k_pixels_b(const Scene *t, int n) {
  each_scene(t, n, 16, [&](const Scene &c) { return c.d.p.enable_bayesian ? far_tiles_x(c.d.p) * far_tiles_y(c.d.p) : 0; },
             [&](const Scene &c, Share sh) { pixels_body(c.d, sh); });
}

// Candidates that the PSDF update may change: the others lie beside the image
// or behind everything in it.  Of the 640x480 PSDF workload's candidate blocks
// 38 % update no voxel, and cost about a third of one that does; a thread here
// drops two thirds of those, and the update takes 771 us with this pass instead
// of 884 us (322x238 at 8 mm: 163 and 186 us).  A bit for each warp's two layers
// dropped another tenth of the warps and took as much longer itself.
//
// The bound is the voxels' box in the camera's axes (cTw may be any matrix) and
// the rectangle that it projects to.  `slack` and the factors are for the
// roundings of the voxels' positions (4 of 2^-24 of the terms' sizes), of their
// pixels (see pixel_of) and of this bound.  Every comparison keeps the block if
// it involves a NaN.
__device__ __forceinline__ bool may_update(const Dev &d, const float *m, int4 cb) {
  const DevParams &p = d.p;
  const float vs = p.voxel_size, h = 0.5f * (MH_BLOCK_SIDE - 1);
  const float w[3] = {((float)cb.x * MH_BLOCK_SIDE + h) * vs, ((float)cb.y * MH_BLOCK_SIDE + h) * vs,
                      ((float)cb.z * MH_BLOCK_SIDE + h) * vs};
  const float r = h * vs;
  float lo[3], hi[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const float *q = m + 4 * a;
    const float c = q[0] * w[0] + q[1] * w[1] + q[2] * w[2] + q[3];
    const float slack = 2e-6f * (fabsf(q[0]) * (fabsf(w[0]) + r) + fabsf(q[1]) * (fabsf(w[1]) + r) +
                                 fabsf(q[2]) * (fabsf(w[2]) + r) + fabsf(q[3]));
    const float e = r * 1.0001f * (fabsf(q[0]) + fabsf(q[1]) + fabsf(q[2])) + slack;
    lo[a] = c - e, hi[a] = c + e;
  }
  if (!(lo[2] > 0.01f)) return true;
  const float near = 1.0f / lo[2], away = 1.0f / hi[2];
  float u0[2], u1[2];
#pragma unroll
  for (int a = 0; a < 2; ++a) {
    const float f = a ? p.fy : p.fx, c = a ? p.cy : p.cx;
    const float s0 = f * lo[a] * (lo[a] < 0.0f ? near : away), s1 = f * hi[a] * (hi[a] > 0.0f ? near : away);
    // a voxel's pixel is the integer part of its quotient + c + 1/2
    const float eps = 0.01f + 1e-5f * (fmaxf(fabsf(s0), fabsf(s1)) + fabsf(c));
    u0[a] = fminf(s0, s1) + c + 0.5f - eps, u1[a] = fmaxf(s0, s1) + c + 0.5f + eps;
    if (!(u1[a] - u0[a] < 128.0f)) return true;
  }
  if (u1[0] <= -1.0f || u1[1] <= -1.0f || u0[0] >= (float)p.width || u0[1] >= (float)p.height) return false;
  const int tw = far_tiles_x(p), x0 = (int)fmaxf(u0[0], 0.0f) / FAR_TILE, y0 = (int)fmaxf(u0[1], 0.0f) / FAR_TILE,
            x1 = min((int)u1[0] / FAR_TILE, tw - 1), y1 = min((int)u1[1] / FAR_TILE, far_tiles_y(p) - 1);
  // a voxel is updated only if depth - z > -tr at its pixel, that is z < far
  const float z = lo[2] - 1e-5f * hi[2];
  for (int y = y0; y <= y1; ++y)
    for (int x = x0; x <= x1; ++x)
      if (!(z > __uint_as_float(__ldg(d.tile_far + y * tw + x)))) return true;
  return false;
}
__device__ __forceinline__ void upd_select_body(const Dev &d, Share sh) {
  __shared__ float cTw[16];
  if (threadIdx.x < 16) cTw[threadIdx.x] = d.fc->cTw[threadIdx.x];
  __syncthreads();
  const int n = *reinterpret_cast<volatile int *>(&d.ctr->cand_count);
  const int stride = sh.stride * blockDim.x;
  for (int base = sh.first * blockDim.x; base < n; base += stride) {
    const int i = base + threadIdx.x;
    int4 cb = make_int4(0, 0, 0, -1);
    if (i < n) cb = d.cand[i];
    const bool keep = cb.w >= 0 && may_update(d, cTw, cb);
    const unsigned m = __ballot_sync(0xffffffffu, keep);
    int slot = 0;
    if (lane_id() == 0 && m) slot = atomicAdd(&d.ctr->upd_count, __popc(m));
    slot = __shfl_sync(0xffffffffu, slot, 0);
    if (keep) d.upd_list[slot + __popc(m & lanemask_lt())] = cb;
  }
}
__global__ void __launch_bounds__(256) k_upd_select(Dev d) { upd_select_body(d, whole_grid()); }
__global__ void __launch_bounds__(256) k_upd_select_b(const Scene *t, int n) {
  each_scene(t, n, 256, [&](const Scene &c) { return c.d.p.enable_bayesian ? count_of(c.d, &Counters::cand_count) : 0; },
             [&](const Scene &c, Share sh) { upd_select_body(c.d, sh); });
}

// UpdateBlocksBayesianKernel (mapping/update_bayesian.cu:103-185).  Per voxel
// the update is division- and transcendental-bound, not load-bound, so the
// default form restates it with 4 IEEE divisions (see below); compat mode
// evaluates the reference's expressions as written.
//
// kPlanned: over the selected candidates and the pixels' records.  Without, over
// all candidates, with the records made per voxel: where the two passes before
// cost more than they save (psdf_update_direct).
template <bool kPlanned> __device__ __forceinline__ void integrate_psdf_body(const Dev &d, Share sh) {
  __shared__ float cTw[16];
  if (threadIdx.x < 16) cTw[threadIdx.x] = d.fc->cTw[threadIdx.x];
  __syncthreads();
  const DevParams &p = d.p;
  const int n = *reinterpret_cast<volatile int *>(kPlanned ? &d.ctr->upd_count : &d.ctr->cand_count);
  const int4 *list = kPlanned ? d.upd_list : d.cand;
  const int t = threadIdx.x;
  if (sh.first == 0 && t == 0) d.ctr->upd_sum += (unsigned)n;
  const int lx = (t & 1) * 4, ly = (t >> 1) & 7, lz = t >> 4;
  int4 next = sh.first < n ? list[sh.first] : make_int4(0, 0, 0, -1);
  for (int c = sh.first; c < n; c += sh.stride) {
    const int4 cb = next;
    if (c + sh.stride < n) next = list[c + sh.stride];
    if (!kPlanned && cb.w < 0) continue;
    const int vx0 = cb.x * MH_BLOCK_SIDE + lx, vy = cb.y * MH_BLOCK_SIDE + ly, vz = cb.z * MH_BLOCK_SIDE + lz;
    const float fx0 = (float)vx0, fy = (float)vy, fz = (float)vz;
    float xs[4], rs[4], ts[4], cs[4];
    bool act[4], any = false;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const F3 cam = voxel_in_camera(p, cTw, fx0 + (float)k, fy, fz);
      const int pix = pixel_of(p, cam);
      act[k] = false;
      if (pix < 0) continue;
      const float4 px = kPlanned ? __ldg(d.pixels + pix) : pixel_record(p, __ldg(d.depth + pix), __ldg(d.inlier + pix));
      const float x = px.x - cam.z;
      const float tr = truncate_dist(p, px.x);
      if (px.x == -__int_as_float(0x7f800000) || x <= -tr) continue;
      xs[k] = x >= 0.0f ? fminf(tr, x) : fmaxf(-tr, x);
      rs[k] = px.y, ts[k] = px.z, cs[k] = px.w;
      act[k] = true;
      any = true;
    }
    if (!__any_sync(0xffffffffu, any)) continue;
    const size_t base = (size_t)cb.w * MH_BLOCK_VOXELS + t * 4;
    float4 S = *reinterpret_cast<const float4 *>(d.sdf + base);
    if (any) {
      float4 W = *reinterpret_cast<const float4 *>(d.w + base);
      float4 A = *reinterpret_cast<const float4 *>(d.a + base);
      float4 B = *reinterpret_cast<const float4 *>(d.b + base);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (!act[k]) continue;
        const float x = xs[k], r = rs[k], t2 = ts[k];
        const float w0 = get(W, k);
        if (w0 == 0.0f) {
          put(S, k, x);
          put(W, k, 1.0f / t2);
          put(A, k, r * 10.0f);
          put(B, k, (1.0f - r) * 10.0f);
          continue;
        }
        const float mu = get(S, k);
        const float a = get(A, k), b = get(B, k);
        if (p.compat) {
          // the reference's expressions as written (update_bayesian.cu:140-180);
          // sqrt(2 pi) is a double there, so the product and the reciprocal of
          // gaussian() are double (geometry_helper.h:30-34)
          const float s2 = 1.0f / w0;
          const float ss2 = 1.0f / (1.0f / s2 + 1.0f / t2);
          const float m = ss2 * (mu / s2 + x / t2);
          const float sv = s2 + t2;
          const double g = 1.0 / (2.5066282746310002 * (double)sqrtf(sv)) * (double)expf(-((x - mu) * (x - mu)) / sv);
          float C1 = (float)((double)r * g);
          float C2 = cs[k];
          const float sum = C1 + C2;
          C1 /= sum;
          C2 /= sum;
          const float f = C1 * (a + 1) / (a + b + 1) + C2 * a / (a + b + 1);
          const float e =
              C1 * (a + 1) * (a + 2) / ((a + b + 1) * (a + b + 2)) + C2 * a * (a + 1) / ((a + b + 1) * (a + b + 2));
          const float nsdf = C1 * m + C2 * mu;
          const float var = C1 * (ss2 + m * m) + C2 * (s2 + mu * mu) - nsdf * nsdf;
          put(S, k, nsdf);
          put(W, k, 1.0f / var);
          const float na = (e - f) / (f - e / f);
          put(A, k, na);
          put(B, k, na * (1.0f - f) / f);
          continue;
        }
        // The same update with 4 divisions instead of 21.  With the stored
        // weight w0 = 1/s^2 and u = w0 sigma^2, q = 1/(1 + u):
        //   the product's variance s~^2 = sigma^2 q, its mean m = q (mu u + x),
        //   1/(s^2 + sigma^2) = w0 q, so gaussian() = exp(-dx^2 w0 q) sqrt(w0 q) / sqrt(2 pi);
        //   c = C1 / (C1 + C2) is the normalised inlier weight, 1 - c the outlier's;
        //   sdf' = mu + c (m - mu);
        //   the variance c s~^2 + (1 - c) s^2 + c (1 - c)(m - mu)^2 (the
        //   reference's C1 (s~^2 + m^2) + C2 (s^2 + mu^2) - sdf'^2 without its
        //   cancellation) gives w' = w0 / (c u q + (1 - c) + c (1 - c)(m - mu)^2 w0);
        //   the Beta moments f, e of the reference give a' = f (e - f) / (f^2 - e)
        //   = (a + c) k and b' = a' (1 - f) / f = (b + 1 - c) k with
        //   k = (c (a - b) - a (b + 1)) / (c^2 (a + b + 2) - (a + 2c)(b + 1)),
        //   which cancels far less than f^2 - e.
        const float u = w0 * t2;
        const float q = 1.0f / (1.0f + u);
        const float m = q * (mu * u + x);
        const float isv = w0 * q;
        const float dx = x - mu;
        // mh_expf is 1 from -2^-25 up; in observed free space (x and mu at the
        // truncation) whole warps stay there
        const float ex = -(dx * dx) * isv;
        const float g = (ex > -0x1p-25f ? 1.0f : mh_expf(ex)) * sqrtf(isv) * 0.398942280401432678f;
        const float C1 = r * g;
        const float c = C1 / (C1 + cs[k]);
        const float oc = 1.0f - c;
        const float dm = m - mu;
        put(S, k, mu + c * dm);
        put(W, k, w0 / (c * u * q + oc + c * oc * (dm * dm) * w0));
        const float b1 = b + 1.0f;
        const float kk = (c * (a - b) - a * b1) / (c * c * (a + b + 2.0f) - (a + 2.0f * c) * b1);
        put(A, k, (a + c) * kk);
        put(B, k, (b1 - c) * kk);
      }
      *reinterpret_cast<float4 *>(d.sdf + base) = S;
      *reinterpret_cast<float4 *>(d.w + base) = W;
      *reinterpret_cast<float4 *>(d.a + base) = A;
      *reinterpret_cast<float4 *>(d.b + base) = B;
      note_wmax(d, cb.w, fmaxf(fmaxf(W.x, W.y), fmaxf(W.z, W.w)));
    }
    __syncwarp();
    note_neg(d, cb.w, S);
  }
}
template <bool kPlanned>
__global__ void __launch_bounds__(128, 8) k_integrate_psdf(Dev d) { integrate_psdf_body<kPlanned>(d, whole_grid()); }
__global__ void __launch_bounds__(128, 8) k_integrate_psdf_b(const Scene *t, int n) {
  each_scene(t, n, 1, [&](const Scene &c) { return c.d.p.enable_bayesian ? count_of(c.d, &Counters::upd_count) : 0; },
             [&](const Scene &c, Share sh) { integrate_psdf_body<true>(c.d, sh); });
}

// PredictOutlierRatioKernel (mapping/update_bayesian.cu:36-101).  The
// per-pixel float max uses an integer atomicMax on the bit pattern, exact for
// the positive ratios involved (all >= 0.01).  Blocks that own no vertex are
// skipped.  The vertex normal is transformed by cTw as a point (with the
// translation), as the reference does (update_bayesian.cu:83-86).
__device__ __forceinline__ void predict_inlier_body(const Dev &d, Share sh) {
  __shared__ float cTw[16];
  if (threadIdx.x < 16) cTw[threadIdx.x] = d.fc->cTw[threadIdx.x];
  __syncthreads();
  const DevParams &p = d.p;
  const int n = *reinterpret_cast<volatile int *>(&d.ctr->vtx_list_count);
  const int t = threadIdx.x;
  const int lx = (t & 1) * 4, ly = (t >> 1) & 7, lz = t >> 4;
  for (int c = sh.first; c < n; c += sh.stride) {
    const int4 cb = d.cand[d.vtx_list[c]];
    const int pg = __ldg(d.page_of + cb.w);
    const size_t base = (size_t)cb.w * MH_BLOCK_VOXELS + t * 4;
    const int4 *vs4 = reinterpret_cast<const int4 *>(d.vtx_slot + ((size_t)pg * MH_BLOCK_VOXELS + t * 4) * 3);
    int4 q0 = vs4[0], q1 = vs4[1], q2 = vs4[2];
    int slots[12] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w, q2.x, q2.y, q2.z, q2.w};
    if (t == 0) atomicAdd(&d.ctr->predict_blocks_sum, 1ull);
    bool has = false;
#pragma unroll
    for (int k = 0; k < 12; ++k) has |= slots[k] > 0;
    if (!has) continue;
    const int vx0 = cb.x * MH_BLOCK_SIDE + lx, vy = cb.y * MH_BLOCK_SIDE + ly, vz = cb.z * MH_BLOCK_SIDE + lz;
#pragma unroll 1
    for (int k = 0; k < 4; ++k) {
      if (slots[3 * k] <= 0 && slots[3 * k + 1] <= 0 && slots[3 * k + 2] <= 0) continue;
      const int pix = pixel_of(p, voxel_in_camera(p, cTw, (float)(vx0 + k), (float)vy, (float)vz));
      if (pix < 0) continue;
      const float depth = __ldg(d.depth + pix);
      if (depth_invalid(p, depth)) continue;
      const int px = pix % p.width, py = pix / p.width;
      const float rx = ((float)px - p.cx) / p.fx, ry = ((float)py - p.cy) / p.fy;
      const F3 pc = f3(depth * rx, depth * ry, depth);
      const float vsdf = d.sdf[base + k], vw = d.w[base + k];
      const F3 npc = normalize3(f3(-pc.x, -pc.y, -pc.z));
#pragma unroll 1
      for (int s = 0; s < 3; ++s) {
        const int vp = slots[3 * k + s];
        if (vp <= 0) continue;
        const Vertex vt = d.vtx[vp];
        const F3 cn = normalize3(mul_pt(cTw, f3(vt.nx, vt.ny, vt.nz)));
        const float cos_a = dot3(npc, cn);
        const F3 cx = mul_pt(cTw, f3(vt.px, vt.py, vt.pz));
        const F3 vec = f3(pc.x - cx.x, pc.y - cx.y, pc.z - cx.z);
        const float pd = dot3(vec, cn);
        const float disk = sqrtf(dot3(vec, vec) - pd * pd);
        const float q = pd - vsdf;
        // the library's own exp (mh_exp.h) unless the reference's arithmetic
        // is asked for
        const float e_dist = -(q * q) * vw, e_disk = -fabsf(disk / vt.radius);
        const float w_dist = p.compat ? expf(e_dist) : mh_expf(e_dist);
        const float w_disk = 0.5f + 0.5f / (1.0f + (p.compat ? expf(e_disk) : mh_expf(e_disk)));
        float w_ang = (cos_a - 0.1736f) / (1.0f - 0.1736f);
        w_ang = fmaxf(w_ang, 0.1f);
        float ir = w_disk * w_dist * w_ang;
        ir = fmaxf(ir, 0.01f);
        atomicMax(reinterpret_cast<int *>(d.inlier + pix), __float_as_int(ir));
      }
    }
  }
}
__global__ void __launch_bounds__(128) k_predict_inlier(Dev d) { predict_inlier_body(d, whole_grid()); }
__global__ void __launch_bounds__(128) k_predict_inlier_b(const Scene *t, int n) {
  each_scene(t, n, 1, [&](const Scene &c) { return c.d.p.enable_bayesian ? count_of(c.d, &Counters::vtx_list_count) : 0; },
             [&](const Scene &c, Share sh) { predict_inlier_body(c.d, sh); });
}

// Candidates owning at least one vertex (and so a mesh page), for the
// inlier prediction; one thread per candidate, warp-ballot compaction.
__device__ __forceinline__ void vtx_select_body(const Dev &d, Share sh) {
  const int n = *reinterpret_cast<volatile int *>(&d.ctr->cand_count);
  const int stride = sh.stride * blockDim.x;
  for (int base = sh.first * blockDim.x; base < n; base += stride) {
    const int i = base + threadIdx.x;
    bool keep = false;
    if (i < n) {
      const int ptr = d.cand[i].w;
      keep = ptr >= 0 && d.nvtx[ptr] > 0 && d.page_of[ptr] >= 0;
    }
    const unsigned m = __ballot_sync(0xffffffffu, keep);
    int slot = 0;
    if (lane_id() == 0 && m) slot = atomicAdd(&d.ctr->vtx_list_count, __popc(m));
    slot = __shfl_sync(0xffffffffu, slot, 0);
    if (keep) d.vtx_list[slot + __popc(m & lanemask_lt())] = i;
  }
}
__global__ void __launch_bounds__(256) k_vtx_select(Dev d) { vtx_select_body(d, whole_grid()); }
__global__ void __launch_bounds__(256) k_vtx_select_b(const Scene *t, int n) {
  each_scene(t, n, 256, [&](const Scene &c) { return c.d.p.enable_bayesian ? count_of(c.d, &Counters::cand_count) : 0; },
             [&](const Scene &c, Share sh) { vtx_select_body(c.d, sh); });
}

// Sensor::Process tail: depth validity (ConvertDepthFormatKernel,
// sensor/preprocess.cu:25-42) and inlier-ratio reset to 0.1 (:10-23).  Raw
// 16-bit depth is read as the reference reads it, through a signed short, so
// raw values of 32768 and above are negative depths and invalid.
__device__ __forceinline__ void preprocess_body(const Dev &d, Share sh, const float *src, const uint16_t *src16, float range_factor) {
  const int n = d.p.width * d.p.height;
  for (int i = sh.first * blockDim.x + threadIdx.x; i < n; i += sh.stride * blockDim.x) {
    float z = src16 ? range_factor * (float)(int16_t)src16[i] : src[i];
    const bool ok = z >= d.p.min_depth_range && z <= d.p.max_depth_range;
    d.depth[i] = ok ? z : -__int_as_float(0x7f800000);
    d.inlier[i] = 0.1f;
  }
}
__global__ void k_preprocess(Dev d, const float *src, const uint16_t *src16, float range_factor) { preprocess_body(d, whole_grid(), src, src16, range_factor); }
__global__ void k_preprocess_b(const Scene *t, int n) {
  each_scene(t, n, 256, [&](const Scene &c) { return (int)(c.d.p.width * c.d.p.height); },
             [&](const Scene &c, Share sh) { preprocess_body(c.d, sh, c.src, nullptr, 0.0f); });
}

// Whether the PSDF update goes over all candidates and makes the pixels' records
// per voxel.  The two passes before the other form cost 8 us, and 20 with 640x480
// pixels; they save about a seventh of the update, which grows with the candidates:
// with the pixels, up to the blocks that fit the view.  The forms are even, us
// without / with the passes, at 64x48, 4 mm (88 / 88); 160x120, 8 mm (68 / 69);
// 240x180, 10 mm (82 / 81); 320x240, 12 mm (80 / 80): 40 pixels for each cubic
// millimetre of a voxel; and at 12 mm for larger images (640x480: 110 / 111), where
// 32 k blocks fit the view.  On one side: 32x24, 20 mm: 10 / 17; 160x120, 16 mm: 31 /
// 37; 640x480, 16 mm: 49 / 67; 640x480, 30 mm: 14 / 43; on the other: 160x120, 4 mm:
// 166 / 155; 640x480, 10 mm: 166 / 160; 640x480, 4 mm: 884 / 771.
bool psdf_update_direct(const mh_params &P) {
  const double v = P.voxel_size, z0 = P.min_depth_range, z1 = P.max_depth_range;
  const double view = std::fabs(P.width / (double)P.fx * (P.height / (double)P.fy)) * (z1 * z1 * z1 - z0 * z0 * z0) / 3.0;
  return (double)P.width * P.height <= 4e10 * v * v * v || view <= 32768.0 * 512.0 * v * v * v;
}

static int grid_persistent(int per_sm) { return mh_sm_count() * per_sm; }

int launch_integrate_simple(const Dev &d, cudaStream_t s) {
  k_integrate_simple<<<mh_resident_grid((const void *)k_integrate_simple, 128, 16), 128, 0, s>>>(d);
  mh_count_launches(1);
  return cudaGetLastError() == cudaSuccess ? MH_OK : MH_ERR_CUDA;
}
int launch_integrate_psdf(const Dev &d, cudaStream_t s) {
  if (d.p.psdf_direct) {
    k_integrate_psdf<false><<<mh_resident_grid((const void *)k_integrate_psdf<false>, 128, 16), 128, 0, s>>>(d);
    mh_count_launches(1);
    return cudaGetLastError() == cudaSuccess ? MH_OK : MH_ERR_CUDA;
  }
  k_pixels<<<std::min((far_tiles_x(d.p) * far_tiles_y(d.p) + 15) / 16, mh_sm_count() * 8), 256, 0, s>>>(d);
  k_upd_select<<<mh_sm_count() * 4, 256, 0, s>>>(d);
  k_integrate_psdf<true><<<mh_resident_grid((const void *)k_integrate_psdf<true>, 128, 16), 128, 0, s>>>(d);
  mh_count_launches(3);
  return cudaGetLastError() == cudaSuccess ? MH_OK : MH_ERR_CUDA;
}
int launch_predict_inlier(const Dev &d, cudaStream_t s) {
  MH_CUDA_TRY(cudaMemsetAsync(&d.ctr->vtx_list_count, 0, sizeof(int), s));
  k_vtx_select<<<grid_persistent(4), 256, 0, s>>>(d);
  k_predict_inlier<<<mh_resident_grid((const void *)k_predict_inlier, 128, 16), 128, 0, s>>>(d);
  mh_count_launches(2);
  return cudaGetLastError() == cudaSuccess ? MH_OK : MH_ERR_CUDA;
}
int launch_preprocess(const Dev &d, const float *src, const uint16_t *src16, float range_factor, cudaStream_t s) {
  k_preprocess<<<grid_persistent(4), 256, 0, s>>>(d, src, src16, range_factor);
  mh_count_launches(1);
  return cudaGetLastError() == cudaSuccess ? MH_OK : MH_ERR_CUDA;
}

// ------------------------------------------------------------------ batched
int launch_batch_preprocess(const Scene *t, int n, cudaStream_t s) {
  k_preprocess_b<<<mh_sm_count() * 4, 256, 0, s>>>(t, n);
  mh_count_launches(1);
  return cudaGetLastError() == cudaSuccess ? MH_OK : MH_ERR_CUDA;
}
int launch_batch_predict(const Scene *t, int n, cudaStream_t s) {
  k_vtx_select_b<<<mh_sm_count() * 4, 256, 0, s>>>(t, n);
  k_predict_inlier_b<<<mh_resident_grid((const void *)k_predict_inlier_b, 128, 16), 128, 0, s>>>(t, n);
  mh_count_launches(2);
  return cudaGetLastError() == cudaSuccess ? MH_OK : MH_ERR_CUDA;
}
// cta_per_sm caps the persistent grid (an autotuned choice)
int launch_batch_integrate(const Scene *t, int n, int has_simple, int has_psdf, int cta_per_sm, cudaStream_t s) {
  if (has_simple) {
    k_integrate_simple_b<<<mh_resident_grid((const void *)k_integrate_simple_b, 128, cta_per_sm), 128, 0, s>>>(t, n);
    mh_count_launches(1);
  }
  if (has_psdf) {
    k_pixels_b<<<mh_sm_count() * 4, 256, 0, s>>>(t, n);
    k_upd_select_b<<<mh_sm_count() * 8, 256, 0, s>>>(t, n);
    k_integrate_psdf_b<<<mh_resident_grid((const void *)k_integrate_psdf_b, 128, cta_per_sm), 128, 0, s>>>(t, n);
    mh_count_launches(3);
  }
  return cudaGetLastError() == cudaSuccess ? MH_OK : MH_ERR_CUDA;
}
// the occupancy queries of the batched persistent grids, made before any
// stream capture
void batch_warm_occupancy() {
  mh_resident_grid((const void *)k_predict_inlier_b, 128, 16);
  mh_resident_grid((const void *)k_integrate_simple_b, 128, 16);
  mh_resident_grid((const void *)k_integrate_psdf_b, 128, 16);
}

// mh_tv.cu -- primal-dual TV-L2 denoising of the input depth frame.
//
// No reference counterpart: the reference's only primal-dual code is a
// volumetric Huber-TV on voxel SDFs that is never called
// (optimize/primal_dual.cu:10-223).  This is Chambolle & Pock (2011),
// Algorithm 1 with theta = 1, on the ROF model
//     min_u  sum_edges |grad u| + lambda/2 * sum_valid (u - f)^2
// with depth in millimetres (the sensor's native unit), forward differences
// over pairs of valid pixels only (invalid pixels are holes with Neumann
// boundaries and stay invalid), tau = sigma = 1/sqrt(8).
//
// Two forms, bit-identical to each other:
//  * k_tv_iter, one launch per iteration (the allocation-free entry point):
//    each thread recomputes the dual update of its own pixel and of its left
//    and upper neighbours (the ones its divergence needs) from the previous
//    iterate, so the dual and primal steps fuse into a single pass with no
//    grid-wide barrier;
//  * k_tv_tile (a volume's frames) and its batch twin k_tv_tile_b: ten
//    iterations per launch on a tile of pixels and a 10-pixel halo, held in
//    registers, so 20 iterations take 2 launches instead of 22.
#include "mh_internal.cuh"
#include "mh_kernels.h"
#include "mh_batch.cuh"
#include "mh_round.cuh"

#include <algorithm>

namespace {

struct TvBuf {
  const float *f;
  const float *u, *ub, *px, *py;
  float *u2, *ub2, *px2, *py2;
  int W, H;
  float lambda;
};

__device__ __forceinline__ bool valid_at(const float *f, int i) { return f[i] > -1e30f; }

// dual update at pixel (x, y) from the previous iterate
__device__ __forceinline__ void dual_at(const TvBuf &b, int x, int y, float sigma, float &ox, float &oy) {
  const int i = y * b.W + x;
  const bool vi = valid_at(b.f, i);
  float gx = 0.0f, gy = 0.0f;
  if (vi && x + 1 < b.W && valid_at(b.f, i + 1)) gx = b.ub[i + 1] - b.ub[i];
  if (vi && y + 1 < b.H && valid_at(b.f, i + b.W)) gy = b.ub[i + b.W] - b.ub[i];
  const float qx = b.px[i] + sigma * gx;
  const float qy = b.py[i] + sigma * gy;
  const float nrm = fmaxf(1.0f, sqrtf(qx * qx + qy * qy));
  ox = qx / nrm;
  oy = qy / nrm;
}

}  // namespace

__device__ __forceinline__ void tv_init_body(const float *depth, float *f, float *u, float *ub, float *px, float *py, int n) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float z = depth[i];
    const bool ok = z > 0.0f && z < 1e30f;
    const float v = ok ? z * 1000.0f : -__int_as_float(0x7f800000);
    f[i] = v;
    u[i] = v;
    ub[i] = v;
    px[i] = 0.0f;
    py[i] = 0.0f;
  }
}
__global__ void k_tv_init(const float *depth, float *f, float *u, float *ub, float *px, float *py, int n) { tv_init_body(depth, f, u, ub, px, py, n); }

__device__ __forceinline__ void tv_iter_body(const TvBuf &b) {
  const float tau = 0.35355339059327373f, sigma = 0.35355339059327373f;
  const int n = b.W * b.H;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int x = i % b.W, y = i / b.W;
    float pxc, pyc;
    dual_at(b, x, y, sigma, pxc, pyc);
    b.px2[i] = pxc;
    b.py2[i] = pyc;
    if (!valid_at(b.f, i)) {
      b.u2[i] = b.f[i];
      b.ub2[i] = b.f[i];
      continue;
    }
    float pxl = 0.0f, pyu = 0.0f, dummy;
    if (x > 0) dual_at(b, x - 1, y, sigma, pxl, dummy);
    if (y > 0) dual_at(b, x, y - 1, sigma, dummy, pyu);
    const float div = (pxc - pxl) + (pyc - pyu);
    const float u0 = b.u[i];
    const float un = (u0 + tau * div + tau * b.lambda * b.f[i]) / (1.0f + tau * b.lambda);
    b.u2[i] = un;
    b.ub2[i] = 2.0f * un - u0;
  }
}
__global__ void __launch_bounds__(256) k_tv_iter(TvBuf b) { tv_iter_body(b); }

__device__ __forceinline__ void tv_out_body(const float *f, const float *u, float *depth, int n, Share sh) {
  for (int i = sh.first * blockDim.x + threadIdx.x; i < n; i += sh.stride * blockDim.x)
    depth[i] = valid_at(f, i) ? u[i] * 0.001f : -__int_as_float(0x7f800000);
}
__global__ void k_tv_out(const float *f, const float *u, float *depth, int n) { tv_out_body(f, u, depth, n, whole_grid()); }
// a batch's TV result after `launches` tiled launches: planes 1-4 hold the
// iterate after an even number of launches, planes 5-8 after an odd number
__global__ void k_tv_out_b(const Scene *t, int n, int launches) {
  each_scene(t, n, 256, [&](const Scene &c) { return (int)(c.d.p.width * c.d.p.height); },
             [&](const Scene &c, Share sh) {
    const size_t np = (size_t)c.d.p.width * c.d.p.height;
    tv_out_body(c.tv, c.tv + np * ((launches & 1) ? 5 : 1), c.d.depth, (int)np, sh);
  });
}

// ------------------------------------------------------------------ tiled
// Up to TV_K iterations per launch for one tile of pixels: the tile and a
// TV_K-pixel halo form a region whose values go stale by one pixel per
// iteration from its edge inwards, so the tile's own pixels stay exact through
// TV_K iterations.  Each value is computed by the same expressions as
// tv_iter_body (the dual of a neighbour is the neighbour's own new dual), so
// the result is bit-identical to running k_tv_iter once per iteration.  The
// first launch initialises from the depth frame (as k_tv_init), the last
// writes the frame back (as k_tv_out); between launches the iterate goes
// through the ping-pong planes.
//
// A thread owns a strip of R rows of one column and keeps its state in
// registers.  Shared memory carries what a strip reads of its neighbours: the
// extrapolated iterate to the right and below, the duals to the left and
// above.  Bound by instruction issue, so validity is kept as bits and norm and
// quotients are the rounded ones of mh_round.cuh, without branches: they are
// those of the operators for depths within 2^-10 .. 2^30 mm (`plain`, for the
// whole region; a dual value below 2^-60, which they may round otherwise,
// cannot change the iterate then).  640x480, 20 iterations: 125 -> 48 us
// (96 us with the operators' division and square root).
#define TV_K 10

struct TvTile {
  const float *depth_in;  // first launch: the depth frame (metres); else null
  float *depth_out;       // last launch: the frame to write; else null
  float *f;               // input plane (written by the first launch)
  const float *u, *ub, *px, *py;  // iterate in (unused by the first launch)
  float *u2, *ub2, *px2, *py2;    // iterate out (unused by the last launch)
  int W, H, iters;
  float lambda;
};

// Region of RW = TW + 2 TV_K columns and RH = R G rows (the tile: RH - 2 TV_K),
// one thread for each column of each of the G strips.
template <int TW, int R, int G> struct TvShape {
  static constexpr int RW = TW + 2 * TV_K, RH = R * G, TH = RH - 2 * TV_K, THREADS = (RW * G + 31) / 32 * 32;
};

template <int TW, int R, int G> __device__ __forceinline__ void tv_tile_body(const TvTile &b, int tile_x, int tile_y) {
  typedef TvShape<TW, R, G> T;
  __shared__ float s_ub[T::RH][T::RW], s_px[T::RH][T::RW], s_py[G][T::RW];
  const float tau = 0.35355339059327373f, sigma = 0.35355339059327373f;
  const float NI = -__int_as_float(0x7f800000);
  const int lx = threadIdx.x % T::RW, g = threadIdx.x / T::RW, ly0 = g * R;
  const int x0 = tile_x * TW - TV_K, y0 = tile_y * T::TH - TV_K, gx = x0 + lx, gy0 = y0 + ly0;
  const bool live = g < G;  // the last warp's surplus threads only keep the barriers
  const float den = 1.0f + tau * b.lambda, rden = 1.0f / den;
  // tf: tau lambda f, the data term
  float tf[R], u[R], ub[R], px[R], py[R];
  unsigned valid = 0, right = 0, below = 0;
  bool plain = den < 0x1p20f;
  if (live) {
#pragma unroll
    for (int j = 0; j < R; ++j) {
      const int gy = gy0 + j;
      float f = NI;  // outside the image: like a hole
      u[j] = ub[j] = NI, px[j] = py[j] = 0.0f;
      if (gx >= 0 && gx < b.W && gy >= 0 && gy < b.H) {
        const int i = gy * b.W + gx;
        if (b.depth_in) {
          const float z = b.depth_in[i];
          const bool ok = z > 0.0f && z < 1e30f;
          f = u[j] = ub[j] = ok ? z * 1000.0f : NI;
          if (lx >= TV_K && lx < TV_K + TW && ly0 + j >= TV_K && ly0 + j < TV_K + T::TH) b.f[i] = f;
        } else {
          f = b.f[i], u[j] = b.u[i], ub[j] = b.ub[i], px[j] = b.px[i], py[j] = b.py[i];
        }
      }
      if (f > -1e30f) valid |= 1u << j, plain = plain && f > 0x1p-10f && f < 0x1p30f;
      tf[j] = tau * b.lambda * f;
      s_px[ly0 + j][lx] = f;
    }
  }
  plain = __syncthreads_and(plain);
  // pairs of valid pixels: to the right and below
  if (live) {
#pragma unroll
    for (int j = 0; j < R; ++j) {
      const bool vi = valid >> j & 1u;
      if (vi && gx + 1 < b.W && lx + 1 < T::RW && s_px[ly0 + j][lx + 1] > -1e30f) right |= 1u << j;
      if (vi && gy0 + j + 1 < b.H && ly0 + j + 1 < T::RH && s_px[ly0 + j + 1][lx] > -1e30f) below |= 1u << j;
      s_ub[ly0 + j][lx] = ub[j];
    }
  }
  __syncthreads();
  const bool has_left = gx > 0 && lx > 0, has_above = gy0 > 0 && ly0 > 0;
  for (int it = 0; it < b.iters; ++it) {
    // dual step (dual_at): forward differences of ub over valid pairs; the
    // norm max(1, sqrt(n2)) is sqrt(max(1, n2))
    if (live) {
#pragma unroll
      for (int j = 0; j < R; ++j) {
        float gxd = 0.0f, gyd = 0.0f;
        if (right >> j & 1u) gxd = s_ub[ly0 + j][lx + 1] - ub[j];
        if (below >> j & 1u) gyd = (j + 1 < R ? ub[(j + 1) % R] : s_ub[ly0 + R][lx]) - ub[j];
        const float qx = px[j] + sigma * gxd;
        const float qy = py[j] + sigma * gyd;
        const float n2 = qx * qx + qy * qy;
        if (plain) {
          const float nrm = sqrt_round(fmaxf(1.0f, n2)), rn = rcp_round(nrm);
          px[j] = mh_div(qx, nrm, rn), py[j] = mh_div(qy, nrm, rn);
        } else {
          const float nrm = fmaxf(1.0f, sqrtf(n2));
          px[j] = qx / nrm, py[j] = qy / nrm;
        }
        s_px[ly0 + j][lx] = px[j];
      }
      s_py[g][lx] = py[R - 1];
    }
    __syncthreads();
    // primal step and extrapolation (tv_iter_body); invalid pixels keep -inf
    if (live) {
#pragma unroll
      for (int j = 0; j < R; ++j) {
        const float pxl = has_left ? s_px[ly0 + j][lx - 1] : 0.0f;
        const float pyu = j > 0 ? py[(j + R - 1) % R] : has_above ? s_py[g - 1][lx] : 0.0f;
        const float div = (px[j] - pxl) + (py[j] - pyu);
        const float u0 = u[j];
        const float num = u0 + tau * div + tf[j];
        const float un = plain ? mh_div(num, den, rden) : num / den;
        if (valid >> j & 1u) {
          u[j] = un;
          ub[j] = 2.0f * un - u0;
          s_ub[ly0 + j][lx] = ub[j];
        }
      }
    }
    __syncthreads();
  }
  if (!live || lx < TV_K || lx >= TV_K + TW || gx >= b.W) return;
#pragma unroll
  for (int j = 0; j < R; ++j) {
    const int gy = gy0 + j;
    if (ly0 + j < TV_K || ly0 + j >= TV_K + T::TH || gy >= b.H) continue;
    const int i = gy * b.W + gx;
    if (b.depth_out) {
      b.depth_out[i] = valid >> j & 1u ? u[j] * 0.001f : NI;
    } else {
      b.u2[i] = u[j], b.ub2[i] = ub[j], b.px2[i] = px[j], b.py2[i] = py[j];
    }
  }
}

// Tile shapes, largest first.  A launch takes the smallest whose tiles fit the
// SMs in one wave: the time of a launch is that of one region, so a small image
// spreads over more SMs although its halos cost more (322x238, 20 iterations:
// 128 -> 32 us; 640x480 with the largest: 48 us).  The batch, whose scenes fill
// the GPU together, takes the largest.
#define TV_SHAPE0 64, 5, 11
#define TV_SHAPE1 32, 4, 10
#define TV_SHAPE2 16, 2, 16
template <int TW, int R, int G>
__global__ void __launch_bounds__(TvShape<TW, R, G>::THREADS) k_tv_tile(TvTile b) {
  tv_tile_body<TW, R, G>(b, blockIdx.x, blockIdx.y);
}
template <int TW, int R, int G> static bool launch_tv_tile(const TvTile &b, bool any, cudaStream_t s) {
  typedef TvShape<TW, R, G> T;
  const dim3 grid((b.W + TW - 1) / TW, (b.H + T::TH - 1) / T::TH);
  if (!any && (long long)grid.x * grid.y > mh_sm_count()) return false;
  k_tv_tile<TW, R, G><<<grid, T::THREADS, 0, s>>>(b);
  return true;
}

typedef TvShape<TV_SHAPE0> TvBatch;
int tv_tile_count(int W, int H) { return ((W + 63) / 64) * ((H + TvBatch::TH - 1) / TvBatch::TH); }

// Launch `launch` (of ceil(iterations / TV_K)) of the tiled TV for every
// active scene: the scenes' tiles are concatenated (Scene::tv_tile0); planes
// 1-4 of a scene's TV scratch hold the iterate after an even number of
// launches, planes 5-8 after an odd number.  Bit-identical to the single
// scene's launches, and so to one launch per iteration.
__global__ void __launch_bounds__(TvBatch::THREADS) k_tv_tile_b(const Scene *t, int n, int total, int launch, int iters, int last,
                                                    float lambda) {
  each_tile(t, n, total, &Scene::tv_tile0, [&](const Scene &c, int lt) {
    const int W = c.d.p.width, H = c.d.p.height;
    const size_t np = (size_t)W * H;
    float *A = c.tv + np * ((launch & 1) ? 5 : 1), *B = c.tv + np * ((launch & 1) ? 1 : 5);
    TvTile b;
    b.depth_in = launch == 0 ? c.d.depth : nullptr;
    b.depth_out = (launch > 0 && last) ? c.d.depth : nullptr;
    b.f = c.tv;
    b.u = A, b.ub = A + np, b.px = A + 2 * np, b.py = A + 3 * np;
    b.u2 = B, b.ub2 = B + np, b.px2 = B + 2 * np, b.py2 = B + 3 * np;
    b.W = W, b.H = H, b.iters = iters, b.lambda = lambda;
    const int tw = (W + 63) / 64;
    tv_tile_body<TV_SHAPE0>(b, lt % tw, lt / tw);
    __syncthreads();  // the next tile reuses the shared arrays
  });
}

int launch_denoise_tv_iterated(const Dev &d, float *tv, float lambda, int iterations, cudaStream_t s);

// tv holds 9 planes of W*H floats: f, (u, ub, px, py) x 2
int launch_denoise_tv(const Dev &d, float *tv, float lambda, int iterations, cudaStream_t s) {
  const int W = d.p.width, H = d.p.height, n = W * H;
  if (iterations <= 0) return launch_denoise_tv_iterated(d, tv, lambda, iterations, s);
  float *A[4] = {tv + (size_t)n, tv + 2 * (size_t)n, tv + 3 * (size_t)n, tv + 4 * (size_t)n};
  float *B[4] = {tv + 5 * (size_t)n, tv + 6 * (size_t)n, tv + 7 * (size_t)n, tv + 8 * (size_t)n};
  int launches = 0;
  for (int done = 0; done < iterations; done += TV_K) {
    TvTile b;
    b.depth_in = done == 0 ? d.depth : nullptr;
    b.iters = std::min(TV_K, iterations - done);
    // the first launch reads the frame, so it never writes it back (other
    // tiles may still be reading their halos)
    b.depth_out = (done > 0 && done + b.iters == iterations) ? d.depth : nullptr;
    b.f = tv;
    b.u = A[0], b.ub = A[1], b.px = A[2], b.py = A[3];
    b.u2 = B[0], b.ub2 = B[1], b.px2 = B[2], b.py2 = B[3];
    b.W = W, b.H = H, b.lambda = lambda;
    if (!launch_tv_tile<TV_SHAPE2>(b, false, s) && !launch_tv_tile<TV_SHAPE1>(b, false, s))
      launch_tv_tile<TV_SHAPE0>(b, true, s);
    ++launches;
    for (int k = 0; k < 4; ++k) std::swap(A[k], B[k]);
  }
  if (iterations <= TV_K) {
    const int g = min((n + 255) / 256, mh_sm_count() * 8);
    k_tv_out<<<g, 256, 0, s>>>(tv, A[0], d.depth, n);
    ++launches;
  }
  mh_count_launches(launches);
  return cudaGetLastError() == cudaSuccess ? MH_OK : MH_ERR_CUDA;
}

// the one-launch-per-iteration form (zero iterations, and the reference
// timing of the tiled form)
int launch_denoise_tv_iterated(const Dev &d, float *tv, float lambda, int iterations, cudaStream_t s) {
  const int W = d.p.width, H = d.p.height, n = W * H;
  const int g = min((n + 255) / 256, mh_sm_count() * 8);
  float *f = tv;
  float *A[4] = {tv + (size_t)n, tv + 2 * (size_t)n, tv + 3 * (size_t)n, tv + 4 * (size_t)n};
  float *B[4] = {tv + 5 * (size_t)n, tv + 6 * (size_t)n, tv + 7 * (size_t)n, tv + 8 * (size_t)n};
  k_tv_init<<<g, 256, 0, s>>>(d.depth, f, A[0], A[1], A[2], A[3], n);
  for (int it = 0; it < iterations; ++it) {
    TvBuf b;
    b.f = f;
    b.u = A[0], b.ub = A[1], b.px = A[2], b.py = A[3];
    b.u2 = B[0], b.ub2 = B[1], b.px2 = B[2], b.py2 = B[3];
    b.W = W, b.H = H, b.lambda = lambda;
    k_tv_iter<<<g, 256, 0, s>>>(b);
    for (int k = 0; k < 4; ++k) {
      float *t = A[k];
      A[k] = B[k];
      B[k] = t;
    }
  }
  k_tv_out<<<g, 256, 0, s>>>(f, A[0], d.depth, n);
  mh_count_launches(2 + iterations);
  return cudaGetLastError() == cudaSuccess ? MH_OK : MH_ERR_CUDA;
}

// ------------------------------------------------------------------ no-alloc
// TV denoising for callers that cannot allocate device memory: the nine
// scratch planes live in a fixed file-scope device array.  See
// mh_denoise_tv_static in include/meshhash.h.
#include <mutex>

static __device__ __align__(256) float g_tv_static_scratch[(size_t)MH_TV_STATIC_MAX_PIXELS * 9];

namespace {
std::mutex g_tv_static_mu;
float *g_tv_static_ptr[64] = {nullptr};  // per device: address of the array above
}  // namespace

extern "C" int mh_denoise_tv_static(const float *depth_in, float *depth_out, int width, int height, float lambda,
                                    int iterations, void *stream) {
  if (!depth_in || !depth_out || width <= 0 || height <= 0 || iterations < 0 || !(lambda > 0.0f))
    return MH_ERR_INVALID;
  if ((long long)width * height > (long long)MH_TV_STATIC_MAX_PIXELS) return MH_ERR_CAPACITY;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return MH_ERR_CUDA;
  cudaStream_t s = (cudaStream_t)stream;
  float *scratch = nullptr;
  {
    // Host code only sees a host-side stand-in for the array, so its device
    // address is looked up with the device current.  Outside a stream
    // capture the lookup runs on every call: after cudaDeviceReset the
    // module is loaded again and the array may sit at another address.
    // While the stream captures, the address found by the last call outside
    // a capture on this device is used.
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &cap) != cudaSuccess) return MH_ERR_CUDA;
    std::lock_guard<std::mutex> lock(g_tv_static_mu);
    if (cap == cudaStreamCaptureStatusNone) {
      void *p = nullptr;
      if (cudaGetSymbolAddress(&p, g_tv_static_scratch) != cudaSuccess || !p) return MH_ERR_CUDA;
      g_tv_static_ptr[dev] = static_cast<float *>(p);
    }
    scratch = g_tv_static_ptr[dev];
    if (!scratch) return MH_ERR_INVALID;
  }
  const int n = width * height;
  const int g = min((n + 255) / 256, mh_sm_count() * 8);
  float *f = scratch;
  float *A[4] = {scratch + (size_t)n, scratch + 2 * (size_t)n, scratch + 3 * (size_t)n, scratch + 4 * (size_t)n};
  float *B[4] = {scratch + 5 * (size_t)n, scratch + 6 * (size_t)n, scratch + 7 * (size_t)n,
                 scratch + 8 * (size_t)n};
  // every plane the iterations read is written here first, so no state from
  // an earlier call leaks into this one
  k_tv_init<<<g, 256, 0, s>>>(depth_in, f, A[0], A[1], A[2], A[3], n);
  for (int it = 0; it < iterations; ++it) {
    TvBuf b;
    b.f = f;
    b.u = A[0], b.ub = A[1], b.px = A[2], b.py = A[3];
    b.u2 = B[0], b.ub2 = B[1], b.px2 = B[2], b.py2 = B[3];
    b.W = width, b.H = height, b.lambda = lambda;
    k_tv_iter<<<g, 256, 0, s>>>(b);
    for (int k = 0; k < 4; ++k) {
      float *t = A[k];
      A[k] = B[k];
      B[k] = t;
    }
  }
  k_tv_out<<<g, 256, 0, s>>>(f, A[0], depth_out, n);
  mh_count_launches(2 + iterations);
  return cudaGetLastError() == cudaSuccess ? MH_OK : MH_ERR_CUDA;
}

// ------------------------------------------------------------------ batched
// The batch's TV: the tiled kernel over all scenes' tiles, TV_K iterations
// per launch (20 iterations: 2 launches instead of 22).
int launch_batch_tv(const Scene *t, int n, int tv_tiles, float lambda, int iterations, cudaStream_t s) {
  if (iterations <= 0 || tv_tiles <= 0) return MH_OK;
  const int launches = (iterations + TV_K - 1) / TV_K;
  const int g = std::max(1, std::min(tv_tiles, mh_sm_count()));
  for (int k = 0; k < launches; ++k) {
    const int iters = std::min(TV_K, iterations - k * TV_K);
    k_tv_tile_b<<<g, TvBatch::THREADS, 0, s>>>(t, n, tv_tiles, k, iters, k == launches - 1 ? 1 : 0, lambda);
  }
  int count = launches;
  if (launches == 1) {
    // one launch reads the frame, so the result is written back separately
    const int g2 = std::max(1, mh_sm_count() * 8);
    k_tv_out_b<<<g2, 256, 0, s>>>(t, n, 1);
    ++count;
  }
  mh_count_launches(count);
  return cudaGetLastError() == cudaSuccess ? MH_OK : MH_ERR_CUDA;
}

// mh_huber.cu -- volumetric Huber-TV smoothing of the fused sdf.
//
// The reference's primal-dual regulariser (optimize/primal_dual.cu:10-223 with
// the neighbour queries of geometry/primal_dual_query.h:15-234), which its
// engines never call, as an optional post-fusion stage over the candidate
// blocks:
//   init   for voxels with inv_sigma2 >= 1e-6: weight = exp(|grad sdf| / voxel)
//          from forward differences (0 when a +x/+y/+z neighbour is missing or
//          unobserved), sdf0 = sdf, sdf_bar = 0, p = 0, mask set;
//   pass 1 (dual)   data error (sdf - sdf0)^2 and Huber(|grad sdf|, 0.02);
//          p = (p + sigma grad sdf_bar) / (1 + sigma alpha), then p /= max(1, |p|);
//   pass 2 (primal) div = sum_i (p(v - e_i) - p(v))_i; sdf -= tau div;
//          sdf = (sdf + lambda w tau sdf0) / (1 + lambda w tau); sdf = sdf0
//          where w > 2; sdf_bar = 2 sdf - sdf_prev.
// Differences use face neighbours that exist, are observed and carry the
// mask; otherwise the gradient (or divergence) is 0, as in the reference.
// The per-voxel state (7 words) lives in arrays laid out like the voxel
// storage, allocated on first use; the mask is an epoch stamp, so voxels not
// initialised by the latest init read as unmasked.  All passes run one CTA per
// candidate block over a face-neighbour table; the iterations' per-voxel flags
// are built once per call, so no pass waits on a hash probe or tests its
// neighbours' weights again.
#include <cstring>

#include "mh_kernels.h"
#include "mh_round.cuh"
#include "mh_volume.h"

namespace {

constexpr float kEps = 1e-6f;     // EPSILON (core/common.h:62)
constexpr float kAlpha = 0.02f;   // Huber threshold (primal_dual.cu:60)

struct PD {
  float *sdf0, *bar, *w, *px, *py, *pz;
  unsigned *mask;
  unsigned epoch;
};

__device__ __forceinline__ int cand_count(const Dev &d) { return *reinterpret_cast<volatile int *>(&d.ctr->cand_count); }

// Face-neighbour table of the candidate list: nbt[6 c + 2 k + (s < 0)] is
// the pool index of the block next to candidate c along axis k, direction
// s (-1 when absent).  One lookup per thread, so the table costs one pass of
// independent hash probes instead of a serial probe per block and pass.
__device__ __forceinline__ void find_faces(const Dev &d, int *nbt) {
  const int n = cand_count(d);
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < 6 * n; t += gridDim.x * blockDim.x) {
    const int c = t / 6, j = t - 6 * c;
    const int4 cb = d.cand[c];
    int q = -1;
    if (cb.w >= 0) {
      const int k = j >> 1, s = (j & 1) ? -1 : 1;
      q = hash_find(d, cb.x + (k == 0) * s, cb.y + (k == 1) * s, cb.z + (k == 2) * s);
    }
    nbt[t] = q;
  }
}
__global__ void __launch_bounds__(256) k_pd_faces(Dev d, int *nbt) { find_faces(d, nbt); }

// neighbour usable by the masked queries: block exists, voxel observed, mask set
__device__ __forceinline__ bool usable(const Dev &d, const PD &pd, long long g) {
  return g >= 0 && d.w[g] >= kEps && pd.mask[g] == pd.epoch;
}

// All passes run one 128-thread CTA per candidate block: thread t holds
// the four voxels x = 4 (t & 1) .. + 3 of row y = t / 2 & 7 of layer z = t / 16,
// so a field moves as one float4 per thread.
__device__ __forceinline__ int first_voxel(int t) { return t * 4; }

// The voxels of a block that the masked queries may use, a byte for each row of
// 8 voxels along x; `known` (cleared before) tells that the block's bytes are of
// this call, `active` whether the candidate has such a voxel at all.  The face
// table is made here too: a launch less in calls of few blocks.
__global__ void __launch_bounds__(128) k_pd_usable(Dev d, PD pd, int *nbt, uint8_t *use, uint8_t *known,
                                                   uint8_t *active) {
  find_faces(d, nbt);
  const int n = cand_count(d), t = threadIdx.x;
  for (int c = blockIdx.x; c < n; c += gridDim.x) {
    const int blk = d.cand[c].w;
    if (blk < 0) {
      if (t == 0) active[c] = 0;
      continue;
    }
    const size_t base = (size_t)blk * MH_BLOCK_VOXELS + first_voxel(t);
    const float4 w = *reinterpret_cast<const float4 *>(d.w + base);
    const uint4 m = *reinterpret_cast<const uint4 *>(pd.mask + base);
    unsigned f = 0;
    if (w.x >= kEps && m.x == pd.epoch) f |= 1u;
    if (w.y >= kEps && m.y == pd.epoch) f |= 2u;
    if (w.z >= kEps && m.z == pd.epoch) f |= 4u;
    if (w.w >= kEps && m.w == pd.epoch) f |= 8u;
    const unsigned hi = __shfl_down_sync(0xffffffffu, f, 1);
    if (!(t & 1)) use[(size_t)blk * 64 + t / 2] = (uint8_t)(f | hi << 4);
    const int any = __syncthreads_or(f != 0u);
    if (t == 0) known[blk] = 1, active[c] = any ? 1 : 0;
  }
}

// What a thread needs to know of a candidate before it can load its part of it: the
// pool block, the voxels' flags and the blocks of the face voxels that it brings in
// (two of 192 at most; side: the faces' place in the table).
struct Visit {
  int c, blk, q[2];
  unsigned f;
  __device__ __forceinline__ void load(const Dev &d, const int *nbt, const uint16_t *flags, int side, int cand) {
    c = cand;
    if (c < 0) return;
    const int t = threadIdx.x;
    blk = d.cand[c].w;
    f = flags[(size_t)c * 128 + t];
    q[0] = __ldg(nbt + 6 * c + 2 * (t >> 6) + side);
    q[1] = t < 64 ? __ldg(nbt + 6 * c + 4 + side) : -1;
  }
};
// Runs visit(Visit) for the active ones of this CTA's candidates, with all 128
// threads.  Their bytes are read 128 at a time, so the others cost next to nothing,
// and the next one's Visit is loaded while the last one is worked on.  (With 200 of
// 49 k candidates initialised, ten iterations take 0.22 ms; with the flags of each
// candidate read in each pass they took 0.39.)
template <class F>
__device__ __forceinline__ void each_active(const Dev &d, const int *nbt, const uint8_t *active, const uint16_t *flags,
                                            int side, F &&visit) {
  __shared__ unsigned bits[4];
  const int n = cand_count(d);
  for (int first = blockIdx.x; first < n; first += 128 * gridDim.x) {
    const int c = first + threadIdx.x * gridDim.x;
    const unsigned b = __ballot_sync(0xffffffffu, c < n && active[c]);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) bits[threadIdx.x >> 5] = b;
    __syncthreads();
    int w = 0;
    unsigned left = bits[0];
    auto next = [&]() {
      while (!left && w < 3) left = bits[++w];
      if (!left) return -1;
      const int k = 32 * w + __ffs(left) - 1;
      left &= left - 1u;
      return first + k * (int)gridDim.x;
    };
    Visit v;
    v.load(d, nbt, flags, side, next());
    while (v.c >= 0) {
      Visit after;
      after.load(d, nbt, flags, side, next());
      visit(v);
      v = after;
    }
  }
}

// Flags of a call, 16 bits a thread: bits 0-3 the voxel is usable, 4-7 its
// three upper face neighbours are usable too, 8-11 its three lower ones.
// Neither pass changes the weights or the mask, so they hold for all
// iterations of the call.  A thread takes a row from the bytes of k_pd_usable:
// reading weights and masks of the faces' voxels, a 32-byte sector each along
// x, took 250 us for 120 k blocks against 134 us for both passes.
__global__ void __launch_bounds__(128) k_pd_flags(Dev d, PD pd, const int *nbt, const uint8_t *use,
                                                  const uint8_t *known, const uint8_t *active, uint16_t *flags) {
  const int n = cand_count(d), row = threadIdx.x & 63, y = row & 7, z = row >> 3;
  for (int c = blockIdx.x * 2 + (threadIdx.x >> 6); c < n; c += gridDim.x * 2) {
    if (!active[c]) continue;
    const int blk = d.cand[c].w;
    unsigned *out = reinterpret_cast<unsigned *>(flags) + (size_t)c * 64 + row;
    // row r of the neighbour `face`, the voxels `want` of it
    auto beyond = [&](int face, int r, unsigned want) -> unsigned {
      const int q = __ldg(nbt + 6 * c + face);
      if (q < 0) return 0u;
      if (known[q]) return use[(size_t)q * 64 + r];
      unsigned f = 0;
      for (int x = 0; x < 8; ++x)
        if ((want >> x & 1u) && usable(d, pd, (long long)q * MH_BLOCK_VOXELS + r * 8 + x)) f |= 1u << x;
      return f;
    };
    const uint8_t *own = use + (size_t)blk * 64;
    const unsigned u = own[row];
    unsigned f = 0u;
    if (u) {
      const unsigned xu = u >> 1 | (u & 128u ? (beyond(0, row, 1u) & 1u) << 7 : 0u);
      const unsigned xl = (u << 1 & 255u) | (u & 1u ? beyond(1, row, 128u) >> 7 : 0u);
      const unsigned yu = y < 7 ? own[row + 1] : beyond(2, row - 7, u), yl = y > 0 ? own[row - 1] : beyond(3, row + 7, u);
      const unsigned zu = z < 7 ? own[row + 8] : beyond(4, row - 56, u), zl = z > 0 ? own[row - 8] : beyond(5, row + 56, u);
      const unsigned up = u & xu & yu & zu, lo = u & xl & yl & zl;
      f = (u & 15u) | (up & 15u) << 4 | (lo & 15u) << 8 | (u >> 4) << 16 | (up >> 4) << 20 | (lo >> 4) << 24;
    }
    *out = f;
  }
}

__device__ __forceinline__ float lane4(const float4 &v, int k) { return k == 0 ? v.x : k == 1 ? v.y : k == 2 ? v.z : v.w; }
__device__ __forceinline__ float4 load4(const float *f, size_t base) { return *reinterpret_cast<const float4 *>(f + base); }
__device__ __forceinline__ void store4(float *f, size_t base, const float *v) {
  *reinterpret_cast<float4 *>(f + base) = make_float4(v[0], v[1], v[2], v[3]);
}

// A block's field with the layers above it on each axis, 9 x 9 x 9 (edges and
// corners unused), and with those below it.
struct Tile9 {
  float v[729];
};
// own voxels of the tile; off = 1 leaves room for the layers below
__device__ __forceinline__ void tile_own(Tile9 &s, int t, int off, const float4 &v) {
  const int i = first_voxel(t);
  float *o = s.v + (i & 7) + off + 9 * (((i >> 3) & 7) + off) + 81 * ((i >> 6) + off);
  o[0] = v.x, o[1] = v.y, o[2] = v.z, o[3] = v.w;
}
// Whether the voxel of the block that faces voxel i of the neighbour's face needs
// it: the flags (16 bits a thread) of the block's last layer (up) or its first.
__device__ __forceinline__ bool face_needed(const uint16_t *flags, int i, int k, bool up) {
  const int a = i & 7, b = i >> 3, in = up ? 7 : 0;
  const int li = k == 0 ? in + 8 * a + 64 * b : k == 1 ? a + 8 * in + 64 * b : a + 8 * b + 64 * in;
  return flags[li >> 2] >> ((up ? 4 : 8) + (li & 3)) & 1u;
}
// 64 voxels of a neighbour's face of axis k: its first layer (up) or its last
__device__ __forceinline__ void tile_face(Tile9 &s, int i, int k, bool up, int q, const float *field) {
  if (q < 0) return;  // no voxel here has the neighbour: the flags say so
  const int a = i & 7, b = i >> 3, in = up ? 0 : 7, out = up ? 8 : 0, off = up ? 0 : 1;
  const int li = k == 0 ? in + 8 * a + 64 * b : k == 1 ? a + 8 * in + 64 * b : a + 8 * b + 64 * in;
  const int o = k == 0 ? out + 9 * (a + off) + 81 * (b + off) : k == 1 ? a + off + 9 * out + 81 * (b + off)
                                                                      : a + off + 9 * (b + off) + 81 * out;
  s.v[o] = __ldg(field + (size_t)q * MH_BLOCK_VOXELS + li);
}

template <int NV> __device__ __forceinline__ void cta_sum(float (&v)[NV], double *acc) {
  __shared__ float red[NV][8];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (int k = 0; k < NV; ++k) {
    float x = v[k];
    for (int o = 16; o; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    if (lane == 0) red[k][wid] = x;
  }
  __syncthreads();
  if (threadIdx.x < NV) {
    double s = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += red[threadIdx.x][w];
    atomicAdd(acc + threadIdx.x, s);
  }
}

// a / b for y = RN(1 / b), b of moderate size: without the operator's tests,
// which send the many zeros down its long way (the sign of a zero is not kept:
// nothing depends on it)
__device__ __forceinline__ float pd_div(float a, float b, float y) {
  const float m = fabsf(a);
  return (m > 0x1p-60f && m < 0x1p60f) || m == 0.0f ? mh_div(a, b, y) : a / b;
}

// The Huber norm of a vector of squared length n2
__device__ __forceinline__ float pd_huber(float n2) {
  const float x = n2 == 0.0f ? 0.0f : n2 > 0x1p-60f && n2 < 0x1p60f ? sqrt_round(n2) : sqrtf(n2);
  return x < kAlpha ? pd_div(0.5f * (x * x), kAlpha, 1.0f / kAlpha) : x - 0.5f * kAlpha;
}

// PrimalDualInit: weights from the gradient, the iterate's start.  Bound by the
// traffic, 36 B a voxel and the faces: 490 us for 120 k blocks, where a thread a
// voxel took 508.
__global__ void __launch_bounds__(128) k_pd_init(Dev d, PD pd, const int *nbt, unsigned *fresh) {
  __shared__ Tile9 sdf, weight;
  const int n = cand_count(d), t = threadIdx.x;
  if (blockIdx.x == 0 && t == 0) *fresh = pd.epoch;
  for (int c = blockIdx.x; c < n; c += gridDim.x) {
    const int blk = d.cand[c].w;
    if (blk < 0) continue;
    const size_t base = (size_t)blk * MH_BLOCK_VOXELS + first_voxel(t);
    const float4 W = load4(d.w, base), S = load4(d.sdf, base);
    const bool any = W.x >= kEps || W.y >= kEps || W.z >= kEps || W.w >= kEps;
    if (!__syncthreads_or(any)) continue;
    tile_own(sdf, t, 0, S), tile_own(weight, t, 0, W);
    for (int i = t; i < 192; i += 128) {
      const int k = i >> 6, q = __ldg(nbt + 6 * c + 2 * k), a = i & 7, b = i >> 3 & 7;
      const int o = k == 0 ? 8 + 9 * a + 81 * b : k == 1 ? a + 72 + 81 * b : a + 9 * b + 648;
      weight.v[o] = 0.0f;
      tile_face(sdf, i & 63, k, true, q, d.sdf);
      tile_face(weight, i & 63, k, true, q, d.w);
    }
    __syncthreads();
    if (any) {
      const int i0 = first_voxel(t), o0 = (i0 & 7) + 9 * ((i0 >> 3) & 7) + 81 * (i0 >> 6);
      float w[4], s0[4];
      unsigned m[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        // what a voxel that is not observed gets is not read: its mask differs
        w[k] = 0.0f, s0[k] = lane4(S, k), m[k] = 0u;
        if (!(lane4(W, k) >= kEps)) continue;
        const float *o = sdf.v + o0 + k, *q = weight.v + o0 + k;
        float gr[3] = {0.0f, 0.0f, 0.0f};
        if (q[1] >= kEps && q[9] >= kEps && q[81] >= kEps) gr[0] = o[1] - s0[k], gr[1] = o[9] - s0[k], gr[2] = o[81] - s0[k];
        const float len = sqrtf(gr[0] * gr[0] + gr[1] * gr[1] + gr[2] * gr[2]);
        w[k] = expf(len / d.p.voxel_size);
        m[k] = pd.epoch;
      }
      const float zero[4] = {0.0f, 0.0f, 0.0f, 0.0f};
      store4(pd.w, base, w), store4(pd.sdf0, base, s0), store4(pd.bar, base, zero);
      store4(pd.px, base, zero), store4(pd.py, base, zero), store4(pd.pz, base, zero);
      *reinterpret_cast<uint4 *>(pd.mask + base) = make_uint4(m[0], m[1], m[2], m[3]);
    }
    __syncthreads();
  }
}

// Dual step (PrimalDualIteratePass1Kernel), with the energies where they are
// asked for.  28 B a voxel (the extrapolated sdf and the dual read, the dual
// written; 8 more for the energies) and the faces; bound by the latency of a block's
// loads, so ten CTAs an SM (48 registers): 361 us for 120 k blocks, 1.45 GB, against
// 390 us with the registers that the compiler takes.  One thread per entry of a list
// of usable voxels took 660 us and read 12 B more a voxel; with the operators'
// divisions this form takes 700 us.  In blocks with few usable voxels the list was
// better: with 35 of 512 in each of 7 k blocks ten iterations take 0.42 ms, and took
// 0.25 ms.  After an init, before the first
// primal step (fresh), the extrapolated sdf is 0 and so is the new dual: there is
// nothing to do.  The device knows that, since graphs may replay the calls.
template <bool kEnergy>
__global__ void __launch_bounds__(128, 10) k_pd_dual(Dev d, PD pd, const int *nbt, const uint8_t *active,
                                                     const uint16_t *flags, const unsigned *fresh, float sigma,
                                                     double *err) {
  __shared__ Tile9 bar, sdf;
  __shared__ uint16_t block_flags[128];
  const float4 none = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  const int t = threadIdx.x;
  const float h = 1.0f + sigma * kAlpha, rh = 1.0f / h;
  const bool h_ok = h > 0x1p-20f && h < 0x1p20f;
  if (!kEnergy && h_ok && *fresh == pd.epoch) return;
  float e[2] = {0.0f, 0.0f};
  each_active(d, nbt, active, flags, 0, [&](const Visit &v) {
    const unsigned f = v.f;
    block_flags[t] = (uint16_t)f;
    __syncthreads();
    const size_t base = (size_t)v.blk * MH_BLOCK_VOXELS + first_voxel(t);
    // a thread without a usable voxel needs none of its own, nor does a neighbour
    float4 B = none, X = none, Y = none, Z = none, S = none, S0 = none;
    if (f) {
      B = load4(pd.bar, base), X = load4(pd.px, base), Y = load4(pd.py, base), Z = load4(pd.pz, base);
      if (kEnergy) S = load4(d.sdf, base), S0 = load4(pd.sdf0, base);
    }
    tile_own(bar, t, 0, B);
    if (kEnergy) tile_own(sdf, t, 0, S);
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      const int i = t + 128 * m, k = i >> 6;
      if (i >= 192 || !face_needed(block_flags, i & 63, k, true)) continue;
      tile_face(bar, i & 63, k, true, v.q[m], pd.bar);
      if (kEnergy) tile_face(sdf, i & 63, k, true, v.q[m], d.sdf);
    }
    __syncthreads();
    const int i0 = first_voxel(t), o0 = (i0 & 7) + 9 * ((i0 >> 3) & 7) + 81 * (i0 >> 6);
    float px[4], py[4], pz[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      px[k] = lane4(X, k), py[k] = lane4(Y, k), pz[k] = lane4(Z, k);
      if (!(f >> k & 1u)) continue;
      const float b = lane4(B, k);
      const float *o = bar.v + o0 + k;
      float gb[3] = {0.0f, 0.0f, 0.0f};
      if (f >> (4 + k) & 1u) gb[0] = o[1] - b, gb[1] = o[9] - b, gb[2] = o[81] - b;
      if (kEnergy) {
        const float s = lane4(S, k);
        const float *os = sdf.v + o0 + k;
        float gs[3] = {0.0f, 0.0f, 0.0f};
        if (f >> (4 + k) & 1u) gs[0] = os[1] - s, gs[1] = os[9] - s, gs[2] = os[81] - s;
        const float dd = fabsf(s - lane4(S0, k));
        e[0] += dd * dd;
        e[1] += pd_huber(gs[0] * gs[0] + gs[1] * gs[1] + gs[2] * gs[2]);
      }
      float x = px[k] + sigma * gb[0], y = py[k] + sigma * gb[1], z = pz[k] + sigma * gb[2];
      if (h_ok) x = pd_div(x, h, rh), y = pd_div(y, h, rh), z = pd_div(z, h, rh);
      else x /= h, y /= h, z /= h;
      // max(1, sqrt(n2)) is sqrt(max(1, n2))
      const float n2 = x * x + y * y + z * z;
      if (n2 < 0x1p60f) {
        const float nrm = sqrt_round(fmaxf(1.0f, n2)), rn = rcp_round(nrm);
        px[k] = pd_div(x, nrm, rn), py[k] = pd_div(y, nrm, rn), pz[k] = pd_div(z, nrm, rn);
      } else {
        const float nrm = fmaxf(1.0f, sqrtf(n2));
        px[k] = x / nrm, py[k] = y / nrm, pz[k] = z / nrm;
      }
    }
    if (f) store4(pd.px, base, px), store4(pd.py, base, py), store4(pd.pz, base, pz);
    __syncthreads();
  });
  if (kEnergy) cta_sum<2>(e, err);
}

// Primal step and extrapolation (PrimalDualIteratePass2Kernel).  Bound by the
// traffic: 32 B a voxel (the dual, sdf, sdf0 and the weight read, sdf and its
// extrapolation written) and the faces: 309 us for 120 k blocks, 1.84 GB at 6.0 TB/s;
// 382 us without the limit to 48 registers.
__global__ void __launch_bounds__(128, 10) k_pd_primal(Dev d, PD pd, const int *nbt, const uint8_t *active,
                                                       const uint16_t *flags, unsigned *fresh, float lambda,
                                                       float tau) {
  __shared__ Tile9 tx, ty, tz;
  __shared__ uint16_t block_flags[128];
  const float4 none = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  const int t = threadIdx.x;
  if (blockIdx.x == 0 && t == 0) *fresh = 0u;
  each_active(d, nbt, active, flags, 1, [&](const Visit &v) {
    const unsigned f = v.f;
    block_flags[t] = (uint16_t)f;
    __syncthreads();
    const size_t base = (size_t)v.blk * MH_BLOCK_VOXELS + first_voxel(t);
    const float4 S = load4(d.sdf, base);  // all of it, for the block's mask
    float4 X = none, Y = none, Z = none, S0 = none, Wt = none;
    if (f) {
      X = load4(pd.px, base), Y = load4(pd.py, base), Z = load4(pd.pz, base);
      S0 = load4(pd.sdf0, base), Wt = load4(pd.w, base);
    }
    tile_own(tx, t, 1, X), tile_own(ty, t, 1, Y), tile_own(tz, t, 1, Z);
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      const int i = t + 128 * m, k = i >> 6;
      if (i >= 192 || !face_needed(block_flags, i & 63, k, false)) continue;
      if (k == 0) tile_face(tx, i & 63, 0, false, v.q[m], pd.px);
      else if (k == 1) tile_face(ty, i & 63, 1, false, v.q[m], pd.py);
      else tile_face(tz, i & 63, 2, false, v.q[m], pd.pz);
    }
    __syncthreads();
    const int i0 = first_voxel(t), o0 = (i0 & 7) + 1 + 9 * (((i0 >> 3) & 7) + 1) + 81 * ((i0 >> 6) + 1);
    float so[4] = {S.x, S.y, S.z, S.w}, bo[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (!(f >> k & 1u)) continue;
      float div = 0.0f;
      if (f >> (8 + k) & 1u) {
        const int o = o0 + k;
        div = (tx.v[o - 1] - lane4(X, k)) + (ty.v[o - 9] - lane4(Y, k)) + (tz.v[o - 81] - lane4(Z, k));
      }
      const float prev = so[k], s0 = lane4(S0, k), w = lane4(Wt, k);
      const float lam = lambda * w;
      float s = prev - tau * div;
      s = (s + lam * tau * s0) / (1.0f + lam * tau);
      if (w > 2.0f) s = s0;
      so[k] = s;
      bo[k] = 2.0f * s - prev;
    }
    // voxels that are not usable keep their sdf, and their extrapolation too: a
    // later call may find them observed again
    if (f) store4(d.sdf, base, so);
    if ((f & 15u) == 15u) {
      store4(pd.bar, base, bo);
    } else {
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (f >> k & 1u) pd.bar[base + k] = bo[k];
    }
    // a warp holds two layers of the block, as in the fusion kernels
    const unsigned neg = neg_bits(make_float4(so[0], so[1], so[2], so[3]));
    if ((t & 31) == 0) reinterpret_cast<uint16_t *>(d.neg + v.blk)[t >> 5] = (uint16_t)neg;
    __syncthreads();
  });
}

}  // namespace

struct mh_pd_state {
  PD pd;
  double *err = nullptr;      // the energies, and after them `known`: cleared together
  int *nbt = nullptr;   // face-neighbour table of the candidate list (6 per candidate)
  uint16_t *flags = nullptr;  // per-voxel flags of the call (128 words per candidate)
  uint8_t *use = nullptr;     // usable voxels, 64 bytes per pool block
  uint8_t *known = nullptr;   // blocks whose bytes this call wrote
  uint8_t *active = nullptr;  // candidates with a usable voxel
  unsigned *fresh = nullptr;  // epoch of an init that no primal step has followed: bar and p are 0
};

static int grid_of(const void *fn, int block = 256) { return mh_resident_grid(fn, block, 2048 / block); }

static int pd_ensure(mh_volume *v) {
  if (v->pd) return MH_OK;
  // 120 GB of state beside 69 GB of voxels
  if (v->hp.value_capacity > (1u << 23)) return MH_ERR_INVALID;
  mh_pd_state *st = new mh_pd_state();
  const size_t nv = (size_t)v->hp.value_capacity * MH_BLOCK_VOXELS;
  float **f[6] = {&st->pd.sdf0, &st->pd.bar, &st->pd.w, &st->pd.px, &st->pd.py, &st->pd.pz};
  bool ok = true;
  for (float **p : f) ok = ok && cudaMalloc((void **)p, sizeof(float) * nv) == cudaSuccess;
  ok = ok && cudaMalloc((void **)&st->pd.mask, sizeof(unsigned) * nv) == cudaSuccess;
  ok = ok && cudaMalloc((void **)&st->err, sizeof(double) * 2 + (size_t)v->hp.value_capacity) == cudaSuccess;
  st->known = reinterpret_cast<uint8_t *>(st->err + 2);
  ok = ok && cudaMalloc((void **)&st->nbt, sizeof(int) * 6 * (size_t)v->hp.value_capacity) == cudaSuccess;
  ok = ok && cudaMalloc((void **)&st->flags, sizeof(uint16_t) * 128 * (size_t)v->hp.value_capacity) == cudaSuccess;
  ok = ok && cudaMalloc((void **)&st->use, 64 * (size_t)v->hp.value_capacity) == cudaSuccess;
  ok = ok && cudaMalloc((void **)&st->active, (size_t)v->hp.value_capacity) == cudaSuccess;
  ok = ok && cudaMalloc((void **)&st->fresh, sizeof(unsigned)) == cudaSuccess;
  ok = ok && cudaMemset(st->pd.mask, 0, sizeof(unsigned) * nv) == cudaSuccess;
  st->pd.epoch = 0;
  v->pd = st;
  if (!ok) {
    cudaGetLastError();  // the failed allocation must not surface at the next launch check
    mh_pd_free(v);
    return MH_ERR_NOMEM;
  }
  return MH_OK;
}

void mh_pd_free(mh_volume *v) {
  mh_pd_state *st = v->pd;
  if (!st) return;
  for (void *p : {(void *)st->pd.sdf0, (void *)st->pd.bar, (void *)st->pd.w, (void *)st->pd.px, (void *)st->pd.py,
                  (void *)st->pd.pz, (void *)st->pd.mask, (void *)st->err, (void *)st->nbt,
                  (void *)st->flags, (void *)st->use, (void *)st->active, (void *)st->fresh})
    if (p) cudaFree(p);
  delete st;
  v->pd = nullptr;
}

extern "C" {

int mh_huber_tv_init(mh_volume *v, void *stream) {
  if (!v) return MH_ERR_INVALID;
  int r = pd_ensure(v);
  if (r != MH_OK) return r;
  mh_pd_state *st = v->pd;
  st->pd.epoch += 1;
  cudaStream_t s = (cudaStream_t)stream;
  k_pd_faces<<<grid_of((const void *)k_pd_faces), 256, 0, s>>>(v->d, st->nbt);
  k_pd_init<<<grid_of((const void *)k_pd_init, 128), 128, 0, s>>>(v->d, st->pd, st->nbt, st->fresh);
  mh_count_launches(2);
  return cudaGetLastError() == cudaSuccess ? MH_OK : MH_ERR_CUDA;
}

int mh_huber_tv_iterate(mh_volume *v, float lambda, float sigma, float tau, int iterations, double *energy,
                        void *stream) {
  if (!v || iterations < 0) return MH_ERR_INVALID;
  if (!v->pd || v->pd->pd.epoch == 0) return MH_ERR_STATE;
  cudaStream_t s = (cudaStream_t)stream;
  mh_pd_state *st = v->pd;
  double last[2] = {0.0, 0.0};
  if (iterations > 0) {
    // the candidate list may have changed since init: rebuild the face table
    // and the flags of this call (neither pass changes w or the mask)
    MH_CUDA_TRY(cudaMemsetAsync(st->err, 0, sizeof(double) * 2 + (size_t)v->hp.value_capacity, s));
    k_pd_usable<<<grid_of((const void *)k_pd_usable, 128), 128, 0, s>>>(v->d, st->pd, st->nbt, st->use, st->known,
                                                                       st->active);
    k_pd_flags<<<grid_of((const void *)k_pd_flags, 128), 128, 0, s>>>(v->d, st->pd, st->nbt, st->use, st->known,
                                                                     st->active, st->flags);
    mh_count_launches(2);
  }
  const int gd = grid_of((const void *)k_pd_dual<false>, 128), ge = grid_of((const void *)k_pd_dual<true>, 128),
            gp = grid_of((const void *)k_pd_primal, 128);
  for (int it = 0; it < iterations; ++it) {
    // only the last pass's energies are returned
    if (it + 1 == iterations)
      k_pd_dual<true><<<ge, 128, 0, s>>>(v->d, st->pd, st->nbt, st->active, st->flags, st->fresh, sigma, st->err);
    else
      k_pd_dual<false><<<gd, 128, 0, s>>>(v->d, st->pd, st->nbt, st->active, st->flags, st->fresh, sigma, nullptr);
    k_pd_primal<<<gp, 128, 0, s>>>(v->d, st->pd, st->nbt, st->active, st->flags, st->fresh, lambda, tau);
    mh_count_launches(2);
  }
  MH_CUDA_TRY(cudaGetLastError());
  if (energy && iterations > 0) {
    MH_CUDA_TRY(cudaMemcpyAsync(last, st->err, sizeof(last), cudaMemcpyDeviceToHost, s));
    MH_CUDA_TRY(cudaStreamSynchronize(s));
    // as the reference prints it: lambda / 2 * data + tv, then data, tv
    energy[0] = last[0] * lambda / 2.0 + last[1];
    energy[1] = last[0];
    energy[2] = last[1];
  }
  return MH_OK;
}

}  // extern "C"

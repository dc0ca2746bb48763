"""Cases over which this framework's speed is measured.

Each case is what one program that uses the library does again and again: a
scanner that fuses one depth frame after another, a rig of cameras stepped as
one batch, a viewer that renders the map, a tracker, an optimiser that takes
gradients through the renderer, a smoother.  Everything runs through the
public host layer (``Volume``, ``Batch``).

Inputs are drawn from the seed: a room (or a floor plan) of its own, a camera
path, and depth frames rendered on the GPU with the sensor's noise (sigma =
0.0012 z^2, 5 % outliers in [0.3, 5] m and 2 % missing pixels; the plain TSDF
case has the Gaussian part only).  The maps that a case starts from are fused
from the frames that come before its own, by the same calls.

Outputs are images in the caller's buffers, poses, gradients and counts.  The
order of the block pool varies from run to run, so gradients of voxels are
returned by block position.
"""
import math

import numpy as np
import torch

from meshhashing_gb300 import Batch, Volume, config
from meshhashing_gb300 import scene as scenes
from meshhashing_gb300.pose import left_update

TV_LAMBDA = 0.1


# ------------------------------------------------------------------ the cases

def listed():
    # A scan is a whole pass of a scanner from an empty map: every frame through the chain (denoising, allocation,
    # fusion, meshing, garbage collection, the model's image), then the counts that the program looks at.
    return [
        # a small plain-TSDF sensor (a robot's ToF camera): launches and latency
        dict(name="scan_tsdf_160", kind="scan", mode="tsdf", plan=False, width=160, height=120, voxel=0.008, frames=15,
             tv=0, host=False, maps="depth"),
        # the plain TSDF workload: 320x240, the circle, 8 mm
        dict(name="scan_tsdf_320", kind="scan", mode="tsdf", plan=False, width=320, height=240, voxel=0.008, frames=45,
             tv=0, host=False, maps="all"),
        # a ragged image from host memory, every map read back to the host, long enough for the surfaces to be meshed
        dict(name="scan_psdf_322_host", kind="scan", mode="psdf", plan=False, width=322, height=238, voxel=0.008,
             frames=60, tv=20, host=True, maps="all"),
        # the PSDF workload: 640x480, 4 mm, frames in device memory
        dict(name="scan_psdf_640", kind="scan", mode="psdf", plan=False, width=640, height=480, voxel=0.004, frames=48,
             tv=20, host=False, maps="all"),
        # the streaming walk through a floor plan, frames from and depth to pinned host memory
        dict(name="scan_plan_640_host", kind="scan", mode="psdf", plan=True, width=640, height=480, voxel=0.005,
             frames=32, tv=20, host=True, maps="depth"),
        # many small and middling scenes advanced together, from empty maps
        dict(name="batch_16", kind="batch", scenes=16, frames=12, tv=20),
        # a viewer: the map of a 640x480 sequence from poses off its path, and a thumbnail of one
        dict(name="render_640", kind="render", width=640, height=480, voxel=0.004, fused=40),
        dict(name="render_161", kind="render", width=161, height=119, voxel=0.008, fused=30),
        # pose and voxel gradients through the renderer, forward and backward
        dict(name="gradient_320", kind="gradient", width=320, height=240, voxel=0.008, fused=24),
        # frame-to-model tracking: 10 Gauss-Newton iterations from a perturbed pose
        dict(name="track_640", kind="track", width=640, height=480, voxel=0.004, fused=64, iterations=10),
        # volumetric Huber-TV of the fused map, then a look at it
        dict(name="smooth_320", kind="smooth", width=320, height=240, voxel=0.006, fused=40, iterations=10),
        # the depth denoiser by itself, to a host image
        dict(name="denoise_640", kind="denoise", width=640, height=480, iterations=20),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(("scan", "scan", "scan", "scan", "batch", "render", "render", "gradient", "track", "smooth",
                       "denoise"))
    width = int(_log(rng, 96, 641))
    height = max(72, min(480, int(width * rng.uniform(0.6, 0.8))))
    # 4 mm at every size; coarser voxels up to 8 mm
    voxel = round(_log(rng, 0.004, 0.008), 5)
    if kind == "scan":
        mode = rng.choice(("psdf", "psdf", "tsdf"))
        host = rng.random() < 0.4
        if host:                # host images have even sides
            width, height = width - width % 2, height - height % 2
        return dict(kind=kind, mode=mode, plan=mode == "psdf" and rng.random() < 0.3, width=width, height=height,
                    voxel=voxel if mode == "psdf" else max(voxel, 0.006), frames=rng.randint(6, 40),
                    tv=rng.choice((0, 5, 20, 23)) if mode == "psdf" else 0, host=host,
                    maps=rng.choice(("depth", "all")))
    if kind == "batch":
        return dict(kind=kind, scenes=rng.randint(3, 16), frames=rng.randint(4, 12), tv=rng.choice((0, 20)))
    if kind == "denoise":
        return dict(kind=kind, width=width, height=height, iterations=rng.randint(3, 30))
    case = dict(kind=kind, width=width, height=height, voxel=max(voxel, 0.006) if kind != "render" else voxel,
                fused=rng.randint(8, 40))
    if kind in ("track", "smooth"):
        case["iterations"] = rng.randint(3, 10)
    return case


def work(case):
    """Bytes that a pass cannot do without.  Blocks in view are estimated from
    the view's volume and the share of it that the outliers have allocated."""
    if case["kind"] == "batch":
        parts = [work(dict(kind="scan", mode="psdf", maps="all", frames=case["frames"], **c)) for c in _mix(case["scenes"])]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    px = case["width"] * case["height"]
    if case["kind"] == "denoise":
        return {"bytes": 8.0 * px, "flops": 30.0 * px * case["iterations"]}
    tsdf = case.get("mode") == "tsdf"
    block = (8 * case["voxel"]) ** 3
    surface = 6.0 * 3 / (8 * case["voxel"]) ** 2
    volume = 7.0 / block                  # between the camera and the surface

    def seen(frames):
        return surface if tsdf else surface + volume * (1.0 - math.exp(-frames * 0.05 * px / volume))

    images = px * (4 if case.get("maps") == "depth" else 36)
    look = surface * (2048 + 16)          # the blocks at the surface that an image shows
    if case["kind"] == "scan":
        n = case["frames"]
        blocks = sum(seen(k + 1) for k in range(n))
        return {"bytes": blocks * 512 * (16 if tsdf else 32) + n * (px * 8 + look + images),
                "flops": blocks * 512 * 60.0 + n * px * 2000.0}
    blocks = seen(case["fused"])
    if case["kind"] == "render":
        return {"bytes": look + images, "flops": px * 2000.0}
    if case["kind"] == "gradient":
        return {"bytes": 2 * look + images + px * 20.0 + blocks * 2048, "flops": px * 5000.0}
    if case["kind"] == "track":
        n = case["iterations"] + 1
        return {"bytes": n * (look + px * 4.0), "flops": n * px * 2000.0}
    # smooth: per observed voxel and iteration sdf, sdf_bar and the dual, read and written, the weight and sdf0 read
    voxels = blocks * 512
    return {"bytes": case["iterations"] * voxels * 48.0 + look + images, "flops": case["iterations"] * voxels * 60.0}


# ------------------------------------------------------------------ inputs

def _render(sc, cam, poses, chunk=16):
    """Noise-free z-depth (F, H, W) of the analytic scene, float64, 0 where nothing is hit."""
    dev = dict(dtype=torch.float64, device="cuda")
    u = (torch.arange(cam.width, **dev) - cam.cx) / cam.fx
    v = (torch.arange(cam.height, **dev) - cam.cy) / cam.fy
    dc = torch.stack([u[None, :].expand(cam.height, -1), v[:, None].expand(-1, cam.width),
                      torch.ones(cam.height, cam.width, **dev)], -1).reshape(-1, 3)
    out = []
    for k in range(0, len(poses), chunk):
        T = torch.tensor(np.stack(poses[k:k + chunk]), **dev)
        o, d = T[:, None, :3, 3], dc @ T[:, :3, :3].transpose(1, 2)
        inv = 1.0 / d
        lo, hi = torch.tensor(sc.room_lo, **dev), torch.tensor(sc.room_hi, **dev)
        t = torch.where(d > 0, (hi - o) * inv, torch.where(d < 0, (lo - o) * inv, torch.inf)).amin(-1)
        a = (d * d).sum(-1)
        for s in sc.spheres:
            oc = o - torch.tensor(s[:3], **dev)
            b, c = (d * oc).sum(-1), (oc * oc).sum(-1) - float(s[3]) ** 2
            disc = b * b - a * c
            sq = disc.clamp(min=0).sqrt()
            t0, t1 = (-b - sq) / a, (-b + sq) / a
            th = torch.where(t0 > 1e-9, t0, torch.where(t1 > 1e-9, t1, torch.inf))
            t = torch.minimum(t, torch.where(disc >= 0, th, torch.inf))
        for bx in sc.boxes:
            t1, t2 = (torch.tensor(bx[:3], **dev) - o) * inv, (torch.tensor(bx[3:], **dev) - o) * inv
            near, far = torch.fmin(t1, t2).amax(-1), torch.fmax(t1, t2).amin(-1)
            th = torch.where(near > 1e-9, near, far)
            t = torch.minimum(t, torch.where((far >= near) & (far > 1e-9), th, torch.inf))
        out.append(torch.where(torch.isfinite(t), t, 0.0))
    return torch.cat(out).reshape(len(poses), cam.height, cam.width)


def _noisy(z, seed, outliers=0.05, zeros=0.02):
    g = torch.Generator("cuda").manual_seed(seed)
    z = torch.where(z > 0, z + torch.randn(z.shape, generator=g, device="cuda", dtype=z.dtype) * 0.0012 * z * z, 0.0)
    if outliers:
        far = torch.rand(z.shape, generator=g, device="cuda", dtype=z.dtype) * 4.7 + 0.3
        z = torch.where(torch.rand(z.shape, generator=g, device="cuda") < outliers, far, z)
        z = torch.where(torch.rand(z.shape, generator=g, device="cuda") < zeros, 0.0, z)
    return z.float()


def _camera(width, height):
    f = 525.0 * width / 640.0
    return scenes.Camera(width, height, f, f, (width - 1) / 2.0, (height - 1) / 2.0)


def _sequence(case, seed, n):
    """n frames (on the device) and their poses; a TSDF case's camera goes round a circle of 60 frames."""
    cam = _camera(case["width"], case["height"])
    if case.get("mode") == "tsdf":
        sc, poses = scenes.room_scene(seed), scenes.circle_trajectory(60)
        first = seed % 60
        poses = [poses[(first + i) % 60] for i in range(n)]
        frames = _noisy(_render(sc, cam, poses), seed, outliers=0.0)
    elif case.get("plan"):
        sc, poses = scenes.floor_plan_scene(seed), scenes.floor_plan_walk(n, seed)
        frames = _noisy(_render(sc, cam, poses), seed)
    else:
        sc, poses = scenes.room_scene(seed, extra=6), scenes.spline_trajectory(n, seed)
        frames = _noisy(_render(sc, cam, poses), seed)
    return cam, frames, [p.astype(np.float32) for p in poses]


def _volume(case, cam, frames):
    """A volume whose pools hold what `frames` frames of this size allocate (with a margin)."""
    v = case["voxel"]
    if case.get("mode") == "tsdf":
        cap = int(2 ** 17 * max(1.0, (0.008 / v) ** 2))
        return Volume(config.make_params(cam.width, cam.height, cam.fx, cam.fy, cam.cx, cam.cy, voxel_size=v,
                                         truncation=3 * v, bayesian=False, bucket_count=1 << 18, value_capacity=cap,
                                         weight_sample=200, max_vertex_count=1 << 21, max_triangle_count=1 << 22))
    k = 53108.0 * (cam.width * cam.height / 307200.0) ** 0.62 * (0.004 / v) ** 1.4
    cap = int(1.8 * k * frames ** 0.62) // 1024 * 1024 + 8192
    buckets = 1 << max(14, (cap - 1).bit_length())
    return Volume(config.make_params(cam.width, cam.height, cam.fx, cam.fy, cam.cx, cam.cy, voxel_size=v,
                                     truncation=3 * v, bayesian=True, bucket_count=buckets, value_capacity=cap,
                                     max_vertex_count=1 << 20, max_triangle_count=1 << 21,
                                     overflow_capacity=max(buckets // 4, 1024),
                                     mesh_page_capacity=min(cap, max(cap // 12, 8192))))


class State:
    pass


def _images(case, cam, host):
    make = (lambda *s: torch.empty(s, pin_memory=True)) if host else (lambda *s: torch.empty(s, device="cuda"))
    out = {"ray_depth": make(cam.height, cam.width)}
    if case.get("maps") != "depth":
        out["ray_vertex"] = make(cam.height, cam.width, 4)
        out["ray_normal"] = make(cam.height, cam.width, 4)
    return out


def _fused(case, seed, more=0):
    """A state with a volume that holds the case's frames, and `more` frames after them."""
    s = State()
    s.cam, frames, s.poses = _sequence(case, seed, case["fused"] + more)
    s.vol = _volume(case, s.cam, case["fused"] + more)
    s.tv = case.get("tv", 20)
    for i in range(case["fused"]):
        s.vol.integrate_frame(frames[i], s.poses[i], on_device=True, tv_iterations=s.tv, tv_lambda=TV_LAMBDA)
    s.frames = frames[case["fused"]:].clone()
    s.poses = s.poses[case["fused"] - (0 if more else 1):]
    return s


def _mix(n):
    """The scenes of a batch: sizes and voxels of the batched-fusion workload in turn, the largest now and then."""
    sizes = ((160, 120), (320, 240), (160, 120), (320, 240), (640, 480))
    return [dict(width=sizes[i % 5][0], height=sizes[i % 5][1], voxel=(0.008, 0.006, 0.004, 0.006)[i % 4])
            for i in range(n)]


class _View:
    """A scene's output buffer as an array; keeps the batch that owns it alive."""

    def __init__(self, owner, ptr, shape):
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=shape, typestr="<f4", data=(ptr, False), version=3)


def _inverse(T):
    return np.linalg.inv(np.asarray(T, np.float64)).astype(np.float32)


def prepare(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng(seed)
    if kind == "scan":
        s = State()
        s.cam, frames, s.poses = _sequence(case, seed, case["frames"])
        s.vol = _volume(case, s.cam, case["frames"])
        s.host, s.tv = case["host"], case["tv"]
        s.images = _images(case, s.cam, s.host)
        s.frames = [f.cpu().pin_memory() if s.host else f for f in frames]
    elif kind == "batch":
        s = State()
        n, total = case["scenes"], case["frames"]
        vols, s.frames, s.poses = [], [], []
        for i, spec in enumerate(_mix(n)):
            c = dict(kind="batch", **spec)
            cam, frames, poses = _sequence(c, seed * 64 + i, total)
            vols.append(_volume(c, cam, total))
            s.frames.append(frames)
            s.poses.append(poses)
        s.batch = Batch(vols, raycast=True)
        s.views = []
        for i, v in enumerate(vols):
            shapes = ((v.RH, v.RW), (v.RH, v.RW, 4), (v.RH, v.RW, 4))
            s.views.append([torch.as_tensor(_View(s.batch, p, sh), device="cuda")
                            for p, sh in zip(s.batch.outputs(i), shapes)])
        s.tv, s.count = case["tv"], total
    elif kind == "render":
        s = _fused(case, seed)
        # off the path by a few centimetres and degrees
        s.cTw = _inverse(left_update(s.poses[0], np.r_[rng.standard_normal(3) * 0.05, rng.standard_normal(3) * 0.05]))
        s.images = _images(case, s.cam, False)
    elif kind == "gradient":
        s = _fused(case, seed)
        s.cTw = _inverse(s.poses[0])
        H, W, cap = s.cam.height, s.cam.width, s.vol.params.value_capacity
        s.depth, s.normal = torch.empty(H, W, device="cuda"), torch.empty(H, W, 4, device="cuda")
        g = torch.Generator("cuda").manual_seed(seed)
        s.g_depth = torch.randn((H, W), generator=g, device="cuda")
        s.g_normal = torch.randn((H, W, 4), generator=g, device="cuda") * 0.01
        # pool index of every block in the order of its position, then the pool's free entries
        probe = torch.zeros(cap, 512, device="cuda")
        probe[:, 0] = torch.arange(cap, device="cuda")
        pos, rows = s.vol.dump_block_field(probe)
        live = rows[:, 0][np.lexsort(pos.T)].astype(np.int64)
        free = np.ones(cap, bool)
        free[live] = False
        s.rows = torch.from_numpy(np.r_[live, np.nonzero(free)[0]]).cuda()
        s.grad = probe
    elif kind == "track":
        s = _fused(case, seed, 1)
        s.start = left_update(s.poses[0], np.r_[rng.standard_normal(3) * 0.02,
                                                rng.standard_normal(3) * math.radians(1.0)])
        s.obs = torch.where((s.frames[0] >= 0.5) & (s.frames[0] <= 4.0), s.frames[0], -torch.inf)
        s.iterations = case["iterations"]
    elif kind == "smooth":
        s = _fused(case, seed)
        s.cTw = _inverse(s.poses[0])
        s.images = _images(case, s.cam, False)
        s.iterations = case["iterations"]
    elif kind == "denoise":
        s = State()
        s.cam, s.frames, s.poses = _sequence(case, seed, 1)
        p = config.make_params(s.cam.width, s.cam.height, s.cam.fx, s.cam.fy, s.cam.cx, s.cam.cy, voxel_size=0.008,
                               truncation=0.024, bayesian=True, bucket_count=1 << 14, value_capacity=1 << 12,
                               max_vertex_count=1 << 14, max_triangle_count=1 << 14)
        s.vol, s.iterations = Volume(p), case["iterations"]
    s.kind = kind
    return s


# ------------------------------------------------------------------ one pass

def run(s):
    if s.kind == "scan":
        s.vol.reset()
        for f, T in zip(s.frames, s.poses):
            s.vol.integrate_frame(f, T, on_device=not s.host, tv_iterations=s.tv, tv_lambda=TV_LAMBDA,
                                  outputs_on_device=not s.host, **s.images)
        st = s.vol.stats()
        return dict(s.images, blocks=st["blocks_allocated"], vertices=st["vertices_allocated"],
                    triangles=st["triangles_allocated"], error=st["error"])
    if s.kind == "batch":
        for v in s.batch.volumes:
            v.reset()
        for k in range(s.count):
            s.batch.step([f[k] for f in s.frames], [p[k] for p in s.poses], on_device=True, tv_iterations=s.tv,
                         tv_lambda=TV_LAMBDA, use_graph=True)
        return s.views
    if s.kind == "render":
        im = s.images
        s.vol.raycast(s.cTw, im["ray_depth"], im["ray_vertex"], im["ray_normal"])
        return im
    if s.kind == "gradient":
        s.vol.raycast(s.cTw, s.depth, None, s.normal)
        s.grad.zero_()
        xi = s.vol.raycast_backward(s.cTw, s.g_depth, s.g_normal, s.grad)
        # the pose gradient sums float32 terms of every pixel
        return dict(depth=s.depth, normal=s.normal, pose=xi.astype(np.float32), sdf=s.grad[s.rows])
    if s.kind == "track":
        T, cost, count = s.vol.refine_pose(s.start, iterations=s.iterations, obs_depth=s.obs, max_residual=0.05)
        return dict(pose=T, cost=np.float32(cost), count=count)   # the cost sums float32 residuals
    if s.kind == "smooth":
        s.vol.huber_tv_init()
        energy = s.vol.huber_tv_iterate(2.0, 8.0, 0.01, s.iterations)
        im = s.images
        s.vol.raycast(s.cTw, im["ray_depth"], im["ray_vertex"], im["ray_normal"])
        return dict(im, energy=energy.astype(np.float32))          # sums of float32 terms
    s.vol.set_frame(s.frames[0], s.poses[0], on_device=True)
    s.vol.denoise_tv(TV_LAMBDA, s.iterations)
    return s.vol.depth()


# ------------------------------------------------------------------ 64 bits
# Values in float64 along the decisions that single precision takes (which
# samples are valid, where the sign changes, which voxels surround a point):
# these are part of what the renderer computes.  Tensors divide tensors here:
# a scalar divisor would become a multiplication by its reciprocal.

class _Map:
    def __init__(self, vol, fields):
        pos, f = vol.dump_blocks(fields)
        order = np.lexsort(pos.T)
        self.pos = torch.from_numpy(pos[order].astype(np.int64)).cuda()
        self.f = {k: torch.from_numpy(f[k]).cuda()[torch.from_numpy(order).cuda()] for k in fields}
        self.vs = torch.tensor(vol.params.voxel_size, device="cuda")
        self.lo, self.hi = self.pos.amin(0) - 1, self.pos.amax(0) + 2
        n = (self.hi - self.lo).tolist()
        self.index = torch.full(n, -1, dtype=torch.int32, device="cuda")
        p = self.pos - self.lo
        self.index[p[:, 0], p[:, 1], p[:, 2]] = torch.arange(len(p), dtype=torch.int32, device="cuda")

    def block(self, b):
        ok = ((b >= self.lo) & (b < self.hi)).all(-1)
        c = torch.where(ok[..., None], b - self.lo, 0)
        return torch.where(ok, self.index[c[..., 0], c[..., 1], c[..., 2]].long(), -1)

    def corners(self, pos):
        """Per point: floor(pos / voxel), the flat index of its eight voxels, and whether all of them exist."""
        q = pos / self.vs
        fl = q.floor()
        fr = q - fl
        def nearest(w):
            w = w / self.vs
            return (w + torch.where(w < 0, -0.5, 0.5)).trunc()
        pc = pos - 0.5 * self.vs
        plain = (fr > 0.01) & (fr < 0.99)
        v0 = torch.where(plain, fl, nearest(pc)).long()
        v1 = torch.where(plain, fl + 1, nearest(pc + self.vs)).long()
        take = torch.tensor([[i >> 2 & 1, i >> 1 & 1, i & 1] for i in range(8)], device="cuda", dtype=torch.bool)
        v = torch.where(take, v1[:, None], v0[:, None])
        b = self.block(v >> 3)
        li = (v[..., 0] & 7) + 8 * (v[..., 1] & 7) + 64 * (v[..., 2] & 7)
        return fl, fr, b.clamp(min=0) * 512 + li, (b >= 0).all(-1)

    @staticmethod
    def blend(fr, v):
        w = torch.stack([1 - fr, fr], -1)
        acc = 0.0
        for i in range(8):
            acc = acc + w[:, 0, i >> 2 & 1] * w[:, 1, i >> 1 & 1] * w[:, 2, i & 1] * v[:, i]
        return acc

    def value32(self, pos):
        _, fr, at, ok = self.corners(pos)
        return self.blend(fr, self.f["sdf"].reshape(-1)[at]), ok

    def value64(self, pos32, pos64, sdf64):
        fl, _, at, ok = self.corners(pos32)
        fr = pos64 / self.vs.double() - fl.double()
        return self.blend(fr, sdf64.reshape(-1)[at]), ok


def _inverse32(m):
    """The 4x4 inverse by cofactors in float32, each product and sum rounded in the order the library states."""
    f, m = np.float32, np.asarray(m, np.float32).reshape(4, 4)
    inv = np.zeros((4, 4), np.float32)
    for r in range(4):
        for c in range(4):
            R, C = [i for i in range(4) if i != c], [j for j in range(4) if j != r]
            s = f(-1.0 if (r + c) & 1 else 1.0)
            e = lambda i, j: m[R[i], C[j]]  # noqa: E731
            t = [s * e(0, 0) * e(1, 1) * e(2, 2), -(s * e(0, 0) * e(1, 2) * e(2, 1)), -(s * e(1, 0) * e(0, 1) * e(2, 2)),
                 s * e(1, 0) * e(0, 2) * e(2, 1), s * e(2, 0) * e(0, 1) * e(1, 2), -(s * e(2, 0) * e(0, 2) * e(1, 1))]
            acc = t[0]
            for x in t[1:]:
                acc = f(acc + x)
            inv[r, c] = acc
    det = f(f(f(m[0, 0] * inv[0, 0] + m[0, 1] * inv[1, 0]) + m[0, 2] * inv[2, 0]) + m[0, 3] * inv[3, 0])
    return inv * f(f(1.0) / det)


def _unit(v):
    one = torch.ones((), dtype=v.dtype, device="cuda")
    return v * (one / (v[:, 0] * v[:, 0] + v[:, 1] * v[:, 1] + v[:, 2] * v[:, 2]).sqrt())[:, None]


def _rays(cam, cTw, dtype):
    wTc = torch.from_numpy(_inverse32(cTw)).cuda().to(dtype)
    n = lambda x: torch.tensor(x, dtype=torch.float32, device="cuda").to(dtype)  # noqa: E731
    u = (torch.arange(cam.width, device="cuda", dtype=dtype) - n(cam.cx)) / n(cam.fx)
    v = (torch.arange(cam.height, device="cuda", dtype=dtype) - n(cam.cy)) / n(cam.fy)
    r = torch.stack([u[None, :].expand(cam.height, -1), v[:, None].expand(-1, cam.width),
                     torch.ones(cam.height, cam.width, device="cuda", dtype=dtype)], -1).reshape(-1, 3)
    cd = _unit(r)
    wd = [wTc[i, 0] * cd[:, 0] + wTc[i, 1] * cd[:, 1] + wTc[i, 2] * cd[:, 2] for i in range(3)]
    return r, cd, wTc[:3, 3], _unit(torch.stack(wd, 1))


def _march(mp, vol, cam, cTw):
    """The rays that hit, and their decisions: the two samples around the zero, the side each secant step replaces."""
    p = vol.params
    _, cd, o, wd = _rays(cam, cTw, torch.float32)
    t, t_max = (torch.full_like(cd[:, 2], x) / cd[:, 2] for x in (p.min_raycast_depth, p.max_raycast_depth))
    ray = torch.arange(len(cd), device="cuda")
    ps, pt = torch.full_like(t, -1.0), torch.zeros_like(t)
    found = []
    while len(ray):
        s, ok = mp.value32(o + t[:, None] * wd[ray])
        at = (ok & (s < 0) & (ps > 0)).nonzero()[:, 0]
        if len(at):
            r, l, h, ls, hs = ray[at], pt[at], t[at], ps[at], s[at]
            good, sides = (ls - hs).abs().lt(p.sample_sdf_threshold) & hs.abs().lt(p.sdf_threshold), []
            for _ in range(3):
                m = l + (ls / (ls - hs)) * (h - l)
                ms, mok = mp.value32(o + m[:, None] * wd[r])
                left = ls * ms > 0
                l, ls = torch.where(left, m, l), torch.where(left, ms, ls)
                h, hs = torch.where(left, h, m), torch.where(left, hs, ms)
                good = good & mok
                sides.append(left)
            found.append([x[good] for x in (r, pt[at], t[at], m, *sides)])
            t[at[good]] = torch.inf
        ps, pt = torch.where(ok, s, ps), torch.where(ok, t, pt)
        t = t + p.raycast_step
        go = t < t_max
        ray, t, t_max, ps, pt = ray[go], t[go], t_max[go], ps[go], pt[go]
    return [torch.cat(x) for x in zip(*found)]


def _look(mp, vol, cam, cTw, sdf64, xi=None):
    """Depth, vertex and normal (float64) of the rays that hit, differentiable in sdf64 and a left pose increment."""
    ray, t0, t1, m32, *sides = _march(mp, vol, cam, cTw)
    _, cd32, o32, wd32 = _rays(cam, cTw, torch.float32)
    r, cd, o, wd = _rays(cam, cTw, torch.float64)
    r, cd, wd, wd32 = r[ray], cd[ray], wd[ray], wd32[ray]
    if xi is not None:
        o = o + torch.linalg.cross(xi[3:], o) + xi[:3]
        wd = wd + torch.linalg.cross(xi[3:].expand_as(wd), wd)
    value = lambda a, b: mp.value64(o32 + a[:, None] * wd32, o + b[:, None] * wd, sdf64)[0]  # noqa: E731
    l32, h32, l, h = t0, t1, t0.double(), t1.double()
    ls, hs = value(l32, l), value(h32, h)
    ls32, hs32 = (mp.value32(o32 + x[:, None] * wd32)[0] for x in (t0, t1))
    for left in sides:
        m32, m = l32 + (ls32 / (ls32 - hs32)) * (h32 - l32), l + ls / (ls - hs) * (h - l)
        ms32, ms = mp.value32(o32 + m32[:, None] * wd32)[0], value(m32, m)
        l32, ls32, h32, hs32 = (torch.where(left, a, b) for a, b in ((m32, l32), (ms32, ls32), (h32, m32), (hs32, ms32)))
        l, ls, h, hs = (torch.where(left, a, b) for a, b in ((m, l), (ms, ls), (h, m), (hs, ms)))
    p32, p = o32 + m32[:, None] * wd32, o + m[:, None] * wd
    g, ok = [], torch.ones(len(ray), dtype=torch.bool, device="cuda")
    for ax in range(3):
        e = torch.zeros(3, device="cuda")
        e[ax] = 0.5 * mp.vs
        (a, oka), (b, okb) = (mp.value64(p32 + k * e, p + k * e.double(), sdf64) for k in (1, -1))
        g.append((a - b) / mp.vs.double())
        ok &= oka & okb
    g = torch.stack(g, 1)
    ok &= (g.detach() != 0).any(1)
    n = torch.where(ok[:, None], -g / torch.where(ok, (g * g).sum(1), 1.0).sqrt()[:, None], 0.0)
    if xi is not None:
        n = n + torch.linalg.cross(n, xi[3:].expand_as(n))
    n = n @ torch.from_numpy(np.array(cTw[:3, :3], np.float64)).cuda().T
    z = m * cd[:, 2]
    return ray, z, r * z[:, None], n


def _picture(cam, ray, x, last=None):
    x = x if last is None else torch.cat([x, torch.full_like(x[:, :1], last)], 1)
    out = torch.full((cam.height * cam.width, *x.shape[1:]), -torch.inf, dtype=torch.float64, device="cuda")
    out[ray] = x
    return out.reshape(cam.height, cam.width, *x.shape[1:])


def exact(case, seed):
    """Scans and tracked poses have no such value: they follow from a long chain of single-precision decisions."""
    if case["kind"] in ("render", "gradient"):
        s = prepare(case, seed)
        mp = _Map(s.vol, ("sdf",))
        sdf = mp.f["sdf"].double()
        if case["kind"] == "render":
            ray, z, v, n = _look(mp, s.vol, s.cam, s.cTw, sdf)
            return dict(ray_depth=_picture(s.cam, ray, z), ray_vertex=_picture(s.cam, ray, v, 1.0),
                        ray_normal=_picture(s.cam, ray, n, 1.0))
        sdf.requires_grad_(True)
        xi = torch.zeros(6, dtype=torch.float64, device="cuda", requires_grad=True)
        ray, z, _, n = _look(mp, s.vol, s.cam, s.cTw, sdf, xi)
        loss = (s.g_depth.reshape(-1)[ray].double() * z).sum() + \
            (s.g_normal.reshape(-1, 4)[ray, :3].double() * n).sum()
        loss.backward()
        return dict(depth=_picture(s.cam, ray, z.detach()), normal=_picture(s.cam, ray, n.detach(), 1.0),
                    pose=xi.grad, sdf=torch.cat([sdf.grad, sdf.grad.new_zeros(len(s.rows) - len(sdf), 512)]))
    if case["kind"] == "smooth":
        return _smooth64(case, seed)
    if case["kind"] == "denoise":
        return _denoise64(case, seed)
    return None


def _smooth64(case, seed):
    """The energies of the last iteration; the images follow from decisions on the smoothed map."""
    s = prepare(case, seed)
    mp = _Map(s.vol, ("sdf", "w"))
    key = lambda p: (p[:, 0] << 42) + (p[:, 1] << 21) + p[:, 2]  # noqa: E731
    cand = torch.from_numpy(s.vol.candidates().astype(np.int64)).cuda()
    seen = torch.isin(key(mp.pos), key(cand))[:, None] & (mp.f["w"] >= 1e-6)      # masked voxels
    mine = torch.nonzero(seen.reshape(-1))[:, 0]
    li, blk = mine & 511, mine >> 9
    v = mp.pos[blk] * 8 + torch.stack([li & 7, li >> 3 & 7, li >> 6], 1)
    def beside(sign):
        out = []
        for ax in range(3):
            q = v.clone()
            q[:, ax] += sign
            b = mp.block(q >> 3)
            out.append(torch.where(b < 0, -1, b * 512 + (q[:, 0] & 7) + 8 * (q[:, 1] & 7) + 64 * (q[:, 2] & 7)))
        return torch.stack(out, 1)
    up, down = beside(1), beside(-1)
    obs, mask = (mp.f["w"] >= 1e-6).reshape(-1), seen.reshape(-1)
    has = lambda q, what: ((q >= 0) & what[q.clamp(min=0)]).all(1)  # noqa: E731
    ok_init, ok_up, ok_down = has(up, obs), has(up, mask), has(down, mask)
    up, down = up.clamp(min=0), down.clamp(min=0)
    sdf = mp.f["sdf"].double().reshape(-1)
    grad = lambda x, ok: torch.where(ok[:, None], x[up] - x[mine, None], 0.0)  # noqa: E731
    w = (grad(sdf, ok_init).square().sum(1).sqrt() / mp.vs.double()).exp()
    s0, bar, p = sdf[mine].clone(), torch.zeros_like(sdf), torch.zeros(3, len(sdf), dtype=torch.float64, device="cuda")
    lam, sigma, tau, alpha = 2.0, float(np.float32(8.0)), float(np.float32(0.01)), float(np.float32(0.02))
    for _ in range(case["iterations"]):
        x = grad(sdf, ok_up).square().sum(1).sqrt()
        data, tv = (sdf[mine] - s0).square().sum(), torch.where(x < alpha, 0.5 * x * x / alpha, x - 0.5 * alpha).sum()
        q = (p[:, mine] + sigma * grad(bar, ok_up).T) / (1 + sigma * alpha)
        p[:, mine] = q / q.square().sum(0).sqrt().clamp(min=1.0)
        div = torch.where(ok_down, sum(p[k][down[:, k]] - p[k][mine] for k in range(3)), 0.0)
        old = sdf[mine]
        new = (old - tau * div + lam * w * tau * s0) / (1 + lam * w * tau)
        new = torch.where(w > 2.0, s0, new)
        sdf[mine], bar[mine] = new, 2 * new - old
    return dict(energy=torch.stack([data * lam / 2 + tv, data, tv]), ray_depth=None, ray_vertex=None, ray_normal=None)


def _denoise64(case, seed):
    """Chambolle and Pock's first algorithm on the ROF model, in millimetres, holes kept."""
    _, frames, _ = _sequence(case, seed, 1)
    z = frames[0]
    ok = (z >= 0.5) & (z <= 4.0)
    f = torch.where(ok, z.double() * 1000.0, 0.0)
    right, below = torch.zeros_like(ok), torch.zeros_like(ok)
    right[:, :-1], below[:-1] = ok[:, :-1] & ok[:, 1:], ok[:-1] & ok[1:]
    u, bar, px, py = f.clone(), f.clone(), torch.zeros_like(f), torch.zeros_like(f)
    tau = 1.0 / math.sqrt(8.0)
    for _ in range(case["iterations"]):
        px = px + tau * torch.where(right, bar.roll(-1, 1) - bar, 0.0)
        py = py + tau * torch.where(below, bar.roll(-1, 0) - bar, 0.0)
        n = (px * px + py * py).sqrt().clamp(min=1.0)
        px, py = px / n, py / n
        left, above = px.roll(1, 1), py.roll(1, 0)
        left[:, 0], above[0] = 0.0, 0.0
        new = (u + tau * (px - left + py - above) + tau * TV_LAMBDA * f) / (1.0 + tau * TV_LAMBDA)
        u, bar = new, 2.0 * new - u
    return torch.where(ok, u * 0.001, -torch.inf)

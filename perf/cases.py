"""The work that programs give this renderer, as cases that can be timed.

A case is a dict of plain values; ``kind`` says which call it makes:

  pick      Renderer.trace_rays: ray queries from host arrays (picking, physics)
  query     Renderer.submit_batch with one query batch, rays and records on the device
  batch     Renderer.submit_batch with many uneven viewports and query batches
  frame     one frame of the context: camera, clipmap, encode_compute or the frame graph
  stream    a frame after a chunk-grid shift with the world kept on the device
  upload    a frame after chunk uploads from the host, its output read back to the host
  sessions  one frame of each of several client views, their images read back
  build     chunks built on the device from the seeded terrain

Worlds, camera heights, sizes and counts are those of vxe/scenes.py, bench.py
and the tests.  ``prepare`` makes a renderer with a resident world of its own
(terrain, poses and rays follow the seed), ``run`` makes one pass.
"""
from __future__ import annotations

import ctypes as C
import math
import sys
from pathlib import Path

import numpy as np
import torch

REPO = Path(__file__).resolve().parent.parent
PKG = REPO / "voxel-engine-v0_b200"
if str(PKG) not in sys.path:
    sys.path.insert(0, str(PKG))

from vxe import _abi as A  # noqa: E402
from vxe.renderer import Renderer  # noqa: E402
from vxe.serve import Session  # noqa: E402
from vxe.world import Clipmap, World, WorldSpec, build_camera, ground_height  # noqa: E402

CHUNK_M = 6.4          # metres of a 64-voxel chunk side
NODES_PER_COLUMN = 1 << 16  # arena nodes per chunk column of a world (all worlds here use less)
CYCLE = 16             # frames of a camera cycle (forth and back over a short path)
MISS = 255             # face of a ray without a hit


# -- the cases --------------------------------------------------------------------
def world_case(nx, ny, nz, caves=0.6, carve=0, features=0):
    """A grid of nx x ny x nz chunks; caves: 3D noise threshold (>= 1: none)."""
    return {"nx": nx, "ny": ny, "nz": nz, "caves": caves, "carve": carve, "features": features}


def listed():
    w2 = world_case(16, 4, 16)                       # the streamed world of the 1080p benchmark
    w5 = world_case(32, 8, 32, caves=0.5)            # the large world
    w1 = world_case(1, 1, 1, caves=2.0, carve=50)    # one carved chunk
    wf = world_case(3, 1, 3, caves=0.62, carve=50, features=3)  # trees and light voxels
    clip2 = {"levels": 5, "res": 256}
    return [
        # A click in an editor or a physics step: a handful of host rays, latency is all of it.
        dict(name="pick_64", kind="pick", rays=64, **w2),
        # One client's line-of-sight or physics query over the whole world.
        dict(name="query_100k", kind="query", rays=100_000, **w2),
        # The mixed launch of a server: 24 viewports and 40 incoherent query batches.
        dict(name="batch_64", kind="batch", viewports=24, queries=40, max_w=1920, max_h=1080, max_rays=1_000_000, **w2),
        # A thumbnail or preview: one chunk, no heightfield, every internal pixel presented.
        dict(name="frame_256x144", kind="frame", width=256, height=144, scale=1.0, mode="plain", levels=0, res=256, **w1),
        # A window of odd size over trees, leaves and local lights.
        dict(name="frame_lights_1001x601", kind="frame", width=1001, height=601, scale=1.0, mode="plain", levels=3,
             res=128, **wf),
        # The engine's default: 1080p presented, traced at half resolution.
        dict(name="frame_1080p", kind="frame", width=1920, height=1080, scale=0.5, mode="plain", **clip2, **w2),
        # High quality: traced at presented resolution, replayed as a graph.
        dict(name="frame_native_graph", kind="frame", width=1920, height=1080, scale=1.0, mode="graph", **clip2, **w2),
        # 4K over the large world with deep caves and a wide heightfield.
        dict(name="frame_4k", kind="frame", width=3840, height=2160, scale=0.5, mode="plain", levels=6, res=512, **w5),
        # A moving camera that crosses a chunk border: one layer of chunks leaves, one is built.
        dict(name="stream_720p", kind="stream", width=1280, height=720, scale=0.5, **clip2, **w2),
        # The same for a host that builds chunks itself and shows the frame elsewhere.
        dict(name="upload_1080p", kind="upload", width=1920, height=1080, scale=0.5, uploads=4, **clip2,
             **world_case(8, 4, 8)),
        # A server's clients: eight small views of different sizes in one launch.
        dict(name="sessions_8", kind="sessions", views=8, min_w=256, max_w=640, min_h=144, max_h=360, scale=1.0,
             **clip2, **w2),
        # A loader fills a region: the chunks of a 16 x 4 strip, four deep.
        dict(name="build_256", kind="build", chunks=256, caves=0.6, carve=0, features=0),
    ]


def log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    world = rng.choice([world_case(16, 4, 16), world_case(16, 4, 16), world_case(8, 4, 8, caves=0.5),
                        world_case(12, 2, 9, caves=2.0, carve=50), world_case(3, 1, 3, caves=0.62, carve=50, features=3)])
    clip = rng.choice([{"levels": 5, "res": 256}, {"levels": 6, "res": 512}, {"levels": 3, "res": 128}])
    kind = rng.choice(["pick", "query", "batch", "frame", "frame", "frame", "stream", "upload", "sessions", "build"])
    if kind == "pick":
        return dict(kind=kind, rays=log_int(rng, 1, 4096), **world)
    if kind == "query":
        return dict(kind=kind, rays=log_int(rng, 1_000, 1_000_000), **world)
    if kind == "batch":
        return dict(kind=kind, viewports=rng.randint(1, 20), queries=rng.randint(1, 36), max_w=rng.randint(200, 1920),
                    max_h=rng.randint(150, 1080), max_rays=log_int(rng, 2_000, 1_000_000), **world)
    if kind == "build":
        return dict(kind=kind, chunks=log_int(rng, 1, 256), caves=rng.choice([0.5, 0.6, 2.0]),
                    carve=rng.choice([0, 50]), features=rng.choice([0, 3]))
    if kind == "sessions":
        return dict(kind=kind, views=rng.randint(1, 8), min_w=256, max_w=rng.randint(300, 640), min_h=144,
                    max_h=rng.randint(160, 360), scale=rng.choice([0.5, 0.75, 1.0]), **clip, **world)
    w = log_int(rng, 160, 2560)
    h = max(90, min(1440, int(w * rng.uniform(0.45, 0.8))))
    size = dict(width=w, height=h, scale=rng.choice([0.5, 0.5, 0.67, 1.0]) if w * h <= 1920 * 1080 else 0.5)
    if kind == "frame":
        return dict(kind=kind, mode=rng.choice(["plain", "plain", "graph"]), **size, **clip, **world)
    if kind == "stream":
        return dict(kind=kind, **size, **clip, **world_case(rng.choice([8, 12, 16]), 4, rng.choice([9, 16])))
    return dict(kind=kind, uploads=rng.randint(1, 10), **size, **clip, **world_case(8, rng.choice([2, 4]), 8))


# -- what a program has in hand -----------------------------------------------------
class State:
    """A renderer, its world and the inputs of a case; views go before the renderer."""

    def __init__(self, case, seed):
        self.case = case
        self.rng = np.random.default_rng(seed)
        f = case.get("features", 0)
        self.spec = WorldSpec(seed=int(seed) & 0x3FFFFFFF, height_min=10 if f else 8, height_max=30 if f else 48,
                              dirt_depth=3, carve_mod=case["carve"], cave_threshold=case["caves"],
                              height_scale_vox=48.0 if f else 64.0, features=f)
        self.r = None
        self.clip = None
        self.views = []
        self.n = 0

    def renderer(self, width, height, scale):
        c = self.case
        chunks = c["nx"] * c["ny"] * c["nz"]
        self.world = World(self.spec, (0, 0, 0), (c["nx"], c["ny"], c["nz"]), c["nx"] * c["nz"] * NODES_PER_COLUMN,
                           chunk_capacity=chunks, mirror=False)
        self.r = Renderer(width, height, scale, node_capacity=self.world.node_capacity, chunk_capacity=chunks,
                          grid_capacity=chunks, clip_levels=max(1, c.get("levels", 0)), clip_res=c.get("res", 256))
        return self.r

    def heights(self):
        """The clipmap state, or the empty uniform of a world without one."""
        c = self.case
        if c.get("levels", 0):
            self.clip = Clipmap(self.spec, c["levels"], c["res"], 1.0)
        else:
            p = A.ClipmapGpu()
            p.res = c.get("res", 256)
            self.r.write_clipmap_updates(p, [])

    def pose(self):
        """A place a few metres over the ground near the middle of the world, and a heading."""
        c = self.case
        u = self.rng.uniform(0.35, 0.65, 2)
        x, z = u[0] * c["nx"] * CHUNK_M, u[1] * c["nz"] * CHUNK_M
        y = 0.1 * ground_height(self.spec, int(x * 10), int(z * 10)) + self.rng.uniform(2.0, 4.5)
        return np.array([x, y, z]), self.rng.uniform(0, 2 * math.pi), self.rng.uniform(-0.3, -0.05)

    def cameras(self, width, height, internal):
        """A cycle of CYCLE frames forth and back along the heading, 0.15 m a frame."""
        pos, yaw, pitch = self.pose()
        if self.case["nx"] == 1:  # a single chunk is looked at from outside
            ang, elev = self.rng.uniform(0, 2 * math.pi), self.rng.uniform(0.35, 0.7)
            to = -np.array([math.cos(elev) * math.sin(ang), math.sin(elev), math.cos(elev) * math.cos(ang)])
            pos, yaw, pitch = CHUNK_M / 2 - 6.7 * to, math.atan2(to[0], to[2]), math.asin(to[1])
        fwd = np.array([math.sin(yaw), 0.0, math.cos(yaw)])
        self.places = [pos + fwd * 0.15 * min(f, CYCLE - f) for f in range(CYCLE)]
        self.look = (yaw, pitch)
        cams, prev = [], None
        for lap in range(2):  # the second lap's first frame follows the first lap's last
            for f in range(CYCLE):
                cam = build_camera(self.places[f], yaw, pitch, (width, height), internal, frame_index=f + 1,
                                   time_s=f / 60.0, world=self.world, prev_view_proj=prev)
                prev = cam.view_proj
                if lap:
                    cams.append(cam)
        return cams

    def rays(self, n):
        """Origins uniform in the world, directions uniform on the sphere."""
        lo, hi = self.world.world_aabb_m()
        d = self.rng.normal(size=(n, 3))
        d /= np.linalg.norm(d, axis=1, keepdims=True)
        return self.rng.uniform(lo, hi, size=(n, 3)).astype(np.float32), d.astype(np.float32)

    def close(self):
        for v in self.views:
            v.close()
        self.views = []
        if self.r is not None:
            self.r.close()
            self.r = None

    def __del__(self):
        try:
            self.close()
        except Exception:
            pass


class _Device:
    """Renderer-owned device memory in the form torch.as_tensor takes; a tensor
    over it keeps `owner` (and so the memory) alive."""

    def __init__(self, owner, ptr, shape):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": "<f4", "version": 2}


def frame_tensors(s, out):
    """The images of a frame as tensors over the renderer's own memory."""
    ih, iw, ph, pw = out.internal_h, out.internal_w, out.present_h, out.present_w
    t = lambda ptr, *shape: torch.as_tensor(_Device(s, ptr, shape), device="cuda")  # noqa: E731
    return {"color": t(out.color, ih, iw, 4), "depth": t(out.depth, ih, iw), "godray": t(out.godray, ih, iw, 4),
            "output": t(out.output, ph, pw, 4)}


def world_camera(s):
    """The context's camera of a program that only traces rays (chunk count, grid)."""
    pos, yaw, pitch = s.pose()
    s.r.write_camera(build_camera(pos, yaw, pitch, (64, 36), (64, 36), 1, 0.0, world=s.world, jitter=False))


def prepare(case, seed):
    s = State(case, seed)
    kind = case["kind"]
    if kind == "build":
        s.r = Renderer(64, 36, 1.0, node_capacity=1 << 12, chunk_capacity=4, grid_capacity=4, clip_levels=1, clip_res=16)
        n = case["chunks"]
        origin = s.rng.integers(-40, 40, 2)
        keys = [(int(origin[0]) + i % 16, (i // 16) % 4, int(origin[1]) + i // 64) for i in range(n)]
        s.coords = torch.tensor(keys, dtype=torch.int32, device="cuda")
        s.params = s.spec.params()
        counts = s.r.build_chunks(s.params, s.coords, node_cap=0)["counts"]
        s.cap = int(counts[:, 0].max())
        # the program's own arena, filled from the front
        rows = min(n, 16 * -(-n // 64)) * NODES_PER_COLUMN
        s.nodes = torch.zeros((rows, 4), dtype=torch.int32, device="cuda")
        s.ropes = torch.zeros((rows, 6), dtype=torch.int32, device="cuda")
        return s
    if kind in ("pick", "query", "batch"):
        s.renderer(64, 36, 1.0)
    else:
        s.renderer(case.get("width", 64), case.get("height", 36), case["scale"])
    if kind == "upload":
        ups = s.world.populate()
        s.r.upload_world(s.world, ups)
        s.uploads = ups
    else:
        s.world.populate_device(s.r)
    if kind in ("pick", "query", "batch"):
        world_camera(s)
        if kind == "pick":
            s.o, s.d = s.rays(case["rays"])
        elif kind == "query":
            prepare_query(s)
        else:
            prepare_batch(s)
        return s
    s.heights()
    if kind == "sessions":
        world_camera(s)
        if s.clip is not None:
            s.clip.update_device(s.r, *s.world.world_aabb_m()[1][[0, 2]] * 0.5)
        s.sessions = []
        mix = np.random.default_rng(case["max_w"])  # the clients' sizes go with the case, their places with the seed
        for i in range(case["views"]):
            w = int(mix.integers(case["min_w"], case["max_w"] + 1))
            h = int(mix.integers(case["min_h"], case["max_h"] + 1))
            pos, yaw, pitch = s.pose()
            s.sessions.append(Session(i, w, h, pos, yaw, pitch, render_scale=case["scale"]))
            s.views.append(s.r.view(w, h, case["scale"]))
    else:
        s.cams = s.cameras(case["width"], case["height"], s.r.internal)
        if kind == "upload":
            s.image = torch.empty((case["height"], case["width"], 4), pin_memory=True).numpy()
    s.r.synchronize()
    return s


def query_request(rays, origins, dirs, out):
    q = A.Request()
    q.kind, q.ray_count, q.tmax = A.REQ_QUERY, rays, 120.0
    q.d_origins, q.d_dirs, q.d_out = origins.data_ptr(), dirs.data_ptr(), out.data_ptr()
    return q


def prepare_query(s):
    o, d = s.rays(s.case["rays"])
    s.o, s.d = torch.from_numpy(o).cuda(), torch.from_numpy(d).cuda()
    s.out = torch.zeros((len(o), 8), dtype=torch.int32, device="cuda")
    s.requests = [query_request(len(o), s.o, s.d, s.out)]
    torch.cuda.synchronize()


def prepare_batch(s):
    c, rng = s.case, s.rng
    sizes = []
    mix = np.random.default_rng(c["max_w"])
    for _ in range(c["viewports"]):
        sizes.append((int(mix.integers(128, c["max_w"] + 1)), int(mix.integers(128, c["max_h"] + 1))))
    for _ in range(c["queries"]):
        sizes.append(int(round(math.exp(mix.uniform(math.log(1e3), math.log(c["max_rays"]))))))
    order = mix.permutation(len(sizes))
    total = sum(v[0] * v[1] if isinstance(v, tuple) else v for v in sizes)
    rays = sum(v for v in sizes if not isinstance(v, tuple))
    s.out = torch.zeros((total, 8), dtype=torch.int32, device="cuda")
    lo, hi = (torch.tensor(v, dtype=torch.float32, device="cuda") for v in s.world.world_aabb_m())
    g = torch.Generator(device="cuda").manual_seed(int(rng.integers(1 << 40)))
    s.o = lo + (hi - lo) * torch.rand((rays, 3), generator=g, device="cuda")
    d = torch.randn((rays, 3), generator=g, device="cuda")
    s.d = d / d.norm(dim=1, keepdim=True)
    s.requests, at, ray = [], 0, 0
    for k in order:
        v = sizes[k]
        if isinstance(v, tuple):
            n = v[0] * v[1]
            pos, yaw, _ = s.pose()
            q = A.Request()
            q.kind, q.width, q.height = A.REQ_VIEWPORT, v[0], v[1]
            q.camera = build_camera(pos, yaw, rng.uniform(-0.45, 0.05), v, v, 1, 0.0, world=s.world, jitter=False)
            q.d_out = s.out[at:].data_ptr()
        else:
            n = v
            q = query_request(n, s.o[ray:], s.d[ray:], s.out[at:])
            ray += n
        s.requests.append(q)
        at += n
    torch.cuda.synchronize()


# -- one pass -------------------------------------------------------------------------
def hit_outputs(records, face, t):
    """Hit records (whole words) and the distances of the rays that hit (0: none)."""
    where = torch.where if isinstance(t, torch.Tensor) else np.where
    return {"records": records, "t": where(face == MISS, t * 0, t)}


def run(s):
    kind, r = s.case["kind"], s.r
    if kind == "pick":
        h = r.trace_rays(s.o, s.d, 120.0)
        return hit_outputs(h.view(np.int32).reshape(-1, 8), h["face"], h["t"])
    if kind in ("query", "batch"):
        r.submit_batch(s.requests, tile=(8, 4), rays_per_thread=1)
        if kind == "batch":
            return s.out
        return hit_outputs(s.out, s.out[:, 5], s.out.view(torch.float32)[:, 0])
    if kind == "build":
        out = r.build_chunks(s.params, s.coords, node_cap=s.cap)
        # the records of each chunk go into the program's arena, packed
        keep = torch.arange(s.cap, device="cuda")[None, :] < out["counts"][:, :1]
        nodes, ropes = out["nodes"][keep], out["ropes"][keep]
        s.nodes[:len(nodes)] = nodes
        s.ropes[:len(nodes)] = ropes[:, :6]
        return {"counts": out["counts"], "macro": out["macro"], "colinfo": out["colinfo"], "nodes": s.nodes,
                "ropes": s.ropes}
    s.n += 1
    if kind == "sessions":
        pairs = []
        for view, client in zip(s.views, s.sessions):
            cam = client.camera(s.world, client.frame, client.prev_vp)
            client.prev_vp = cam.view_proj
            client.frame = (client.frame + 1) % CYCLE
            pairs.append((view, cam))
        r.render_views_async(0, pairs)
        r.batch_wait(0)
        return [view.read_image(A.IMG_OUTPUT) for view in s.views]
    f = (s.n - 1) % CYCLE
    cam = s.cams[f]
    x, z = float(s.places[f][0]), float(s.places[f][2])
    if kind == "stream":
        s.world.shift_device(r, 1 if s.n % 2 else -1, 0, 0)
        cam = build_camera(s.places[f], *s.look, r.present, r.internal, f + 1, f / 60.0, world=s.world,
                           prev_view_proj=s.cams[f - 1].view_proj)
    if kind == "upload":
        n = s.case["uploads"]
        r.apply_chunk_uploads([s.uploads[(s.n * n + i) % len(s.uploads)] for i in range(n)])
        r.write_clipmap_updates(*s.clip.update(x, z))
        r.write_camera(cam)
        r.encode_compute(sync=False)
        r.read_image_wait(r.read_image_async(A.IMG_OUTPUT, s.image))
        return s.image
    if s.clip is not None:
        s.clip.update_device(r, x, z)
    r.write_camera(cam)
    return frame_tensors(s, r.render_frame_graph() if s.case.get("mode") == "graph" else r.encode_compute())


# -- what a pass cannot do without ----------------------------------------------------
def work(case):
    """Bytes of the pass's inputs and outputs, each once.  The world's records
    that the rays meet depend on the view and are left out, and so is the
    traversal's arithmetic, which is scalar and follows the data: no flops."""
    kind = case["kind"]
    column = 22_000 * 48 + 2048 * 4 + 16 * 4  # nodes and ropes of a surface chunk, its column and macro words
    frame = 0
    if kind in ("frame", "stream", "upload"):
        present = case["width"] * case["height"]
        internal = present * case["scale"] ** 2
        # color, depth; primary-hit, shadow, local-light and godray histories in and out; output, its history
        frame = internal * (16 + 4 + 2 * (16 + 4 + 16 + 16)) + present * (16 + 2 * 16)
    if kind in ("pick", "query"):
        n = case["rays"] * (24 + 32)
    elif kind == "batch":
        mean = (case["max_rays"] - 1e3) / math.log(case["max_rays"] / 1e3) if case["max_rays"] > 1e3 else 1e3
        pixels = (128 + case["max_w"]) / 2 * (128 + case["max_h"]) / 2
        n = case["viewports"] * pixels * 32 + case["queries"] * mean * (24 + 32)
    elif kind == "build":
        n = case["chunks"] * (column / 4 + 8 + 12)  # one chunk in four of the strip holds the surface
    elif kind == "sessions":
        pixels = (case["min_w"] + case["max_w"]) / 2 * (case["min_h"] + case["max_h"]) / 2
        n = case["views"] * pixels * (case["scale"] ** 2 * 124 + 48 + 16)
    elif kind == "stream":
        n = frame + case["ny"] * case["nz"] * column / case["ny"]
    elif kind == "upload":
        n = frame + case["uploads"] * column / case["ny"] + case["width"] * case["height"] * 16
    else:
        n = frame
    return {"bytes": float(n), "flops": 0.0}


# -- ray distances in 64 bits ----------------------------------------------------------
def _mix32(v):
    v = v & 0xFFFFFFFF
    v = ((v ^ (v >> 16)) * 0x7FEB352D) & 0xFFFFFFFF
    v = ((v ^ (v >> 15)) * 0x846CA68B) & 0xFFFFFFFF
    return v ^ (v >> 16)


def _lattice(seed, *ixyz):
    """Uniform numbers in [0, 1) at integer lattice points (int64 tensors, 32-bit wrap)."""
    mul = (0x9E3779B1, 0x85EBCA6B) if len(ixyz) == 2 else (0x9E3779B1, 0x85EBCA6B, 0xC2B2AE35)
    v = torch.full_like(ixyz[0], seed & 0xFFFFFFFF)
    for i, m in zip(ixyz, mul):
        v = v ^ (((i & 0xFFFFFFFF) * m) & 0xFFFFFFFF)
    return _mix32(v).double() / 4294967296.0


def _noise(seed, *xyz):
    """Value noise with smoothstep interpolation, x innermost."""
    base = [torch.floor(v) for v in xyz]
    fade = [(v - b) * (v - b) * (3.0 - 2.0 * (v - b)) for v, b in zip(xyz, base)]
    at = [b.long() for b in base]

    def corner(axis, shift):
        if axis < 0:
            return _lattice(seed, *[a + k for a, k in zip(at, shift)])
        lo, hi = (corner(axis - 1, (k,) + shift) for k in (0, 1))
        return lo + (hi - lo) * fade[axis]

    return corner(len(xyz) - 1, ())


def _solid(s):
    """The dense solid grid [x, y, z] of the world (voxels), in 64-bit arithmetic."""
    c, p = s.case, s.spec
    nx, ny, nz = c["nx"] * 64, c["ny"] * 64, c["nz"] * 64
    x = torch.arange(nx, device="cuda").double()[:, None].expand(nx, nz)
    z = torch.arange(nz, device="cuda").double()[None, :].expand(nx, nz)
    total, norm, amp, spacing = torch.zeros((nx, nz), dtype=torch.float64, device="cuda"), 0.0, 1.0, p.height_scale_vox
    for o in range(4):
        total += amp * _noise(p.seed + 0x9E37 * (o + 1), x / spacing, z / spacing)
        norm, amp, spacing = norm + amp, amp * 0.5, spacing * 0.5
    ground = (p.height_min + torch.floor(total / norm * (p.height_max - p.height_min + 1))).clamp(p.height_min, p.height_max)
    solid = torch.zeros((nx, ny, nz), dtype=torch.bool, device="cuda")
    for y in range(min(ny, p.height_max + 1)):
        layer = y <= ground
        yy = torch.full_like(x, float(y))
        if p.cave_threshold < 1.0:
            k = p.seed ^ 0xCA7E5EED
            v = (_noise(k, x / 16, yy / 16, z / 16) + 0.5 * _noise(k + 7, x / 8, yy / 8, z / 8)) / 1.5
            layer = layer & ~(v > float(np.float32(p.cave_threshold)))
        if p.carve_mod:
            h = _mix32(torch.full_like(x, 0).long() ^ (p.seed ^ 0x5EED) ^ ((x.long() * 0x9E3779B1) & 0xFFFFFFFF)
                       ^ ((y * 0x85EBCA6B) & 0xFFFFFFFF) ^ ((z.long() * 0xC2B2AE35) & 0xFFFFFFFF))
            layer = layer & ~(h % p.carve_mod == 0)
        solid[:, y] = layer
    return solid


def exact(case, seed):
    """Distances of ray queries: a 64-bit cell walk (Amanatides-Woo) over the
    dense voxels.  Frames, hit records of marched grass and built chunks have
    no value of that kind; nor has a world with trees here."""
    if case["kind"] not in ("pick", "query") or case["features"]:
        return None
    s = State(case, seed)
    s.world = World(s.spec, (0, 0, 0), (case["nx"], case["ny"], case["nz"]), 1, chunk_capacity=1, mirror=False)
    s.pose()  # as prepare(): the rays follow the pose
    o, d = (torch.from_numpy(v).cuda().double() for v in s.rays(case["rays"]))
    solid = _solid(s)
    size = torch.tensor(solid.shape, device="cuda").double()
    vs = 0.1
    o, step = o / vs, torch.where(d > 0, 1, -1)
    cell = torch.minimum(torch.floor(o), size - 1).clamp(min=0).long()
    nxt = torch.where(d != 0, (cell + (d > 0) - o) / d, torch.inf)
    delta = torch.where(d != 0, (1.0 / d).abs(), torch.inf)
    t = torch.zeros(len(o), dtype=torch.float64, device="cuda")
    found = torch.zeros(len(o), dtype=torch.float64, device="cuda")
    live = torch.arange(len(o), device="cuda")
    for _ in range(int(size.sum()) + 3):
        hit = solid[cell[:, 0], cell[:, 1], cell[:, 2]]
        found[live[hit]] = t[hit] * vs
        axis = nxt.argmin(dim=1, keepdim=True)
        t = nxt.gather(1, axis)[:, 0]
        cell = cell.scatter_add(1, axis, step.gather(1, axis))
        nxt = nxt.scatter_add(1, axis, delta.gather(1, axis))
        on = ~hit & (t * vs <= 120.0) & ((cell >= 0) & (cell < size)).all(dim=1)
        t, cell, nxt, delta, step, live = (v[on] for v in (t, cell, nxt, delta, step, live))
        if not len(live):
            break
    if case["kind"] == "pick":
        found = found.cpu().numpy()
    return {"records": None, "t": found}

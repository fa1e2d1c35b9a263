"""The calls that the engine's speed is measured on: every traversal kernel through the entry
points that a renderer calls, the scene updates that it makes each frame, and the BVH build.

A case is a dict of plain values. ``listed()`` names the ones that stand for a use each, ``draw``
makes more of the same ranges, ``prepare`` makes what a program holds before the call (scene,
rays, plan), ``run`` makes one call, ``work`` says what the call cannot do without, and ``exact``
gives the hits in 64-bit arithmetic by testing every triangle, where that is short enough.

Scenes are those of ``renderlab_b200.scenes`` (cluster soup, jittered cubes, many instanced
meshes), generated here on the GPU from the case's seed.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from renderlab_b200 import api as A

DEV = "cuda"
FAR = 1.0e3          # closest-hit and any-hit tmax where the caller sets one: past every scene here
EXACT_PAIRS = 1.5e11  # ray-triangle pairs that exact() tests at most


# ---------------------------------------------------------------- the cases

def listed() -> list:
    return [
        # A light or probe query between passes: one small batch of visibility rays through the
        # seam's own function and its default kernel, over some 900 boxes under a top level.
        # Latency and launches count.
        dict(name="visible_small", kind="seam", fn="visible", side=30, rays=4096),
        # The plain method's own workload: 10,000 jittered cubes merged into one mesh, 1024 x 1024
        # primary rays, closest hit, default kernel.
        dict(name="primary_cubes", kind="seam", fn="closest", side=100, rays=1 << 20),
        # Coherent camera rays at the size of the plain-kernel-at-scale workload: 1M triangles,
        # 2048 x 2048 pixels in 8 x 4 tiles, the packet walk.
        dict(name="primary_packet", kind="trace", layout=1, tris=1_000_000, rays=1 << 22, source="primary",
             mode=0, kernel="wide8p"),
        # Diffuse GI rays of the same workload: one cosine-hemisphere ray from each camera hit.
        dict(name="gi_hemisphere", kind="trace", layout=1, tris=1_000_000, rays=1 << 22, source="gi", mode=0,
             kernel="wide8"),
        # Shadow rays toward 16 point lights, any hit, an odd count (a screen with sky in it).
        dict(name="shadow_rays", kind="trace", layout=1, tris=250_000, rays=838_861, source="shadow", mode=2,
             kernel="wide8"),
        # The GI cache's gather: 16,384 cells of 64 directions (the 1.05M rays of the reference's
        # 1080p gather), closest hit, over a world of instanced meshes.
        dict(name="gi_gather", kind="cells", meshes=8, instances=400, tri_lo=200, tri_hi=5000, cells=16_384, mode=0,
             rotate=True),
        # The GI cache's light visibility: every cell against 40 lights, packed into words.
        dict(name="gi_lights", kind="lights", tris=250_000, cells=16_384, lights=40, kernel="fast"),
        # A frame's uneven batches of mixed modes over many overlapping instances, replayed as one
        # captured plan (the batching workload at a tenth of its instances and batches' sum).
        dict(name="batches_instanced", kind="batches", meshes=16, instances=1000, tri_lo=2000, tri_hi=20_000, batches=32,
             n_lo=1000, n_hi=200_000, kernel="wide8", order="none", plan=True),
        # A caller whose rays and hits live in host memory: camera, GI and shadow batches of one
        # step through the host pipeline, copies included.
        dict(name="host_step", kind="host", tris=250_000, rays=2_000_000),
        # A deforming mesh: refit its boxes for this frame's vertices, then trace a quarter-size frame.
        dict(name="deforming_mesh", kind="refit", layout=1, tris=250_000, rays=65_536),
        # Rigid motion: 2,500 instances get new placements, then a small frame is traced.
        dict(name="moving_instances", kind="move", layout=0, side=50, rays=65_536),
        # A runtime mesh's BVH from its triangles (host arrays in, host records out).
        dict(name="blas_build", kind="build", tris=250_000, median=False),
    ]


def _log(rng, lo, hi) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(("seam", "trace", "trace", "trace", "cells", "lights", "batches", "host", "refit", "move", "build"))
    if kind == "seam":
        return dict(kind=kind, fn=rng.choice(("visible", "closest")), side=rng.randint(4, 100), rays=_log(rng, 200, 1 << 20))
    if kind == "trace":
        source = rng.choice(("primary", "gi", "shadow"))
        kernels = ("plain", "fast", "wide8", "wide8p") if source == "primary" else ("plain", "fast", "wide8")
        return dict(kind=kind, layout=rng.choice((0, 1)), tris=_log(rng, 2000, 400_000), rays=_log(rng, 1000, 2_000_000),
                    source=source, mode=2 if source == "shadow" else rng.choice((0, 0, 1)), kernel=rng.choice(kernels))
    if kind == "cells":
        return dict(kind=kind, meshes=rng.randint(1, 12), instances=rng.randint(1, 500), tri_lo=100,
                    tri_hi=_log(rng, 200, 10_000), cells=_log(rng, 50, 16_384), mode=rng.choice((0, 0, 1)),
                    rotate=rng.random() < 0.5)
    if kind == "lights":
        return dict(kind=kind, tris=_log(rng, 5000, 300_000), cells=_log(rng, 50, 16_384), lights=rng.randint(1, 64),
                    kernel=rng.choice(("fast", "fast", "wide8")))
    if kind == "batches":
        return dict(kind=kind, meshes=rng.randint(1, 16), instances=rng.randint(2, 600), tri_lo=500,
                    tri_hi=_log(rng, 1000, 20_000), batches=rng.randint(1, 48), n_lo=100, n_hi=_log(rng, 500, 100_000),
                    kernel=rng.choice(("fast", "wide8", "wide8")), order=rng.choice(("none", "none", "origin", "octant")),
                    plan=rng.random() < 0.5)
    if kind == "host":
        return dict(kind=kind, tris=_log(rng, 5000, 300_000), rays=_log(rng, 5000, 2_000_000))
    if kind == "refit":
        return dict(kind=kind, layout=rng.choice((0, 1)), tris=_log(rng, 500, 300_000), rays=_log(rng, 1000, 200_000))
    if kind == "move":
        return dict(kind=kind, layout=rng.choice((0, 1)), side=rng.randint(3, 50), rays=_log(rng, 1000, 200_000))
    return dict(kind=kind, tris=_log(rng, 100, 300_000), median=rng.random() < 0.25)


# ---------------------------------------------------------------- scenes and rays, on the GPU

def _gen(seed: int, salt: int) -> torch.Generator:
    g = torch.Generator(device=DEV)
    g.manual_seed((seed * 1_000_003 + salt) & 0x7FFFFFFF)
    return g


def _uniform(g, *shape):
    return torch.rand(*shape, generator=g, device=DEV, dtype=torch.float64)


def _unit(g, n):
    u = _uniform(g, n, 2)
    z, phi = 2.0 * u[:, 0] - 1.0, 2.0 * math.pi * u[:, 1]
    r = torch.sqrt((1.0 - z * z).clamp_min(0.0))
    return torch.stack([r * torch.cos(phi), r * torch.sin(phi), z], dim=1)


def _clusters(g, n, per_cluster=500, half=100.0, radius=5.0):
    """The cluster soup: (n, 3, 3) float32 vertices, unshared."""
    k = (n + per_cluster - 1) // per_cluster
    centres = (2.0 * _uniform(g, k, 3) - 1.0) * half
    a = centres[torch.arange(n, device=DEV) // per_cluster] + _unit(g, n) * (radius * _uniform(g, n, 1) ** (1.0 / 3.0))
    normal = torch.randn(n, 2, generator=g, device=DEV, dtype=torch.float64)
    length = torch.exp(math.log(0.5) + 0.8 * normal)
    b, c = a + _unit(g, n) * length[:, 0:1], a + _unit(g, n) * length[:, 1:2]
    return torch.stack([a, b, c], dim=1).float()


_CORNERS = [[x, y, z] for z in (-0.5, 0.5) for y in (-0.5, 0.5) for x in (-0.5, 0.5)]
_FACES = [0, 2, 1, 1, 2, 3, 4, 5, 6, 5, 7, 6, 0, 1, 4, 1, 5, 4, 2, 6, 3, 3, 6, 7, 0, 4, 2, 2, 4, 6, 1, 3, 5, 3, 7, 5]


def _cube_models(g, side):
    """side x side cubes on a grid of spacing 2: jitter, scale and yaw; (n, 3, 4) float64."""
    n = side * side
    u = _uniform(g, n, 4)
    at = torch.arange(n, device=DEV)
    cx = ((at % side).double() - (side - 1) / 2.0) * 2.0 + (u[:, 0] * 0.6 - 0.3)
    cz = ((at // side).double() - (side - 1) / 2.0) * 2.0 + (u[:, 1] * 0.6 - 0.3)
    scale, yaw = 0.5 + u[:, 2], u[:, 3] * 2.0 * math.pi
    m = torch.zeros(n, 3, 4, device=DEV, dtype=torch.float64)
    m[:, 0, 0], m[:, 0, 2] = torch.cos(yaw) * scale, torch.sin(yaw) * scale
    m[:, 1, 1] = scale
    m[:, 2, 0], m[:, 2, 2] = -torch.sin(yaw) * scale, torch.cos(yaw) * scale
    m[:, 0, 3], m[:, 1, 3], m[:, 2, 3] = cx, 0.5 * scale, cz
    return m


class _Instances:
    """What pack_scene takes: models, world-to-object rows, mesh ids (host float32 / uint32)."""

    def __init__(self, model, mesh):
        a, t = model[:, :, :3], model[:, :, 3]
        ai = torch.linalg.inv(a)
        rows = torch.cat([ai, -torch.einsum("nij,nj->ni", ai, t)[:, :, None]], dim=2)
        self.model, self.rows = model.float().cpu().numpy(), rows.float().cpu().numpy()
        self.mesh = np.asarray(mesh, np.uint32)

    def __len__(self):
        return len(self.mesh)


def _identity():
    m = torch.zeros(1, 3, 4, device=DEV, dtype=torch.float64)
    m[0, 0, 0] = m[0, 1, 1] = m[0, 2, 2] = 1.0
    return _Instances(m, [0])


def _placed(g, n, n_meshes, half):
    """n instances of n_meshes meshes: random rotations, scales 0.5 to 4, anywhere in the box."""
    q = torch.randn(n, 4, generator=g, device=DEV, dtype=torch.float64)
    q = q / q.norm(dim=1, keepdim=True)
    w, x, y, z = q.unbind(1)
    rot = torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w),
                       2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w),
                       2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)], dim=1).reshape(n, 3, 3)
    scale = 0.5 + 3.5 * _uniform(g, n)
    at = (2.0 * _uniform(g, n, 3) - 1.0) * half
    mesh = torch.randint(0, n_meshes, (n,), generator=g, device=DEV).cpu().numpy()
    return _Instances(torch.cat([rot * scale[:, None, None], at[:, :, None]], dim=2), mesh)


def _pinhole(n, eye, forward, fov_deg=60.0):
    """n unit directions through the pixel centres of a square image, in 8 x 4 tiles."""
    side = max(8, 8 * math.ceil(math.sqrt(n) / 8))
    f = torch.tensor(forward, device=DEV, dtype=torch.float64)
    f = f / f.norm()
    up0 = torch.tensor([0.0, 1.0, 0.0], device=DEV, dtype=torch.float64)
    right = torch.linalg.cross(up0, f)
    right = right / right.norm()
    up = torch.linalg.cross(f, right)
    i = torch.arange(n, device=DEV)
    tile, pix = i // 32, i % 32
    x = (tile % (side // 8)) * 8 + pix % 8
    y = (tile // (side // 8)) * 4 + pix // 8
    k = math.tan(math.radians(fov_deg) / 2.0)
    u = ((x.double() + 0.5) / side * 2.0 - 1.0) * k
    v = (1.0 - (y.double() + 0.5) / side * 2.0) * k
    d = f[None, :] + u[:, None] * right[None, :] + v[:, None] * up[None, :]
    d = d / d.norm(dim=1, keepdim=True)
    return torch.tensor(eye, device=DEV, dtype=torch.float64).expand(n, 3), d


def _rays(o, d, tmin, tmax):
    r = torch.empty(o.shape[0], 8, device=DEV, dtype=torch.float32)
    r[:, 0:3], r[:, 3], r[:, 4:7], r[:, 7] = o, tmin, d, tmax
    return r


def _cluster_camera(g, n):
    """A camera outside the cluster box, a little off its axis."""
    jitter = ((_uniform(g, 3) - 0.5) * 20.0).tolist()
    return _rays(*_pinhole(n, [jitter[0], jitter[1], -250.0 + jitter[2]], [0.0, 0.0, 1.0]), 0.0, FAR)


def _cube_camera(g, n, side):
    lift = 0.4 * side * (1.0 + 0.1 * float(_uniform(g, 1)))
    eye = [0.0, lift, -1.7 * lift]
    return _rays(*_pinhole(n, eye, [0.0, -0.5, 0.866]), 0.0, FAR)


def _mesh_arrays(tri):
    """(positions, indices) host arrays of an unshared triangle soup (n, 3, 3)."""
    pos = tri.reshape(-1, 3).cpu().numpy()
    return pos, np.arange(len(pos), dtype=np.uint32)


def _hits_of(engine, scene, rays, tri):
    """The surface points and unit normals (toward the ray's side) that `rays` meet, in ray order."""
    h = engine.trace(scene, rays, A.CLOSEST, "fast")
    prim_at, hit = (2, h[:, 1] != -1) if scene.layout == A.LAYOUT_GI else (2, h[:, 1] != 0)
    t, prim = h[:, 0].view(torch.float32)[hit].double(), h[:, prim_at][hit].long()
    r = rays[hit].double()
    v = tri[prim].double()
    n = torch.linalg.cross(v[:, 1] - v[:, 0], v[:, 2] - v[:, 0])
    n = n / n.norm(dim=1, keepdim=True).clamp_min(1e-30)
    n = torch.where((n * r[:, 4:7]).sum(1, keepdim=True) > 0.0, -n, n)
    return r[:, 0:3] + r[:, 4:7] * t[:, None], n


def _tmin(p):
    return 1e-4 * p.abs().amax(dim=1).clamp_min(1.0)


def _hemisphere(g, p, n, count):
    """One cosine-weighted ray from each point in turn."""
    k = torch.arange(count, device=DEV) % p.shape[0]
    p, n = p[k], n[k]
    u = _uniform(g, count, 2)
    r, phi = torch.sqrt(u[:, 0]), 2.0 * math.pi * u[:, 1]
    helper = torch.zeros_like(n)
    helper[:, 1] = (n[:, 0].abs() > 0.9).double()
    helper[:, 0] = 1.0 - helper[:, 1]
    t = torch.linalg.cross(helper, n)
    t = t / t.norm(dim=1, keepdim=True)
    b = torch.linalg.cross(n, t)
    d = t * (r * torch.cos(phi))[:, None] + b * (r * torch.sin(phi))[:, None] + n * torch.sqrt((1.0 - u[:, 0]).clamp_min(0.0))[:, None]
    return _rays(p, d, _tmin(p), FAR)


def _to_lights(g, p, count, half=100.0, n_lights=16):
    """Rays from the points in turn toward point lights in the scene's box, up to the light."""
    lights = (2.0 * _uniform(g, n_lights, 3) - 1.0) * half
    p = p[torch.arange(count, device=DEV) % p.shape[0]]
    v = lights[torch.randint(0, n_lights, (count,), generator=g, device=DEV)] - p
    dist = v.norm(dim=1).clamp_min(1e-30)
    return _rays(p, v / dist[:, None], _tmin(p), dist * (1.0 - 1e-4))


def _octahedral(n):
    """Unit normals as the cells keep them: octahedral, two signed 16-bit halves."""
    p = n[:, :2] / n.abs().sum(dim=1, keepdim=True)
    sign = torch.where(p >= 0.0, 1.0, -1.0).double()
    q = torch.where(n[:, 2:3] >= 0.0, p, (1.0 - p.flip(1).abs()) * sign)
    s = torch.round(q.clamp(-1.0, 1.0) * 32767.0).long() & 0xFFFF
    return (s[:, 0] | (s[:, 1] << 16)).to(torch.int64)


def _i32(x):
    """Integers in [0, 2^32) as int32 words."""
    return torch.where(x >= 1 << 31, x - (1 << 32), x).to(torch.int32)


def _cells(g, p, n, count, edge=0.5):
    k = (torch.arange(count, device=DEV) * max(1, p.shape[0] // count)) % p.shape[0]
    out = torch.zeros(count, 8, device=DEV, dtype=torch.int32)
    out[:, 0:3] = p[k].float().view(torch.int32)
    out[:, 3] = torch.full((count,), edge, device=DEV).view(torch.int32)
    out[:, 4] = _i32(_octahedral(n[k]))
    out[:, 5] = _i32(torch.randint(0, 1 << 32, (count,), generator=g, device=DEV))
    return out


def _lights(g, count, half=100.0):
    """Point, spot and directional lights (80-byte records) around the scene."""
    f = torch.zeros(count, 20, device=DEV, dtype=torch.float32)
    f[:, 0:3] = (2.0 * _uniform(g, count, 3) - 1.0) * half
    f[:, 3] = 50.0 + 300.0 * _uniform(g, count)
    f[:, 4:7] = _unit(g, count)
    f[:, 7] = 0.2 + 0.5 * _uniform(g, count)
    f[:, 8:11] = 0.1 + _uniform(g, count, 3)
    words = f.view(torch.int32).clone()
    words[:, 12:16] = 0
    words[:, 12] = torch.randint(1, 3, (count,), generator=g, device=DEV) * (torch.arange(count, device=DEV) % 8 != 0)
    return words


# ---------------------------------------------------------------- states

_engine = None


def _the_engine():
    """A program has one engine on its device."""
    global _engine
    if _engine is None:
        _engine = A.Engine(0)
    return _engine


class _State:
    """What a program holds for one case; gives its scene back when dropped."""

    def __init__(self, case, seed):
        self.case, self.kind, self.engine = case, case["kind"], _the_engine()
        self.plan = self.scene = None
        self.gen = _gen(seed, 1)

    def upload(self, layout, meshes, instances, kernel="plain", primitives=True):
        self.scene = self.engine.upload(layout, A.pack_scene(layout, meshes, instances, primitives=[primitives] * len(meshes)))
        if kernel.startswith("wide8"):
            self.scene.prepare(kernel)

    def upload_soup(self, layout, tris, kernel="plain"):
        self.tri = _clusters(self.gen, tris)
        pos, idx = _mesh_arrays(self.tri)
        self.upload(layout, [A.Blas.build_device(self.engine, pos, idx)], _identity(), kernel)

    def upload_world(self, layout, case, half, kernel="plain"):
        """case["meshes"] cluster meshes of log-uniform size under case["instances"] placements."""
        lo, hi = math.log(case["tri_lo"]), math.log(case["tri_hi"])
        counts = torch.exp(lo + (hi - lo) * _uniform(self.gen, case["meshes"])).round().long().tolist()
        arrays = [_mesh_arrays(_clusters(self.gen, max(1, c), half=10.0)) for c in counts]
        meshes = [A.Blas.build_device(self.engine, p, i) for p, i in arrays]
        self.upload(layout, meshes, _placed(self.gen, case["instances"], len(meshes), half), kernel)

    def __del__(self):
        try:
            if self.plan is not None:
                self.plan.close()
            if self.scene is not None:
                torch.cuda.synchronize()
                self.scene.release()
        except Exception:
            pass


def _merged_cubes(g, side):
    """(n * 8, 3) float32 positions and the triangle list of side x side cubes in one mesh."""
    m = _cube_models(g, side)
    v = torch.einsum("nij,kj->nki", m[:, :, :3], torch.tensor(_CORNERS, device=DEV, dtype=torch.float64)) + m[:, None, :, 3]
    idx = np.asarray(_FACES, np.uint32)[None, :] + (np.arange(side * side, dtype=np.uint32) * 8)[:, None]
    return v.reshape(-1, 3).float(), idx.reshape(-1).astype(np.uint32)


def _seam_inputs(s):
    """Closest: the cubes merged into one mesh, seen by a camera. Visible: the same cubes as
    instances of one box, rays between points above and among them."""
    c = s.case
    if c["fn"] == "closest":
        s.positions, s.indices = _merged_cubes(s.gen, c["side"])
        s.rays = _cube_camera(s.gen, c["rays"], c["side"])
    else:
        s.models = _cube_models(s.gen, c["side"])
        n, half = c["rays"], float(c["side"])
        box = torch.tensor([half, 1.5, half], device=DEV, dtype=torch.float64)
        a, b = ((2.0 * _uniform(s.gen, n, 3) - 1.0) * box for _ in range(2))
        a[:, 1] += 1.5
        b[:, 1] += 1.5
        dist = (b - a).norm(dim=1).clamp_min(1e-3)
        s.rays = _rays(a, (b - a) / dist[:, None], 0.0, dist)


def _refit_inputs(s):
    """The soup, and the same vertices drawn toward the centre by a wave (inside the old box)."""
    c = s.case
    s.tri = _clusters(s.gen, c["tris"])
    p = s.tri.reshape(-1, 3).double()
    s.moved = (p * (1.0 - 0.05 * (1.0 + torch.sin(0.1 * p.flip(1))))).float()
    s.rays = _cluster_camera(s.gen, c["rays"])


def _move_inputs(s):
    c = s.case
    s.models = _cube_models(s.gen, c["side"])
    s.next = s.models.clone()
    s.next[:, :, 3] += 0.2 * (_uniform(s.gen, s.next.shape[0], 3) - 0.5)
    s.rays = _cube_camera(s.gen, c["rays"], c["side"])


def prepare(case, seed):
    s, c = _State(case, seed), case
    e, g = s.engine, s.gen
    if s.kind == "seam":
        _seam_inputs(s)
        if c["fn"] == "closest":
            blas = A.Blas.build_device(e, s.positions.cpu().numpy(), s.indices)
            s.upload(A.LAYOUT_GI, [blas], _identity())
        else:
            cube = A.Blas(np.asarray(_CORNERS, np.float32), np.asarray(_FACES, np.uint32))
            s.upload(A.LAYOUT_GI, [cube], _Instances(s.models, np.zeros(len(s.models))))
        s.o, s.d, s.tmax = s.rays[:, 0:3].contiguous(), s.rays[:, 4:7].contiguous(), s.rays[:, 7].contiguous()
    elif s.kind == "trace":
        s.upload_soup(c["layout"], c["tris"], c["kernel"])
        s.rays = _cluster_camera(g, c["rays"])
        if c["source"] != "primary":
            p, n = _hits_of(e, s.scene, s.rays, s.tri)
            s.rays = _hemisphere(g, p, n, c["rays"]) if c["source"] == "gi" else _to_lights(g, p, c["rays"])
    elif s.kind in ("cells", "lights"):
        if s.kind == "lights":
            s.upload_soup(A.LAYOUT_GI, c["tris"], c["kernel"])
            p, n = _hits_of(e, s.scene, _cluster_camera(g, 4 * c["cells"]), s.tri)
            s.cells, s.lights = _cells(g, p, n, c["cells"]), _lights(g, c["lights"])
        else:
            half = 15.0 * c["instances"] ** (1.0 / 3.0)
            s.upload_world(A.LAYOUT_GI, c, half)
            d = _unit(g, 4 * c["cells"])
            r = _rays((2.0 * _uniform(g, len(d), 3) - 1.0) * half, d, 0.0, FAR)
            h = A.decode_gi(e.trace(s.scene, r, A.CLOSEST, "fast"))
            hit = h["inst"] != -1
            n = h["normal"][hit].double()
            n = torch.where((n * d[hit]).sum(1, keepdim=True) > 0.0, -n, n)
            p = (r[:, 0:3] + r[:, 4:7] * h["t"][:, None])[hit].double()
            s.cells = _cells(g, p, n, c["cells"])
    elif s.kind == "batches":
        half = 25.0 * c["instances"] ** (1.0 / 3.0)
        s.upload_world(A.LAYOUT_REFLECTION, c, half, c["kernel"])
        s.batches = []
        for k in range(c["batches"]):  # log-spaced sizes and alternating modes, in a scattered order
            j = k * 7919 % c["batches"]
            n = int(round(c["n_lo"] * (c["n_hi"] / c["n_lo"]) ** ((j + 0.5) / c["batches"])))
            s.batches.append((_rays((2.0 * _uniform(g, n, 3) - 1.0) * half, _unit(g, n), 0.0, FAR), 2 if j % 2 else 0))
        if c["plan"]:
            s.plan = e.plan(s.scene, s.batches, c["kernel"], order=c["order"])
    elif s.kind == "host":
        s.upload_soup(A.LAYOUT_REFLECTION, c["tris"], "wide8")
        n = c["rays"]
        camera = _cluster_camera(g, n // 2)
        p, nrm = _hits_of(e, s.scene, camera, s.tri)
        parts = [(camera, 0, "wide8p"), (_hemisphere(g, p, nrm, n * 3 // 10), 0, "wide8"), (_to_lights(g, p, n // 5), 2, "wide8")]
        s.batches = []
        for r, mode, kernel in parts:
            words = A.hit_words(A.LAYOUT_REFLECTION, mode)
            out = torch.zeros((len(r), words) if words > 1 else (len(r),), dtype=torch.int32, pin_memory=True)
            s.batches.append((r.cpu().pin_memory(), mode, kernel, out))
    elif s.kind == "refit":
        _refit_inputs(s)
        pos, idx = _mesh_arrays(s.tri)
        s.upload(c["layout"], [A.Blas.build_device(e, pos, idx)], _identity())
        s.indices = torch.from_numpy(idx.view(np.int32)).to(DEV)
    elif s.kind == "move":
        _move_inputs(s)
        cube = A.Blas(np.asarray(_CORNERS, np.float32), np.asarray(_FACES, np.uint32))
        mesh = np.zeros(len(s.models))
        s.upload(c["layout"], [cube], _Instances(s.models, mesh))
        s.boxes = A.object_boxes(c["layout"], [cube])
        s.instances = _Instances(s.next, mesh)
    else:
        s.positions, s.indices = _mesh_arrays(_clusters(g, c["tris"]))
        s.nodes = np.zeros((max(c["tris"], 1), 16), np.uint32)  # a mesh cache with room for any tree
    return s


def _closest(layout, h):
    """A closest-hit record as a shading pass reads it: the distance only where something was hit."""
    t = h[:, 0].view(torch.float32)
    if layout == A.LAYOUT_GI:
        return {"t": torch.where(h[:, 1] != -1, t, 0.0), "ids": h[:, 1:5], "uv": h[:, 5:7].view(torch.float32),
                "normal": h[:, 7:10].view(torch.float32)}
    return {"t": torch.where(h[:, 1] != 0, t, 0.0), "ids": h[:, 1:3], "uv": h[:, 3:5].view(torch.float32)}


def run(s):
    c, e = s.case, s.engine
    if s.kind == "seam":
        if c["fn"] == "visible":
            return A.gi_visible_within(e, s.scene, s.o, s.d, s.tmax)
        h = A.gi_closest(e, s.scene, s.o, s.d, 0.0, FAR)
        return {"t": torch.where(h["inst"] != -1, h["t"], 0.0), "inst": h["inst"], "tri": h["tri"], "uv": h["bary"],
                "normal": h["normal"]}
    if s.kind == "trace":
        h = e.trace(s.scene, s.rays, c["mode"], c["kernel"])
        return h if c["mode"] else _closest(c["layout"], h)
    if s.kind == "cells":
        h = e.trace_gi_cells(s.scene, s.cells, c["mode"], c["rotate"])
        return h if c["mode"] else _closest(A.LAYOUT_GI, h)
    if s.kind == "lights":
        return e.trace_gi_lights(s.scene, s.cells, s.lights, c["kernel"])
    if s.kind == "batches":
        if s.plan is None:
            return e.trace_batches(s.scene, s.batches, c["kernel"])
        s.plan.launch()
        return s.plan.hits
    if s.kind == "host":
        out = e.trace_host_batches(s.scene, s.batches)
        return [x if x.dim() == 1 else {"t": x[:, 0].view(torch.float32), "ids": x[:, 1:3], "uv": x[:, 3:5].view(torch.float32)}
                for x in out]
    if s.kind == "refit":
        s.scene.refit(0, s.moved, s.indices if c["layout"] == A.LAYOUT_REFLECTION else None)
        return _closest(c["layout"], e.trace(s.scene, s.rays, A.CLOSEST, "fast"))
    if s.kind == "move":
        s.scene.move_instances(s.instances, s.boxes)
        return _closest(c["layout"], e.trace(s.scene, s.rays, A.CLOSEST, "fast"))
    blas = A.Blas.build_device(e, s.positions, s.indices, c["median"])
    nodes = blas.nodes()
    s.nodes[:len(nodes)] = nodes
    return {"count": len(nodes), "nodes": s.nodes, "indices": blas.bvh_indices()}


# ---------------------------------------------------------------- what a call cannot do without

def work(case):
    """Rays in, hits out, and the packed scene once (or the part of it that so few rays can read:
    some ten nodes and four triangles each); per ray a walk of log4(triangles) nodes of four boxes."""
    c, k = case, case["kind"]
    hit = {0: {0: 40, 1: 4, 2: 4}, 1: {0: 20, 1: 4, 2: 4}}

    def walk(rays, tris, ray_bytes):
        scene = min(62.0 * tris, rays * (10 * 64.0 + 4 * 48.0))
        return {"bytes": rays * ray_bytes + scene, "flops": rays * (80.0 * math.log(max(tris, 4), 4) + 100.0)}

    if k == "seam":
        return walk(c["rays"], 12 * c["side"] ** 2, 28 + (1 if c["fn"] == "visible" else 40))
    if k == "trace":
        return walk(c["rays"], c["tris"], 32 + hit[c["layout"]][c["mode"]])
    if k == "cells":
        mean = 0.5 * (c["tri_lo"] + c["tri_hi"]) * c["meshes"]
        return walk(64 * c["cells"], mean, 0.5 + hit[0][c["mode"]])
    if k == "lights":
        return walk(c["cells"] * c["lights"], c["tris"], 32.0 / c["lights"] + 0.125)
    if k == "batches":
        mean = 0.5 * (c["tri_lo"] + c["tri_hi"]) * c["meshes"]
        ratio = c["n_hi"] / c["n_lo"]
        return walk(c["batches"] * (c["n_hi"] - c["n_lo"]) / math.log(ratio), mean, 32 + 12)
    if k == "host":
        return walk(c["rays"], c["tris"], 32 + 0.8 * 20 + 0.2 * 4)
    if k == "refit":
        w = walk(c["rays"], c["tris"], 32 + hit[c["layout"]][0])
        return {"bytes": w["bytes"] + c["tris"] * (36.0 + 36.0 + 20.0), "flops": w["flops"] + 60.0 * c["tris"]}
    if k == "move":
        w = walk(c["rays"], 12 * c["side"] ** 2, 32 + hit[c["layout"]][0])
        return {"bytes": w["bytes"] + c["side"] ** 2 * (96.0 + 72.0 + 43.0), "flops": w["flops"]}
    n = c["tris"]
    return {"bytes": n * (36.0 + 12.0 + 12.0 + 20.0), "flops": 60.0 * n * math.log2(max(n / 6.0, 2.0))}


# ---------------------------------------------------------------- the hits in 64 bits

def _brute(rays, tri, pairs_at_once=1 << 27):
    """The nearest triangle of each ray by testing all of them in float64 (Moller-Trumbore over
    double-precision matrix products of the ray's and the triangles' Pluecker coordinates, the
    chosen triangle's values by the direct formula): (hit, t, u, v, triangle)."""
    o, d = rays[:, 0:3].double(), rays[:, 4:7].double()
    tmin, tmax = rays[:, 3].double(), rays[:, 7].double()
    a, b, c = tri.double().unbind(1)
    n = torch.linalg.cross(b - a, c - a)
    ray6 = torch.cat([d, torch.linalg.cross(o, d)], dim=1)
    edge = [torch.cat([torch.linalg.cross(p, q), q - p], dim=1).T.contiguous() for p, q in ((a, b), (b, c), (c, a))]
    plane = torch.cat([n, (n * a).sum(1, keepdim=True)], dim=1).T.contiguous()
    o4 = torch.cat([-o, torch.ones_like(o[:, :1])], dim=1)
    step = max(1, min(len(o), pairs_at_once // max(1, len(a))))
    best_t, best_i = torch.full_like(tmin, math.inf), torch.zeros(len(o), dtype=torch.long, device=DEV)
    for k in range(0, len(o), step):
        s = slice(k, k + step)
        w = [ray6[s] @ x for x in edge]
        low, high = torch.minimum(torch.minimum(w[0], w[1]), w[2]), torch.maximum(torch.maximum(w[0], w[1]), w[2])
        inside = (low >= 0.0) | (high <= 0.0)
        t = (o4[s] @ plane) / (d[s] @ plane[:3])
        t = torch.where(inside & (t > tmin[s, None]) & (t < tmax[s, None]), t, math.inf)
        best_t[s], best_i[s] = t.min(dim=1)
    hit = torch.isfinite(best_t)
    a, b, c = a[best_i], b[best_i], c[best_i]
    e1, e2, at = b - a, c - a, o - a
    p, q = torch.linalg.cross(d, e2), torch.linalg.cross(at, e1)
    det = (e1 * p).sum(1)
    u, v, t = ((x * y).sum(1) / det for x, y in ((at, p), (d, q), (e2, q)))
    zero = torch.zeros_like(t)
    return hit, torch.where(hit, t, zero), torch.where(hit, u, zero), torch.where(hit, v, zero), best_i


def exact(case, seed):
    """Closest hits of camera rays in float64; None for flags and words (whole values), and where
    testing every triangle is too long."""
    c, k = case, case["kind"]
    s = _State(case, seed)
    if k == "seam" and c["fn"] == "closest":
        if 12.0 * c["side"] ** 2 * c["rays"] > EXACT_PAIRS:
            return None
        _seam_inputs(s)
        tri, layout = s.positions[torch.from_numpy(s.indices.astype(np.int64)).to(DEV)].reshape(-1, 3, 3), 0
    elif k == "trace" and c["source"] == "primary" and c["mode"] == 0:
        if 1.0 * c["tris"] * c["rays"] > EXACT_PAIRS:
            return None
        tri, layout = _clusters(s.gen, c["tris"]), c["layout"]
        s.rays = _cluster_camera(s.gen, c["rays"])
    elif k == "refit":
        if 1.0 * c["tris"] * c["rays"] > EXACT_PAIRS:
            return None
        _refit_inputs(s)
        tri, layout = s.moved.reshape(-1, 3, 3), c["layout"]
    elif k == "move":
        if 12.0 * c["side"] ** 2 * c["rays"] > EXACT_PAIRS:
            return None
        _move_inputs(s)
        # where the engine's float32 world-to-object rows put the box's corners
        rows = torch.from_numpy(_Instances(s.next, np.zeros(len(s.next))).rows).to(DEV).double()
        inv = torch.linalg.inv(rows[:, :, :3])
        corner = torch.tensor(_CORNERS, device=DEV, dtype=torch.float64)[None] - rows[:, None, :, 3]
        world = torch.einsum("nij,nkj->nki", inv, corner)
        tri, layout = world[:, torch.tensor(_FACES, device=DEV)].reshape(-1, 3, 3), c["layout"]
    else:
        return None
    hit, t, u, v, i = _brute(s.rays, tri)
    out = {"t": t, "uv": torch.stack([u, v], dim=1)}
    if layout == A.LAYOUT_GI:
        x = tri.double()[i]
        n = torch.linalg.cross(x[:, 1] - x[:, 0], x[:, 2] - x[:, 0])
        out["normal"] = torch.where(hit[:, None], n / n.norm(dim=1, keepdim=True), 0.0)
    return out

"""The calls this renderer is measured on: ray casts, renders, gradients and scene builds.

Every case goes through the package's public entry points.  The sizes are those of the repository's
own workloads (scenes.py, bench.py, the tests) and of the calls around them: a pick of a few rays, a
preview frame, ragged block counts, progressive frames.  Scenes:
  * "room":  the 2x2x2 room with an icosphere of radius 0.6 and one light (closed: every ray hits)
  * "open":  the displaced icosphere on a ground plane under four lights (rays leave the scene)
  * "mesh":  the displaced icosphere alone (casts)
The sphere is turned by a rotation drawn from the seed, so every seed has another octree, and the
materials, rays and cameras are the seed's as well.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

import dumbray_gb300 as dr
from dumbray_gb300 import scenes

DEV = "cuda"
FLT_MAX = 3.4028234663852886e38
EPS = 0.000005          # the renderer's VECTOR_EPSILON
EXACT_PAIRS = 1.5e10    # ray-triangle pairs that a 64-bit brute force gets through in some seconds


def listed():
    return [
        # picking an object under a cursor, line-of-sight probes: a few rays, one launch
        dict(name="cast_pick", kind="cast", scene="room", level=5, tree="reference", split=0, rays=61, coherent=False,
             cull=True, counted=False, ignore=False),
        # light baking and visibility queries: an odd number of rays that leave surfaces, with
        # traversal statistics
        dict(name="cast_counted", kind="cast", scene="open", level=6, tree="physical", split=8, rays=100003,
             coherent=False, cull=False, counted=True, ignore=True),
        # the ray-cast benchmark: 1080p primary rays on the reference's octree
        dict(name="cast_primary", kind="cast", scene="mesh", level=8, tree="reference", split=0, rays=1920 * 1080,
             coherent=True, cull=True, counted=False, ignore=False),
        # the ray-cast benchmark: 8M incoherent rays
        dict(name="cast_incoherent", kind="cast", scene="mesh", level=8, tree="physical", split=8, rays=8388608,
             coherent=False, cull=True, counted=False, ignore=False),
        # a preview frame with DumbRenderer's defaults (1 sample, 2 bounces), ragged block grid
        dict(name="preview_reference", kind="render", mode="reference", scene="room", level=5, tree="reference", split=0,
             width=161, height=91, sx=1, sy=1, depth=2, lens="stochastic", iteration=1),
        # the plain path-trace configuration: room, 256x256, 16 spp, depth 4
        dict(name="room_physical", kind="render", mode="physical", scene="room", level=5, tree="reference", split=0,
             width=256, height=256, sx=4, sy=4, depth=4, lens="pinhole", iteration=1),
        # one progressive iteration of the drop-in path at full HD (DumbRenderer's estimator)
        dict(name="twin_hd", kind="render", mode="reference", scene="open", level=8, tree="reference", split=0,
             width=1920, height=1080, sx=2, sy=2, depth=8, lens="stochastic", iteration=1),
        # the full path trace at full HD, 16 of its 64 samples
        dict(name="path_hd", kind="render", mode="physical", scene="open", level=8, tree="physical", split=4,
             width=1920, height=1080, sx=4, sy=4, depth=8, lens="pinhole", iteration=1),
        # a later progressive iteration through the fisheye lens, odd resolution, blended
        dict(name="fisheye_blend", kind="render", mode="physical", scene="open", level=7, tree="physical", split=8,
             width=1283, height=717, sx=3, sy=3, depth=8, lens="fisheye", iteration=3),
        # uneven scenes, resolutions and sample counts in one batch, replayed as a graph
        dict(name="batch_mixed", kind="batch", jobs=10, max_tris=60000, max_side=512, max_spp=16, depth=6, split=4),
        # one optimiser step of the differentiable workload: image, loss, gradients
        dict(name="gradient", kind="gradient", level=7, width=512, height=512, sx=4, sy=4, depth=5),
        # an edited mesh: the scene is made again from host arrays (octree built on the GPU) and looked at
        dict(name="rebuild", kind="rebuild", scene="mesh", level=6, tree="physical", split=4, rays=320 * 180, coherent=True,
             cull=True, counted=False, ignore=False),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["cast", "cast", "cast", "render", "render", "render", "render", "batch", "gradient", "rebuild"])
    if kind == "cast":
        scene = rng.choice(["room", "open", "mesh"])
        tree = rng.choice(["reference", "physical"])
        level = rng.randint(3, 7)
        return dict(kind="cast", scene=scene, level=level, tree=tree,
                    split=0 if tree == "reference" else rng.choice([3, 4, 6, 8, 12]), rays=_log(rng, 1, 4000000),
                    coherent=rng.random() < 0.4, cull=rng.random() < 0.6, counted=rng.random() < 0.3,
                    ignore=rng.random() < 0.3)
    if kind == "render":
        mode = rng.choice(["reference", "physical"])
        scene = rng.choice(["room", "open"])
        tree = "reference" if mode == "reference" else rng.choice(["reference", "physical"])
        s = rng.randint(1, 4)
        side = _log(rng, 40, 1200)
        width = max(17, int(side * rng.uniform(0.8, 1.6)))
        return dict(kind="render", mode=mode, scene=scene, level=rng.randint(3, 7), tree=tree,
                    split=0 if tree == "reference" else rng.choice([3, 4, 6, 8, 12]), width=width,
                    height=max(9, side), sx=s, sy=rng.randint(1, s), depth=rng.randint(1, 8),
                    lens="stochastic" if mode == "reference" else rng.choice(["pinhole", "fisheye", "spherical"]),
                    iteration=rng.choice([1, 1, 2, 5]))
    if kind == "batch":
        return dict(kind="batch", jobs=rng.randint(2, 10), max_tris=_log(rng, 3000, 60000),
                    max_side=rng.choice([128, 256, 512]), max_spp=rng.choice([4, 16]), depth=rng.randint(2, 6),
                    split=rng.choice([3, 4, 8]))
    if kind == "gradient":
        side = _log(rng, 48, 400)
        return dict(kind="gradient", level=rng.randint(3, 7), width=side + rng.randint(0, 31), height=side,
                    sx=rng.randint(1, 4), sy=rng.randint(1, 4), depth=rng.randint(1, 5))
    tree = rng.choice(["reference", "physical"])
    return dict(kind="rebuild", scene=rng.choice(["room", "open", "mesh"]), level=rng.randint(2, 6), tree=tree,
                split=0 if tree == "reference" else rng.choice([3, 4, 8, 12]), rays=_log(rng, 1000, 100000), coherent=True,
                cull=True, counted=False, ignore=False)


# ---- inputs ----------------------------------------------------------------------------------------

@functools.lru_cache(maxsize=None)
def _sphere(level, displaced):
    return scenes.displaced_icosphere(level) if displaced else scenes.icosphere(level)


def _turned(tris, rng, radius):
    q = rng.normal(size=4)
    w, x, y, z = q / np.linalg.norm(q)
    r = np.array([[1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w)],
                  [2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w)],
                  [2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)]], np.float32)
    return ((tris.reshape(-1, 3) * np.float32(radius)) @ r.T).reshape(-1, 3, 3)


def _room(level, rng):
    walls = scenes.box((2.0, 2.0, 2.0), inward=True)
    light = scenes.quad((0.0, 0.999, 0.0), (0.5, 0.5), (0.0, -1.0, 0.0))
    tris = np.concatenate([walls, _turned(_sphere(level, False), rng, 0.6), light])
    mat = np.zeros(len(tris), np.int32)
    mat[:2] = 1
    mat[-2:] = 2
    return tris, mat


def _open(level, rng):
    mesh = _turned(_sphere(level, True), rng, 1.0)
    ground = scenes.quad((0.0, -1.2, 0.0), (40.0, 40.0), (0.0, 1.0, 0.0))
    lights = [scenes.quad((x, 3.0, z), (1.0, 1.0), (0.0, -1.0, 0.0)) for x in (-2.0, 2.0) for z in (-2.0, 2.0)]
    tris = np.concatenate([mesh, ground] + lights)
    kind = rng.integers(0, 100, len(tris))
    mat = np.where(kind < 60, 0, np.where(kind < 85, 1, 2)).astype(np.int32)
    mat[len(mesh):] = 0
    return tris, mat


def _geometry(case, rng):
    if case["scene"] == "mesh":
        tris = _turned(_sphere(case["level"], True), rng, 1.0)
        return tris, np.zeros(len(tris), np.int32)
    return (_room if case["scene"] == "room" else _open)(case["level"], rng)


def _epsilon(case):
    return dr.PHYSICAL_TREE if case["tree"] == "physical" else 0.0


def _rays(case, seed):
    """Origins and directions on the GPU: a pinhole grid, or origins in the scene's box with uniform directions."""
    n, g = case["rays"], torch.Generator(DEV).manual_seed(seed)
    room = case["scene"] == "room"
    if case["coherent"]:
        w = max(1, int(math.sqrt(n * 16 / 9)))
        i = torch.arange(n, device=DEV)
        x, y = (i % w + 0.5) / w - 0.5, 0.5 - (i // w + 0.5) / max(1, -(-n // w))
        turn = float(torch.rand(1, generator=g, device=DEV)) * 2 * math.pi
        d = torch.stack([x * 16 / 9, y, torch.full_like(x, 0.8660254)], 1)
        c, s = math.cos(turn), math.sin(turn)
        rot = torch.tensor([[c, 0, s], [0, 1, 0], [-s, 0, c]], device=DEV)
        at = torch.tensor([0.0, 0.0, -0.95 if room else -3.0], device=DEV)
        o, d = (rot @ at).expand(n, 3), torch.nn.functional.normalize(d, dim=1) @ rot.T
    else:
        o = (torch.rand(n, 3, generator=g, device=DEV) - 0.5) * (1.98 if room else 2.2)
        d = torch.nn.functional.normalize(torch.randn(n, 3, generator=g, device=DEV), dim=1)
    return o.contiguous(), d.contiguous()


def _ignored(case, seed, n_tris):
    if not case["ignore"]:
        return None
    g = torch.Generator(DEV).manual_seed(seed + 1)
    return torch.randint(-1, n_tris, (case["rays"],), generator=g, device=DEV, dtype=torch.int32)


LENSES = {"stochastic": (dr.LENS_SIMPLE_STOCHASTIC, 60.0, 60.0), "pinhole": (dr.LENS_PINHOLE, 60.0, 60.0),
          "fisheye": (dr.LENS_FISHEYE, 180.0, 180.0), "spherical": (dr.LENS_SPHERICAL, 200.0, 180.0)}


def _view(room, rng):
    """Camera position and (right, up, forward), float32."""
    turn = rng.uniform(0.0, 2.0 * math.pi)
    away, height = (0.97, 0.0) if room else (3.4, 0.6)
    p = np.array([away * math.sin(turn), height, -away * math.cos(turn)])
    f = np.array([0.0, 0.0 if room else -0.15, 0.0]) - p
    f /= np.linalg.norm(f)
    r = np.cross([0.0, 1.0, 0.0], f)
    r /= np.linalg.norm(r)
    return [v.astype(np.float32) for v in (p, r, np.cross(f, r), f)]


def _inputs(case, seed):
    """Everything a render needs, as plain arrays."""
    rng = np.random.default_rng(seed)
    tris, mat = _geometry(case, rng)
    room, n = case["scene"] == "room", len(tris)
    s = dict(tris=tris, mat=mat, view=_view(room, rng), seed=int(rng.integers(1, 1 << 31)), room=room)
    if case["mode"] == "physical":
        if room:
            s["albedo"] = np.array([[0.7, 0.7, 0.7], [0.7, 0.1, 0.1], [0.0, 0.0, 0.0]], np.float32)[mat]
        else:
            s["albedo"] = rng.uniform(0.2, 0.8, (n, 3)).astype(np.float32)
            s["albedo"][-10:-8], s["albedo"][-8:] = 0.5, 0.0
        s["emission"] = np.zeros((n, 3), np.float32)
        s["emission"][-2 if room else -8:] = 10.0
        s["roughness"] = rng.uniform(0.05, 0.4, n).astype(np.float32)
        s["kinds"] = ["lambert"] * 3 if room else ["lambert", "mirror", "glossy"]
    else:  # emitters become spherical lights
        keep = n - (2 if room else 8)
        s["tris"], s["mat"] = tris[:keep], mat[:keep]
        if room:
            s["kinds"] = [("dumb", (0.7, 0.7, 0.7), (0.2, 0.2, 0.2), 8.0, 0.0), ("dumb", (0.7, 0.1, 0.1), (0.2, 0.2, 0.2), 8.0, 0.0)]
            s["lights"] = [((0.625,) * 3, (0.0, 0.8, 0.0), 0.05)]
        else:
            s["kinds"] = [("dumb", (0.5, 0.5, 0.5), (0.2, 0.2, 0.2), 8.0, 0.0), ("stochastic", (0.9, 0.9, 0.9), 0.0, 1.0, 64.0),
                          ("dumb", (1.0, 1.0, 1.0), (0.6, 0.6, 0.6), 48.0, 1.0)]
            s["lights"] = [((31.415926,) * 3, (x, 2.95, z), 0.3) for x in (-2.0, 2.0) for z in (-2.0, 2.0)]
    return s


def _scene(case, s):
    if case["mode"] == "physical":
        make = dict(lambert=dr.lambert, mirror=dr.mirror, glossy=dr.glossy)
        scene = dr.Scene(s["tris"], mat_id=s["mat"], materials=[make[k]() for k in s["kinds"]], split_threshold=case["split"],
                         box_epsilon=_epsilon(case), device_build=True)
        scene.set_triangle_params(s["albedo"], s["emission"], s["roughness"])
        return scene
    mats = [dr.dumb_based(diffuse=k[1], fresnel=k[2], specular=k[3], metal=k[4]) if k[0] == "dumb" else dr.simple_stochastic(*k[1:])
            for k in s["kinds"]]
    return dr.Scene(s["tris"], mat_id=s["mat"], materials=mats, lights=[dr.spherical_light(*l) for l in s["lights"]],
                    split_threshold=case["split"], box_epsilon=_epsilon(case), device_build=True)


def _camera(lens, view):
    kind, a, b = LENSES[lens]
    return dr.camera(kind, position=view[0], angle=(a, b), basis=view[1:])


def _prior(width, height, seed):
    """A frame buffer that holds the earlier iterations' mean."""
    g = torch.Generator(DEV).manual_seed(seed)
    fb = dr.new_frame_buffer(width, height, DEV)
    return fb.copy_(torch.rand(fb.shape, generator=g, device=DEV))


def _gradient_inputs(case, seed):
    rng = np.random.default_rng(seed)
    walls = scenes.box((2.0, 2.0, 2.0), inward=True)
    tris = np.concatenate([walls, _turned(_sphere(case["level"], False), rng, 0.6)])
    n = len(tris)
    emission = np.zeros((n, 3), np.float32)
    emission[len(walls) + rng.choice(n - len(walls), size=64, replace=False)] = 10.0
    return dict(tris=tris, mat=np.zeros(n, np.int32), kinds=["lambert"], emission=emission, room=True,
                albedo=rng.uniform(0.1, 0.9, (n, 3)).astype(np.float32), roughness=np.full(n, 0.2, np.float32),
                view=_view(True, rng), seed=int(rng.integers(1, 1 << 31)))


def _target(case, seed):
    return _prior(case["width"], case["height"], seed + 1) * 0.3


def _job_sizes(case):
    """Side and samples per pixel of a batch's jobs: every mix of the two in turn."""
    sides = [r for r in (128, 256, 512) if r <= case["max_side"]]
    spps = [p for p in (1, 4, 16) if p <= case["max_spp"]]
    return [(sides[i % len(sides)], spps[(i + i // len(sides)) % len(spps)]) for i in range(case["jobs"])]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "cast":
        tris, mat = _geometry(case, np.random.default_rng(seed))
        scene = dr.Scene(tris, mat_id=mat, materials=[dr.lambert()] * 3, split_threshold=case["split"],
                         box_epsilon=_epsilon(case), device_build=True)
        o, d = _rays(case, seed)
        return dict(case=case, scene=scene, o=o, d=d, ignore=_ignored(case, seed, len(tris)))
    if kind == "render":
        s = _inputs(case, seed)
        w, h = case["width"], case["height"]
        fb = _prior(w, h, seed) if case["iteration"] > 1 else dr.new_frame_buffer(w, h, DEV)
        params = dr.render_params(w, h, dr.MODE_REFERENCE if case["mode"] == "reference" else dr.MODE_PHYSICAL,
                                  samples=(case["sx"], case["sy"]), max_bounces=case["depth"], iteration=case["iteration"], seed=s["seed"])
        return dict(case=case, scene=_scene(case, s), camera=_camera(case["lens"], s["view"]), fb=fb, params=params,
                    renderer=dr.Renderer(), blocks=dr.block_count(w, h))
    if kind == "batch":
        jobs = []
        for j, (size, spp) in zip(scenes.batch_workload(case["jobs"], seed=seed, max_tris=case["max_tris"]), _job_sizes(case)):
            scene = dr.Scene(j["tris"], mat_id=j["mat_id"], materials=[dr.lambert(), dr.mirror(), dr.glossy()],
                             split_threshold=case["split"], box_epsilon=dr.PHYSICAL_TREE, device_build=True)
            scene.set_triangle_params(j["albedo"], j["emission"], j["roughness"])
            cam = dr.camera(dr.LENS_PINHOLE, position=j["cam_pos"], target=j["cam_target"], angle=60.0)
            side = math.isqrt(spp)
            params = dr.render_params(size, size, dr.MODE_PHYSICAL, samples=(side, side), max_bounces=case["depth"],
                                      seed=seed * 101 + j["seed"])
            jobs.append((scene, cam, params, dr.new_frame_buffer(size, size, DEV), 0, dr.block_count(size, size)))
        return dict(case=case, jobs=jobs, batch=dr.Batch(jobs), renderer=dr.Renderer())
    if kind == "gradient":
        s = _gradient_inputs(case, seed)
        scene = dr.Scene(s["tris"], mat_id=s["mat"], materials=[dr.lambert()], box_epsilon=dr.PHYSICAL_TREE, device_build=True)
        scene.set_triangle_params(s["albedo"], s["emission"], s["roughness"])
        params = dr.render_params(case["width"], case["height"], dr.MODE_PHYSICAL, samples=(case["sx"], case["sy"]),
                                  max_bounces=case["depth"], seed=s["seed"])
        return dict(case=case, scene=scene, camera=_camera("pinhole", s["view"]), params=params, renderer=dr.Renderer(1 << 20),
                    albedo=torch.from_numpy(s["albedo"]).to(DEV).requires_grad_(True),
                    emission=torch.from_numpy(s["emission"]).to(DEV).requires_grad_(True), target=_target(case, seed))
    tris, mat = _geometry(case, np.random.default_rng(seed))
    o, d = _rays(case, seed)
    return dict(case=case, tris=tris, mat=mat, epsilon=_epsilon(case), materials=[dr.lambert()] * 3, o=o, d=d)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "cast":
        return dr.cast(state["scene"], state["o"], state["d"], ignore=state["ignore"], cull_backfaces=case["cull"],
                       counted=case["counted"])
    if kind == "render":
        state["renderer"].render_blocks(state["scene"], state["camera"], state["fb"], 0, state["blocks"], state["params"])
        return state["fb"]
    if kind == "batch":
        state["batch"].render(state["renderer"], use_graph=True)
        return [j[3] for j in state["jobs"]]
    if kind == "gradient":
        image = dr.render_differentiable(state["scene"], state["camera"], state["params"], state["albedo"], state["emission"],
                                         state["renderer"])
        loss = ((image - state["target"]) ** 2).sum()
        return (image.detach(),) + torch.autograd.grad(loss, (state["albedo"], state["emission"]))
    scene = dr.Scene(state["tris"], mat_id=state["mat"], materials=state["materials"], split_threshold=case["split"],
                     box_epsilon=state["epsilon"], device_build=True)
    return dr.cast(scene, state["o"], state["d"], cull_backfaces=case["cull"])


# ---- what a pass cannot do without -----------------------------------------------------------------

BOX_FLOPS, TRIANGLE_FLOPS, SHADE_FLOPS = 18.0, 60.0, 150.0


def _triangles(case):
    n = 20 * 4 ** case["level"]
    return n + {"room": 14, "open": 10, "mesh": 0}[case.get("scene", "room")]


def _cast_flops(casts, triangles):
    """A cast goes down one path of an 8-way tree, eight boxes a level, and tests the triangle it hits."""
    return casts * (8 * BOX_FLOPS * max(1.0, math.log(triangles, 8)) + TRIANGLE_FLOPS)


def _render_work(paths, pixels, triangles, depth, closed, lights):
    """Closed scenes keep every path to its last bounce; in the open ones about 1.6 vertices a path are hit."""
    vertices = depth + 1.0 if closed else min(1.6, depth + 1.0)
    casts = paths * (vertices + vertices * lights)
    # geometry, materials and shading records once, the frame buffer once
    return dict(bytes=36.0 * triangles + 32.0 * triangles + 16.0 * pixels,
                flops=_cast_flops(casts, triangles) + SHADE_FLOPS * paths * vertices)


def work(case):
    kind = case["kind"]
    if kind == "cast":
        n = _triangles(case)
        per_ray = 24 + 8 + (8 if case["counted"] else 0) + (4 if case["ignore"] else 0)
        return dict(bytes=float(per_ray * case["rays"] + 36 * min(n, case["rays"])), flops=_cast_flops(case["rays"], n))
    if kind == "render":
        lights = 4 if case["mode"] == "reference" and case["scene"] == "open" else 1
        pixels = case["width"] * case["height"]
        return _render_work(pixels * case["sx"] * case["sy"], pixels, _triangles(case), case["depth"], case["scene"] == "room", lights)
    if kind == "batch":
        sizes = _job_sizes(case)
        triangles = case["jobs"] * (case["max_tris"] - 1000) / math.log(case["max_tris"] / 1000)  # log-uniform from 1000
        return _render_work(sum(r * r * p for r, p in sizes), sum(r * r for r, _ in sizes), triangles, case["depth"], False, 1)
    if kind == "gradient":
        n, pixels = 20 * 4 ** case["level"] + 12, case["width"] * case["height"]
        w = _render_work(pixels * case["sx"] * case["sy"], pixels, n, case["depth"], True, 1)
        # forward and replay; the gradients are written, the target image is read
        return dict(bytes=2 * w["bytes"] + 24.0 * n + 32.0 * pixels, flops=2 * w["flops"])
    n = _triangles(case)
    # geometry and material ids in, a tree of about as many bytes out; a triangle is clipped once a level, some 200 operations
    return dict(bytes=2 * 40.0 * n + 32.0 * case["rays"], flops=200.0 * n * max(1.0, math.log(n, 8)) + _cast_flops(case["rays"], n))


# ---- the same in 64 bits, by brute force -----------------------------------------------------------

def _t(x):
    return torch.as_tensor(np.asarray(x), device=DEV).double()


def _dot(a, b):
    return (a * b).sum(-1)


def _unit(a):
    return a / a.norm(dim=-1, keepdim=True)


class _Mesh:
    """Triangles with the renderer's predicate: plane test, then the three edge angles with their tolerance."""

    def __init__(self, tris):
        v = _t(tris)
        self.a, self.b, self.c = v[:, 0], v[:, 1], v[:, 2]
        self.ab, self.bc, self.ca = self.b - self.a, self.c - self.b, self.a - self.c
        self.n = torch.linalg.cross(self.ab, self.c - self.a)      # plane normal of the cast
        self.unit = _unit(-self.n)                                  # outward: (c - a) x (b - a)
        self.area = 0.5 * self.n.norm(dim=1)
        self.edges = []
        for p, e, f in ((self.a, self.ab, self.ca), (self.b, self.bc, self.ab), (self.c, self.ca, self.bc)):
            self.edges.append((p, e, -_dot(e, f) / f.norm(dim=1)))

    def cast(self, o, d, ignore=None, cull=False):
        """(distance in units of |d|, triangle), inf and -1 where nothing is hit."""
        t_all = torch.full((len(o),), math.inf, dtype=torch.float64, device=DEV)
        i_all = torch.full((len(o),), -1, dtype=torch.int64, device=DEV)
        T = len(self.a)
        step = max(1, int(1.2e8 // T))
        ids = torch.arange(T, device=DEV)
        for r in range(0, len(o), step):
            O, D = o[r:r + step], d[r:r + step]
            dp = _dot(self.a, self.n) - O @ self.n.T
            dirp = D @ self.n.T
            t = dp / dirp
            ok = dp * dirp > 0
            if cull:
                ok &= dp >= -EPS
            if ignore is not None:
                ok &= ids != ignore[r:r + step, None]
            for p, e, y in self.edges:
                x = O @ e.T - _dot(p, e) + t * (D @ e.T)
                # |o + t d - p|^2, expanded
                od = _dot(O, D)[:, None] - D @ p.T
                oo = _dot(O, O)[:, None] - 2 * (O @ p.T) + _dot(p, p)
                q = (oo + t * (2 * od + t * _dot(D, D)[:, None])).clamp_min(0)
                ok &= (x / q.sqrt() + 32 * EPS >= y) | (q == 0)
            t = torch.where(ok, t, math.inf)
            best, at = t.min(dim=1)
            t_all[r:r + step] = best
            i_all[r:r + step] = torch.where(best.isinf(), -1, at)
        return t_all, i_all


def _hash(x):
    x = x & 0xFFFFFFFF
    x = x ^ (x >> 16)
    x = (x * 0x7feb352d) & 0xFFFFFFFF
    x = x ^ (x >> 15)
    x = (x * 0x846ca68b) & 0xFFFFFFFF
    return x ^ (x >> 16)


def _random(key, bounce, dim):
    u = _hash(_hash(key + 0x9E3779B9 * (bounce * 128 + dim + 1)))
    return (u >> 8).double() / 16777216.0


def _paths(case, s):
    """Pixel coordinates, sample index within the pixel and random key of every path; the slot of its pixel."""
    w, h, spp = case["width"], case["height"], case["sx"] * case["sy"]
    i = torch.arange(w * h * spp, device=DEV)
    pixel, k = i // spp, i % spp
    x, y = pixel % w, pixel // w
    base = _hash(torch.tensor((s["seed"] ^ 0x2545F491) & 0xFFFFFFFF, device=DEV))
    key = _hash(_hash(base ^ pixel) + (case.get("iteration", 1) - 1) * spp + k)
    slot = ((y // 16) * -(-w // 8) + x // 8) * 128 + (y % 16) * 8 + x % 8
    return x.double(), y.double(), k, key, slot


def _world(s, v):
    r, u, f = (_t(a) for a in s["view"][1:])
    return v[:, :1] * r + v[:, 1:2] * u + v[:, 2:] * f


def _frame(case, seed, image):
    """Blended with the prior image as a later iteration is; alpha 1."""
    nb, w, h = -(-case["width"] // 8) * -(-case["height"] // 16), case["width"], case["height"]
    fb = torch.zeros(nb * 128, 4, dtype=torch.float64, device=DEV)
    k = case.get("iteration", 1)
    if k > 1:
        g = torch.Generator(DEV).manual_seed(seed)
        fb = torch.rand((nb * 128, 4), generator=g, device=DEV).double()
    slot = torch.arange(nb * 128, device=DEV)
    block, at = slot // 128, slot % 128
    inside = ((block % -(-w // 8)) * 8 + at % 8 < w) & ((block // -(-w // 8)) * 16 + at // 8 < h)
    new = torch.cat([image, torch.ones(nb * 128, 1, dtype=torch.float64, device=DEV)], 1)
    return torch.where(inside[:, None], new / k + fb * (1 - 1 / k), fb)


def _mis(a, b):
    return a * a / (a * a + b * b)


def _ggx_d(c, a):
    return a * a / (math.pi * (c * c * (a * a - 1) + 1) ** 2)


def _ggx_g(c, a):
    return 2 * c / (c + (a * a + (1 - a * a) * c * c).sqrt())


def _basis(n):
    s = torch.where(n[:, 2] >= 0, 1.0, -1.0)
    a = -1 / (s + n[:, 2])
    b = n[:, 0] * n[:, 1] * a
    return (torch.stack([1 + s * n[:, 0] ** 2 * a, s * b, -s * n[:, 0]], 1), torch.stack([b, s + n[:, 1] ** 2 * a, -n[:, 1]], 1))


def _physical(case, s, albedo, emission):
    """Mean radiance per slot: emission hits and sampled lights, each weighted against the other."""
    mesh = _Mesh(s["tris"])
    x, y, _, key, slot = _paths(case, s)
    w, h = case["width"], case["height"]
    sx = (x + _random(key, 1023, 0) - 0.5 * w) / h
    sy = (0.5 * h - (y + _random(key, 1023, 1))) / h
    lens = case.get("lens", "pinhole")
    _, ang0, ang1 = LENSES[lens]
    alive = torch.ones_like(sx, dtype=torch.bool)
    if lens == "fisheye":
        theta, phi = (sx * sx + sy * sy).sqrt() * math.radians(ang0), torch.atan2(sy, sx)
        alive = theta <= math.pi
        d = torch.stack([theta.sin() * phi.cos(), theta.sin() * phi.sin(), theta.cos()], 1)
    elif lens == "spherical":
        u, v = sx * math.radians(ang0), sy * math.radians(ang1)
        d = torch.stack([u.sin() * v.cos(), v.sin(), u.cos() * v.cos()], 1)
    else:
        d = _unit(torch.stack([sx, sy, torch.full_like(sx, 0.5 / math.tan(math.radians(ang0) / 2))], 1))
    d = _unit(_world(s, d))
    o = _t(s["view"][0]).expand_as(d)
    keep = alive.nonzero()[:, 0]
    o, d, key, slot = o[keep], d[keep], key[keep], slot[keep]
    thr = torch.ones_like(d)
    prev, pdf, delta = torch.full_like(key, -1), torch.zeros_like(d[:, 0]), torch.ones_like(key, dtype=torch.bool)
    em0 = _t(s["emission"])
    power = em0.sum(1) * mesh.area
    lit = (em0.sum(1) > 0).nonzero()[:, 0]
    cdf, total = power[lit].cumsum(0), float(power.sum())
    light_pdf = em0.sum(1) / total
    kinds = torch.tensor([("lambert", "mirror", "glossy").index(k) for k in s["kinds"]], device=DEV)[torch.as_tensor(s["mat"], device=DEV).long()]
    rough = _t(s["roughness"])
    nb = -(-w // 8) * -(-h // 16)
    image = torch.zeros(nb * 128, 3, dtype=torch.float64, device=DEV)
    for b in range(case["depth"] + 1):
        t, tri = mesh.cast(o, d, prev)
        hit = (tri >= 0).nonzero()[:, 0]
        o, d, key, slot, thr, pdf, delta, t, tri = (v[hit] for v in (o, d, key, slot, thr, pdf, delta, t, tri))
        if not len(tri):
            break
        p, wo, out = o + d * t[:, None], -d, mesh.unit[tri]
        n = torch.where(_dot(out, wo)[:, None] < 0, -out, out)
        cosl = _dot(out, wo)
        em = emission[tri]
        shows = (em0[tri].sum(1) > 0) & (cosl > 0)
        pl = light_pdf[tri] * t * t * _dot(d, d) / cosl
        weight = torch.where(delta, torch.ones_like(t), _mis(pdf, pl)).where(shows, torch.zeros_like(t))
        image = image.index_add(0, slot, thr * em * weight[:, None])
        if b == case["depth"]:
            break
        alb, kind, alpha = albedo[tri], kinds[tri], rough[tri].clamp_min(1e-3)
        # a point of a light
        u = _random(key, b, 3) * total
        li = lit[torch.searchsorted(cdf, u).clamp_max(len(lit) - 1)]
        su = _random(key, b, 4).sqrt()
        ba, bb = 1 - su, _random(key, b, 5) * su
        lv = mesh.a[li] * ba[:, None] + mesh.b[li] * bb[:, None] + mesh.c[li] * (1 - ba - bb)[:, None] - p
        wi = _unit(lv)
        cl, ci = -_dot(mesh.unit[li], wi), _dot(n, wi)
        pl = light_pdf[li] * _dot(lv, lv) / cl
        half = _unit(wi + wo)
        nh, no = _dot(n, half), _dot(n, wo)
        spec = _ggx_d(nh, alpha) * _ggx_g(no, alpha) * _ggx_g(ci, alpha) / (4 * no * ci)
        gl = kind == 2
        f = torch.where(gl, spec, torch.full_like(spec, 1 / math.pi))
        pb = torch.where(gl, _ggx_d(nh, alpha) * nh / (4 * _dot(wo, half).abs()), ci / math.pi)
        go = ((kind != 1) & (cl > 0) & (ci > 0)).nonzero()[:, 0]
        tl, il = mesh.cast(p[go], lv[go], tri[go])
        go = go[(il < 0) | (il == li[go]) | ~(tl < 0.999)]
        k = (f * ci / pl * _mis(pl, pb))[go]
        image = image.index_add(0, slot[go], thr[go] * alb[go] * emission[li[go]] * k[:, None])
        # the next direction
        u1, u2 = _random(key, b, 1), _random(key, b, 2)
        T, B = _basis(n)
        phi, r = 2 * math.pi * u2, u1.sqrt()
        z = (1 - u1).clamp_min(0).sqrt()
        nd = T * (r * phi.cos())[:, None] + B * (r * phi.sin())[:, None] + n * z[:, None]
        scale, npdf = torch.ones_like(z), z / math.pi
        mi = kind == 1
        nd = torch.where(mi[:, None], d - n * (2 * _dot(d, n))[:, None], nd)
        ct = ((1 - u2) / (1 + (alpha * alpha - 1) * u2)).sqrt()
        st, phi = (1 - ct * ct).clamp_min(0).sqrt(), 2 * math.pi * u1
        half = T * (st * phi.cos())[:, None] + B * (st * phi.sin())[:, None] + n * ct[:, None]
        oh = _dot(wo, half)
        gd = half * (2 * oh)[:, None] - wo
        gc = _dot(n, gd)
        nd = torch.where(gl[:, None], gd, nd)
        scale = torch.where(gl, _ggx_g(no, alpha) * _ggx_g(gc, alpha) * oh.abs() / (no * ct), scale)
        npdf = torch.where(gl, _ggx_d(ct, alpha) * ct / (4 * oh.abs()), npdf)
        on = (~gl | (gc > 0)).nonzero()[:, 0]
        thr = (thr * alb * scale[:, None])[on]
        o, d, key, slot, prev, pdf, delta = p[on], _unit(nd[on]), key[on], slot[on], tri[on], npdf[on], mi[on]
    return image / (case["sx"] * case["sy"])


def _on_sphere(u, v, radius):
    cos = 1 - 2 * v
    sin = (1 - cos * cos).clamp_min(0).sqrt()
    a = 2 * math.pi * u
    return torch.stack([sin * a.cos(), sin * a.sin(), cos], 1) * radius


def _mirrored(v, n):
    return v - n * (2 * _dot(v, n) / _dot(n, n))[:, None]


class _Shaders:
    """The two reference shaders on flat normals: material columns gathered by triangle."""

    def __init__(self, s, mesh):
        self.mesh, self.mat = mesh, torch.as_tensor(s["mat"], device=DEV).long()
        k = s["kinds"]
        self.dumb = torch.tensor([m[0] == "dumb" for m in k], device=DEV)
        self.color = _t([m[1] for m in k])
        self.fresnel = _t([m[2] if m[0] == "dumb" else (0.0,) * 3 for m in k])
        self.spec = _t([m[3] if m[0] == "dumb" else 8.0 for m in k])
        self.metal = _t([m[4] if m[0] == "dumb" else 0.0 for m in k])
        total = [max(1.0, m[2] + m[3]) if m[0] != "dumb" else 1.0 for m in k]
        self.diff = _t([m[2] / q if m[0] != "dumb" else 0.0 for m, q in zip(k, total)])
        self.gloss = _t([m[3] / q if m[0] != "dumb" else 0.0 for m, q in zip(k, total)])
        self.shine = _t([m[4] if m[0] != "dumb" else 1.0 for m in k])

    def request(self, tri, ray, key, b):
        """(direction, kind of sample, whether there is one)."""
        m, n = self.mat[tri], self.mesh.unit[tri]
        dumb, metal = self.dumb[m], _random(key, b, 0) <= self.metal[m]
        point = _on_sphere(_random(key, b, 1), _random(key, b, 2), 1.0)
        point = torch.where(_dot(point, n)[:, None] < 0, -point, point)
        refl = _mirrored(ray, n)
        soft = _unit(point * self.diff[m][:, None] + refl * self.gloss[m][:, None])
        r = _unit(refl)
        side = torch.where(_dot(r, n)[:, None] < 0, -n, n)
        a = _unit(torch.linalg.cross(r, _t([1.0, 0.0, 0.0]).expand_as(r)))
        c = torch.linalg.cross(r, a)
        lobe, todo = torch.zeros_like(r), torch.ones_like(metal)
        for k in range(32):
            cos = _random(key, b, 8 + 2 * k) ** (1 / self.spec[m])
            sin = (1 - cos * cos).sqrt()
            ac = (_random(key, b, 9 + 2 * k) * 2 * math.pi).cos()
            v = r * cos[:, None] + (a * ac[:, None] + c * (1 - ac * ac).clamp_min(0).sqrt()[:, None]) * sin[:, None]
            lobe = torch.where(todo[:, None], v, lobe)
            todo = todo & (_dot(v, side) < 0)
            if not bool((todo & dumb & metal).any()):
                break
        d = torch.where(dumb[:, None], torch.where(metal[:, None], lobe, point), soft)
        return d, torch.where(dumb, torch.where(metal, 1, 2), 0), ~(dumb & metal & (_dot(n, ray) >= 0))

    def reflect(self, tri, photon, observer, direct, sample):
        """Share of the photon's colour that leaves toward the observer."""
        m, n = self.mat[tri], self.mesh.unit[tri]
        wi, w0 = -_unit(photon), _unit(observer)
        wh = _unit(w0 + wi)
        metal, spec = self.metal[m], self.spec[m]
        f5 = (1 - _dot(wh, wi)) ** 5
        fr = self.fresnel[m]
        brdf = fr + (1 - fr) * f5[:, None]
        if direct:
            nh, n0, ni, oh = _dot(n, wh), _dot(n, w0), _dot(n, wi), _dot(w0, wh)
            g = torch.minimum(torch.ones_like(nh), torch.minimum(2 * nh * n0 / oh, 2 * nh * ni / oh))
            brdf = brdf * ((spec + 2) / (2 * math.pi) * nh ** spec * g / (4 * n0 * ni))[:, None]
        brdf = brdf.nan_to_num(0.0).clamp(0, 1)
        diffuse = self.color[m] * ((1 - metal) * _dot(n, wi))[:, None]
        if direct:
            c = (brdf * metal[:, None] + diffuse).clamp(0, 1)
        else:
            c = torch.where((sample == 1)[:, None], brdf, torch.where((sample == 2)[:, None], diffuse / (1 - metal).clamp_min(1e-30)[:, None], 0.0))
        c = torch.where((_dot(n, observer) < 0)[:, None], 0.0, c)
        if not direct:
            c = torch.where((_dot(n, photon) > 0)[:, None], 1.0, c)
        refl = _mirrored(photon, n)
        rc = (_dot(refl, n) / refl.norm(dim=1)).clamp_min(0)
        oc = (_dot(observer, refl) / (observer.norm(dim=1) * refl.norm(dim=1))).clamp_min(0)
        soft = self.color[m] * (self.diff[m] * rc + self.gloss[m] * oc ** self.shine[m])[:, None]
        return torch.where(self.dumb[m][:, None], c, soft)


def _reference(case, s):
    """DumbRenderer's estimator: one indirect sample a layer, one photon a light, photons pass what reflects them on."""
    mesh = _Mesh(s["tris"])
    sh = _Shaders(s, mesh)
    x, y, k, key, slot = _paths(case, s)
    w, h, fx, fy = case["width"], case["height"], case["sx"], case["sy"]
    i, j = (k // fy).double(), (k % fy).double()
    px = (x - w / 2) / h + (i + _random(key, 1023, 0)) / (h * fx)
    py = (h / 2 - y) / h + (j + _random(key, 1023, 1)) / (h * fy)
    d = _world(s, torch.stack([px, py, torch.full_like(px, 0.5 / math.tan(math.radians(30.0)))], 1))
    o = _t(s["view"][0]).expand_as(d)
    thr, prev = torch.ones_like(d), torch.full_like(key, -1)
    nb = -(-w // 8) * -(-h // 16)
    image = torch.zeros(nb * 128, 3, dtype=torch.float64, device=DEV)
    for b in range(case["depth"] + 1):
        t, tri = mesh.cast(o, d, prev, cull=True)
        hit = (tri >= 0).nonzero()[:, 0]
        o, d, key, slot, thr, t, tri = (v[hit] for v in (o, d, key, slot, thr, t, tri))
        if not len(tri):
            break
        p = o + d * t[:, None]
        for li, (color, position, radius) in enumerate(s["lights"]):
            e = _on_sphere(_random(key, b, 72 + 3 * li), _random(key, b, 73 + 3 * li), radius)
            e = e * _random(key, b, 74 + 3 * li)[:, None] + _t(position)
            ld = _unit(p - e)
            lc = _t(color) / _dot(p - e, p - e)[:, None]
            c = thr * sh.reflect(tri, ld, -d, True, None)
            go = (c.sum(1) != 0).nonzero()[:, 0]
            q, r, ign = e[go], ld[go], torch.full_like(go, -1)
            lc, c, goal, at, where = lc[go], c[go], tri[go], p[go], slot[go]
            for _ in range(64):
                if not len(q):
                    break
                tl, il = mesh.cast(q, r, ign, cull=True)
                f = q + r * tl.where(il >= 0, torch.zeros_like(tl))[:, None]
                there = (il >= 0) & ((il == goal) | (_dot(f - at, f - at) <= 8 * EPS))
                image = image.index_add(0, where[there], (c * lc)[there])
                lc = lc * sh.reflect(il.clamp_min(0), r, r, True, None)
                on = ((il >= 0) & ~there & (lc.sum(1) > EPS)).nonzero()[:, 0]
                q, r, ign = f[on] + r[on] * (64 * EPS), r[on], il[on]
                lc, c, goal, at, where = lc[on], c[on], goal[on], at[on], where[on]
        if b == case["depth"]:
            break
        nd, kind, on = sh.request(tri, d, key, b)
        thr = thr * sh.reflect(tri, -nd, -d, False, kind)
        on = on.nonzero()[:, 0]
        o, d, prev, key, slot, thr = p[on], nd[on], tri[on], key[on], slot[on], thr[on]
    return image / (fx * fy)


def exact(case, seed):
    """Triangle numbers and counts have no such value; the large scenes would take minutes."""
    kind = case["kind"]
    if kind in ("cast", "rebuild"):
        if case["rays"] * _triangles(case) > EXACT_PAIRS:
            return None
        tris, _ = _geometry(case, np.random.default_rng(seed))
        o, d = _rays(case, seed)
        t, _ = _Mesh(tris).cast(o.double(), d.double(), _ignored(case, seed, len(tris)), case["cull"])
        t = t.clamp_max(FLT_MAX)
        return (None, t, None, None) if case["counted"] else (None, t)
    if kind in ("render", "gradient"):
        casts = work(case)["flops"] / _cast_flops(1, _triangles(case))
        if casts * _triangles(case) > EXACT_PAIRS:
            return None
    if kind == "render":
        s = _inputs(case, seed)
        if case["mode"] == "reference":
            return _frame(case, seed, _reference(case, s))
        return _frame(case, seed, _physical(case, s, _t(s["albedo"]), _t(s["emission"])))
    if kind == "gradient":
        s = _gradient_inputs(case, seed)
        albedo, emission = _t(s["albedo"]).requires_grad_(True), _t(s["emission"]).requires_grad_(True)
        image = _frame(case, seed, _physical(case, s, albedo, emission))
        loss = ((image - _target(case, seed).double()) ** 2).sum()
        return (image.detach(),) + torch.autograd.grad(loss, (albedo, emission))
    return None

"""Timed cases of the ray-query and path-tracing engine, through its public classes.

A case is a scene (an icosphere field over a ground quad, the recipe of
``sort_b200.scenes``, generated here on the GPU from the seed), a tree over it
and one pass of a query, a render, a batch list, a request mix or a build:

  closest  Accelerator.GetIntersect on rays in device memory
  any      Accelerator.GetAttenuation (shadow rays) on rays in device memory
  host     Accelerator.GetIntersect on page-locked host rays, results in host memory
  batch    Batcher.run: uneven ray batches over several resident scenes
  render   PathTracer.Render: whole frames, depth 5
  serve    RenderServer: a closed set of render requests of uneven sizes
  build    Accelerator.Build of a scene and its first rays

Ray kinds: camera (coherent primary rays, one per pixel, jittered), bounce
(cosine-weighted diffuse rays from camera hits: incoherent) and shadow (from
camera hits towards a 2 x 2 light above the scene).
"""
import functools
import math

import numpy as np
import torch

from sort_b200 import Batch, Batcher, Hits, Obvh, Qbvh, _lib, scenes
from sort_b200.pathtracer import PathTracer
from sort_b200.server import RenderServer

BUILDERS = {"host": _lib.SG_BUILDER_HOST, "gpu": _lib.SG_BUILDER_GPU, "lbvh": _lib.SG_BUILDER_LBVH,
            "ploc": _lib.SG_BUILDER_PLOC}
NODES = {"fp32": _lib.SG_NODES_FP32, "q8": _lib.SG_NODES_QUANT8}
FLT_MAX = 3.4028234663852886e38
DEPTH = 5  # bounces of every render


def listed():
    return [
        # An interactive pick or a probe grid: a few thousand rays, where the launch and the
        # slowest ray's latency are the whole cost.
        {"name": "closest_4k", "op": "closest", "spheres": 64, "level": 3, "width": 8, "nodes": "fp32",
         "builder": "gpu", "kind": "camera", "rays": 4099},
        # The ray-cast benchmark: coherent primary rays, one per pixel of 1024 x 1024, over a
        # tree that fits in L2.
        {"name": "raycast_82k", "op": "closest", "spheres": 64, "level": 3, "width": 4, "nodes": "fp32",
         "builder": "gpu", "kind": "camera", "rays": 1 << 20},
        # The headline: incoherent closest-hit on 21M triangles.
        {"name": "closest_21m", "op": "closest", "spheres": 1024, "level": 5, "width": 8, "nodes": "fp32",
         "builder": "gpu", "kind": "bounce", "rays": 1 << 22},
        # Its shadow rays.
        {"name": "shadow_21m", "op": "any", "spheres": 1024, "level": 5, "width": 8, "nodes": "fp32",
         "builder": "gpu", "kind": "shadow", "rays": 1 << 22},
        # 8-bit child boxes, and a batch of an ordinary odd size: a bounce of a frame that is
        # rendered by the caller's own integrator.
        {"name": "closest_q8_1m", "op": "closest", "spheres": 64, "level": 5, "width": 8, "nodes": "q8",
         "builder": "host", "kind": "bounce", "rays": 700_001},
        # A caller whose rays live in host memory, as SORT's integrators' do.
        {"name": "host_closest_5m", "op": "host", "spheres": 256, "level": 5, "width": 8, "nodes": "fp32",
         "builder": "gpu", "kind": "bounce", "rays": 2_000_003},
        # Many uneven batches over scenes of 10k to 2M triangles in one run.
        {"name": "batch_mix", "op": "batch", "scenes": 5, "width": 8, "nodes": "fp32", "batches": 24,
         "rays_max": 1 << 20},
        # A 1080p frame.
        {"name": "render_1080p", "op": "render", "spheres": 256, "level": 5, "width": 8, "nodes": "fp32",
         "pixels_x": 1920, "pixels_y": 1080, "spp": 2},
        # A preview tile: launches and their latency count.
        {"name": "render_tile", "op": "render", "spheres": 20, "level": 4, "width": 8, "nodes": "fp32",
         "pixels_x": 161, "pixels_y": 91, "spp": 4},
        # A render service's request mix on two resident scenes.
        {"name": "serve_mix", "op": "serve", "spheres": 50, "level": 5, "width": 8, "nodes": "fp32", "requests": 24,
         "pixels_max": 960, "spp_max": 16},
        # Loading a 5M-triangle scene with SORT's tree, and its first rays.
        {"name": "build_sah_5m", "op": "build", "spheres": 256, "level": 5, "width": 8, "nodes": "fp32",
         "builder": "gpu", "kind": "camera", "rays": 1 << 16},
        # Rebuilding a changing scene every frame with the fast builder, and its first rays.
        {"name": "build_lbvh_1m", "op": "build", "spheres": 64, "level": 5, "width": 8, "nodes": "fp32",
         "builder": "lbvh", "kind": "camera", "rays": 1 << 16},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["closest", "closest", "closest", "any", "any", "host", "batch", "render", "render", "serve",
                     "build"])
    level = rng.choice([3, 4, 5])
    per = 20 * 4 ** level
    most = {"closest": 20_971_520, "any": 20_971_520, "host": 5_242_880, "build": 5_242_880, "render": 5_242_880,
            "serve": 1_024_000, "batch": 0}[op]
    c = {"op": op, "width": rng.choice([4, 8, 8]), "nodes": rng.choice(["fp32", "fp32", "fp32", "q8"])}
    if op != "batch":
        c["spheres"] = min(_log(rng, 8, 1024), most // per)
        c["level"] = level
    if op in ("closest", "any", "host", "build"):
        c["builder"] = rng.choice(["gpu", "gpu", "lbvh", "ploc"])
        if c["builder"] in ("lbvh", "ploc"):
            c["nodes"] = "fp32"
        c["kind"] = "shadow" if op == "any" else rng.choice(["camera", "bounce"])
        c["rays"] = _log(rng, 4096, {"closest": 1 << 22, "any": 1 << 22, "host": 2_000_000, "build": 1 << 17}[op])
    elif op == "batch":
        c["scenes"] = rng.randint(2, 5)
        c["batches"] = rng.randint(3, 24)
        c["rays_max"] = _log(rng, 1 << 15, 1 << 20)
    elif op == "render":
        s = rng.random()
        c["pixels_x"] = int(round(64 * (1920 / 64) ** s))
        c["pixels_y"] = int(round(64 * (1080 / 64) ** s))
        c["spp"] = max(1, min(rng.choice([1, 2, 4, 16]), 2 * 1920 * 1080 // (c["pixels_x"] * c["pixels_y"])))
    else:
        c["requests"] = rng.randint(4, 24)
        c["pixels_max"] = _log(rng, 128, 960)
        c["spp_max"] = rng.choice([1, 4, 16])
    return c


# ---- scenes -----------------------------------------------------------------------

def _gen(seed, k=0):
    g = torch.Generator(device="cuda")
    g.manual_seed(1_000_003 * int(seed) + k)
    return g


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64)


@functools.lru_cache(maxsize=4)
def _ball(level):
    v, f = scenes.icosphere(level)
    return torch.from_numpy(v[f].reshape(-1, 3)).cuda()  # (20 * 4**level * 3, 3)


def _field(spheres, level, g):
    """sphere_field's recipe on the GPU: (triangles, 9) float32, the ground quad last."""
    ball = _ball(level)
    centres = _rand(g, spheres, 3) * 20.0 - 10.0
    q = torch.randn(spheres, 4, generator=g, device="cuda", dtype=torch.float64)
    w, x, y, z = (q / q.norm(dim=1, keepdim=True)).unbind(1)
    rot = torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w),
                       2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w),
                       2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)], 1).reshape(-1, 3, 3)
    rot = rot * (_rand(g, spheres) * 1.5 + 0.5)[:, None, None]
    out = torch.empty(spheres * ball.shape[0] // 3 + 2, 9, device="cuda", dtype=torch.float32)
    body = out[:-2].view(spheres, -1, 3)
    for a in range(0, spheres, 64):  # 64 spheres at a time: bounded double-precision temporaries
        part = torch.einsum("vk,sjk->svj", ball, rot[a:a + 64]) + centres[a:a + 64, None, :]
        body[a:a + 64] = part.float()
    h, gy = 60.0, -11.0
    out[-2:] = torch.tensor([[-h, gy, -h, h, gy, h, -h, gy, h], [-h, gy, -h, h, gy, -h, h, gy, h]], device="cuda")
    return out


def _camera(n, g):
    """n camera rays: one jittered ray per pixel of the smallest square that holds n."""
    side = math.isqrt(n - 1) + 1
    k = torch.arange(n, device="cuda", dtype=torch.float64)
    py = torch.floor(k / side)
    px = k - py * side
    jit = _rand(g, 2, n)
    half = math.tan(math.radians(45.0) * 0.5)
    d = torch.stack([((px + jit[0]) / side * 2 - 1) * half, (1 - (py + jit[1]) / side * 2) * half, -torch.ones_like(k)])
    rays = torch.empty(8, n, device="cuda", dtype=torch.float32)
    rays[0:2] = 0.0
    rays[2] = 30.0
    rays[3:6] = (d / d.norm(dim=0)).float()
    rays[6] = 0.0
    rays[7] = FLT_MAX
    return rays


def _secondary(tri, cam, hits, kind, g):
    """One bounce or shadow ray per camera ray (a camera ray that missed takes another's hit)."""
    n = cam.shape[1]
    found = torch.nonzero(hits.prim >= 0).flatten()
    src = torch.arange(n, device="cuda")
    if found.numel() < n:
        lost = torch.nonzero(hits.prim < 0).flatten()
        src[lost] = found[torch.randint(found.numel(), (lost.numel(),), generator=g, device="cuda")]
    o = cam[0:3, src].double()
    d = cam[3:6, src].double()
    p = o + d * hits.t[src].double()
    rays = torch.empty(8, n, device="cuda", dtype=torch.float32)
    rays[0:3] = p.float()
    if kind == "shadow":
        u = _rand(g, 2, n) * 2 - 1
        to = torch.stack([u[0], torch.full_like(u[0], 15.0), u[1]]) - p
        dist = to.norm(dim=0)
        rays[3:6] = (to / dist).float()
        rays[6] = 0.01
        rays[7] = (dist - 0.01).float()
        return rays
    v = tri[hits.prim[src].long()].double().view(n, 3, 3)
    nrm = torch.linalg.cross(v[:, 2] - v[:, 0], v[:, 1] - v[:, 0]).T
    nrm = nrm / nrm.norm(dim=0).clamp_min(1e-30)
    nrm = torch.where((nrm * d).sum(0) > 0, -nrm, nrm)
    u = _rand(g, 2, n)
    r, phi = u[0].sqrt(), 2 * math.pi * u[1]
    up = torch.tensor([0.0, 1.0, 0.0], device="cuda", dtype=torch.float64)[:, None].expand(3, n)
    side = torch.tensor([1.0, 0.0, 0.0], device="cuda", dtype=torch.float64)[:, None].expand(3, n)
    tx = torch.linalg.cross(torch.where(nrm[0].abs() > 0.9, up, side), nrm, dim=0)
    tx = tx / tx.norm(dim=0)
    tz = torch.linalg.cross(nrm, tx, dim=0)
    w = tx * (r * phi.cos()) + nrm * (1 - u[0]).clamp_min(0).sqrt() + tz * (r * phi.sin())
    rays[3:6] = (w / w.norm(dim=0)).float()
    rays[6] = 1e-4
    rays[7] = FLT_MAX
    return rays


def _accel(c, builder):
    return (Qbvh if c["width"] == 4 else Obvh)(node_format=NODES[c["nodes"]], builder=BUILDERS[builder])


def _rays(acc, tri, kind, n, g):
    cam = _camera(n, g)
    return cam if kind == "camera" else _secondary(tri, cam, acc.GetIntersect(cam), kind, g)


def _tracer(c, spheres, level, seed, k):
    """A path-tracing scene: per-sphere materials, the area light's two triangles appended."""
    tri = np.concatenate([_field(spheres, level, _gen(seed, k)).cpu().numpy(),
                          scenes.light_triangles(scenes.AREA_LIGHT)])
    mat, table = scenes.instance_materials(spheres, level, seed=int(seed) % 100_003 + k)
    mat = np.concatenate([mat, np.array([-1, -1], np.int32)])
    return PathTracer(tri, mat, table, scenes.AREA_LIGHT, width=c["width"], node_format=NODES[c["nodes"]])


BATCH_SCENES = [(8, 3), (40, 3), (40, 4), (50, 5), (100, 5)]  # the batch workload's smaller scenes, 10k .. 2M


def prepare(case, seed):
    c, op = case, case["op"]
    if op in ("closest", "any", "host"):
        g = _gen(seed)
        tri = _field(c["spheres"], c["level"], g)
        acc = _accel(c, c["builder"])
        acc.Build(tri.cpu().numpy())
        rays = _rays(acc, tri, c["kind"], c["rays"], g)
        if op != "host":
            return {"op": op, "acc": acc, "rays": rays}
        n = c["rays"]
        pinned = torch.empty(8, n, dtype=torch.float32, pin_memory=True)
        pinned.copy_(rays)
        res = [torch.empty(n, dtype=t, pin_memory=True) for t in (torch.int32,) + (torch.float32,) * 3]
        return {"op": op, "acc": acc, "rays": pinned.numpy(), "out": Hits(*(x.numpy() for x in res)),
                "keep": (pinned, res)}
    if op == "build":
        g = _gen(seed)
        tri = _field(c["spheres"], c["level"], g)
        rays = _camera(c["rays"], g)
        if c["kind"] == "bounce":
            acc = _accel(c, c["builder"])
            acc.Build(tri.cpu().numpy())
            rays = _secondary(tri, rays, acc.GetIntersect(rays), "bounce", g)
        return {"op": op, "case": dict(c), "tri": tri.cpu().numpy(), "rays": rays}
    if op == "batch":
        g = _gen(seed)
        pick = np.random.default_rng(int(seed))
        accs, tris = [], []
        for k in range(c["scenes"]):
            tris.append(_field(*BATCH_SCENES[k], g))
            accs.append(_accel(c, "gpu"))
            accs[-1].Build(tris[-1].cpu().numpy())
        batches = []
        # Sizes log-uniform from 4,096 to rays_max, scene uniform, kinds as a renderer mixes them.
        # They belong to the case: another seed draws other scenes and rays, not other sizes.
        plan = np.random.default_rng(c["batches"] * 1_000_003 + c["rays_max"])
        for _ in range(c["batches"]):
            n = int(np.exp(plan.uniform(np.log(4096), np.log(max(c["rays_max"], 4097)))))
            s, kind = int(plan.integers(c["scenes"])), ("camera", "bounce", "bounce", "shadow")[plan.integers(4)]
            batches.append(Batch(accs[s], _rays(accs[s], tris[s], kind, n, g), any=kind == "shadow"))
        order = pick.permutation(len(batches))
        return {"op": op, "batcher": Batcher(max_batches=64), "batches": [batches[k] for k in order], "accs": accs}
    if op == "render":
        return {"op": op, "pt": _tracer(c, c["spheres"], c["level"], seed, 0), "case": dict(c),
                "seed": int(seed) % (1 << 31)}
    # serve: two scenes, the second with a tenth of the first's spheres; sizes belong to the case
    pts = [_tracer(c, max(1, c["spheres"] // (1 if k == 0 else 10)), c["level"], seed, k) for k in range(2)]
    srv = RenderServer(path_slots=1 << 20, pixel_budget=1 << 23, samples_per_claim=64)
    for pt in pts:
        srv.add_scene(pt)
    plan = np.random.default_rng(c["requests"] * 1_000_003 + c["pixels_max"])
    reqs = []
    for k in range(c["requests"]):
        w = int(round(64 * (c["pixels_max"] / 64) ** plan.random()))
        h = max(1, w * 9 // 16)
        spp = int(min(c["spp_max"], plan.choice([1, 4, 16])))
        img = torch.empty(h, w, 3, dtype=torch.float32, pin_memory=True)
        reqs.append((int(plan.integers(2)), w, h, spp, int(seed) % (1 << 20) + k, img))
    return {"op": op, "srv": srv, "reqs": reqs}


def run(s):
    op = s["op"]
    if op == "closest":
        h = s["acc"].GetIntersect(s["rays"])
        return [h.prim, h.t, h.u, h.v]
    if op == "any":
        return s["acc"].GetAttenuation(s["rays"])
    if op == "host":
        h = s["acc"].GetIntersect(s["rays"], out=s["out"])
        return [h.prim, h.t, h.u, h.v]
    if op == "batch":
        done = s["batcher"].run(s["batches"])
        return [torch.cat([b.hits.prim for b in done if not b.any] or [torch.empty(0, device="cuda")]),
                torch.cat([b.hits.t for b in done if not b.any] or [torch.empty(0, device="cuda")]),
                torch.cat([b.occluded for b in done if b.any] or [torch.empty(0, device="cuda")])]
    if op == "render":
        c = s["case"]
        return s["pt"].Render(scenes.CAMERA, c["pixels_x"], c["pixels_y"], c["spp"], DEPTH, seed=s["seed"])
    if op == "serve":
        tickets = [s["srv"].submit(sc, scenes.CAMERA, w, h, spp, DEPTH, seed=seed, image=img.numpy())
                   for sc, w, h, spp, seed, img in s["reqs"]]
        return [s["srv"].wait(t)[0] for t in tickets]
    acc = _accel(s["case"], s["case"]["builder"])
    acc.Build(s["tri"])
    h = acc.GetIntersect(s["rays"])
    i = acc.info()
    return [h.prim, h.t, h.u, h.v, [i["interior_nodes"], i["leaves"], i["depth"]], list(i["bbox"])]


def _triangles(c):
    return c["spheres"] * 20 * 4 ** c["level"] + 2


def _trace_work(tri, rays, width, io):
    """Rays in, answers out, each node and triangle of the tree at most once, and per ray the box
    and triangle tests of SORT's traversal: 13.4 nodes and 19.2 triangles on 21M triangles
    (OBVH), growing with the depth of the tree."""
    depth = math.log2(max(tri, 16)) / 24.3
    nodes, tests = 13.4 * depth * (8 / width) ** 0.6, 19.2 * depth
    per_ray = nodes * width * 28 + tests * 36
    tree = tri * 36 + tri / 17.0 * 224
    return {"bytes": rays * io + min(tree, rays * per_ray), "flops": rays * (nodes * width * 12 + tests * 45)}


def work(case):
    c, op = case, case["op"]
    if op in ("closest", "any", "host"):
        return _trace_work(_triangles(c), c["rays"], c["width"], 33 if op == "any" else 48)
    if op == "build":
        tri = _triangles(c)
        w = _trace_work(tri, c["rays"], c["width"], 48)
        # 36 bytes a triangle in; 48-byte records and about a seventeenth of a 224-byte node out
        return {"bytes": w["bytes"] + tri * (36 + 48 + 13), "flops": w["flops"] + tri * 20 * math.log2(tri)}
    if op == "batch":
        mean = (c["rays_max"] - 4096) / max(1e-9, math.log(max(c["rays_max"], 4097) / 4096))
        parts = [_trace_work(BATCH_SCENES[k][0] * 20 * 4 ** BATCH_SCENES[k][1], mean * c["batches"] / c["scenes"],
                             c["width"], 44) for k in range(c["scenes"])]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    if op == "render":
        samples = c["pixels_x"] * c["pixels_y"] * c["spp"]
        w = _trace_work(_triangles(c), samples * 3.4, c["width"], 0)  # about 3.4 rays a sample
        return {"bytes": w["bytes"] + 12 * c["pixels_x"] * c["pixels_y"], "flops": w["flops"] + samples * 2500}
    mean = sum((64 * (c["pixels_max"] / 64) ** ((k + 0.5) / 16)) ** 2 * 9 / 16 for k in range(16)) / 16
    samples = c["requests"] * mean * (1 + min(4, c["spp_max"]) + min(16, c["spp_max"])) / 3
    w = _trace_work(_triangles(c), samples * 3.4, c["width"], 0)
    return {"bytes": w["bytes"] + 12 * mean * c["requests"], "flops": w["flops"] + samples * 2500}


def exact(case, seed):
    """Brute force over every triangle in 64 bits, for batches where that is quick: the nearest
    distance per ray (the largest float where there is none). Which of two triangles that are hit
    within rounding of each other is named is the tree's business, and u, v follow it: None."""
    c = case
    if c["op"] != "closest" or c["rays"] * _triangles(c) > 6e8 or c["kind"] != "camera":
        return None
    g = _gen(seed)
    tri = _field(c["spheres"], c["level"], g).double().view(-1, 3, 3)
    rays = _camera(c["rays"], g).double()
    best = torch.full((c["rays"],), FLT_MAX, device="cuda", dtype=torch.float64)
    e1, e2 = tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    step = max(1, 20_000_000 // tri.shape[0])
    for a in range(0, c["rays"], step):  # Moeller and Trumbore's test, every ray against every triangle
        o, d = rays[0:3, a:a + step].T[:, None, :], rays[3:6, a:a + step].T[:, None, :]
        p = torch.linalg.cross(d, e2[None], dim=2)
        det = (p * e1).sum(2)
        q0 = o - tri[None, :, 0]
        u = (p * q0).sum(2) / det
        q = torch.linalg.cross(q0, e1[None].expand_as(q0), dim=2)
        v = (q * d).sum(2) / det
        t = (q * e2).sum(2) / det
        t = torch.where((det != 0) & (u >= 0) & (v >= 0) & (u + v <= 1) & (t > 0), t, best.new_tensor(FLT_MAX))
        best[a:a + step] = t.amin(1)
    return [None, best, None, None]

"""What this library is measured on: ray queries, renders, batches and the radiance cache.

Every case goes through the public Python API (ptb200).  A case is a dict of plain values with a
``kind``; ``prepare`` makes what a program holds before the call (scene, renderer, network, ray
buffers), ``run`` makes the one call that is timed, ``work`` states the bytes and operations the
call cannot do without, and ``exact`` gives the answer in 64 bits where plain torch can.
"""
from __future__ import annotations

import functools
import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "cuda-path-tracer_b200"))
import ptb200 as pt  # noqa: E402

# The scenes: the Cornell box (23 primitives), displaced spheres at the sizes of the batch
# workload, the 1M-triangle procedural scene (its walked arrays fit in L2) and a cloud of spheres
# and small random triangles like the traversal microbenchmark's (its walked arrays do not).
SCENES = {
    "cornell": None,
    "spheres10k": dict(sphere_count=2, segments=51, rings=51, seed=11),
    "spheres65k": dict(sphere_count=4, segments=90, rings=92, seed=12),
    "spheres200k": dict(sphere_count=6, segments=129, rings=130, seed=13),
    "procedural1m": dict(),
    "soup2m": dict(sphere_count=32, box_size=1.0, radius_min=0.03, radius_max=0.08, floor=0, light_fraction=0.0,
                   random_triangles=1 << 19, seed=3),
}
TRIANGLES = {"cornell": 20, "spheres10k": 10204, "spheres65k": 65524, "spheres200k": 199696, "procedural1m": 1048580,
             "soup2m": 2621440}
BOX = (0.0, 0.0, 0.0), (10.0, 10.0, 10.0)     # scene box of the network cases


@functools.lru_cache(maxsize=8)
def host_scene(name: str, width: int, height: int):
    """(FlatScene, camera) of a scene, built once per process."""
    if SCENES[name] is None:
        return pt.cornell_box(width, height)
    return pt.procedural_scene(width, height, **SCENES[name])


def listed() -> list[dict]:
    return [
        # a picking or line-of-sight query of an interactive tool: a few rays, latency only
        dict(name="query-pick", kind="query", scene="cornell", mode="closest", rays=64, mix="box"),
        # the headline query: 2^25 rays, half camera rays and half bounce rays, on the 1M-triangle scene
        dict(name="query-closest-1m", kind="query", scene="procedural1m", mode="closest", rays=1 << 25, mix="camera+bounce"),
        # occlusion rays of a baking or visibility pass, an odd count, each with its own tmax
        dict(name="query-shadow-1m", kind="query", scene="procedural1m", mode="any", rays=3_000_017, mix="shadow"),
        # incoherent rays on a scene whose tree does not fit in L2
        dict(name="query-soup", kind="query", scene="soup2m", mode="closest", rays=1 << 22, mix="surface"),
        # rays and answers in host memory: the whole call with its copies
        dict(name="query-host", kind="host", scene="procedural1m", mode="closest", rays=1_500_003),
        # the drop-in form of the reference's validation query: full 56-byte records, host arrays
        dict(name="query-compat", kind="compat", scene="spheres65k", rays=100_003),
        # the small render of the reference's own demo scene
        dict(name="render-cornell", kind="render", scene="cornell", width=320, height=200, samples=16, depth=8, mis=True),
        # the large render: 1M triangles, a quarter of the benchmark's 64 samples
        dict(name="render-1m", kind="render", scene="procedural1m", width=960, height=600, samples=16, depth=8, mis=True),
        # jobs of uneven size and scene in one launch
        dict(name="batch-6", kind="batch", jobs=6, samples=8, side=256),
        # one cached frame at 1080p with the network as it is (a final render after training)
        dict(name="cached-1080p", kind="cached", scene="procedural1m", width=1920, height=1080, depth=12, spf=4),
        # the cache network alone: a query batch, and the gradients of a training batch
        dict(name="net-query-2m", kind="net-query", count=1 << 21),
        dict(name="net-gradients-64k", kind="net-gradients", count=1 << 16),
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    """One more case: sizes over the logarithm of the listed ranges."""
    kind = rng.choice(["query", "query", "query", "host", "compat", "render", "render", "batch", "cached", "net-query",
                       "net-gradients"])
    if kind == "query":
        scene = rng.choice(["cornell", "spheres10k", "spheres65k", "procedural1m", "soup2m"])
        if scene == "cornell":
            return dict(kind=kind, scene=scene, mode=rng.choice(["closest", "any"]), rays=_log_int(rng, 1, 1 << 22), mix="box")
        mode = rng.choice(["closest", "any"])
        mix = "shadow" if mode == "any" else rng.choice(["camera+bounce", "surface"])
        return dict(kind=kind, scene=scene, mode=mode, rays=_log_int(rng, 16, 1 << (22 if scene == "soup2m" else 24)), mix=mix)
    if kind == "host":
        return dict(kind=kind, scene=rng.choice(["spheres10k", "procedural1m"]), mode=rng.choice(["closest", "any"]),
                    rays=_log_int(rng, 100, 1 << 21))
    if kind == "compat":
        return dict(kind=kind, scene=rng.choice(["cornell", "spheres10k", "spheres65k"]), rays=_log_int(rng, 100, 1 << 19))
    if kind == "render":
        scene = rng.choice(["cornell", "spheres10k", "spheres65k", "procedural1m"])
        big = scene == "procedural1m"
        return dict(kind=kind, scene=scene, width=_log_int(rng, 40, 960 if big else 480), height=_log_int(rng, 30, 600 if big else 300),
                    samples=_log_int(rng, 1, 16), depth=rng.choice([4, 8, 12, 50]), mis=rng.random() < 0.8)
    if kind == "batch":
        return dict(kind=kind, jobs=rng.randint(1, 6), samples=_log_int(rng, 1, 8), side=_log_int(rng, 40, 256))
    if kind == "cached":
        return dict(kind=kind, scene=rng.choice(["spheres65k", "procedural1m"]), width=_log_int(rng, 120, 1920),
                    height=_log_int(rng, 80, 1080), depth=rng.choice([4, 8, 12]), spf=rng.choice([1, 2, 4]))
    if kind == "net-query":
        return dict(kind=kind, count=_log_int(rng, 1, 1 << 21))
    return dict(kind=kind, count=_log_int(rng, 64, 1 << 17))


# ---------------------------------------------------------------- inputs
def _generator(seed: int) -> torch.Generator:
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _box_rays(count: int, seed: int) -> torch.Tensor:
    """Rays from random points inside the Cornell box in random directions, as (count, 7) floats."""
    g = _generator(seed)
    rays = torch.zeros((count, 7), device="cuda")
    rays[:, 0:3] = torch.rand(count, 3, device="cuda", generator=g) * 0.9 + 0.05
    rays[:, 3:6] = torch.nn.functional.normalize(torch.randn(count, 3, device="cuda", generator=g), dim=1)
    return rays


def _query_rays(case: dict, scene, cam, seed: int):
    """(rays (n, 7) float32, tmax or None) on the GPU."""
    n, mix = case["rays"], case["mix"]
    if mix == "box":
        rays = _box_rays(n, seed)
        tmax = torch.rand(n, device="cuda", generator=_generator(seed + 7)) + 0.05 if case["mode"] == "any" else None
        return rays, tmax
    rays = torch.empty((n, 7), dtype=torch.float32, device="cuda")
    if mix == "shadow":
        tmax = torch.empty(n, dtype=torch.float32, device="cuda")
        scene.surface_rays_device(seed, 0, n, rays, tmax=tmax)
        return rays, tmax
    if mix == "surface":
        scene.surface_rays_device(seed, 0, n, rays)
        return rays, None
    half = (n + 1) // 2                      # camera rays, then bounce rays from their hits
    hits = torch.empty((half, 4), dtype=torch.int32, device="cuda")
    pt.camera_rays_device(cam, 960, 600, seed, 0, half, rays)
    scene.query_device(rays, half, hits)
    if n > half:
        scene.bounce_rays_device(rays, hits, n - half, seed + 1, 0, rays[half:])
    torch.cuda.synchronize()
    return rays, None


def _net_inputs(count: int, seed: int):
    """Cache queries (count, 13), positive targets (count, 3) and weights like the network's own initial ones."""
    g = _generator(seed)
    q = torch.zeros((count, 13), device="cuda")
    q[:, 0:3] = torch.rand(count, 3, device="cuda", generator=g) * 10
    q[:, 3:6] = torch.nn.functional.normalize(torch.randn(count, 3, device="cuda", generator=g), dim=1)
    q[:, 6:9] = torch.nn.functional.normalize(torch.randn(count, 3, device="cuda", generator=g), dim=1)
    q[:, 9:12] = 0.2 + 0.6 * torch.rand(count, 3, device="cuda", generator=g)
    q[:, 12] = torch.rand(count, device="cuda", generator=g)
    targets = -torch.log(torch.rand(count, 3, device="cuda", generator=g) * 0.999 + 1e-3)
    return q, targets, _weights(seed)


def _weights(seed: int) -> np.ndarray:
    r = np.random.default_rng(int(seed))
    w = r.uniform(-1, 1, pt.CACHE_WEIGHTS)
    w[:5 * 4096] *= math.sqrt(6 / 128)
    w[5 * 4096:] *= math.sqrt(6 / 67)
    return w.astype(np.float32)


def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    state = dict(case)
    if kind == "query":
        flat, cam = host_scene(case["scene"], 960, 600)
        scene = pt.Scene(flat)
        rays, tmax = _query_rays(case, scene, cam, seed)
        state.update(device=scene, buffer=rays, tmax=tmax, hits=torch.zeros((case["rays"], 4), dtype=torch.int32, device="cuda"),
                     flag=pt.QUERY_ANY if case["mode"] == "any" else pt.QUERY_CLOSEST)
    elif kind in ("host", "compat"):
        flat, cam = host_scene(case["scene"], 960, 600)
        scene = pt.Scene(flat)
        n = case["rays"]
        rays, _ = _query_rays(dict(rays=n, mix="box" if case["scene"] == "cornell" else "camera+bounce", mode="closest"), scene, cam, seed)
        host = np.empty(n, pt.RAY)
        host.view(np.float32).reshape(n, 7)[:] = rays.cpu().numpy()
        state.update(device=scene, buffer=host, flag=pt.QUERY_ANY if case.get("mode") == "any" else pt.QUERY_CLOSEST)
    elif kind == "render":
        flat, cam = host_scene(case["scene"], case["width"], case["height"])
        state.update(camera=cam, renderer=pt.CudaRenderer(flat, cam, case["width"], case["height"], seed, direct_light=case["mis"],
                                                          max_depth=case["depth"]))
    elif kind == "batch":
        names = ["cornell", "spheres10k", "spheres65k", "spheres200k"]
        scenes, jobs, side = [], [], case["side"]
        for k in range(case["jobs"]):
            width, height = side + 61 * k, max(1, side - 13 * k)
            flat, cam = host_scene(names[k % 4], width, height)
            scenes.append(flat)
            jobs.append(dict(scene=k, camera=cam, width=width, height=height, samples=case["samples"] + k % 3,
                             max_depth=4 + 2 * (k % 5), seed=seed + k))
        state["batch"] = pt.Batch(scenes, jobs)
    elif kind == "cached":
        flat, cam = host_scene(case["scene"], case["width"], case["height"])
        renderer = pt.CachedRenderer(flat, cam, case["width"], case["height"], seed=seed, max_depth=case["depth"], train=False,
                                     samples_per_frame=case["spf"])
        renderer.cache().set_weights(_weights(seed))
        state["renderer"] = renderer
    else:
        q, targets, weights = _net_inputs(case["count"], seed)
        net = pt.RadianceCache(*BOX, seed=seed)
        net.set_weights(weights)
        state.update(net=net, queries=q, targets=targets, rgb=torch.zeros((case["count"], 3), device="cuda"))
    torch.cuda.synchronize()
    return state


# ---------------------------------------------------------------- the timed call
def _split(hits: torch.Tensor) -> dict:
    """pt_hit records as (distance, primitive id, primitive type, error)."""
    return dict(t=hits.view(torch.float32)[:, 0], id=hits[:, 1], type=hits[:, 2], error=hits[:, 3])


def run(state: dict):
    kind = state["kind"]
    if kind == "query":
        state["device"].query_device(state["buffer"], state["rays"], state["hits"], mode=state["flag"], tmax=state["tmax"])
        if state["mode"] == "any":           # any-hit answers whether a ray is blocked; which occluder is found is not defined
            return dict(blocked=state["hits"][:, 2] != 0, error=state["hits"][:, 3])
        return _split(state["hits"])
    if kind == "host":
        hits = state["device"].query(state["buffer"], mode=state["flag"])
        if state["mode"] == "any":
            return dict(blocked=hits["primitive_type"] != 0, error=hits["error"])
        return dict(t=hits["t"], id=hits["primitive_id"], type=hits["primitive_type"], error=hits["error"])
    if kind == "compat":
        out = state["device"].query_compat(state["buffer"])
        words = out.view(np.float32).reshape(-1, 14)
        return dict(record=words[:, 0:9], ids=words.view(np.int32)[:, 9:14])
    if kind == "render":
        renderer = state["renderer"]
        renderer.reset(state["camera"])
        renderer.add_samples(state["samples"])
        return dict(sums=renderer.sums(), rays=renderer.rays_traced())
    if kind == "batch":
        batch = state["batch"]
        batch.run()
        return [batch.sums(k) for k in range(state["jobs"])]
    if kind == "cached":
        renderer = state["renderer"]
        renderer.clear()
        renderer.frames(1)
        return renderer.sums()
    if kind == "net-query":
        state["net"].query(state["queries"], state["count"], state["rgb"])
        return state["rgb"]
    loss, gradient = state["net"].gradients(state["queries"], state["targets"], state["count"])
    return dict(loss=loss, gradient=gradient)


# ---------------------------------------------------------------- what a pass cannot do without
def _ray_flops(triangles: int) -> float:
    """A walk straight to its hit: four child boxes per level of a four-wide tree (six subtractions and products and the
    comparisons of a slab test each), then two triangles."""
    return 4 * 18 * max(1.0, math.log(triangles, 4)) + 2 * 45


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind in ("query", "host", "compat"):
        n, tris = case["rays"], TRIANGLES[case["scene"]]
        out = 56 if kind == "compat" else 16
        scene = min(36 * tris, 256 * n)       # a small batch touches only the part of the scene around its rays
        return dict(bytes=n * (28 + out + (4 if case.get("mode") == "any" and kind == "query" else 0)) + scene, flops=n * _ray_flops(tris))
    if kind == "render":
        paths = case["width"] * case["height"] * case["samples"]
        return dict(bytes=case["width"] * case["height"] * 28, flops=paths * 2.5 * (_ray_flops(TRIANGLES[case["scene"]]) + 200))
    if kind == "batch":
        names = ["cornell", "spheres10k", "spheres65k", "spheres200k"]
        total, pixels = 0.0, 0
        for k in range(case["jobs"]):
            px = (case["side"] + 61 * k) * max(1, case["side"] - 13 * k)
            pixels += px
            total += px * (case["samples"] + k % 3) * 2.5 * (_ray_flops(TRIANGLES[names[k % 4]]) + 200)
        return dict(bytes=pixels * 28, flops=total)
    if kind == "cached":
        px = case["width"] * case["height"]
        return dict(bytes=px * 28, flops=px * case["spf"] * 2.5 * (_ray_flops(TRIANGLES[case["scene"]]) + 200))
    n = case["count"]
    if kind == "net-query":
        return dict(bytes=n * 64 + 43008, flops=n * 2.0 * 20672)
    return dict(bytes=n * 64 + 43008 + 82688, flops=n * 6.0 * 20672)


# ---------------------------------------------------------------- the answer in 64 bits
def _exact_closest(flat, rays: torch.Tensor) -> torch.Tensor:
    """Closest distance of each ray over every primitive in float64 (0 for a miss)."""
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a).astype(np.float64)).cuda()  # noqa: E731
    v0, v1, v2 = (d(flat.triangles[k]) for k in ("v0", "v1", "v2"))
    e1, e2 = v1 - v0, v2 - v0
    out = []
    step = max(1, int(2e7) // max(1, len(v0)))
    for part in rays.double().split(step):
        o, dd = part[:, None, 0:3], part[:, None, 3:6]
        p = torch.cross(dd.expand(-1, len(v0), -1), e2[None].expand(len(part), -1, -1), dim=2)
        det = (e1[None] * p).sum(2)
        tv = o - v0[None]
        u = (tv * p).sum(2) / det
        q = torch.cross(tv, e1[None].expand(len(part), -1, -1), dim=2)
        v = (dd * q).sum(2) / det
        t = (e2[None] * q).sum(2) / det
        size = torch.linalg.norm(torch.cross(e1, e2, dim=1), dim=1)
        ok = (det.abs() > 1e-7 * size[None] * torch.linalg.norm(part[:, 3:6], dim=1)[:, None]) & (u >= 0) & (u <= 1) & (v >= 0) & (u + v <= 1) & (t > 1e-3)
        best = torch.where(ok, t, torch.inf).min(dim=1).values
        for sphere in flat.spheres:
            c, r = d(sphere["center"]), float(sphere["radius"])
            oc = part[:, 0:3] - c
            a, b = (part[:, 3:6] ** 2).sum(1), (oc * part[:, 3:6]).sum(1)
            disc = b * b - a * ((oc * oc).sum(1) - r * r)
            root = torch.sqrt(disc.clamp(min=0))
            near, far = (-b - root) / a, (-b + root) / a
            s = torch.where(near > 1e-3, near, far)
            best = torch.minimum(best, torch.where((disc > 0) & (s > 1e-3), s, torch.inf))
        out.append(torch.where(torch.isinf(best), 0.0, best))
    return torch.cat(out)


def _encode64(q: torch.Tensor) -> torch.Tensor:
    """The network's 64 inputs in float64: 6 octaves of sin and cos per axis, 16 spherical harmonics, 7 features."""
    q = q.double()
    p = q[:, 0:3] / 10.0
    freq = []
    for axis in range(3):
        for octave in range(6):
            a = math.pi * (2 ** octave) * p[:, axis]
            freq += [torch.sin(a), torch.cos(a)]
    x, y, z = q[:, 3], q[:, 4], q[:, 5]
    c = lambda v: math.sqrt(v / math.pi)  # noqa: E731
    sh = [torch.full_like(x, 0.5 * c(1)), -0.5 * c(3) * y, 0.5 * c(3) * z, -0.5 * c(3) * x,
          0.5 * c(15) * x * y, -0.5 * c(15) * y * z, 0.25 * c(5) * (3 * z * z - 1), -0.5 * c(15) * x * z, 0.25 * c(15) * (x * x - y * y),
          -0.25 * c(17.5) * y * (3 * x * x - y * y), 0.5 * c(105) * x * y * z, -0.25 * c(10.5) * y * (5 * z * z - 1),
          0.25 * c(7) * z * (5 * z * z - 3), -0.25 * c(10.5) * x * (5 * z * z - 1), 0.25 * c(105) * z * (x * x - y * y),
          -0.25 * c(17.5) * x * (x * x - 3 * y * y)]
    zeros = torch.zeros((len(q), 5), dtype=torch.float64, device=q.device)
    return torch.cat([torch.stack(freq + sh, dim=1), q[:, 6:13], zeros], dim=1)


def _forward64(w: torch.Tensor, q: torch.Tensor) -> torch.Tensor:
    h = _encode64(q)
    for layer in range(5):
        h = torch.relu(h @ w[layer * 4096:(layer + 1) * 4096].view(64, 64))
    return torch.exp(h @ w[5 * 4096:].view(64, 3))


def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind == "query" and case["scene"] == "cornell" and case["mode"] == "closest":
        flat, _ = host_scene("cornell", 960, 600)
        return dict(t=_exact_closest(flat, _box_rays(case["rays"], seed)), id=None, type=None, error=None)
    if kind == "net-query":
        q, _, weights = _net_inputs(case["count"], seed)
        w = torch.from_numpy(weights).cuda().double()
        return torch.cat([_forward64(w, part) for part in q.split(1 << 18)])
    if kind == "net-gradients":
        q, targets, weights = _net_inputs(case["count"], seed)
        w = torch.from_numpy(weights).cuda().double().requires_grad_(True)
        total = 0.0
        for part, want in zip(q.split(1 << 16), targets.split(1 << 16)):
            y = _forward64(w, part)
            loss = ((y - want.double()) ** 2 / (y.detach() ** 2 + 0.01)).sum() / (3 * case["count"])
            loss.backward()
            total += float(loss.detach())
        return dict(loss=total, gradient=w.grad.cpu().numpy())
    return None

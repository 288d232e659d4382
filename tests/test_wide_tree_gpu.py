"""The four-wide collapse on trees where it can go wrong: zero-area boxes, scales that leave the float
range when squared, single-child chains, mixed primitive types, and every size around a node's and a
leaf's capacity.  Answers are compared with the brute-force scan, which uses no boxes."""
from __future__ import annotations

import numpy as np
import pytest

import ptb200 as pt

pytestmark = pytest.mark.gpu


def cloud(triangles: int, spheres: int, scale: float = 1.0, flat: int = 0) -> pt.FlatScene:
    """Random small primitives; `flat` axes are squeezed to a plane (1) or a line (2) of positions."""
    g = np.random.default_rng(100 * triangles + spheres)
    tri = np.zeros(triangles, pt.TRIANGLE)
    c = g.uniform(-1, 1, (triangles, 3))
    if flat:
        c[:, :flat] = 0.25
    for k in ("v0", "v1", "v2"):
        p = c + g.normal(0, 0.15, (triangles, 3))
        if flat:
            p[:, :flat] = 0.25
        tri[k] = p * scale
    sph = np.zeros(spheres, pt.SPHERE)
    sph["center"], sph["radius"] = g.uniform(-1, 1, (spheres, 3)) * scale, g.uniform(0.02, 0.3, spheres) * scale
    mats, tex = np.zeros(1, pt.MATERIAL), np.zeros(1, pt.TEXTURE)
    return pt.FlatScene(tri, sph if spheres else None, None, mats, tex).build_bvh()


def chained(scene: pt.FlatScene, links: int) -> pt.FlatScene:
    """The same scene below `links` branches that store one child twice."""
    head = np.zeros(links, pt.NODE)
    root = scene.nodes[scene.root]
    for k in range(links):
        head[k] = (root["minimum"], root["maximum"], 0, k + 1 if k + 1 < links else links + scene.root, 0, -1)
        head[k]["right"] = head[k]["left"]
    tail = scene.nodes.copy()
    inner = tail["type"] == 0
    tail["left"][inner] += links
    tail["right"][inner] += links
    return pt.FlatScene(scene.triangles, scene.spheres, np.concatenate([head, tail]), scene.materials, scene.textures, None, 0,
                        scene.max_depth + links)


CASES = ([("n%d" % n, lambda n=n: cloud(n, 0)) for n in (1, 2, 3, 4, 5, 8, 9, 16, 17, 33, 65, 300)] +
         [("mixed%d_%d" % (t, s), lambda t=t, s=s: cloud(t, s)) for t, s in ((1, 1), (4, 4), (5, 3), (40, 37), (200, 9))] +
         [("tiny", lambda: cloud(100, 20, 1e-12)), ("huge", lambda: cloud(100, 20, 1e12)),
          ("plane", lambda: cloud(120, 0, 1.0, 1)), ("line", lambda: cloud(120, 0, 1.0, 2)),
          ("chain1", lambda: chained(cloud(50, 10), 1)), ("chain9", lambda: chained(cloud(3, 0), 9))])


@pytest.mark.parametrize("name,make", CASES, ids=[c[0] for c in CASES])
def test_every_primitive_is_reached(name, make):
    import torch
    scene = make()
    nodes, bad = pt.layout_check(scene)
    assert nodes >= 1 and bad == 0
    size = max(float(np.abs(scene.triangles["v0"]).max()), 1e-30)
    g = np.random.default_rng(7)
    n = 4000
    rays = np.zeros(n, pt.RAY)
    rays["origin"] = g.uniform(-2, 2, (n, 3)) * size
    target = scene.triangles["v0"][g.integers(0, len(scene.triangles), n)] * 0.9 + scene.triangles["v1"][g.integers(0, len(scene.triangles), n)] * 0.1
    rays["direction"] = np.where(g.random((n, 1)) < 0.7, (target - rays["origin"]) / size, g.normal(size=(n, 3)))
    d = torch.from_numpy(rays.view(np.uint8).copy()).cuda()
    dev = pt.Scene(scene)
    tmin = 1e-3 * size if name == "tiny" else 1e-3
    got, want = (torch.zeros(n * 16, dtype=torch.uint8, device="cuda") for _ in range(2))
    for mode in (pt.QUERY_CLOSEST, pt.QUERY_ANY):
        dev.query_device(d, n, got, mode=mode, tmin=tmin)
        dev.query_device(d, n, want, mode=mode, tmin=tmin, brute=True)
        torch.cuda.synchronize()
        a, b = got.cpu().numpy().view(pt.HIT), want.cpu().numpy().view(pt.HIT)
        if mode == pt.QUERY_CLOSEST:
            assert a.tobytes() == b.tobytes()
        else:
            assert ((a["primitive_type"] != 0) == (b["primitive_type"] != 0)).all()

"""Queries from pageable memory, which worker threads move through pinned chunks, against the device
query and the one-thread form: the same bytes around the chunk sizes, with every optional array, from
several threads at once."""
from __future__ import annotations

import threading

import numpy as np
import pytest

import ptb200 as pt

pytestmark = pytest.mark.gpu
STAGED = 1 << 19                     # kStagedMin of pt_query.cu


@pytest.fixture(scope="module")
def scene():
    flat, cam = pt.procedural_scene(160, 100, sphere_count=4, segments=40, rings=21, seed=6)
    return flat, cam, pt.Scene(flat)


def device_hits(dev, rays, mode, tmax):
    import torch
    d = torch.from_numpy(rays.view(np.uint8).copy()).cuda()
    t = None if tmax is None else torch.from_numpy(tmax).cuda()
    out = torch.zeros(len(rays) * 16, dtype=torch.uint8, device="cuda")
    dev.query_device(d, len(rays), out, mode=mode, tmax=t)
    torch.cuda.synchronize()
    return out.cpu().numpy().view(pt.HIT)


@pytest.mark.parametrize("count", [STAGED - 1, STAGED, STAGED + 7, 3 * STAGED + 1025])
def test_host_query_equals_device_query(scene, count):
    import torch
    flat, cam, dev = scene
    rays = pt.camera_rays(cam, 160, 100, 3, 0, count)
    tmax = np.random.default_rng(1).uniform(5, 20, count).astype(np.float32)
    want = device_hits(dev, rays, pt.QUERY_CLOSEST, tmax)
    assert dev.query(rays, tmax=tmax).tobytes() == want.tobytes()
    pt.query_walk(0)                 # the single-loop walk's counters do not depend on the split
    try:
        hits, stats = dev.query(rays, tmax=tmax, stats=True)
        assert hits.tobytes() == want.tobytes()
        pinned = torch.empty(count * 28, dtype=torch.uint8, pin_memory=True)
        pinned.numpy()[:] = rays.view(np.uint8)
        out, st = (torch.empty(count * k, dtype=torch.uint8, pin_memory=True) for k in (16, 8))
        pt.check(pt.library().pt_query_rays(dev.handle, pinned.data_ptr(), count, 0, 0.001, tmax.ctypes.data, out.data_ptr(),
                                            st.data_ptr()))
        assert out.numpy().tobytes() == want.tobytes() and st.numpy().tobytes() == stats.tobytes()
    finally:
        pt.query_walk(1)
    blocked = dev.query(rays, mode=pt.QUERY_ANY, tmax=tmax)["primitive_type"] != 0
    assert (blocked == (want["primitive_type"] != 0)).all()


@pytest.mark.parametrize("brute", [False, True])
def test_compat_query_in_parts(scene, brute):
    flat, cam, dev = scene
    rays = pt.camera_rays(cam, 160, 100, 9, 0, 70001)
    if brute:
        rays = rays[:20000]
    whole = dev.query_compat(rays, brute=brute)
    assert whole["hit"].any()
    for n in (1, 31, 32, 33, 8191, 8192, 8193, 16385):
        assert dev.query_compat(rays[:n], brute=brute).tobytes() == whole[:n].tobytes()


def test_threads_on_one_and_two_scenes(scene):
    flat, cam, dev = scene
    other = pt.Scene(flat)
    rays = pt.camera_rays(cam, 160, 100, 5, 0, STAGED + 100)
    want, compat = dev.query(rays).tobytes(), dev.query_compat(rays[:40000]).tobytes()
    wrong = []

    def work(s):
        for _ in range(3):
            if s.query(rays).tobytes() != want or s.query_compat(rays[:40000]).tobytes() != compat:
                wrong.append(s)

    threads = [threading.Thread(target=work, args=(s,)) for s in (dev, other, dev, other)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
    other.close()
    assert dev.query(rays).tobytes() == want

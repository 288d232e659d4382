"""The caller's arrays in the queries on host memory (pt_query_rays, pt_query_rays_compat): whatever memory
they are, the call's answer or error is that of plain copies."""
from __future__ import annotations

import numpy as np
import pytest

import ptb200 as pt

pytestmark = pytest.mark.gpu
STAGED = 1 << 19                     # rays from which pt_query_rays copies through worker threads
RECORD = 56                          # bytes of a pt_trace_result
CUDA_ERROR = 3                       # PT_CUDA_ERROR


@pytest.fixture(scope="module")
def scene():
    flat, cam = pt.procedural_scene(160, 100, sphere_count=4, segments=40, rings=21, seed=6)
    return cam, pt.Scene(flat)


def query(dev, rays, count, hits, tmax=None, stats=None):
    return pt.library().pt_query_rays(dev.handle, rays, count, 0, 0.001, tmax, hits, stats)


def compat(dev, rays, count, results):
    return pt.library().pt_query_rays_compat(dev.handle, rays, count, 0, results)


@pytest.mark.parametrize("count", [1000, STAGED - 1, STAGED])
def test_device_pointers_give_the_copies_error(scene, count):
    """A device pointer in place of any of the arrays is what a copy of the stated direction makes of it: an error,
    or the answer.  It never reaches a host access."""
    import torch
    cam, dev = scene
    rays = pt.camera_rays(cam, 160, 100, 3, 0, count)
    tmax = np.full(count, 50.0, np.float32)
    want, want_stats = dev.query(rays, tmax=tmax, stats=True)
    host = dict(rays=rays, hits=np.zeros(count, pt.HIT), tmax=tmax, stats=np.zeros(count, pt.RAY_STATS))
    for name in host:
        on_device = torch.from_numpy(host[name].view(np.uint8).reshape(-1).copy()).cuda()
        at = {k: on_device.data_ptr() if k == name else v.ctypes.data for k, v in host.items()}
        status = query(dev, at["rays"], count, at["hits"], at["tmax"], at["stats"])
        assert status in (CUDA_ERROR, 0), name
        if status == 0:
            got = on_device.cpu().numpy().view(pt.HIT) if name == "hits" else host["hits"]
            assert got.tobytes() == want.tobytes(), name
    records = np.zeros(count * RECORD, np.uint8)
    full = dev.query_compat(rays).view(np.uint8)
    for device_rays in (True, False):
        on_device = torch.from_numpy((rays.view(np.uint8) if device_rays else records).copy()).cuda()
        status = compat(dev, on_device.data_ptr() if device_rays else rays.ctypes.data, count,
                        records.ctypes.data if device_rays else on_device.data_ptr())
        assert status in (CUDA_ERROR, 0)
        if status == 0:
            assert (records if device_rays else on_device.cpu().numpy()).tobytes() == full.tobytes()
    hits, _ = dev.query(rays, tmax=tmax, stats=True)      # the scene is usable afterwards
    assert hits.tobytes() == want.tobytes()


@pytest.mark.parametrize("count", [777, STAGED, 2 * STAGED])
def test_answers_written_over_the_rays(scene, count):
    """Hits over the rays they answer, and full records over their rays."""
    cam, dev = scene
    rays = pt.camera_rays(cam, 160, 100, 3, 0, count)
    want = dev.query(rays)
    memory = rays.view(np.uint8).copy()
    assert query(dev, memory.ctypes.data, count, memory.ctypes.data) == 0
    assert memory[:count * 16].tobytes() == want.tobytes()
    full = dev.query_compat(rays).view(np.uint8).tobytes()
    memory = np.zeros(count * RECORD, np.uint8)
    memory[:count * 28] = rays.view(np.uint8)
    assert compat(dev, memory.ctypes.data, count, memory.ctypes.data) == 0
    assert memory.tobytes() == full


@pytest.mark.parametrize("count", [1000, 100_003])
def test_full_records_of_rays_still_being_copied(scene, count):
    """Pinned rays that work queued on the default stream is still to write."""
    import torch
    cam, dev = scene
    rays = pt.camera_rays(cam, 160, 100, 3, 0, count)
    want = dev.query_compat(rays).view(np.uint8).tobytes()
    on_device = torch.from_numpy(rays.view(np.uint8).copy()).cuda()
    pinned = torch.zeros(count * 28, dtype=torch.uint8, pin_memory=True)
    results = np.zeros(count * RECORD, np.uint8)
    torch.cuda.synchronize()
    torch.cuda._sleep(40_000_000)                        # about 20 ms
    pinned.copy_(on_device, non_blocking=True)
    assert compat(dev, pinned.data_ptr(), count, results.ctypes.data) == 0
    assert results.tobytes() == want

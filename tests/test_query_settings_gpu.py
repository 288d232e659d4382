"""pt_query_tuning's settings reach the launch at every batch size: the counter form is a memset and a kernel, the
forms without a counter one kernel.  Counted as the nodes of a captured call."""
from __future__ import annotations

import ctypes as C

import pytest

import ptb200 as pt

pytestmark = pytest.mark.gpu


def nodes_of(call) -> int:
    """Graph nodes that `call(stream)` issues (captured, not run)."""
    import torch
    cuda = C.CDLL("libcuda.so.1")
    s = torch.cuda.Stream()
    graph, count = C.c_void_p(), C.c_size_t()
    assert cuda.cuStreamBeginCapture_v2(C.c_void_p(s.cuda_stream), 1) == 0      # thread-local capture
    try:
        call(s.cuda_stream)
    finally:
        assert cuda.cuStreamEndCapture(C.c_void_p(s.cuda_stream), C.byref(graph)) == 0
    assert cuda.cuGraphGetNodes(graph, None, C.byref(count)) == 0
    assert cuda.cuGraphDestroy(graph) == 0
    return count.value


@pytest.mark.parametrize("small", [True, False], ids=["shared-memory scene", "tree"])
def test_refill_and_block_settings_ask_for_the_general_walk(small):
    import torch
    flat, cam = pt.cornell_box(64, 40) if small else pt.procedural_scene(64, 40, sphere_count=2, segments=16, rings=9, seed=2)
    dev, n = pt.Scene(flat), 2560
    rays = torch.empty((n, 7), dtype=torch.float32, device="cuda")
    pt.camera_rays_device(cam, 64, 40, 3, 0, n, rays)
    hits = torch.zeros((n, 4), dtype=torch.int32, device="cuda")

    def call(stream=0):
        dev.query_device(rays, n, hits, stream=stream)

    # (refill, blocks per SM) -> nodes; a block count leaves a tree's small batches without a counter
    want = {(24, 0): 1, (8, 0): 2, (24, 2): 1, (32, 4): 2}
    try:
        answers = []
        for (refill, blocks), nodes in want.items():
            pt.query_tuning(1, refill, blocks)
            call()                                       # loads the kernel
            torch.cuda.synchronize()
            answers.append(hits.clone())
            assert nodes_of(call) == nodes, (refill, blocks)
    finally:
        pt.query_tuning()
    assert all(torch.equal(a, answers[0]) for a in answers)

"""Memory that kernels on a non-blocking stream read is cleared on that stream, or the function that clears it
ends with a device synchronisation: a memset on the default stream is asynchronous to the host, and a
non-blocking stream does not wait for it."""
from __future__ import annotations

import re
import threading
from pathlib import Path

import numpy as np
import pytest

import ptb200 as pt

CSRC = Path(pt.__file__).resolve().parents[1] / "csrc"


@pytest.mark.parametrize("name", ["pt_batch.cu", "pt_cache_render.cu", "pt_query.cu", "pt_render.cu"])
def test_default_stream_memsets_are_waited_for(name):
    text = (CSRC / name).read_text()
    for m in re.finditer(r"cudaMemset\(", text):
        rest = text[m.end():]
        end = re.search(r"\n(?:    )?\}", rest)          # of the enclosing function or member function
        assert "cudaDeviceSynchronize()" in rest[:end.start()], f"{name}: line {text[:m.start()].count(chr(10)) + 1}"


@pytest.mark.gpu
def test_batch_beside_a_busy_default_stream():
    """Batches of the one-kernel form created and run while another thread keeps the default stream busy."""
    import torch
    flat, _ = pt.procedural_scene(64, 40, sphere_count=4, segments=24, rings=13, seed=2, glass_fraction=0.5)
    _, cam = pt.procedural_scene(520, 400, sphere_count=4, segments=24, rings=13, seed=2)
    jobs = [dict(scene=0, camera=cam, width=520, height=400, samples=2, max_depth=5, seed=3)]    # 208,000 pixels

    def render():
        b = pt.Batch([flat], jobs)
        b.run()
        out = b.sums(0).tobytes()
        b.close()
        return out

    want = render()
    assert np.frombuffer(want, np.float32).max() > 0
    stop = threading.Event()

    def busy():
        while not stop.is_set():
            for _ in range(4):
                torch.cuda._sleep(1_000_000)             # about half a millisecond each
            torch.cuda.current_stream().synchronize()

    t = threading.Thread(target=busy)
    t.start()
    try:
        for _ in range(6):
            assert render() == want
    finally:
        stop.set()
        t.join()

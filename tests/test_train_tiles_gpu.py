"""The training kernel around its tile edges (two 128-row tiles per pass, one pass per SM before a second
one): gradients against the FP64 oracle with the bars of test_mlp_gpu.py."""
from __future__ import annotations

import numpy as np
import pytest

import ptb200 as pt
import mlp_oracle as mo
from test_mlp_gpu import HI, LO, queries, target_fn, to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 3, 127, 129, 255, 256, 257, 385, 513, 148 * 256 - 1, 148 * 256 + 130])
def test_gradients_match_oracle_at_tile_edges(n):
    cache = pt.RadianceCache(LO, HI, seed=5)
    q = queries(n, 200 + n)
    t = target_fn(q)
    dq, dt = to_dev(q), to_dev(t)
    loss, g = cache.gradients(dq, dt, n)
    want_loss, want = mo.loss_and_grad(cache.weights(), mo.encode(q, LO, HI), t)
    assert abs(loss - want_loss) <= 2e-2 * abs(want_loss)
    offsets = [0] + [4096 * (l + 1) for l in range(5)] + [pt.CACHE_WEIGHTS]
    for l in range(6):
        a, b = g[offsets[l]:offsets[l + 1]].astype(np.float64), want[offsets[l]:offsets[l + 1]].astype(np.float64)
        cos = float(a @ b / max(1e-30, np.linalg.norm(a) * np.linalg.norm(b)))
        rel = float(np.linalg.norm(a - b) / max(1e-30, np.linalg.norm(b)))
        assert cos > 0.999 and rel < 2e-2, (l, cos, rel)
    again = cache.gradients(dq, dt, n)              # deterministic
    assert again[0] == loss and np.array_equal(again[1], g)


@pytest.mark.parametrize("n", [1, 127, 128, 129, 1024, 1025, 148 * 128, 148 * 128 + 1, 148 * 7 * 128 + 5, 148 * 8 * 128,
                               148 * 8 * 128 * 2 + 77])
def test_forward_at_tile_edges_and_unaligned_queries(n):
    """Whole tiles come by bulk copy, partial tiles and queries off a 16-byte boundary by plain loads: the same bits
    wherever a query lies, nothing written past the last one, and the oracle's values."""
    import torch
    cache = pt.RadianceCache(LO, HI, seed=9)
    q = queries(n, n)
    want = None
    for shift in (0, 1, 4):                        # 52-byte records: shifts of 0, 52 and 208 bytes
        raw = torch.zeros((n + 8) * 52, dtype=torch.uint8, device="cuda")
        raw[shift * 52:(shift + n) * 52] = to_dev(q)
        out = torch.full((n * 3 + 64,), -7.0, dtype=torch.float32, device="cuda")
        cache.query(raw[shift * 52:], n, out)
        cache.sync()
        got = out.cpu().numpy()
        assert (got[3 * n:] == -7.0).all()
        if want is None:
            want = got
            m = min(n, 4096)
            ref = mo.forward(cache.weights(), mo.encode(q[:m], LO, HI))
            assert (np.abs(got[:3 * m].reshape(m, 3) - ref) / np.maximum(np.abs(ref), 1e-6)).max() < 2e-2
        assert got.tobytes() == want.tobytes()

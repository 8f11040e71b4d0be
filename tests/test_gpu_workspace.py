"""Ray queries reuse one device workspace of the context: calls of any size in
any order answer as a first call of that size does, below, at and above the
size that is kept (64 MiB, 48 bytes per ray)."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KEPT = (64 << 20) // 48


def test_ray_queries_of_changing_sizes(srt):
    ctx = srt.Context(0)
    b = srt.SceneBuilder()
    b.add_preset(srt.PRESET_CORNELL_BOX)
    scene = b.build(ctx)
    n = KEPT + 3
    rng = np.random.default_rng(2)
    rays = np.zeros((n, 8), np.float32)
    rays[:, :3] = rng.uniform(-0.5, 0.5, (n, 3))
    rays[:, 3] = 1e-3
    rays[:, 4:7] = rng.normal(size=(n, 3))
    rays[:, 7] = 1e9
    ref = scene.trace(rays[:4096])
    for k in (1, 33, 4096, KEPT, 7, n, 5, KEPT + 1, 0, 4096):
        got = scene.trace(rays[:k])
        assert len(got) == k
        m = min(k, 4096)
        assert np.array_equal(got[:m].view(np.uint32), ref[:m].view(np.uint32))
    scene.close()
    ctx.close()

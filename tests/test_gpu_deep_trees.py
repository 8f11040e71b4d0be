"""Scenes of triangles whose sizes and places fall off geometrically: the cost
recurrence gives them more than 32 levels, opening the largest child does not.
They are built, their trees are complete, and rays go down them."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_collapse import _check

pytestmark = pytest.mark.gpu


def _spiral(n, seed, mode, ratio, size, per):
    g = np.random.default_rng(seed)
    s = ratio ** (np.arange(n) // per).astype(np.float64)
    c = np.zeros((n, 3))
    if mode == 1:
        c[:, 0] = s
    elif mode == 2:
        c = s[:, None] * g.random((n, 3))
        c[:, 0] = s
    p = c[:, None, :] + (s * size)[:, None, None] * (g.random((n, 3, 3)) - 0.5)
    v = np.zeros((3 * n, 8), np.float32)
    v[:, :3] = p.reshape(-1, 3)
    v[:, 6] = 1.0
    return v


@pytest.mark.parametrize("seed,n,mode,width,leaf,ratio,size,per", [
    (235, 422, 1, 8, 1, 0.33982352645143954, 0.25089844111386667, 4),
    (803, 488, 2, 8, 2, 0.53560647035532, 6.85378940567406e-05, 3),
    (1213, 523, 1, 7, 1, 0.7059193191125301, 4.4527511790881236e-05, 2),
    (256, 828, 1, 7, 3, 0.8968175752271239, 0.0016032775145707503, 1),
    (374, 130, 2, 4, 2, 0.4583578467666648, 1.796615402633463e-06, 1),
    (1064, 200, 2, 5, 2, 0.3855702307296464, 0.4273760427914073, 2),
])
def test_deep_scene_is_built(srt, ctx, seed, n, mode, width, leaf, ratio, size, per):
    v = _spiral(n, seed, mode, ratio, size, per)
    b = srt.SceneBuilder()
    m = b.add_material([0.5, 0.5, 0.5, 1], [0, 0, 0, 0])
    b.add_instance(b.add_mesh(v, np.arange(3 * n, dtype=np.uint32)), m, np.eye(4))
    ctx.set_bvh_width(width)
    ctx.set_bvh_leaf_size(leaf)
    try:
        scene = b.build(ctx)
    finally:
        ctx.set_bvh_width(8)
        ctx.set_bvh_leaf_size(2)
    assert scene.info()["depth"] <= 32
    _check(*scene.read_bvh(), n, width, leaf)
    # rays down the whole chain: no stack overflow (the answers are those of sizes below a float's step)
    target = v[:, :3].reshape(n, 3, 3).mean(1)
    rays = np.zeros((n, 8), np.float32)
    rays[:, :3] = target[0] + [0.0, 1.0, 0.0]
    rays[:, 4:7] = target - rays[:, :3]
    rays[:, 7] = 100.0
    assert len(scene.trace(rays)) == n
    scene.close()

"""Pooled triangle tests of the persistent kernels (pool_tris): a stack of
overlapping sheets gives a lane up to 24 pending triangles per node visit (many
rounds of 32 per warp) and hits of one ray on several lanes of a round.  With
more rays than the eight-lane launches take, the frame must equal, bit for bit,
the one whose bounces all run in the tail kernel."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sheets(n):
    g = np.random.default_rng(n)
    v = np.zeros((3 * n, 8), np.float32)
    c = g.uniform(-0.05, 0.05, (n, 1, 3))
    v[:, :3] = (c + 0.3 * np.array([[-1, -1, 0], [1, -1, 0], [0, 1, 0]])).reshape(-1, 3)
    v[:, 6] = 1.0
    return v, np.arange(3 * n, dtype=np.uint32)


def _frame(srt, ctx, n, leaf, tail, w=400, h=300):
    b = srt.SceneBuilder()
    cam = srt.CameraController(*b.add_preset(srt.PRESET_CORNELL_BOX))
    m = b.add_material([0.5, 0.5, 0.5, 1], [0, 0, 0, 0])
    b.add_instance(b.add_mesh(*_sheets(n)), m, np.eye(4))
    ctx.set_bvh_leaf_size(leaf)
    try:
        scene = b.build(ctx)
    finally:
        ctx.set_bvh_leaf_size(2)
    r = srt.Renderer(ctx, scene, w, h, srt.default_params(photons_per_frame=1 << 17, max_depth=5, seed=3))
    r.set_tail(tail)
    r.render(cam.build_uniform(w / h, 0))
    out = r.read_accum(), r.read_photons(), {k: r.stats()[k] for k in ("rays_closest", "rays_shadow", "rays_photon")}
    r.close()
    scene.close()
    return out


@pytest.mark.parametrize("n,leaf", [(1, 1), (24, 3), (257, 3), (1000, 1), (1000, 2)])
def test_stacked_triangles(srt, ctx, n, leaf):
    a, b = _frame(srt, ctx, n, leaf, 0), _frame(srt, ctx, n, leaf, 1)
    assert a[2] == b[2]
    assert np.array_equal(a[0].view(np.uint32), b[0].view(np.uint32))
    assert np.array_equal(a[1].view(np.uint8), b[1].view(np.uint8))

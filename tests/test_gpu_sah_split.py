"""The binned split of one warp per task (k_sah_split) and the partition with
one atomic per warp and child (k_sah_partition): complete trees at counts around
the small-range limit (64), one and several warps and blocks, for primitives
spread in a box, on a line (one axis to bin), in two far clusters (empty bins)
and all on one point (split by position)."""
from __future__ import annotations

import numpy as np
import pytest
from test_gpu_collapse import _check

pytestmark = pytest.mark.gpu


def _triangles(kind, n):
    g = np.random.default_rng(n)
    c = {"box": g.uniform(-1, 1, (n, 3)), "line": np.outer(g.uniform(-1, 1, n), [0.0, 1.0, 0.0]),
         "clusters": g.uniform(-0.01, 0.01, (n, 3)) + np.where(g.random(n) < 0.1, 5.0, -5.0)[:, None],
         "point": np.zeros((n, 3))}[kind]
    v = np.zeros((3 * n, 8), np.float32)
    corner = np.array([[0.02, 0, 0], [-0.01, 0.02, 0], [-0.01, -0.02, 0]])
    v[:, :3] = (c[:, None, :] + corner).reshape(-1, 3)
    v[:, 6] = 1.0
    return v, np.arange(3 * n, dtype=np.uint32)


@pytest.mark.parametrize("kind", ["box", "line", "clusters", "point"])
@pytest.mark.parametrize("n", [2, 3, 4, 5, 31, 33, 63, 64, 65, 66, 129, 257, 1025, 9001])
def test_split_trees_are_complete_and_answer_alike(srt, ctx, kind, n):
    b = srt.SceneBuilder()
    m = b.add_material([0.5, 0.5, 0.5, 1], [0, 0, 0, 0])
    b.add_instance(b.add_mesh(*_triangles(kind, n)), m, np.eye(4))
    g = np.random.default_rng(1)
    rays = np.zeros((2000, 8), np.float32)
    rays[:, :3] = g.uniform(-1.2, 1.2, (2000, 3)) * ([1, 1, 0] if kind != "clusters" else [5, 5, 0]) - [0, 0, 9]
    rays[:, 3], rays[:, 6], rays[:, 7] = 1e-3, 1.0, 1e9
    hits = {}
    for builder in (srt.BVH_SAH, srt.BVH_LBVH):
        ctx.set_bvh_builder(builder)
        try:
            scene = b.build(ctx)
        finally:
            ctx.set_bvh_builder(srt.BVH_SAH)
        nodes, tris = scene.read_bvh()
        _check(nodes, tris, n, 8, 2)
        hits[builder] = scene.trace(rays)
        scene.close()
    assert np.array_equal(hits[srt.BVH_SAH].view(np.uint32), hits[srt.BVH_LBVH].view(np.uint32))

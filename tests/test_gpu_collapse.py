"""The wide tree that the cost recurrence picks (collapse_costs, k_collapse),
decoded on the host: every triangle lies in exactly one leaf, every node is
reached exactly once, no node has more than `width` children or leaves of more
than `leaf` triangles, and a child's quantised box holds the triangles below it;
for every width and leaf size, both builders, and triangle counts around the
smallest trees."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(nodes, tris, n_tris, width, leaf):
    w = nodes  # [n, 20] uint32
    by = np.ascontiguousarray(w).view(np.uint8).reshape(len(w), 80)
    seen_tri, seen_node = np.zeros(n_tris, int), np.zeros(len(w), int)
    lo, hi = tris[:, [0, 1, 2]].copy(), tris[:, [0, 1, 2]].copy()
    for k in (4, 8):
        lo, hi = np.minimum(lo, tris[:, k:k + 3]), np.maximum(hi, tris[:, k:k + 3])

    def walk(i):
        seen_node[i] += 1
        p = w[i, :3].view(np.float32).astype(np.float64)
        scale = 2.0 ** (by[i, 12:15].astype(int) - 127)
        imask, base, tbase, meta = int(by[i, 15]), int(w[i, 4]), int(w[i, 5]), by[i, 24:32]
        assert np.count_nonzero(meta) <= width
        nlo, nhi, rank = np.full(3, np.inf), np.full(3, -np.inf), 0
        for s in range(8):
            if meta[s] == 0:
                continue
            if (imask >> s) & 1:
                clo, chi = walk(base + rank)
                rank += 1
            else:
                c, o = int(meta[s]) >> 5, int(meta[s]) & 31
                assert 1 <= c <= leaf
                r = slice(tbase + o, tbase + o + c)
                seen_tri[r] += 1
                clo, chi = lo[r].min(0), hi[r].max(0)
            qlo = p + scale * np.array([by[i, 32 + 8 * a + s] for a in range(3)])
            qhi = p + scale * np.array([by[i, 56 + 8 * a + s] for a in range(3)])
            assert np.all(qlo <= clo) and np.all(qhi >= chi)
            nlo, nhi = np.minimum(nlo, clo), np.maximum(nhi, chi)
        return nlo, nhi

    walk(0)
    assert np.all(seen_tri == 1) and np.all(seen_node == 1)
    ids = np.sort(tris[:, 3].view(np.uint32))
    np.testing.assert_array_equal(ids, np.arange(n_tris))


def _soup(n, seed):
    g = np.random.default_rng(seed)
    v = np.zeros((3 * n, 8), np.float32)
    v[:, :3] = (g.uniform(-1, 1, (n, 1, 3)) + g.normal(0, 0.05, (n, 3, 3))).reshape(-1, 3)
    v[:, 6] = 1.0
    return v, np.arange(3 * n, dtype=np.uint32)


@pytest.mark.parametrize("builder", [0, 1])
@pytest.mark.parametrize("width,leaf", [(8, 2), (8, 1), (8, 3), (5, 2), (3, 3), (2, 1), (2, 3)])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 9, 17, 700])
def test_collapsed_tree_is_complete(srt, ctx, builder, width, leaf, n):
    b = srt.SceneBuilder()
    m = b.add_material([0.5, 0.5, 0.5, 1], [0, 0, 0, 0])
    b.add_instance(b.add_mesh(*_soup(n, n)), m, np.eye(4))
    ctx.set_bvh_builder(builder)
    ctx.set_bvh_width(width)
    ctx.set_bvh_leaf_size(leaf)
    try:
        scene = b.build(ctx)
    finally:
        ctx.set_bvh_builder(srt.BVH_SAH)
        ctx.set_bvh_width(8)
        ctx.set_bvh_leaf_size(2)
    nodes, tris = scene.read_bvh()
    _check(nodes, tris, n, width, leaf)
    scene.close()

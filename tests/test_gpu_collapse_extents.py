"""Tree builds over triangles of extreme size: with one triangle far larger than
the rest the tree is complete and rays answer alike with both builders; an
infinite corner is refused and the context stays usable; a triangle with NaN
corners is never hit and changes no other answer; corners near the largest
float end in a tree or an error."""
from __future__ import annotations

import numpy as np
import pytest
from conftest import random_rays
from test_gpu_collapse import _check, _soup

pytestmark = pytest.mark.gpu

N = 700


def _build(srt, ctx, v, builder):
    b = srt.SceneBuilder()
    m = b.add_material([0.5, 0.5, 0.5, 1], [0, 0, 0, 0])
    b.add_instance(b.add_mesh(v, np.arange(len(v), dtype=np.uint32)), m, np.eye(4))
    ctx.set_bvh_builder(builder)
    try:
        return b.build(ctx)
    finally:
        ctx.set_bvh_builder(srt.BVH_SAH)


def _with_last(corners):
    v, _ = _soup(N, 5)
    v[-3:, :3] = corners
    return v


def _rays():
    return random_rays(4096, np.random.default_rng(3))


@pytest.mark.parametrize("extent", [1e18, 1e19, 1e20])
def test_one_huge_triangle(srt, ctx, extent):
    v = _with_last([[-extent, -extent, 2.0], [extent, -extent, 2.0], [0.0, extent, 2.0]])
    got = []
    for builder in (srt.BVH_SAH, srt.BVH_LBVH):
        scene = _build(srt, ctx, v, builder)
        _check(*scene.read_bvh(), N, 8, 2)
        got.append(scene.trace(_rays()))
        scene.close()
    assert np.array_equal(got[0].view(np.uint32), got[1].view(np.uint32))
    if extent < 1e19:  # (beyond it the edge functions overflow: no builder finds the triangle)
        assert np.count_nonzero(got[0]["prim"] == N - 1) > 100


@pytest.mark.parametrize("builder", [0, 1])
@pytest.mark.parametrize("corners", [[[np.inf, 0, 0], [1, 0, 0], [0, 1, 0]],
                                     [[0, -np.inf, 0], [0, np.inf, 0], [1, 0, 0]]])
def test_an_infinite_corner_is_refused(srt, ctx, builder, corners):
    with pytest.raises(srt.SrtError) as e:
        _build(srt, ctx, _with_last(corners), builder)
    assert e.value.status == 3  # SRT_ERR_CUDA
    _build(srt, ctx, _soup(N, 5)[0], builder).close()


@pytest.mark.parametrize("builder", [0, 1])
@pytest.mark.parametrize("corners", [[[np.nan, 0, 0], [0.1, 0, 0], [0, 0.1, 0]], [[np.nan] * 3] * 3,
                                     [[-np.inf] * 3, [np.inf] * 3, [0, 0, 0]]])  # 0 x inf: NaN in world space
def test_a_nan_triangle_is_never_hit(srt, ctx, builder, corners):
    ref = _build(srt, ctx, _soup(N, 5)[0][:-3], builder)
    scene = _build(srt, ctx, _with_last(corners), builder)
    a, b = ref.trace(_rays()), scene.trace(_rays())
    assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
    ref.close()
    scene.close()


@pytest.mark.parametrize("corner", [-3.36e38, -3.39e38, -3.4e38, -3.402e38, 3.402e38])
def test_corners_near_the_largest_float_end(srt, ctx, corner):
    try:
        _build(srt, ctx, _with_last([[corner, 0, 0], [0, 1, 0], [1, 0, 1]]), srt.BVH_SAH).close()
    except srt.SrtError as e:
        assert e.status == 3
    _build(srt, ctx, _soup(N, 5)[0], srt.BVH_SAH).close()

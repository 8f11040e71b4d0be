"""The radix sort by itself (srt_test_sort): stable over whole tiles of 4096, at
their edges and at more tiles than two look-back windows of 5, up to the
largest photon grid; and where its tile numbers were drawn by another launch it
reports that and writes nothing past its arrays.  What sorts reports a sort that
gave up instead of using its result."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TILE = 4096


def _pairs(n, bits):
    g = np.random.default_rng(n + bits)
    return g.integers(0, 1 << bits, n, dtype=np.uint32), np.arange(n, dtype=np.uint32)


@pytest.mark.parametrize("n", [1, TILE - 1, TILE, TILE + 1, 5 * TILE, 5 * TILE + 1, 10 * TILE + 1, 1 << 20])
@pytest.mark.parametrize("bits", [5, 23, 32])
def test_sort_is_stable(srt, ctx, n, bits):
    keys, vals = _pairs(n, bits)
    k, v = srt.sort_check(ctx, keys, vals, bits)
    order = np.argsort(keys, kind="stable")
    np.testing.assert_array_equal(k, keys[order])
    np.testing.assert_array_equal(v, vals[order])


@pytest.mark.parametrize("n,first", [(TILE, 1), (5 * TILE, 1), (5 * TILE, 3), (5 * TILE, 5), (10 * TILE + 1, 4),
                                     (10 * TILE + 1, 11), (10 * TILE + 1, 245), (TILE, 0x7FFFFFFF)])
def test_tile_numbers_of_another_launch(srt, ctx, n, first):
    keys, vals = _pairs(n, 23)
    with pytest.raises(srt.SrtError) as e:
        srt.sort_check(ctx, keys, vals, 23, first)
    assert e.value.status == 4  # SRT_ERR_TIMEOUT
    k, _ = srt.sort_check(ctx, keys, vals, 23)
    np.testing.assert_array_equal(k, np.sort(keys))


def test_lbvh_build_reports_a_sort_that_gave_up(srt, ctx, monkeypatch):
    b = srt.SceneBuilder()
    b.add_preset(srt.PRESET_CORNELL_BOX)
    ctx.set_bvh_builder(srt.BVH_LBVH)
    try:
        scene = b.build(ctx)
        monkeypatch.setenv("SRT_FAULT", "sort")
        for build in (lambda: b.build(ctx), lambda: scene.rebuild_bvh(8)):
            with pytest.raises(srt.SrtError) as e:
                build()
            assert e.value.status == 4  # SRT_ERR_TIMEOUT
        monkeypatch.delenv("SRT_FAULT")
        scene.rebuild_bvh(8)
        b.build(ctx).close()
        scene.close()
    finally:
        ctx.set_bvh_builder(srt.BVH_SAH)


def _frames(srt, ctx, scene, cam, w, h, flags, n=2):
    r = srt.Renderer(ctx, scene, w, h, srt.default_params(max_depth=6, photons_per_frame=1 << 14, flags=flags))
    try:
        for f in range(n):
            r.render(cam.build_uniform(w / h, f))
        return r.read_accum()
    finally:
        r.close()


@pytest.mark.parametrize("size", [(63, 65), (64, 64), (17, 241), (8193, 1)])  # 4095, 4096, 4097, 8193 paths
def test_ray_sort_changes_no_image(srt, ctx, size):
    b = srt.SceneBuilder()
    cam = srt.CameraController(*b.add_preset(srt.PRESET_CORNELL_BOX))
    scene = b.build(ctx)
    plain = _frames(srt, ctx, scene, cam, *size, 0)
    assert np.array_equal(_frames(srt, ctx, scene, cam, *size, srt.FLAG_RAY_SORT), plain)
    scene.close()


def test_frame_reports_a_ray_sort_that_gave_up(srt, ctx, monkeypatch):
    b = srt.SceneBuilder()
    cam = srt.CameraController(*b.add_preset(srt.PRESET_CORNELL_BOX))
    scene = b.build(ctx)
    plain = _frames(srt, ctx, scene, cam, 64, 48, 0)
    monkeypatch.setenv("SRT_FAULT", "sort")
    with pytest.raises(srt.SrtError) as e:
        _frames(srt, ctx, scene, cam, 64, 48, srt.FLAG_RAY_SORT)
    assert e.value.status == 4  # SRT_ERR_TIMEOUT
    monkeypatch.delenv("SRT_FAULT")
    assert np.array_equal(_frames(srt, ctx, scene, cam, 64, 48, srt.FLAG_RAY_SORT), plain)
    scene.close()

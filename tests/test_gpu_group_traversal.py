"""One ray on eight lanes (group_step): launches of few rays and the tail
kernel.  A ray's answer does not depend on the tree or on how it was traced,
so frames are compared bit for bit between trees (8 and 2 children per node:
the 16- and the 32-entry stack; single-triangle leaves) and between the
bounce-by-bounce frame and the tail, at ray counts from one to above the
switch to one ray per lane (2 rays per resident group of 8 lanes)."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _frame(srt, ctx, preset, w, h, tail, width=8, leaf=2):
    b = srt.SceneBuilder()
    cam = srt.CameraController(*b.add_preset(preset))
    ctx.set_bvh_width(width)
    ctx.set_bvh_leaf_size(leaf)
    try:
        scene = b.build(ctx)
    finally:
        ctx.set_bvh_width(8)
        ctx.set_bvh_leaf_size(2)
    r = srt.Renderer(ctx, scene, w, h, srt.default_params(photons_per_frame=1 << 14, max_depth=10, seed=5))
    r.set_tail(tail)
    for f in range(2):
        r.render(cam.build_uniform(w / h, f))
    out = r.read_accum(), r.read_photons(), {k: r.stats()[k] for k in ("rays_closest", "rays_shadow", "rays_photon")}
    r.close()
    scene.close()
    return out


@pytest.mark.parametrize("w,h", [(1, 1), (3, 3), (33, 1), (97, 61), (330, 260)])
@pytest.mark.parametrize("preset", [0, 3])
def test_frames_do_not_depend_on_the_tree_or_the_tail(srt, ctx, preset, w, h):
    ref = _frame(srt, ctx, preset, w, h, 0)
    for kw in ({"tail": 1}, {"tail": 4}, {"tail": 0, "width": 2, "leaf": 1}, {"tail": 1, "width": 2, "leaf": 3}):
        got = _frame(srt, ctx, preset, w, h, **kw)
        np.testing.assert_array_equal(got[0], ref[0], err_msg=str(kw))
        np.testing.assert_array_equal(got[1], ref[1], err_msg=str(kw))
        assert got[2] == ref[2], kw

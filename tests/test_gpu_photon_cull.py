"""The emission cull (k_photon_emit): emitted rays that meet no leaf box with a
scattering triangle are answered without a closest hit.  What is stored must
not depend on the tree the cull walks: the photons of a frame are compared,
bit for bit, between the default tree, a binary tree (deeper than the small
traversal stack for the larger scenes) and an LBVH with single-triangle
leaves."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

W, H, N = 40, 24, 40_001  # an odd photon count: the last emission block is partial


def _photons(srt, ctx, preset, seed, rebuild=None):
    b = srt.SceneBuilder()
    cam = srt.CameraController(*b.add_preset(preset, seed))
    scene = b.build(ctx)
    r = srt.Renderer(ctx, scene, W, H, srt.default_params(photons_per_frame=N, max_depth=4, seed=3))
    r.render(cam.build_uniform(W / H, 0))
    if rebuild:
        scene.rebuild_bvh(rebuild)
        r.render(cam.build_uniform(W / H, 0))  # the same frame again on the new tree
    ph, st, depth = r.read_photons(), r.stats(), scene.info()["depth"]
    r.close()
    scene.close()
    return ph, st, depth


# every material kind; all surfaces diffuse (indirect room: nothing is stored); many scattering instances
@pytest.mark.parametrize("preset,seed", [(0, 0), (1, 0), (2, 0), (3, 0), (4, 0), (5, 0), (6, 2)])
def test_stored_photons_do_not_depend_on_the_culling_tree(srt, ctx, preset, seed):
    ref, st, _ = _photons(srt, ctx, preset, seed)
    assert st["rays_photon"] >= N  # every emitted ray counts, culled or traced
    if preset == 5:
        assert len(ref) == 0 and st["rays_photon"] == N
    else:
        assert len(ref) > 0
    got, _, depth = _photons(srt, ctx, preset, seed, rebuild=2)
    np.testing.assert_array_equal(got, ref)
    if preset == 3:
        assert depth > 16  # the 32-entry stack
    try:
        ctx.set_bvh_builder(srt.BVH_LBVH)
        ctx.set_bvh_leaf_size(1)
        got, _, _ = _photons(srt, ctx, preset, seed)
    finally:
        ctx.set_bvh_builder(srt.BVH_SAH)
        ctx.set_bvh_leaf_size(2)
    np.testing.assert_array_equal(got, ref)

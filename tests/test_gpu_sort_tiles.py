"""The radix sort (k_rs_pass) and the photon deposit (k_deposit) at the edges of
their tiles (4096 pairs; 8192 emitters) and over several look-back windows (16
and 32 tiles): the grid's keys and ranges against the CPU oracle, bit for bit,
and the stored photons of N emitters as the first of those of more emitters (a
photon depends on its emitter's id and the frame alone, and photons are stored
in emitter order)."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 31, 33, 255, 4095, 4096, 4097, 8192, 12289, 65537, 16 * 4096, 16 * 4096 + 1, 200_001])
@pytest.mark.parametrize("spread,bits", [(0.01, 22), (0.7, 22), (0.3, 26), (0.3, 4)])
def test_grid_keys_at_tile_edges(srt, orc, ctx, n, spread, bits):
    g = np.random.default_rng(n + bits)
    ph = np.zeros((n, 8), np.float32)
    ph[:, :3] = g.normal(0.0, spread, (n, 3))
    ph[:, 3] = 550.0
    ph[:, 4] = 1.0
    ph[:, 7] = np.where(g.random(n) < 0.02, 0.0, 1.0)  # some in the sentinel bucket
    keys, ranges = srt.photon_grid_build(ctx, ph, 5, 0.02, bits)
    o_keys, o_ranges = orc.photon_grid_build(ph, 5, 0.02, bits)
    np.testing.assert_array_equal(keys, o_keys)
    np.testing.assert_array_equal(ranges, o_ranges.reshape(ranges.shape))


def test_deposit_at_tile_edges(srt, ctx):
    b = srt.SceneBuilder()
    cam = srt.CameraController(*b.add_preset(srt.PRESET_CAUSTIC_SLAB))
    scene = b.build(ctx)

    def photons(n):
        r = srt.Renderer(ctx, scene, 24, 16, srt.default_params(photons_per_frame=n, max_depth=3))
        for f in (3, 4):  # the second map is built ahead, on the other set
            r.render(cam.build_uniform(1.5, f))
        out, stored = r.read_photons(), r.stats()["photons_stored"]
        r.close()
        return out, stored

    ref, _ = photons(600_000)
    assert len(ref) > 100_000
    last = 0
    for n in (1, 15, 17, 8191, 8192, 8193, 33 * 8192 - 1, 33 * 8192 + 1, 500_000):
        got, stored = photons(n)
        assert last <= len(got) <= n and stored >= len(got)
        np.testing.assert_array_equal(got, ref[: len(got)])
        last = len(got)
    scene.close()

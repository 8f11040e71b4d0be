"""Light samples read a per-light frame (unit normal, area) and the path's
radiance at the first light's temperature (path_blackbody): lights of
different temperatures, the first one's and another emitter seen directly, and
a light that moves, against the CPU oracle.  Tolerances as the frame tests of
test_gpu_parity.py: pixels within 1e-3 relative except where a path took
another branch (a draw within rounding of its threshold), at least 97 %."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

W, H, N = 48, 32, 1 << 14


def _t(x, y, z, sx, sy, sz, flip=False):
    m = np.diag([sx, sy, sz, 1.0])
    if flip:  # half a turn about x: facing down
        m[1, 1], m[2, 2] = -sy, -sz
    m[:3, 3] = x, y, z
    return m


def _scene(srt, temps, first_x):
    b = srt.SceneBuilder()
    white = b.add_material([0.7, 0.7, 0.7, 1], [0, 0, 0, 0])
    red = b.add_material([0.65, 0.05, 0.05, 1], [0, 0, 0, 0])
    metal = b.add_material([0.9, 0.8, 0.7, 1], [1, 0.2, 0, 0])
    emit = [b.add_material([t, 2.0, 0, 1], [3, 0, 0, 0]) for t in temps]
    plane = b.add_mesh(*srt.geometry("plane"))
    cube = b.add_mesh(*srt.geometry("cube"))
    for k, t in enumerate(temps):
        b.add_light_instance(plane, emit[k], _t(first_x if k == 0 else 0.5, 0.9, -0.2 * k, 0.4, 1, 0.4, True),
                             [0.0, t, 2.0, 0.0])
    b.add_instance(plane, white, _t(0, -1, 0, 3, 1, 3))
    b.add_instance(cube, red, _t(-0.4, -0.6, -0.2, 0.5, 0.8, 0.5))
    b.add_instance(cube, metal, _t(0.4, -0.7, 0.1, 0.5, 0.5, 0.5))
    return b


@pytest.mark.parametrize("temps", [(6500.0,), (3000.0, 6500.0), (6500.0, 6500.0, 2500.0)])
@pytest.mark.parametrize("tail", [0, 1])
def test_lights_of_several_temperatures_match_the_oracle(srt, orc, ctx, temps, tail):
    b = _scene(srt, temps, -0.5)
    scene = b.build(ctx)
    # the first light moves to the place of a fresh scene's
    moved = _scene(srt, temps, -0.2)
    scene.update_instances([0], _t(-0.2, 0.9, 0.0, 0.4, 1, 0.4, True).T.reshape(1, 16))
    o = orc.OracleScene(moved.arrays())
    p = srt.default_params(photons_per_frame=N, max_depth=6)
    r = srt.Renderer(ctx, scene, W, H, p)
    r.set_tail(tail)
    u = srt.camera_uniform([0.0, 0.0, 3.0], -np.pi / 2, 0.0, W / H, 0)
    r.render(u)
    g = r.read_accum()[..., :3]
    ref, _, _, counts = o.render_frame(u, W, H, p)
    ref = ref[..., :3]
    # light samples behind the surface are not traced, but counted: the oracle traces them
    assert abs(r.stats()["rays_shadow"] - int(counts[2])) <= 0.01 * int(counts[2])
    ok = (np.abs(g - ref) <= 1e-3 * np.maximum(np.abs(ref), 1e-3)).all(-1)
    assert ref.mean() > 0 and ok.mean() >= 0.97, ok.mean()
    r.close()
    scene.close()
    o.close()

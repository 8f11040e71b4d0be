"""Ray queries from two threads on one context: only one call at a time holds
the context's workspace, the other brings its own, and each answers as it does
alone, whatever sizes meet."""
from __future__ import annotations

import threading

import numpy as np
import pytest
from conftest import random_rays

pytestmark = pytest.mark.gpu


def test_ray_queries_from_two_threads(srt):
    ctx = srt.Context(0)
    b = srt.SceneBuilder()
    b.add_preset(srt.PRESET_CORNELL_BOX)
    scene = b.build(ctx)
    rays = [random_rays(50_000, np.random.default_rng(k)) for k in range(2)]
    ref = [scene.trace(r) for r in rays]
    bad: list = []

    def work(k, sizes):
        try:
            for i, n in enumerate(sizes):
                any_hit = i % 3 == 2
                got = scene.trace(rays[k][:n], any_hit=any_hit)
                if any_hit:
                    same = np.array_equal(got["prim"] == 0xFFFFFFFF, ref[k][:n]["prim"] == 0xFFFFFFFF)
                else:
                    same = np.array_equal(got.view(np.uint32), ref[k][:n].view(np.uint32))
                if not same:
                    bad.append((k, i, n))
        except Exception as e:  # (an exception in a thread would be lost)
            bad.append((k, repr(e)))

    sizes = [int(x) for x in np.random.default_rng(7).integers(1, 50_000, 120)]
    threads = [threading.Thread(target=work, args=(k, sizes[::-1] if k else sizes)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
    scene.close()
    ctx.close()

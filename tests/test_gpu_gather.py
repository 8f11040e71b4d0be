"""The photon gather (gather, gather_range) against a restatement of
shader.wgsl:297-342 in float32, every operation rounded on its own in the
shader's order, over the general form (four weights for every photon within
the radius): the sums agree bit for bit, also where the kernel leaves photons
out because they would add zeros, and where it must not (a non-finite energy, a
radius that is not positive)."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

F = np.float32


def _reference(keys, photons, queries, cap, r0, sr, norm):
    """frame 0: the radius is r0.  keys: sorted (hash << 32 | index)."""
    out = np.zeros((len(queries), 4), F)
    h, idx = (keys >> np.uint64(32)).astype(np.uint32), (keys & np.uint64(0xFFFFFFFF)).astype(np.int64)
    r, sr = F(r0), F(sr)
    r2 = F(r * r)
    with np.errstate(all="ignore"):
        density = F(F(F(3.0) / F(F(3.14159265359) * r2)) * F(F(1.0) / sr)) * F(F(1.0) / F(norm))
        for q, (qh, row) in enumerate(queries):
            lo, hi = np.searchsorted(h, qh, "left"), np.searchsorted(h, qh, "right")
            total = np.zeros(4, F)
            for i in range(hi - 1, max(lo, hi - cap) - 1, -1):
                p = photons[idx[i]]
                dd = (row[:3] - p[:3]).astype(F)
                d2 = F(F(F(dd[0] * dd[0]) + F(dd[1] * dd[1])) + F(dd[2] * dd[2]))
                nd = F(F(F(row[3] * p[4]) + F(row[4] * p[5])) + F(row[5] * p[6]))
                if not (d2 < r2 and nd > 0):
                    continue
                e = F(p[7] * F(F(1.0) - F(F(np.sqrt(d2)) / r)))
                w = (F(1.0) - (np.abs(row[6:10] - p[3]).astype(F) / sr).astype(F)).astype(F)
                w = np.where(w > 0, w, F(0.0))  # NaN -> 0, as fmaxf
                total = (total + (w * e).astype(F)).astype(F)
            out[q] = (total * density).astype(F)
    return out


@pytest.mark.parametrize("cap", [0, 1, 31, 32, 33, 64, 500])
@pytest.mark.parametrize("sr,energy", [(20.0, "finite"), (150.0, "finite"), (20.0, "inf"), (20.0, "nan"),
                                       (-3.0, "finite"), (float("inf"), "finite")])
def test_gather_matches_the_general_form_bit_for_bit(srt, ctx, cap, sr, energy):
    g = np.random.default_rng(7)
    n, nq = 3000, 60
    ph = np.zeros((n, 8), F)
    ph[:, :3] = g.normal(0.0, 0.02, (n, 3))  # crowded cells
    ph[:, 3] = g.uniform(380.0, 780.0, n)
    ph[:, 4:7] = g.normal(size=(n, 3))
    ph[:, 7] = g.uniform(0.1, 1.0, n)
    ph[5::97, 7] = 0.0  # not in the grid
    if energy != "finite":
        ph[:: 400, 7] = np.inf if energy == "inf" else np.nan
    q = np.zeros((nq, 10), F)
    q[:, :3] = ph[g.integers(0, n, nq), :3] + g.normal(0.0, 0.002, (nq, 3))
    q[:, 3:6] = g.normal(size=(nq, 3))
    hero = g.uniform(380.0, 780.0, nq)
    q[:, 6:10] = 380.0 + np.mod(hero[:, None] - 380.0 + 100.0 * np.arange(4), 400.0)
    keys, _ = srt.photon_grid_build(ctx, ph, 0)
    # the queries' buckets: keys of photons placed at the query points
    at = np.zeros((nq, 8), F)
    at[:, :3], at[:, 7] = q[:, :3], 1.0
    qk, _ = srt.photon_grid_build(ctx, at, 0)
    bucket = np.zeros(nq, np.uint32)
    bucket[(qk & np.uint64(0xFFFFFFFF)).astype(np.int64)] = (qk >> np.uint64(32)).astype(np.uint32)
    p = srt.default_params(gather_cap=cap, spectral_radius=sr, photons_per_frame=n)
    got = srt.photon_gather(ctx, ph, q, 0, p)
    ref = _reference(keys, ph, list(zip(bucket, q)), cap, 0.02, sr, n)
    if cap > 0 and energy == "finite" and np.isfinite(sr):  # (an infinite radius has a density of zero)
        assert np.count_nonzero(ref) > 0
    np.testing.assert_array_equal(got, ref)

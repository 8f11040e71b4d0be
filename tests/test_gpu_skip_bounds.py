"""What shading may leave out because it adds zeros: only where every component
of the factor is a number below the bound, so that a NaN or an infinity in one
of the four wavelengths reaches the image."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bound", [1e15, np.inf])
def test_every_component_counts(srt, ctx, bound):
    odd = np.array([0.0, -0.0, 0.25, -0.25, 1e14, 1e15, -1e15, 3e38, -3e38, np.inf, -np.inf, np.nan], np.float32)
    rows = []
    for k in range(4):
        for x in odd:
            f = np.array([0.5, 0.0, 1.0, 0.25], np.float32)
            f[k] = x
            rows.append([*f, bound])
    rows.append([np.nan] * 4 + [bound])
    rows = np.array(rows, np.float32)
    with np.errstate(invalid="ignore"):
        want = np.all(np.abs(rows[:, :4]) < np.float32(bound), axis=1)
    got = srt.device_math(ctx, 9, rows)[:, 0]
    np.testing.assert_array_equal(got, want.astype(np.uint32))

"""The allocation-free photon grid at the edges of its sort's tiles (4096
photons), at more tiles than one and two look-back windows (5 tiles), up to its
largest set, and for small sets right after it (leftover scratch words would
show): the keys and ranges of the CPU oracle."""
from __future__ import annotations

import numpy as np
import pytest
from test_zz_no_alloc import _call, _photons

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [4, 22, 26])
def test_tile_edges_in_a_row(srt, orc, bits):
    torch = pytest.importorskip("torch")
    stream = torch.cuda.current_stream().cuda_stream
    d_ranges = torch.full((1 << bits, 2), 0x7FFFFFFF, dtype=torch.int32, device="cuda")
    for n in (1, 4095, 4096, 4097, 5 * 4096, 5 * 4096 + 1, 10 * 4096 + 1, 1 << 20, 33, 4097, (1 << 20) - 1, 2):
        ph = _photons(n, n + bits, 0.4)
        d_ph = torch.from_numpy(ph).cuda()
        d_keys = torch.zeros(n, dtype=torch.int64, device="cuda")
        assert _call(srt.lib(), stream, d_ph, n, 3, bits, d_keys, d_ranges) == 0
        torch.cuda.synchronize()
        o_keys, o_ranges = orc.photon_grid_build(ph, 3, 0.02, bits)
        assert np.array_equal(d_keys.cpu().numpy().view(np.uint64), o_keys)
        ranges = d_ranges.cpu().numpy().view(np.uint32)
        assert np.array_equal(ranges, o_ranges.reshape(ranges.shape))

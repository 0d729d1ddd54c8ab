"""8-connected vertical whole-image sweeps, which run in segments of 128 rows:
heights at and around the segment edges, paths that cross many of them
(straight, diagonal, along a strip's edge), against the restatement."""
import numpy as np
import pytest

import iwpp
import oracle

pytestmark = pytest.mark.gpu
NP = {0: np.uint8, 1: np.uint16, 2: np.int32}
TW = {0: 128, 1: 64, 2: 32}


def _dev(a):
    import torch
    return torch.from_numpy(a.view(np.int16) if a.dtype == np.uint16 else a.copy()).cuda()


@pytest.mark.parametrize("dt", [0, 1, 2])
@pytest.mark.parametrize("h", [1, 7, 64, 127, 128, 129, 136, 257, 641, 1100])
def test_tall_8_connected_sweeps(dt, h):
    rng = np.random.default_rng(h * 10 + dt)
    info = np.iinfo(NP[dt])
    levels = np.linspace(info.min, info.max, 9).astype(np.int64)
    for w in (1, 5, TW[dt], 2 * TW[dt] + 3):
        mask = levels[rng.integers(0, 8, (h, w))].astype(NP[dt])
        y = np.arange(h)
        mask[:, w // 2] = info.max                      # a straight path
        mask[y, np.minimum(y % (2 * w), w - 1)] = info.max  # diagonals, then along the edge
        mask[y, np.maximum(w - 1 - y, 0)] = levels[7]
        marker = np.full((h, w), info.min, NP[dt])
        at = rng.random((h, w)) < 0.01
        marker[at] = mask[at]
        marker[0], marker[-1] = mask[0], mask[-1]
        for d in (1, 3):
            tm, tk = _dev(marker), _dev(mask)
            iwpp.sweep(tm, tk, d, 8)
            got = tm.cpu().numpy().view(NP[dt])
            assert np.array_equal(got, oracle.sweep(marker, mask, d, 8)), (w, d)

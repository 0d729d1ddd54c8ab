"""Vertical whole-image sweeps by strips (8-connected, and 4-connected of rows off
the 16-byte boundary), which run in one walk up to 384 rows and above that in
segments of 128: heights at and around those, paths that cross many of them
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
@pytest.mark.parametrize("h", [1, 7, 64, 383, 384, 385, 392, 512, 513, 641, 1100])
def test_strip_sweeps(dt, h):
    rng = np.random.default_rng(h * 10 + dt)
    info = np.iinfo(NP[dt])
    levels = np.linspace(info.min, info.max, 9).astype(np.int64)
    for w in (1, 5, TW[dt], 2 * TW[dt] + 3, TW[dt] + 4):
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
            for conn in (4, 8):
                tm, tk = _dev(marker), _dev(mask)
                iwpp.sweep(tm, tk, d, conn)
                got = tm.cpu().numpy().view(NP[dt])
                assert np.array_equal(got, oracle.sweep(marker, mask, d, conn)), (w, d, conn)

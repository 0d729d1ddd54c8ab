"""Vertical sweeps by strips whose fronts run down many segments: the settle
step's walk through rows copied ahead, and the last strip's partial words,
which are loaded whole and stored pixel by pixel: nothing outside the image is
written, and what lies there does not get in."""
import numpy as np
import pytest

import iwpp
import oracle

pytestmark = pytest.mark.gpu
NP = {0: np.uint8, 1: np.uint16, 2: np.int32}


@pytest.mark.parametrize("dt", [0, 1, 2])
@pytest.mark.parametrize("h", [385, 512, 777, 1289, 4224, 4225, 8321])
@pytest.mark.parametrize("extra", [0, 1, 2, 3])
def test_one_front_down_the_whole_height(dt, h, extra):
    import torch
    lib = iwpp.load()
    bpp = np.dtype(NP[dt]).itemsize
    tw = 128 // bpp
    info = np.iinfo(NP[dt])
    rng = np.random.default_rng(h * 4 + extra)
    for w in (extra + 1, tw + extra, 2 * tw + 4 // bpp * 3 + extra):
        # rows in a wider buffer full of the type's largest value
        stride = -(-(w + 3) * bpp // 4) * 4 // bpp
        bufs = []
        mask = rng.integers(info.max // 2, info.max, (h, w), endpoint=True).astype(NP[dt])
        marker = np.full((h, w), info.min, NP[dt])
        marker[0] = mask[0] // 3
        marker[-1] = mask[-1] // 4
        marker[rng.random((h, w)) < 0.001] = 7
        marker = np.minimum(marker, mask)
        for a in (marker, mask):
            b = np.full((h, stride), info.max, NP[dt])
            b[:, :w] = a
            bufs.append(b)
        for d in (1, 3):
            for conn in (4, 8):
                m, k = (torch.from_numpy(b.view(np.uint8).copy()).cuda() for b in bufs)
                pitch = stride * bpp
                assert lib.iwpp_sweep(m.data_ptr(), k.data_ptr(), pitch, pitch, w, h, dt, conn, d, None) == 0
                got = m.cpu().numpy().view(NP[dt])
                assert np.array_equal(got[:, :w], oracle.sweep(marker, mask, d, conn)), (w, d, conn)
                assert np.all(got[:, w:] == info.max), (w, d, conn)
                assert np.array_equal(k.cpu().numpy().view(NP[dt]), bufs[1])

"""Staging copies of rows of more than one piece (1024 bytes): widths around the
pieces' ends, every byte offset, a few very wide rows."""
import numpy as np
import pytest

import iwpp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w", [1023, 1024, 1025, 1027, 1029, 2047, 2048, 2053, 4099, 100003])
def test_clip_of_wide_rows_at_any_offset(w):
    # clip goes through the copies in both directions and changes few pixels
    import torch
    lib = iwpp.load()
    h = 5
    rng = np.random.default_rng(w)
    for off_m, off_k, pad in ((0, 1, 0), (1, 0, 1), (2, 3, 2), (3, 2, 3), (1, 1, 0)):
        pitch = w + pad if (w + pad) % 4 else w + pad + 1  # off the word boundary
        bm, bk = (rng.integers(0, 256, off + h * pitch + 8, dtype=np.uint8) for off in (off_m, off_k))
        want = bm.copy()
        for y in range(h):
            a = slice(off_m + y * pitch, off_m + y * pitch + w)
            want[a] = np.minimum(bm[a], bk[off_k + y * pitch:off_k + y * pitch + w])
        m, k = torch.from_numpy(bm).cuda(), torch.from_numpy(bk).cuda()
        assert lib.iwpp_clip(m.data_ptr() + off_m, k.data_ptr() + off_k, pitch, pitch, w, h, 0, None) == 0
        assert np.array_equal(m.cpu().numpy(), want), (off_m, off_k, pitch)
        assert np.array_equal(k.cpu().numpy(), bk)

"""What the warps of a visit stored is published by the first warp, after the
barrier that ends the visit: fronts that rise in the last warp's rows first,
by eight, four and two warps per tile, again and again."""
import numpy as np
import pytest

import iwpp
import oracle

pytestmark = pytest.mark.gpu


# 64-row tiles: 72, 1056 and 2080 of them on 152 multiprocessors
@pytest.mark.parametrize("w, h", [(1100, 500), (4096, 2111), (4224, 4037)])
@pytest.mark.parametrize("conn", [4, 8])
def test_fronts_that_start_in_a_tiles_last_rows(w, h, conn):
    import torch
    rng = np.random.default_rng(17 * w + conn)
    mask = rng.integers(150, 256, (h, w), dtype=np.uint8)
    marker = np.zeros_like(mask)
    rows = np.arange(63, h, 64 * 4)
    marker[rows[:, None], np.arange(0, w, 517)[None, :]] = 240
    marker = np.minimum(marker, mask)
    want = oracle.reconstruct(marker, mask, conn)
    k = torch.from_numpy(mask).cuda()
    m = torch.from_numpy(marker).cuda()
    cfg = iwpp.Config.make(tile_rows=64)
    for variant in ("async", "mutex", "double", "unique"):
        for _ in range(4):
            out = m.clone()
            iwpp.reconstruct(out, k, connectivity=conn, variant=variant, config=cfg)
            assert np.array_equal(out.cpu().numpy(), want), variant

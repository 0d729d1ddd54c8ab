"""The solvers of one warp per tile: four workers per CTA, each on a tile of its
own, that share a mutex buffer and arrive at the round barrier one by one:
fewer tiles than workers, a few more, and as many workers as tiles."""
import numpy as np
import pytest

import iwpp
import oracle
from iwpp import synth

pytestmark = pytest.mark.gpu
NP = {0: np.uint8, 1: np.uint16, 2: np.int32}
TW = {0: 128, 1: 64, 2: 32}


def _dev(a):
    import torch
    return torch.from_numpy(a.view(np.int16) if a.dtype == np.uint16 else a.copy()).cuda()


@pytest.mark.parametrize("solver", [1, 3])
@pytest.mark.parametrize("variant", ["async", "unique", "double", "mutex"])
@pytest.mark.parametrize("dt, tiles_x, tiles_y", [(0, 1, 1), (0, 3, 1), (1, 2, 2), (2, 5, 1), (0, 7, 3), (1, 17, 16),
                                                  (2, 30, 20)])
def test_workers(solver, variant, dt, tiles_x, tiles_y):
    w, h = tiles_x * TW[dt] - 3, tiles_y * 32 - 5
    for conn, sparse in ((4, False), (8, False), (8, True)):
        mask = synth.noise_mask(w, h, dt, 100 * tiles_x + tiles_y + conn, 3.0, 6)
        marker = synth.sparse_marker(mask, 5, 0.002) if sparse else synth.hdome_marker(mask, 60)
        want = oracle.reconstruct(marker, mask, conn)
        for grid, rows in ((0, 32), (0, 64), (1, 32), (3, 32)):
            m, k = _dev(marker), _dev(mask)
            cfg = iwpp.Config.make(solver=solver, grid_ctas=grid, tile_rows=rows)
            iwpp.reconstruct(m, k, connectivity=conn, variant=variant, config=cfg)
            assert np.array_equal(m.cpu().numpy().view(NP[dt]), want), (conn, sparse, grid, rows)

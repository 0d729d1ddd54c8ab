"""grid_ctas below, at and above what each kernel keeps resident: the limit
chooses the warps per tile and the default tile height, never the result."""
import numpy as np
import pytest

import iwpp
import oracle
from iwpp import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w, h, conn", [(300, 200, 8), (1024, 1030, 4), (4224, 4037, 8)])
def test_limited_grids(w, h, conn):
    import torch
    mask = synth.noise_mask(w, h, synth.U8, w + conn, 4.0, 40)
    marker = synth.hdome_marker(mask, 40)
    want = torch.from_numpy(oracle.reconstruct(marker, mask, conn)).cuda()
    k = torch.from_numpy(mask).cuda()
    m = torch.from_numpy(marker).cuda()
    for variant in ("async", "unique", "double", "mutex"):
        for grid in (2, 3, 151, 153, 456, 457, 912, 913):
            if w > 4000 and grid < 151 and variant != "async":
                continue
            out = m.clone()
            iwpp.reconstruct(out, k, connectivity=conn, variant=variant, config=iwpp.Config.make(grid_ctas=grid))
            assert torch.equal(out, want), (variant, grid)

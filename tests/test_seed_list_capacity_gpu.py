"""The double queue started from a seed list that is longer than its capacity:
every tile on the list has to be visited all the same."""
import numpy as np
import pytest

import iwpp
import oracle
from iwpp import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("front_passes, init_passes", [(1, 0), (1, 2), (3, -1)])
@pytest.mark.parametrize("capacity", [1, 16, 255])
@pytest.mark.parametrize("conn", [4, 8])
def test_a_seed_list_longer_than_the_queue(front_passes, init_passes, capacity, conn):
    import torch
    # 256 tiles of 128 x 32, nearly all with a pixel to raise
    mask = synth.noise_mask(1024, 1024, synth.U8, 41 + conn, 2.0, 60)
    marker = synth.hdome_marker(mask, 40)
    k = torch.from_numpy(mask).cuda()
    out = torch.from_numpy(marker).cuda()
    cfg = iwpp.Config.make(tile_rows=32, queue_capacity=capacity, front_passes=front_passes,
                           init_passes=init_passes, max_restarts=100000)
    iwpp.reconstruct(out, k, connectivity=conn, variant="double", config=cfg)
    assert np.array_equal(out.cpu().numpy(), oracle.reconstruct(marker, mask, conn))

"""The engine's kernels for many tiles: jobs large enough in 64-row tiles that
four and two warps share a tile (the smaller sizes of the other files run with
eight, or four per 32-row tile), narrow ragged images so that every tile has a
tile edge or an image edge in it, bit for bit against the oracle."""
import numpy as np
import pytest

import iwpp
import oracle
from iwpp import synth

pytestmark = pytest.mark.gpu
NP = {0: np.uint8, 1: np.uint16, 2: np.int32}
TW = {0: 128, 1: 64, 2: 32}  # pixels of a tile row


def _run(marker, mask, conn, variant):
    import torch

    def dev(a):
        return torch.from_numpy(a.view(np.int16) if a.dtype == np.uint16 else a.copy()).cuda()

    m, k = dev(marker.copy()), dev(mask)
    st = iwpp.reconstruct(m, k, connectivity=conn, variant=variant, config=iwpp.Config.make(tile_rows=64))
    return m.cpu().numpy().view(marker.dtype), st


@pytest.mark.parametrize("dt", [0, 1, 2])
@pytest.mark.parametrize("conn", [4, 8])
@pytest.mark.parametrize("tiles_x,tiles_y,extra_w,extra_h", [(2, 521, 3, 5), (3, 641, -1, 0), (1, 2001, -3, 63)])
def test_warps_per_tile(dt, conn, tiles_x, tiles_y, extra_w, extra_h):
    w, h = tiles_x * TW[dt] + extra_w, tiles_y * 64 + extra_h
    rng = np.random.default_rng(dt * 100 + conn * 10 + tiles_x)
    info = np.iinfo(NP[dt])
    # few levels, so that plateaus, dead ends and diagonal links abound; rows
    # of a serpentine corridor at the top level cross every tile boundary
    levels = np.linspace(info.min, info.max, 7).astype(np.int64)
    mask = levels[rng.integers(0, 6, (h, w))].astype(NP[dt])
    mask[40::173] = info.max
    marker = np.full((h, w), info.min, NP[dt])
    at = rng.random((h, w)) < 0.002
    marker[at] = mask[at]
    marker[40::346, 0] = info.max
    ref = oracle.reconstruct(marker, mask, conn)
    for variant in ("async", "unique"):
        out, st = _run(marker, mask, conn, variant)
        assert st.tiles == -(-w // TW[dt]) * -(-h // 64) and st.status == 0
        assert np.array_equal(out, ref), (variant, int((out != ref).sum()))


@pytest.mark.parametrize("conn", [4, 8])
def test_mixed_batch_many_tiles(conn):
    # a batch of every pixel type in one job of the two-warp shape
    pairs, refs = [], []
    import torch
    for i, (dt, w, h) in enumerate([(0, 131, 30000), (1, 257, 20000), (2, 65, 18000), (0, 1, 7), (1, 64, 64)]):
        mask = synth.noise_mask(w, h, dt, 70 + i, 2.0, 40)
        marker = synth.hdome_marker(mask, 20 + 9 * i)
        refs.append(oracle.reconstruct(marker, mask, conn))
        pairs.append([torch.from_numpy(a.view(np.int16) if dt == 1 else a).cuda() for a in (marker, mask)] + [conn])
    iwpp.reconstruct_batch(pairs, config=iwpp.Config.make(tile_rows=64))
    for (m, _, _), ref in zip(pairs, refs):
        assert np.array_equal(m.cpu().numpy().view(ref.dtype), ref)

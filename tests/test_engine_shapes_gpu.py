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


@pytest.mark.parametrize("dt", [0, 1])
@pytest.mark.parametrize("conn", [4, 8])
@pytest.mark.parametrize("off_m,off_k", [(1, 0), (0, 1), (3, 2), (2, 2)])
def test_rows_off_the_word_boundary(dt, conn, off_m, off_k):
    # views at an odd pixel of a larger buffer and of odd pitches: rows start
    # at every byte of a word, one word, part of a word and several tiles wide;
    # nothing around the view changes
    import torch
    rng = np.random.default_rng(off_m * 10 + off_k + conn)
    for w, h, pad_m, pad_k in ((1, 3, 0, 2), (3, 40, 2, 0), (TW[dt] - 1, 33, 0, 0), (2 * TW[dt] + 5, 130, 3, 1),
                               (3 * TW[dt] + 2, 67, 1, 4)):
        mask = synth.noise_mask(w, h, dt, 5 + w, 1.5, 3)
        marker = synth.hdome_marker(mask, 60)
        ref = oracle.reconstruct(marker, mask, conn)
        t = torch.uint8 if dt == 0 else torch.int16

        def view(a, off, pad):
            buf = torch.from_numpy(rng.integers(0, 120, (w + pad) * h + off, dtype=np.int64)).to(t).cuda()
            v = torch.as_strided(buf, (h, w), (w + pad, 1), off)
            v.copy_(torch.from_numpy(a.view(np.int16) if dt == 1 else a))
            return buf, v

        (bm, m), (bk, k) = view(marker, off_m, pad_m), view(mask, off_k, pad_k)
        before = bm.clone()
        for variant in ("async", "unique"):
            for solver in (0, 1):
                bm.copy_(before)
                iwpp.reconstruct(m, k, connectivity=conn, variant=variant, config=iwpp.Config.make(solver=solver))
                assert np.array_equal(m.cpu().numpy().view(ref.dtype), ref), (w, h, variant, solver)
                around = torch.ones_like(bm, dtype=torch.bool)
                torch.as_strided(around, (h, w), (w + pad_m, 1), off_m).fill_(False)
                assert torch.equal(bm[around], before[around]), (w, h, variant, solver)


@pytest.mark.parametrize("tile_rows,height", [(32, 300), (64, 700), (64, 15000), (64, 26000)])
@pytest.mark.parametrize("variant", ["mutex", "double", "unique", "async"])
def test_batch_of_both_connectivities(variant, tile_rows, height):
    # the kernels that look the connectivity up, at every warp count of a tile
    import torch
    pairs, refs = [], []
    for i, (dt, conn, w) in enumerate([(0, 4, 129), (1, 8, 63), (2, 4, 33), (0, 8, 127), (1, 4, 1), (2, 8, 31)]):
        mask = synth.noise_mask(w, height - 97 * i if i < 4 else 65, dt, 90 + i, 2.0, 40)
        marker = synth.hdome_marker(mask, 15 + 9 * i)
        refs.append(oracle.reconstruct(marker, mask, conn))
        pairs.append([torch.from_numpy(a.view(np.int16) if dt == 1 else a).cuda() for a in (marker, mask)] + [conn])
    iwpp.reconstruct_batch(pairs, variant=variant, config=iwpp.Config.make(tile_rows=tile_rows))
    for (m, _, _), ref in zip(pairs, refs):
        assert np.array_equal(m.cpu().numpy().view(ref.dtype), ref)

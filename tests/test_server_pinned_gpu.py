"""The server's planes in pinned host memory, which one kernel a batch reads and
writes in place: rows with a pitch, planes on any byte a pixel may start on,
bursts of more copies than a launch holds, and pinned planes beside pageable
ones.  Every result is the oracle's, the bytes around it stay, and what was
read is what it was."""
import numpy as np
import pytest

import iwpp
import oracle
from iwpp import synth

pytestmark = pytest.mark.gpu
NP = {0: np.uint8, 1: np.uint16, 2: np.int32}
GUARD = 0xA5


class Plane:
    """An h x w image `shift` bytes into a buffer full of GUARD, with `pad` more pixels a row."""

    def __init__(self, h, w, dt, shift, pad, pinned):
        import torch
        bpp = np.dtype(NP[dt]).itemsize
        size = 64 + shift + h * (w + pad) * bpp + 64
        self.buf = torch.full((size,), GUARD, dtype=torch.uint8, pin_memory=pinned)
        self.bytes = self.buf.numpy()
        at = 64 + shift
        self.image = np.ndarray((h, w), NP[dt], self.bytes.data, at, ((w + pad) * bpp, bpp))
        inside = np.zeros(size, bool)
        for y in range(h):
            inside[at + y * (w + pad) * bpp:at + y * (w + pad) * bpp + w * bpp] = True
        self.around = ~inside

    def guarded(self):
        return bool(np.all(self.bytes[self.around] == GUARD))


def _burst(specs, lanes):
    """specs: (h, w, dt, shifts, pads, pinned) per request, the last three for marker, mask, result."""
    with iwpp.Server(lanes=lanes) as server:
        jobs = []
        for i, (h, w, dt, shifts, pads, pinned) in enumerate(specs):
            mask = synth.noise_mask(w, h, dt, 50 + i, 3.0, 4)
            marker = synth.hdome_marker(mask, 40) if i % 2 else synth.sparse_marker(mask, i, 0.01)
            planes = [Plane(h, w, dt, s, p, pin) for s, p, pin in zip(shifts, pads, pinned)]
            planes[0].image[:], planes[1].image[:] = marker, mask
            jobs.append((planes, marker, mask))
        tickets = [server.submit(p[0].image, p[1].image, 8, out=p[2].image) for p, _, _ in jobs]
        for t in tickets:
            server.wait(t)
    for (planes, marker, mask), spec in zip(jobs, specs):
        assert np.array_equal(planes[2].image, oracle.reconstruct(marker, mask, 8)), spec
        assert np.array_equal(planes[0].image, marker) and np.array_equal(planes[1].image, mask), spec
        assert all(p.guarded() for p in planes), spec


@pytest.mark.parametrize("dt", [0, 1, 2])
@pytest.mark.parametrize("w", [1, 3, 5, 31, 130, 257])
def test_pitches_and_byte_offsets(dt, w):
    bpp = np.dtype(NP[dt]).itemsize
    steps = [s for s in range(0, 5) if s % bpp == 0]
    specs = [(37, w, dt, (a, b, c), (pad, 2 * pad, pad + 1), (True, True, True))
             for a, b, c in ((s, t, u) for s in steps for t in steps[:2] for u in steps) for pad in (0, 3)]
    _burst(specs, lanes=1)


@pytest.mark.parametrize("lanes", [1, 3])
def test_pinned_planes_beside_pageable_ones(lanes):
    specs = []
    for i in range(48):
        pinned = (bool(i & 1), bool(i & 2), bool(i & 4))
        specs.append((20 + 7 * i, 600 - 11 * i, i % 2, (2 * (i % 3), 0, 2), (i % 4, 0, 1), pinned))
    _burst(specs, lanes)

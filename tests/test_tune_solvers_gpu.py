"""The autotuner times a kernel once: solver 2 is the same one as solver 0, so
what it records is 0 or 1."""
import numpy as np
import pytest

import iwpp
from iwpp import synth

pytestmark = pytest.mark.gpu


def test_no_configuration_is_timed_under_two_names():
    import torch
    for i in range(10):
        mask = synth.noise_mask(200 + 100 * i, 300, synth.U8, i, 3.0, 5)
        m = torch.from_numpy(synth.hdome_marker(mask, 30)).cuda()
        res = iwpp.autotune([(m, torch.from_numpy(np.ascontiguousarray(mask)).cuda(), 8)], repeats=1)
        iwpp.tune_clear()
        assert res["solver"] in (0, 1), res

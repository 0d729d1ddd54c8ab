"""stats.launches counts the same kernels for a job whichever way it is run,
the copies of rows off the word boundary among them."""
import ctypes

import pytest

import iwpp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w, count", [(128, 1), (131, 1), (131, 2), (131, 40)])
def test_launches_of_a_synchronous_call_an_asynchronous_one_and_a_plan(w, count):
    import torch
    lib = iwpp.load()
    g = torch.Generator(device="cuda")
    g.manual_seed(w + count)
    masks = [torch.randint(0, 256, (70, w), dtype=torch.uint8, device="cuda", generator=g) for _ in range(count)]
    pairs = [((k.to(torch.int16) - 30).clamp_(min=0).to(torch.uint8), k, 8) for k in masks]
    h = iwpp.Handle()
    sync = iwpp.reconstruct_batch([(m.clone(), k, c) for m, k, c in pairs], handle=h)
    arr = (iwpp.Image * count)(*[iwpp.Image(m.data_ptr(), k.data_ptr(), w, w, w, 70, 0, c) for m, k, c in pairs])
    again = iwpp.Stats()
    torch.cuda.synchronize()
    assert lib.iwpp_reconstruct_batch_async(h.ptr, arr, count, iwpp.DEFAULT, None, None) == 0
    assert lib.iwpp_handle_sync(h.ptr, ctypes.byref(again)) == 0
    plan = iwpp.Plan(h, [(m.clone(), k, c) for m, k, c in pairs])
    plan.launch()
    planned = plan.sync()
    # the engine and its initialisation; in and out, 64 copies a launch
    copies = 0 if w % 4 == 0 else -(-2 * count // 64) + -(-count // 64)
    assert (sync.launches, again.launches, planned.launches) == (2 + copies,) * 3
    plan.close()
    h.close()

"""iwpp_reconstruct_noalloc takes no device memory after its first call,
whichever kernel a later call's connectivity and tile count choose."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

SCRIPT = """
import torch, iwpp
lib = iwpp.load()
# 64-row tiles by eight, four and two warps
sizes = [(300, 200), (4096, 2112), (4224, 4037)]
planes = {}
for w, h in sizes:
    g = torch.Generator(device="cuda"); g.manual_seed(w)
    k = torch.randint(0, 256, (h, w), dtype=torch.uint8, device="cuda", generator=g)
    m = (k.to(torch.int16) - 40).clamp_(min=0).to(torch.uint8)
    planes[w, h] = (m, m.clone(), m.clone(), k)
torch.cuda.synchronize()
w, h = sizes[0]
m, o, _, k = planes[w, h]
assert lib.iwpp_reconstruct_noalloc(o.data_ptr(), k.data_ptr(), w, w, w, h, 0, 8, None) == 0
torch.cuda.synchronize()
free, _ = torch.cuda.mem_get_info()
for conn in (4, 8):
    for w, h in sizes:
        m, o, r, k = planes[w, h]
        (o if conn == 4 else r).copy_(m)
        torch.cuda.synchronize()
        assert lib.iwpp_reconstruct_noalloc((o if conn == 4 else r).data_ptr(), k.data_ptr(), w, w, w, h, 0, conn,
                                            None) == 0
        assert torch.cuda.mem_get_info()[0] >= free, (conn, w, h, free - torch.cuda.mem_get_info()[0])
for w, h in sizes:
    m, o, r, k = planes[w, h]
    for conn, got in ((4, o), (8, r)):
        want = m.clone()
        iwpp.reconstruct(want, k, connectivity=conn)
        assert torch.equal(got, want), (conn, w, h)
print("same memory, same bytes")
"""


def test_no_later_call_takes_memory():
    # a process of its own: no kernel of the library is loaded before
    env = dict(os.environ, PYTHONPATH=os.pathsep.join(p for p in sys.path if p))
    r = subprocess.run([sys.executable, "-c", SCRIPT], capture_output=True, text=True, timeout=300, env=env)
    assert r.returncode == 0, r.stderr[-2000:]
    assert "same memory, same bytes" in r.stdout

"""rmq_query_idx_static's first call on a device, with no queries and a small
array, prepares the device for every later one: in a fresh process, the next
call needs other kernels (more sizes of windows, more queries), takes no device
memory, can be made inside a stream capture, and is exact."""
from __future__ import annotations

import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parents[1]

CHILD = """
import ctypes, sys, time
sys.path.insert(0, "gpu-rmq_gb300")
import torch
import rmq_gb300 as R
P, U = ctypes.c_void_p, ctypes.c_uint64
f = R.lib().rmq_query_idx_static
f.argtypes, f.restype = [P, U, U, P, U, P, P, P], ctypes.c_int
n, q = 1 << 22, (1 << 18) + int(sys.argv[1])
g = torch.Generator(device="cuda").manual_seed(4)
v = torch.randint(0, 1000, (n,), generator=g, device="cuda").float()
length = torch.exp(torch.rand(q, generator=g, device="cuda") * 15.2).long().clamp(1, n)
l = (torch.rand(q, generator=g, device="cuda", dtype=torch.float64) * (n - length + 1)).long()
lr = torch.stack([l, l + length - 1], 1).to(torch.int32).contiguous()
bm, bi = R.bruteforce(v, lr)
oi, om = torch.zeros(q, dtype=torch.int32, device="cuda"), torch.zeros(q, device="cuda")
assert f(v.data_ptr(), 100, 0, None, 0, oi.data_ptr(), None, None) == R.RMQ_OK
torch.cuda.synchronize()
if sys.argv[2] == "captured":
    s = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(s):
        graph.capture_begin()
        st = f(v.data_ptr(), n, 0, lr.data_ptr(), q, oi.data_ptr(), om.data_ptr(), s.cuda_stream)
        graph.capture_end()
    graph.replay()
else:
    free = torch.cuda.mem_get_info()[0]
    t = time.perf_counter()
    st = f(v.data_ptr(), n, 0, lr.data_ptr(), q, oi.data_ptr(), om.data_ptr(), None)
    t = time.perf_counter() - t
    torch.cuda.synchronize()
    assert torch.cuda.mem_get_info()[0] == free
    print(f"enqueued in {t * 1e6:.0f} us")
assert st == R.RMQ_OK, st
torch.cuda.synchronize()
assert torch.equal(oi, bi) and torch.equal(om.view(torch.int32), bm.view(torch.int32))
"""


@pytest.mark.parametrize("how", ["captured", "plain"])
@pytest.mark.parametrize("more", [0, 5])
def test_first_call_prepares_every_later_one(cuda, more, how):
    r = subprocess.run([sys.executable, "-c", CHILD, str(more), how], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    print(r.stdout)

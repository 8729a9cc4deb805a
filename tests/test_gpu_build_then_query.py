"""Builds followed at once by queries that are scheduled before the build ends
(rmq_query_idx_static, rmq_batch_run_per_array), again and again over the same
tables with other values, unsynchronised (GPU): no result is an older build's.
Sizes on both sides of every line between the build's kernels."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

import rmq_gb300 as R
from test_gpu_window import _queries

pytestmark = pytest.mark.gpu

SIZES = [1, 255, 256, 257, 4095, 4096, 4097, 4128, 16_383, 16_384, 16_385, 16_416, 65_537, 300_007, (1 << 20) - 1,
         1 << 20, (1 << 20) + 1, (1 << 21) + 33, (1 << 22) - 7, 1 << 22]


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("q", [3000, (1 << 18) + 3])
def test_alternating_arrays_static(cuda, n, q):
    import torch
    f = R.lib().rmq_query_idx_static
    f.argtypes = [ctypes.c_void_p, ctypes.c_uint64, ctypes.c_uint64, ctypes.c_void_p, ctypes.c_uint64,
                  ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p]
    f.restype = ctypes.c_int
    rng = np.random.default_rng(n)
    values = [torch.from_numpy(rng.integers(0, 1 << 20, n).astype(np.float32)).to(cuda) for _ in range(3)]
    dq = torch.from_numpy(_queries(n, q, rng).view(np.int32)).to(cuda)
    expect = [R.bruteforce(v, dq) for v in values]
    rounds = 30 if q < 10_000 else 3
    outs = [[(torch.zeros(q, dtype=torch.int32, device=cuda), torch.zeros(q, device=cuda)) for _ in values]
            for _ in range(rounds)]
    stream = torch.cuda.current_stream().cuda_stream
    for row in outs:
        for v, (i, m) in zip(values, row):
            assert f(v.data_ptr(), n, 0, dq.data_ptr(), q, i.data_ptr(), m.data_ptr(), stream) == R.RMQ_OK
    torch.cuda.synchronize()
    for row in outs:
        for (bm, bi), (i, m) in zip(expect, row):
            assert torch.equal(i, bi) and torch.equal(m.view(torch.int32), bm.view(torch.int32))


def test_per_array_loop_over_changing_values(cuda):
    import torch
    rng = np.random.default_rng(8)
    sizes = SIZES[:-4]
    offs, total = R.pack_offsets(sizes)
    qs = [_queries(n, 500, rng) for n in sizes]
    qo = np.arange(len(sizes) + 1, dtype=np.uint64) * 500
    dq = torch.from_numpy(np.concatenate(qs).view(np.int32)).to(cuda)
    host = [rng.integers(0, 1 << 20, total).astype(np.float32) for _ in range(2)]
    v = torch.empty(total, device=cuda)
    new = [torch.from_numpy(h).to(cuda) for h in host]
    expect = []
    for x in new:
        expect.append([R.bruteforce(x[int(o):int(o) + n], dq[500 * k:500 * (k + 1)])
                       for k, (o, n) in enumerate(zip(offs, sizes))])
    q = dq.shape[0]
    for with_index in (True, False):
        with R.Batch(v, offs, sizes, with_index=with_index) as b:
            i, m = torch.zeros(q, dtype=torch.int32, device=cuda), torch.zeros(q, device=cuda)
            b.set_queries(dq, qo, i if with_index else None, m)
            got = []
            for step in range(6):
                v.copy_(new[step % 2])
                b.run_per_array()
                got.append((i.clone(), m.clone()))
            torch.cuda.synchronize()
            for step, (i_, m_) in enumerate(got):
                bm = torch.cat([e[0] for e in expect[step % 2]])
                assert torch.equal(m_.view(torch.int32), bm.view(torch.int32))
                if with_index:
                    assert torch.equal(i_, torch.cat([e[1] for e in expect[step % 2]]))

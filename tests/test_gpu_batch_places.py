"""Batches whose results lie in page-locked memory, and batches without argmin
tables (GPU): every path and CTA size gives the oracle's results."""
from __future__ import annotations

import numpy as np
import pytest

import rmq_gb300 as R
from test_gpu_batch import _check, _expected, _make_batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("with_index", [True, False])
@pytest.mark.parametrize("pinned", [True, False])
def test_batch_results_anywhere(cuda, pinned, with_index):
    import torch
    rng = np.random.default_rng(31)
    sizes = [1, 2, 7, 8, 9, 17, 63, 64, 65, 255, 257, 4097, 8193, 100_003] + \
            [int(x) for x in np.exp(rng.uniform(np.log(1 << 10), np.log(1 << 20), 30))]
    dv, dq, offs, arrays, qs, qo = _make_batch(cuda, sizes, 31)
    k = int(np.flatnonzero(np.diff(qo.astype(np.int64)) > 40)[0])
    emin, eidx = _expected(arrays, qs, qo)
    at = int(qo[k]) + 33
    dq[at] = torch.tensor([sizes[k], sizes[k] + 1], dtype=torch.int32)  # invalid
    emin[at], eidx[at] = np.nan, R.NO_POS
    emin.view(np.uint32)[at] = 0x7FC00000
    q = qs.shape[0]
    where = dict(pin_memory=True) if pinned else dict(device=cuda)
    out_min = torch.empty(q, dtype=torch.float32, **where)
    out_idx = torch.empty(q, dtype=torch.int32, **where)
    with R.Batch(dv, offs, sizes, with_index=with_index) as b:
        for block in (32, 128, 512):
            b.set_tuning(64, block)
            for idx in ([out_idx, None] if with_index else [None]):
                b.set_queries(dq, qo, idx, out_min)
                for call in ("run", "run_per_array", "query"):
                    out_min.fill_(-1)
                    out_idx.fill_(-1)
                    torch.cuda.synchronize()
                    getattr(b, call)()
                    torch.cuda.synchronize()
                    _check(out_min, out_idx if idx is not None else torch.from_numpy(eidx.view(np.int32)), emin, eidx,
                           f"{call}, {block} threads")

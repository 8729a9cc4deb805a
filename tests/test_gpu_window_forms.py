"""The coarser forms of the window tables (GPU): a handle above 2^22 entries
takes no more memory than the levels that its scan threshold and reduction
factor plan, and answers as the scan does, for values in every order; the
server keeps its arrays to what levels took, too."""
from __future__ import annotations

import numpy as np
import pytest

import rmq_gb300 as R
from oracle import oracle
from test_gpu_window import KINDS, _queries, _values

pytestmark = pytest.mark.gpu

# rf_log, t, with_index, index_bits: all forms, with and without positions
CONFIGS = [(3, 0, True, 32), (3, 1 << 22, True, 32), (4, 0, True, 32), (5, 0, True, 32), (3, 0, False, 32),
           (3, 1 << 22, False, 32), (4, 0, False, 32), (5, 0, False, 32), (3, 1 << 30, True, 32),
           (3, 1 << 30, False, 32), (4, 0, True, 64), (5, 0, True, 64), (5, 0, False, 64)]


def _planned(n, t, rf_log, with_index, bits):
    info = R.plan_layout(n, t, rf_log, "vl")
    if info.num_levels == 1:
        return 0
    top = info.num_levels - 1
    entries = (info.level_offset[top] + info.level_size[top] + 31) // 32 * 32
    return entries * (4 + (bits // 8 if with_index else 0))


@pytest.mark.parametrize("n", [(1 << 22) + 1, 5_000_011, (1 << 24) + 13, (1 << 24) + (1 << 23) + 4096])
@pytest.mark.parametrize("kind", KINDS)
def test_every_form_matches_scan(cuda, n, kind):
    import torch
    rng = np.random.default_rng(n * 11 + KINDS.index(kind))
    dv = torch.from_numpy(_values(kind, n, rng)).to(cuda)
    for q in (777, (1 << 18) + 5):
        qs = _queries(n, q, rng)
        if q == 777:
            qs[5] = (n - 1, 0)  # invalid
        dq = torch.from_numpy(qs.view(np.int32)).to(cuda)
        dq64 = torch.from_numpy(qs.astype(np.int64)).to(cuda)
        bm, bi = R.bruteforce(dv, dq)
        bits, valid = bm.view(torch.int32), bi != -1
        for rf_log, t, with_index, index_bits in CONFIGS:
            with R.Hierarchy(dv, rf_log=rf_log, t=t, with_index=with_index, index_bits=index_bits) as h:
                planned = _planned(n, t, rf_log, with_index, index_bits)
                assert h.info().level_bytes <= (planned or n // 9)
                wide = index_bits == 64
                m = h.query64(dq64) if wide else h.query(dq)
                assert torch.equal(m.view(torch.int32), bits), (rf_log, t, with_index, index_bits)
                if with_index or planned == 0:
                    i, m = h.query_idx64(dq64, with_min=True) if wide else h.query_idx(dq, with_min=True)
                    assert torch.equal(m.view(torch.int32), bits), (rf_log, t, with_index, index_bits)
                    assert torch.equal(i[valid], bi[valid].to(i.dtype)) and bool((i[~valid] == -1).all())


@pytest.mark.parametrize("t", [8, 64, 1 << 18, 1 << 21])
def test_served_arrays(cuda, t):
    """Arrays with several levels, one level and none at the server's scan threshold."""
    rng = np.random.default_rng(t)
    arrays = [_values("ties", n, rng) for n in (1, 50, 64, 65, 1000, 65_537, 300_001, (1 << 21) + 9)]
    with R.Server(hbm_budget_bytes=64 << 20, t=t) as s:
        for a in arrays:
            i = s.register_host(a)
            qs = _queries(a.size, 3000, rng)
            idx, mins = np.empty(3000, np.uint32), np.empty(3000, np.float32)
            assert s.wait(s.submit(i, qs, idx, mins))[0] == R.RMQ_OK
            assert np.array_equal(idx, oracle.rmq_argmin(a, qs)) and mins.tobytes() == oracle.rmq_min(a, qs).tobytes()
        # what values and levels took, a granule of 256 bytes each; arrays without levels half as much again at most
        took = 0
        for a in arrays:
            levels = _planned(a.size, t, 3, False, 32)
            took += (4 * a.size + 255) // 256 * 256 + 2 * ((levels + 255) // 256 * 256 if levels else a.size // 4 + 256)
        assert s.stats()["resident_bytes"] <= took

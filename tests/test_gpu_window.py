"""The window tables of VL handles (GPU): sizes at the edges of blocks, strides,
windows, build tiles and table forms, lengths at the edges of the query's
routes, values in the orders that defeat the covering windows (sorted, tied,
constant, signed zeros, +inf), with and without argmin tables, 32- and 64-bit
positions, few and many queries.  Every result equals the brute-force scan."""
from __future__ import annotations

import numpy as np
import pytest

import rmq_gb300 as R

pytestmark = pytest.mark.gpu

SIZES = [1, 8, 9, 31, 33, 127, 128, 129, 255, 256, 257, 511, 513, 4097, 65_535, 65_536, 65_537,
         (1 << 22) - 1, 1 << 22, (1 << 22) + 1, (1 << 22) + 65, 9_000_001, (1 << 24) + 13]
KINDS = ["random", "ascending", "descending", "ties", "zeros", "inf"]
LENGTHS = [1, 2, 7, 8, 9, 15, 16, 17, 31, 33, 63, 65, 127, 128, 129, 223, 224, 225, 255, 256, 257, 319, 321, 447, 449,
           511, 512, 513, 1023, 1025, 4095, 4097, 8191, 8193, 65_535, 65_537, 1 << 20, 1 << 22]


def _values(kind, n, rng):
    if kind == "random":
        return rng.random(n, dtype=np.float32) - np.float32(0.5)
    if kind in ("ascending", "descending"):
        a = np.arange(n, dtype=np.float32)
        return a if kind == "ascending" else a[::-1].copy()
    if kind == "ties":
        return rng.integers(0, 100, n).astype(np.float32)
    if kind == "zeros":
        return np.where(rng.random(n) < 0.01, np.where(rng.random(n) < 0.5, -0.0, 0.0), 1.0).astype(np.float32)
    a = np.full(n, np.inf, np.float32)
    a[rng.integers(0, n, n // 1000 + 1)] = 3.0
    return a


def _queries(n, q, rng):
    length = np.minimum(n, np.where(rng.random(q) < 0.7, rng.choice(LENGTHS, q) + rng.integers(-1, 2, q),
                                    np.exp(rng.uniform(0, np.log(n + 1), q)).astype(np.int64)))
    length = np.clip(length, 1, n)
    l = (rng.random(q) * (n - length + 1)).astype(np.int64)
    l = np.where(rng.random(q) < 0.3, np.minimum(l & ~np.int64(31), n - length), l)
    return np.stack([l, l + length - 1], 1).astype(np.uint32)


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("kind", KINDS)
def test_window_tables_match_scan(cuda, n, kind):
    import torch
    rng = np.random.default_rng(n * 7 + KINDS.index(kind))
    dv = torch.from_numpy(_values(kind, n, rng)).to(cuda)
    for q in (777, (1 << 18) + 5):  # below and above the few-queries kernel's limit
        qs = _queries(n, q, rng)
        if q == 777:
            qs[5] = (n - 1, 0) if n > 1 else (0, 1)  # invalid
        dq = torch.from_numpy(qs.view(np.int32)).to(cuda)
        bm, bi = R.bruteforce(dv, dq)
        with R.Hierarchy(dv) as h:
            i, m = h.query_idx(dq, with_min=True)
            only = h.query(dq)
        with R.Hierarchy(dv, with_index=False) as h:
            bare = h.query(dq)
        with R.Hierarchy(dv, index_bits=64) as h:
            i64, m64 = h.query_idx64(torch.from_numpy(qs.astype(np.int64)).to(cuda), with_min=True)
        torch.cuda.synchronize()
        bits = bm.view(torch.int32)
        for name, got in (("min", m), ("min only", only), ("min-only handle", bare), ("64-bit min", m64)):
            assert torch.equal(got.view(torch.int32), bits), name
        assert torch.equal(i, bi)
        valid = bi != -1
        assert torch.equal(i64[valid], bi[valid].to(torch.int64)) and bool((i64[~valid] == -1).all())


@pytest.mark.parametrize("n", [7, 40, 5000, 300_007])
def test_positions_without_argmin_arrays(cuda, n):
    """A handle without argmin arrays whose plan is level 0 alone (t >= n) still answers positions."""
    import torch
    rng = np.random.default_rng(n)
    dv = torch.from_numpy(_values("ties", n, rng)).to(cuda)
    for q in (777, (1 << 18) + 5):
        dq = torch.from_numpy(_queries(n, q, rng).view(np.int32)).to(cuda)
        _, bi = R.bruteforce(dv, dq)
        with R.Hierarchy(dv, t=1 << 20, with_index=False) as h:
            assert torch.equal(h.query_idx(dq), bi)


def test_many_queries_into_page_locked_memory_and_captured(cuda):
    """Above the few-queries limit: results in page-locked host memory through the device call, and a captured launch."""
    import torch
    n, q = 100_003, (1 << 18) + 77
    rng = np.random.default_rng(3)
    dv = torch.from_numpy(_values("random", n, rng)).to(cuda)
    dq = torch.from_numpy(_queries(n, q, rng).view(np.int32)).to(cuda)
    bm, bi = R.bruteforce(dv, dq)
    with R.Hierarchy(dv) as h:
        hi, hm = torch.empty(q, dtype=torch.int32).pin_memory(), torch.empty(q).pin_memory()
        assert h.query_idx_raw(dq.data_ptr(), q, hi.data_ptr(), hm.data_ptr()) == R.RMQ_OK
        torch.cuda.synchronize()
        assert torch.equal(hi, bi.cpu()) and torch.equal(hm.view(torch.int32), bm.cpu().view(torch.int32))
        di, dm = torch.zeros(q, dtype=torch.int32, device=cuda), torch.zeros(q, device=cuda)
        s = torch.cuda.Stream()
        s.wait_stream(torch.cuda.current_stream())
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            h.query_idx(dq, out_idx=di, out_min=dm, with_min=True)
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(di, bi) and torch.equal(dm.view(torch.int32), bm.view(torch.int32))

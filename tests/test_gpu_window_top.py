"""Window tables at the largest sizes (GPU): 32-bit handles up to 0xFFFFFF00
entries, whose positions end just below 2^32, and 64-bit handles beyond 2^33,
where a query can be longer than the two largest windows; always more queries
than the few-queries kernel takes."""
from __future__ import annotations

import numpy as np
import pytest

import rmq_gb300 as R

pytestmark = pytest.mark.gpu

Q = (1 << 18) + 4099
MAX_N = 0xFFFFFF00


def _bits(x):
    import torch
    return x.view(torch.int32)


def _local(n, q, rng):
    """Queries over n entries, most of them short, many at the end."""
    length = np.where(rng.random(q) < 0.7, rng.integers(1, 640, q), rng.integers(1, n + 1, q))
    l = np.where(rng.random(q) < 0.5, n - length - rng.integers(0, 64, q), rng.integers(0, n, q))
    l = np.clip(l, 0, n - length)
    return np.stack([l, l + length - 1], 1).astype(np.int64)


def _pairs(lr, cuda, dtype=np.int32):
    import torch
    return torch.from_numpy(np.ascontiguousarray(lr).astype(np.uint32 if dtype == np.int32 else np.int64).view(dtype)).to(cuda)


@pytest.mark.parametrize("n", [MAX_N, MAX_N - 1, MAX_N - 0x15B])
def test_last_entries_of_32_bit_handles(cuda, n):
    """Short queries at the end of the largest 32-bit handles equal the scan of the tail alone."""
    import torch
    rng = np.random.default_rng(n)
    v = torch.empty(n, dtype=torch.float32, device=cuda)
    R.gen_values_device(v, 77)
    t0 = (n - 4096) & ~7
    v[t0:] = torch.from_numpy(rng.integers(0, 50, n - t0).astype(np.float32)).to(cuda)
    local = _local(n - t0, Q, rng)
    bm, bi = R.bruteforce(v[t0:], _pairs(local, cuda))
    dq = _pairs(local + t0, cuda)
    for with_index, rf_log in ((True, 3), (False, 3), (True, 5), (False, 5)):
        with R.Hierarchy(v, with_index=with_index, rf_log=rf_log, index_bits=32) as h:
            m = h.query(dq)
            assert torch.equal(_bits(m), _bits(bm))
            if with_index:
                i, m = h.query_idx(dq, with_min=True)
                assert torch.equal(_bits(m), _bits(bm)) and torch.equal(i, bi + (t0 - (1 << 32)))


def test_long_queries_of_the_largest_32_bit_handle(cuda):
    """Lengths up to n (windows of 2^32, the build's last kernel): 32- and 64-bit
    handles agree on every query, and torch's scan with both on some."""
    import torch
    n = MAX_N
    rng = np.random.default_rng(5)
    v = torch.empty(n, dtype=torch.float32, device=cuda)
    R.gen_values_device(v, 78)
    length = np.where(rng.random(Q) < 0.5, rng.integers(1, n + 1, Q), np.exp(rng.uniform(0, np.log(n), Q)).astype(np.int64))
    l = (rng.random(Q) * (n - length + 1)).astype(np.int64)
    lr = np.stack([l, l + length - 1], 1)
    lr[:4] = [(0, n - 1), (1, n - 2), (n // 2 - 5, n - 1), (0, (1 << 31) + 7)]
    with R.Hierarchy(v, index_bits=32) as h, R.Hierarchy(v, index_bits=64) as h64, R.Hierarchy(v, with_index=False) as hm:
        i, m = h.query_idx(_pairs(lr, cuda), with_min=True)
        i64, m64 = h64.query_idx64(_pairs(lr, cuda, np.int64), with_min=True)
        bare = hm.query(_pairs(lr, cuda))
        assert torch.equal(i.to(torch.int64) & 0xFFFFFFFF, i64) and torch.equal(_bits(m), _bits(m64))
        assert torch.equal(_bits(m), _bits(bare))
    for k in list(range(4)) + list(rng.integers(0, Q, 12)):
        lo, hi = int(lr[k, 0]), int(lr[k, 1])
        assert int(i64[k]) == lo + int(torch.argmin(v[lo:hi + 1]))


def test_64_bit_handle_past_2_pow_33_entries(cuda):
    """n = 2^33 + 2^25 + 8: queries across 2^32 equal a 32-bit handle's on that
    part, and queries longer than two windows of 2^32 equal torch's scan, with
    and without argmin tables."""
    import torch
    n = (1 << 33) + (1 << 25) + 8
    rng = np.random.default_rng(6)
    v = torch.empty(n, dtype=torch.float32, device=cuda)
    R.gen_values_device(v, 79)
    w0, wn = (1 << 32) - (1 << 25), 1 << 26
    local = _local(wn, Q, rng)
    long = np.array([(0, n - 1), (1, n - 1), (12_345, n - 6), (3, (1 << 33) + 900), ((1 << 25) - 9, n - 1),
                     ((1 << 32) - 5, (1 << 32) + 5), (7, (1 << 32) + 1000), (1 << 31, n - 77)], dtype=np.int64)
    many = np.tile(long, (Q // len(long) + 1, 1))
    expect = torch.tensor([int(a) + int(torch.argmin(v[int(a):int(b) + 1])) for a, b in long], device=cuda)
    for with_index, rf_log in ((True, 3), (False, 3), (True, 5)):
        with R.Hierarchy(v, with_index=with_index, rf_log=rf_log) as h, R.Hierarchy(v[w0:w0 + wn]) as part:
            pi, pm = part.query_idx(_pairs(local, cuda), with_min=True)
            at = expect.repeat(Q // len(long) + 1)
            if with_index:
                i, m = h.query_idx64(_pairs(local + w0, cuda, np.int64), with_min=True)
                assert torch.equal(i, pi.to(torch.int64) + w0)
                j, k = h.query_idx64(_pairs(many, cuda, np.int64), with_min=True)
                assert torch.equal(j, at)
            else:
                m, k = h.query64(_pairs(local + w0, cuda, np.int64)), h.query64(_pairs(many, cuda, np.int64))
            assert torch.equal(_bits(m), _bits(pm)) and torch.equal(_bits(k), _bits(v[at]))

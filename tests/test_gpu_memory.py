"""What handles and batches report as their device memory is what they take (GPU)."""
from __future__ import annotations

import numpy as np
import pytest

import rmq_gb300 as R

pytestmark = pytest.mark.gpu

GRANULE = 2 << 20  # of a device allocation


def _taken(make):
    import torch
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    made = make()
    return made, before - torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("variant,rf_log,t,with_index,bits", [
    ("vl", 3, 0, True, 32), ("vl", 4, 0, True, 32), ("vl", 5, 0, True, 32), ("vl", 3, 0, False, 32),
    ("vl", 5, 0, False, 32), ("vl", 3, 1 << 26, True, 32), ("vl", 3, 0, True, 64), ("vl", 5, 0, False, 64),
    ("cl", 3, 0, True, 32), ("cl", 5, 0, False, 32)])
def test_handle_reports_what_it_takes(cuda, variant, rf_log, t, with_index, bits):
    import torch
    v = torch.rand(1 << 26, device=cuda)
    cfg = dict(variant=variant, rf_log=rf_log, t=t, with_index=with_index, index_bits=bits)
    R.Hierarchy(v, **cfg).close()  # loads the kernels
    h, taken = _taken(lambda: R.Hierarchy(v, **cfg))
    with h:
        assert abs(taken - h.info().level_bytes) <= GRANULE + 65536


@pytest.mark.parametrize("with_index", [True, False])
def test_batch_reports_what_it_takes(cuda, with_index):
    import torch
    sizes = [1 << 20] * 63 + [12_345]
    offs, total = R.pack_offsets(sizes)
    v = torch.rand(total, device=cuda)
    R.Batch(v, offs, sizes, with_index=with_index).close()
    b, taken = _taken(lambda: R.Batch(v, offs, sizes, with_index=with_index))
    with b:
        assert abs(taken - b.info().level_bytes) <= GRANULE + 65536

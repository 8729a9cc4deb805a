"""bench.py's targets are held against the bytes that the roofline counts (CPU)."""
from __future__ import annotations

import bench


def test_mixture_target_is_a_fraction_of_the_roofline():
    subs = {"mixture_n2e26": {"roofline": {"frac": 0.13, "canonical_frac": 1.04}}}
    out = bench.targets_summary(subs)["plain_mixture_n2e26_frac"]
    assert out["value"] == 0.13 and out["met"] is False
    subs["mixture_n2e26"]["roofline"]["frac"] = 0.61
    assert bench.targets_summary(subs)["plain_mixture_n2e26_frac"]["met"] is True

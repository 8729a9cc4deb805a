"""The calls a user of this library makes, as cases that can be timed and compared.

A case names one call form of the Python binding (which only forwards to the C
ABI) with its sizes, length law and options:

  query    Hierarchy.query / query_idx / query_idx64 on device buffers, on a
           handle built beforehand
  oneshot  build, one query call and release of a hierarchy over new values
  host     Hierarchy.query_idx_host_raw: queries and results in page-locked
           host memory
  batch    Batch.run: build and queries of many arrays in one graph launch
  served   Server.submit / wait: a burst of requests on resident arrays

Values are uniform in [0, 1); `ties` sets that fraction of the entries to the
smallest value.  Query lengths follow the laws of the benchmark (bench.py):
uniform in [1, n], lognormal(median, sigma) clamped to [1, n], or the mixture
of uniform, lognormal(2^13, 1) and lognormal(2^5, 0.7) by thirds.
"""
from __future__ import annotations

import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "gpu-rmq_gb300"))

import rmq_gb300 as R  # noqa: E402

DEV = "cuda:0"


def listed() -> list[dict]:
    return [
        # a caller that asks a few questions at a time: launch and call latency
        {"name": "tiny", "kind": "query", "n": 10_007, "q": 256, "law": "uniform", "out": "both"},
        # the reference's CPU comparison size: one array, one small batch of queries
        {"name": "small_uniform", "kind": "query", "n": 1 << 20, "q": 1 << 16, "law": "uniform", "t": 64, "out": "both"},
        # the benchmark's headline workload: many medium-length queries
        {"name": "headline", "kind": "query", "n": 1 << 26, "q": 1 << 26, "law": "medium", "t": 1 << 10, "out": "both"},
        # mixed lengths on one array, with repeated minima
        {"name": "mixture", "kind": "query", "n": 1 << 26, "q": 1 << 26, "law": "mixture", "t": 64, "ties": 0.01,
         "out": "both"},
        # the benchmark's largest array
        {"name": "large_mixture", "kind": "query", "n": 1 << 28, "q": 1 << 27, "law": "mixture", "t": 64, "ties": 0.01,
         "out": "both"},
        # minima only, lengths up to the whole array, a size that is no multiple of anything
        {"name": "uniform_min", "kind": "query", "n": 50_000_017, "q": 30_000_001, "law": "uniform", "out": "min"},
        # positions only, short windows
        {"name": "short_argmin", "kind": "query", "n": 1 << 26, "q": 1 << 25, "law": "short", "out": "idx"},
        # 64-bit positions (arrays beyond 2^32 entries use this form; here at a smaller size)
        {"name": "wide", "kind": "query", "n": (1 << 26) + 8_191, "q": 1 << 25, "law": "medium", "bits": 64,
         "out": "both"},
        # values that are queried once and replaced: build, query, release
        {"name": "oneshot", "kind": "oneshot", "n": 20_000_003, "q": 1 << 20, "law": "medium", "out": "both"},
        # queries and results in page-locked host memory
        {"name": "host_pinned", "kind": "host", "n": 1 << 24, "q": 1 << 22, "law": "medium", "out": "both"},
        # many arrays of very different sizes, rebuilt and queried together
        {"name": "batch", "kind": "batch", "arrays": 384, "lo": 1 << 10, "hi": 1 << 20, "per": 4, "cap": 1 << 20,
         "out": "both"},
        # a server's burst: requests of 1 to 2^16 queries on resident arrays
        {"name": "served", "kind": "served", "arrays": 32, "lo": 1 << 16, "hi": 1 << 21, "requests": 256,
         "cap": 1 << 16, "out": "both"},
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["query"] * 5 + ["oneshot", "host", "batch", "served"])
    if kind == "batch":
        return {"kind": kind, "arrays": _log_int(rng, 16, 384), "lo": _log_int(rng, 100, 5_000),
                "hi": _log_int(rng, 50_000, 1 << 20), "per": rng.choice([1, 2, 4]), "cap": 1 << 20,
                "out": rng.choice(["both", "both", "idx", "min"])}
    if kind == "served":
        return {"kind": kind, "arrays": _log_int(rng, 4, 32), "lo": _log_int(rng, 5_000, 1 << 16),
                "hi": _log_int(rng, 1 << 17, 1 << 21), "requests": _log_int(rng, 32, 256),
                "cap": _log_int(rng, 1 << 10, 1 << 16), "out": "both"}
    case = {"kind": kind, "law": rng.choice(["uniform", "medium", "mixture", "short"]),
            "ties": rng.choice([0.0, 0.0, 0.01])}
    if kind == "oneshot":
        return dict(case, n=_log_int(rng, 1 << 16, 1 << 27), q=_log_int(rng, 1 << 10, 1 << 22), out="both")
    if kind == "host":
        return dict(case, n=_log_int(rng, 1 << 16, 1 << 26), q=_log_int(rng, 1 << 10, 1 << 24),
                    out=rng.choice(["both", "idx"]))
    n = _log_int(rng, 1_000, 1 << 28)
    bits = 64 if rng.random() < 0.2 else 32
    return dict(case, n=n, q=_log_int(rng, 100, 1 << 26), bits=bits, t=rng.choice([0, 32, 64, 1 << 10]),
                out="both" if bits == 64 else rng.choice(["both", "idx", "min"]))


# ---- inputs, from the seed alone ---------------------------------------------

def _generator(seed: int) -> torch.Generator:
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _values(n: int, ties: float, g: torch.Generator) -> torch.Tensor:
    v = torch.rand(n, generator=g, device=DEV)
    if ties:
        v[torch.rand(n, generator=g, device=DEV) < ties] = v.min()
    return v


def _lognormal(n, q: int, median, sigma: float, g: torch.Generator) -> torch.Tensor:
    z = torch.randn(q, generator=g, device=DEV)
    length = torch.exp(z * sigma + (torch.log(median) if isinstance(median, torch.Tensor) else math.log(median)))
    length = length.round().clamp(1.0, 3e9).to(torch.int64)
    return torch.minimum(length, n) if isinstance(n, torch.Tensor) else length.clamp(max=n)


def _lengths(n: int, q: int, law: str, g: torch.Generator) -> torch.Tensor:
    if law == "uniform":
        return (torch.rand(q, generator=g, device=DEV, dtype=torch.float64) * n).to(torch.int64).clamp(max=n - 1) + 1
    if law == "medium":
        return _lognormal(n, q, 8192.0, 1.0, g)
    if law == "short":
        return _lognormal(n, q, 32.0, 0.7, g)
    length = _lengths(n, q, "uniform", g)
    which = torch.rand(q, generator=g, device=DEV)
    length = torch.where(which < 2 / 3, _lengths(n, q, "medium", g), length)
    return torch.where(which < 1 / 3, _lengths(n, q, "short", g), length)


def _pairs(n, length: torch.Tensor, g: torch.Generator, dtype=torch.int32) -> torch.Tensor:
    room = n - length + 1
    l = (torch.rand(length.numel(), generator=g, device=DEV, dtype=torch.float64) * room).to(torch.int64)
    l = torch.minimum(l, room - 1)
    lr = torch.empty((length.numel(), 2), dtype=dtype, device=DEV)
    lr[:, 0] = l
    lr[:, 1] = l + length - 1
    return lr


def _inputs(case: dict, seed: int) -> tuple[torch.Tensor, torch.Tensor]:
    """Values and queries of one array."""
    g = _generator(seed)
    n = case["n"]
    v = _values(n, case.get("ties", 0.0), g)
    lr = _pairs(n, _lengths(n, case["q"], case["law"], g), g, torch.int64 if case.get("bits") == 64 else torch.int32)
    return v, lr


def _many(case: dict, seed: int):
    """Packed values, array offsets and sizes, packed local queries and their
    offsets, for the batched and served forms.  The array sizes and query
    counts belong to the case; the seed gives the values and the queries."""
    g = _generator(seed)
    rng = np.random.default_rng([case["arrays"], case["lo"], case["hi"]])
    sizes = np.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"]), case["arrays"])).astype(np.uint64)
    ends = np.cumsum((sizes + np.uint64(7)) // np.uint64(8) * np.uint64(8))  # every array on a 32-byte boundary
    offs = np.concatenate([np.zeros(1, dtype=np.uint64), ends[:-1]])
    v = torch.rand(int(ends[-1]), generator=g, device=DEV)
    if case["kind"] == "batch":
        owner = np.arange(case["arrays"])
        counts = np.minimum(case["per"] * sizes, case["cap"]).astype(np.int64)
    else:
        owner = rng.integers(0, case["arrays"], case["requests"])
        counts = np.exp(rng.uniform(0.0, math.log(case["cap"]), case["requests"])).astype(np.int64)
    qo = np.zeros(counts.size + 1, dtype=np.uint64)
    qo[1:] = np.cumsum(counts)
    n = torch.from_numpy(sizes[owner].astype(np.int64)).to(DEV).repeat_interleave(torch.from_numpy(counts).to(DEV))
    median = n.to(torch.float32).sqrt() if case["kind"] == "batch" else 8192.0
    lr = _pairs(n, _lognormal(n, n.numel(), median, 1.0, g), g)
    return v, offs, sizes, owner, lr, qo


def _outputs(q: int, out: str, pinned: bool = False) -> tuple[torch.Tensor | None, torch.Tensor | None]:
    where = {"pin_memory": True} if pinned else {"device": DEV}
    idx = torch.zeros(q, dtype=torch.int32, **where) if out != "min" else None
    mins = torch.zeros(q, dtype=torch.float32, **where) if out != "idx" else None
    return idx, mins


# ---- prepare / run -------------------------------------------------------------

def _close(state) -> None:
    for key in ("handle", "batch", "server"):
        if key in state:
            state[key].close()


class State(dict):
    """What a user's program holds between calls; releases its handle with itself."""

    def __del__(self):
        _close(self)


def prepare(case: dict, seed: int) -> State:
    kind = case["kind"]
    s = State(kind=kind, out=case["out"])
    if kind == "batch":
        v, offs, sizes, _, lr, qo = _many(case, seed)
        s["idx"], s["min"] = _outputs(lr.shape[0], case["out"])
        s["batch"] = R.Batch(v, offs, sizes)
        s["batch"].set_queries(lr, qo, s["idx"], s["min"])
    elif kind == "served":
        v, offs, sizes, owner, lr, qo = _many(case, seed)
        host = v.cpu().numpy()
        s["lr"] = lr.cpu().pin_memory()
        s["idx"], s["min"] = _outputs(lr.shape[0], case["out"], pinned=True)
        s["server"] = R.Server(hbm_budget_bytes=1 << 30)
        ids = [s["server"].register_host(host[int(o):int(o) + int(n)]) for o, n in zip(offs, sizes)]
        lr_h, idx_h, min_h = (s[k].numpy().view(d) for k, d in (("lr", np.uint32), ("idx", np.uint32), ("min", np.float32)))
        s["requests"] = [(ids[a], lr_h[int(b):int(e)], idx_h[int(b):int(e)], min_h[int(b):int(e)])
                         for a, b, e in zip(owner, qo[:-1], qo[1:])]
        one = np.zeros((1, 2), dtype=np.uint32)
        for i in ids:  # every array resident and built
            s["server"].wait(s["server"].submit(i, one, np.empty(1, np.uint32)))
    else:
        s["values"], s["lr"] = _inputs(case, seed)
        s["wide"] = case.get("bits") == 64
        s["cfg"] = {"t": case.get("t", 0), "index_bits": case.get("bits", 32)}
        s["idx"], s["min"] = _outputs(case["q"], case["out"], pinned=kind == "host")
        if kind == "host":
            s["lr"] = s["lr"].cpu().pin_memory()
        if kind != "oneshot":
            s["handle"] = R.Hierarchy(s["values"], **s["cfg"])
    return s


def _query(h: R.Hierarchy, s: State):
    if s["wide"]:
        return h.query_idx64(s["lr"], with_min=True)
    if s["out"] == "min":
        return h.query(s["lr"], out=s["min"])
    return h.query_idx(s["lr"], out_idx=s["idx"], out_min=s["min"], with_min=s["out"] == "both")


def run(s: State):
    kind = s["kind"]
    if kind == "query":
        return _query(s["handle"], s)
    if kind == "oneshot":
        with R.Hierarchy(s["values"], **s["cfg"]) as h:
            return _query(h, s)
    if kind == "host":
        mins = s["min"].data_ptr() if s["min"] is not None else None
        st = s["handle"].query_idx_host_raw(s["lr"].data_ptr(), s["lr"].shape[0], s["idx"].data_ptr(), mins)
        if st != R.RMQ_OK:
            raise R.RMQError(st, "rmq_query_idx_host")
    elif kind == "batch":
        s["batch"].run()
    else:
        for rid in [s["server"].submit(*r) for r in s["requests"]]:
            st, _ = s["server"].wait(rid)
            if st != R.RMQ_OK:
                raise R.RMQError(st, "rmq_server_wait")
    return [x for x in (s["idx"], s["min"]) if x is not None]


# ---- what a pass cannot do without, and its exact results ------------------------

def work(case: dict) -> dict:
    """Bytes: every query read once, every result written once, and of the
    values what the pass needs: all of them where it builds, else at least the
    two 32-byte pieces at each query's ends, and no more than the array."""
    out = {"both": 8, "idx": 4, "min": 4}[case["out"]]
    if case["kind"] in ("batch", "served"):
        # means of the log-uniform laws
        lo, hi = case["lo"], case["hi"]
        mean = (hi - lo) / math.log(hi / lo)
        if case["kind"] == "batch":
            cut = min(hi, max(lo, case["cap"] / case["per"]))
            q = case["arrays"] * (case["per"] * (cut - lo) + case["cap"] * math.log(hi / cut)) / math.log(hi / lo)
            return {"bytes": 4 * mean * case["arrays"] + (8 + out) * q, "flops": 0}
        q = case["requests"] * (case["cap"] - 1) / math.log(case["cap"])
        return {"bytes": min(4 * mean * case["arrays"], 64 * q) + (8 + out) * q, "flops": 0}
    n, q = case["n"], case["q"]
    pair = 8
    if case.get("bits") == 64:
        pair, out = 16, 12
    values = 4 * n if case["kind"] == "oneshot" else min(4 * n, 64 * q)
    return {"bytes": values + (pair + out) * q, "flops": 0}


def _range_min(v: torch.Tensor, l: torch.Tensor, r: torch.Tensor) -> torch.Tensor:
    """min(v[l..r]) in float64, from the minima of all windows of 2^k entries."""
    out = torch.empty(l.numel(), dtype=torch.float64, device=v.device)
    k_of = (torch.log2((r - l + 1).to(torch.float64)) + 1e-12).to(torch.uint8)
    win, k = v.to(torch.float64), 0
    while True:
        at = torch.nonzero(k_of == k).flatten()
        if at.numel():
            out[at] = torch.minimum(win[l[at]], win[r[at] - (1 << k) + 1])
        if (2 << k) > v.numel():
            return out
        win = torch.minimum(win[:-(1 << k)], win[1 << k:])
        k += 1


def exact(case: dict, seed: int):
    """The minima as 64-bit values; positions are whole numbers."""
    if case["out"] == "idx":
        return None
    if case["kind"] in ("batch", "served"):
        v, offs, _, owner, lr, qo = _many(case, seed)
        counts = np.diff(qo.astype(np.int64))
        base = torch.from_numpy(offs[owner].astype(np.int64)).to(DEV).repeat_interleave(torch.from_numpy(counts).to(DEV))
    else:
        (v, lr), base = _inputs(case, seed), 0
    mins = _range_min(v, lr[:, 0].to(torch.int64) + base, lr[:, 1].to(torch.int64) + base)
    if case["kind"] == "query" and case["out"] == "min":
        return mins
    return [mins] if case["out"] == "min" else [None, mins]

"""The work a user of this package has it do, as timed cases.

Each case is one call of a public entry point on data of a size and kind that
the package's configurations, tests and benchmark name: the LSD sorts (32- and
64-bit integers, float32, key + payload), the batched segmented sort, digit
histograms, radix select and the 64-bit sum, on device tensors, and the sort
of page-locked host memory.  Sorts work in place, so a pass first copies the
input into the buffer to be sorted, as a caller does who still needs the input.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import parallelalgorithms_gb300 as pa
from parallelalgorithms_gb300 import batched

_ITEM = {"u32": 4, "u64": 8, "f32": 4, "kv_u32": 8, "kv_u64": 12}
_ZIPF_RANKS = 1 << 20


def listed():
    return [
        # one small array per call: latency and launches are all that counts
        {"name": "sort_u32_4k", "op": "sort", "type": "u32", "n": 4096, "dist": "uniform"},
        # a medium array of odd length, a typical request of a service
        {"name": "sort_u32_1m", "op": "sort", "type": "u32", "n": 1_000_003, "dist": "uniform"},
        # the headline: 100M uniform 32-bit keys, resident on the device
        {"name": "sort_u32_100m", "op": "sort", "type": "u32", "n": 100_000_000, "dist": "uniform"},
        # row numbers or timestamps that are already in order
        {"name": "sort_u32_100m_presorted", "op": "sort", "type": "u32", "n": 100_000_000, "dist": "presorted"},
        # measurements: normal floats with signed zeros, infinities and denormals among them
        {"name": "sort_f32_100m", "op": "sort", "type": "f32", "n": 100_000_000, "dist": "normal"},
        # 64-bit hashes or identifiers alone, an odd length
        {"name": "sort_u64_33m", "op": "sort", "type": "u64", "n": 33_333_333, "dist": "uniform"},
        # an index build: 64-bit keys, few of them very frequent, with the row number as payload
        {"name": "sort_kv_u64_100m_zipf", "op": "sort", "type": "kv_u64", "n": 100_000_000, "dist": "zipf"},
        # thousands of arrays of uneven size in one call, replayed from a plan
        {"name": "batched_4096", "op": "batched", "segments": 4096, "lo": 1000, "hi": 4_000_000},
        # the median of 100M keys
        {"name": "select_u32_100m", "op": "select", "type": "u32", "n": 100_000_000, "dist": "uniform", "share": 0.5},
        # every byte digit's counts, as a caller's own radix code wants them
        {"name": "hist_u32_100m", "op": "hist", "type": "u32", "n": 100_000_000, "dist": "uniform"},
        # a checksum-like total
        {"name": "sum_u32_100m", "op": "sum", "type": "u32", "n": 100_000_000, "dist": "uniform"},
        # the whole call on page-locked host memory: copy in, sort, copy out
        {"name": "host_sort_u32_100m", "op": "host_sort", "type": "u32", "n": 100_000_000, "dist": "uniform"},
    ]


def _log_uniform(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))


def draw(rng):
    op = rng.choice(["sort", "sort", "sort", "sort", "batched", "select", "hist", "sum", "host_sort", "inplace"])
    if op == "batched":
        return {"op": op, "segments": _log_uniform(rng, 16, 4096), "lo": 1000, "hi": _log_uniform(rng, 50_000, 4_000_000)}
    n = _log_uniform(rng, 1000, 100_000_000) | 1
    if op == "sort":
        kind = rng.choice(["u32", "u32", "f32", "u64", "kv_u32", "kv_u64"])
        dist = "normal" if kind == "f32" else rng.choice(["uniform", "uniform", "presorted", "zipf", "constant"])
        return {"op": op, "type": kind, "n": n, "dist": dist}
    dist = rng.choice(["uniform", "uniform", "presorted", "zipf"])
    case = {"op": op, "type": "u32", "n": n, "dist": dist}
    if op == "select":
        case["share"] = rng.uniform(0.0, 1.0)
    return case


# ---- inputs -----------------------------------------------------------------
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _mix64(x):
    """A 64-bit hash of x (numpy uint64), so that frequent values lie anywhere in the range."""
    with np.errstate(over="ignore"):
        x = x + np.uint64(0x9E3779B97F4A7C15)
        x = (x ^ (x >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        x = (x ^ (x >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        return x ^ (x >> np.uint64(31))


def _keys(kind, n, dist, seed):
    """n keys on the GPU: torch.int32 / int64 hold the unsigned 32- and 64-bit keys."""
    g = _generator(seed)
    wide = kind.endswith("u64")
    dtype = torch.int64 if wide else torch.int32
    if dist == "normal":
        x = torch.randn(n, generator=g, device="cuda", dtype=torch.float32)
        u = torch.rand(n, generator=g, device="cuda")
        special = [0.0, -0.0, math.inf, -math.inf]
        for i, v in enumerate(special):  # 1 % each
            x[(u >= 0.01 * i) & (u < 0.01 * (i + 1))] = v
        tiny = (u >= 0.04) & (u < 0.05)  # 1 % denormals
        x[tiny] = (torch.rand(int(tiny.sum()), generator=g, device="cuda") - 0.5) * 2e-38
        return x
    if dist == "presorted":
        start = int(torch.randint(0, 1 << 20, (1,), generator=g, device="cuda"))
        return torch.arange(start, start + n, dtype=dtype, device="cuda")
    if dist == "constant":
        return torch.randint(0, 1 << 31 if not wide else 1 << 62, (1,), generator=g, device="cuda").to(dtype).expand(n).contiguous()
    if dist == "zipf":  # rank r with weight r ** -1.1, each rank a hashed value
        cdf = torch.arange(1, _ZIPF_RANKS + 1, device="cuda", dtype=torch.float64).pow(-1.1).cumsum(0)
        cdf /= cdf[-1].clone()
        value = torch.from_numpy(_mix64(np.arange(_ZIPF_RANKS, dtype=np.uint64) + np.uint64(seed)).view(np.int64)).cuda()
        out = torch.empty(n, dtype=dtype, device="cuda")
        for lo in range(0, n, 1 << 24):
            hi = min(n, lo + (1 << 24))
            r = torch.searchsorted(cdf, torch.rand(hi - lo, generator=g, device="cuda", dtype=torch.float64))
            v = value[r.clamp_(max=_ZIPF_RANKS - 1)]
            out[lo:hi] = v if wide else (v >> 32).to(dtype)
        return out
    if wide:
        return torch.randint(-(1 << 63), (1 << 63) - 1, (n,), generator=g, device="cuda", dtype=dtype)
    return torch.randint(-(1 << 31), 1 << 31, (n,), generator=g, device="cuda", dtype=dtype)


def _offsets(case, seed):
    r = np.random.RandomState(int(seed) % (1 << 32))
    # log-uniform sizes at even strides, in another order for each seed: the same work for all of them
    sizes = np.exp(np.linspace(math.log(case["lo"]), math.log(case["hi"]), case["segments"])).astype(np.uint64)
    off = np.zeros(sizes.size + 1, np.uint64)
    off[1:] = np.cumsum(sizes[r.permutation(sizes.size)])
    return off


def prepare(case, seed):
    if case["op"] == "batched":
        off = _offsets(case, seed)
        src = _keys("u32", int(off[-1]), "uniform", seed)
        return {"case": case, "src": src, "keys": torch.empty_like(src), "tmp": torch.empty_like(src),
                "off": off, "plan": batched.SegmentedSortPlan(off)}
    n, kind = case["n"], case["type"]
    src = _keys(kind, n, case["dist"], seed)
    s = {"case": case, "src": src}
    if case["op"] == "sort":
        s["keys"], s["tmp"] = torch.empty_like(src), torch.empty_like(src)
        if kind.startswith("kv"):
            s["rows"] = torch.arange(n, dtype=torch.int32, device="cuda")
            s["vals"], s["tmp_vals"] = torch.empty_like(s["rows"]), torch.empty_like(s["rows"])
    elif case["op"] == "inplace":
        s["keys"] = torch.empty_like(src)
    elif case["op"] == "host_sort":
        s["host"] = torch.empty(n, dtype=src.dtype, pin_memory=True)
        s["array"] = s["host"].numpy().view(np.uint32)
    return s


# ---- one pass ----------------------------------------------------------------
def run(s):
    case = s["case"]
    op = case["op"]
    if op == "sort":
        s["keys"].copy_(s["src"])
        if "vals" in s:
            s["vals"].copy_(s["rows"])
            pa.sort(s["keys"], s["vals"], s["tmp"], s["tmp_vals"])
            return [s["keys"], s["vals"]]
        pa.sort(s["keys"], tmp_keys=s["tmp"])
        return s["keys"]
    if op == "batched":
        s["keys"].copy_(s["src"])
        s["plan"].run(s["keys"], s["tmp"], torch.cuda.current_stream().cuda_stream)
        return s["keys"]
    if op == "inplace":
        s["keys"].copy_(s["src"])
        pa.parallel_hybrid_inplace_msd_radix_sort(s["keys"])
        return s["keys"]
    if op == "host_sort":  # the keys arrive in page-locked memory, from the device here
        s["host"].copy_(s["src"], non_blocking=True)
        pa.SortRadixPar(s["array"])
        return s["host"]
    if op == "select":
        return pa.select(s["src"], _rank(case))
    if op == "hist":
        return pa.HistogramByteComponentsParallel(s["src"], 0, case["n"] - 1)
    return pa.SumParallelNonRecursive(s["src"], 0, case["n"])


def _rank(case):
    return min(case["n"] - 1, int(case["n"] * case["share"]))


def work(case):
    """Every input read once, every output written once."""
    if case["op"] == "batched":
        return {"bytes": 8 * int(_offsets(case, 0)[-1]), "flops": 0}
    n = case["n"]
    if case["op"] in ("sort", "inplace", "host_sort"):
        return {"bytes": 2 * n * _ITEM[case["type"]], "flops": 0}
    return {"bytes": 4 * n, "flops": 0}


# ---- the same in plain torch --------------------------------------------------
def _unsigned_order(x):
    """Signed values in the order of x's bits read as unsigned."""
    return x ^ torch.tensor(torch.iinfo(x.dtype).min, dtype=x.dtype, device=x.device)


def exact(case, seed):
    if case["op"] == "batched":
        off = _offsets(case, seed).astype(np.int64)
        x = _unsigned_order(_keys("u32", int(off[-1]), "uniform", seed))
        for lo, hi in zip(off[:-1], off[1:]):
            x[lo:hi] = torch.sort(x[lo:hi])[0]
        return _unsigned_order(x)
    src = _keys(case["type"], case["n"], case["dist"], seed)
    op = case["op"]
    if op == "hist":
        out = np.zeros((8, 256), np.uint64)
        for d in range(4):
            out[d] = torch.bincount((src >> (8 * d)) & 255, minlength=256).cpu().numpy().astype(np.uint64)
        return out
    if op == "sum":
        return int((src.to(torch.int64) & 0xFFFFFFFF).sum())
    if case["type"] == "f32":  # total order: -0.0 before +0.0
        b = src.view(torch.int32)
        b = torch.sort(torch.where(b < 0, b ^ 0x7FFFFFFF, b))[0]
        return torch.where(b < 0, b ^ 0x7FFFFFFF, b).view(torch.float32).to(torch.float64)
    keys, rows = torch.sort(_unsigned_order(src), stable=True)
    keys = _unsigned_order(keys)
    if op == "select":
        return int(keys[_rank(case)]) & 0xFFFFFFFF
    return [keys, rows.to(torch.int32)] if case["type"].startswith("kv") else keys

"""Performance cases: the work that programs hand to this library, through its Python entry points.

Sizes and distributions come from the benchmark configurations and the tests: 32-bit and 64-bit sorts of
2^25 to 2^28 elements with uniform, low-entropy and Zipf keys, streaming scans and by-key algorithms of up to
2^28 elements, and the small and odd-sized calls of programs that sort or compact a few thousand to a few
million elements at a time.

A sort works in place, so a pass sorts a fresh copy of the unsorted arrays (a program that keeps its input
does the same); the copy is part of the pass.
"""
import math

import numpy as np
import torch

import thrust_b200 as tb
from thrust_b200 import _capi as capi

DEVICE = "cuda:0"

# storage dtype of a tensor, code passed to the library, bytes
_KEYS = {
    "u8": (torch.uint8, capi.U8, 1), "i16": (torch.int16, capi.I16, 2),
    "i32": (torch.int32, capi.I32, 4), "u32": (torch.int32, capi.U32, 4),
    "i64": (torch.int64, capi.I64, 8), "u64": (torch.int64, capi.U64, 8),
    "f32": (torch.float32, capi.F32, 4), "f64": (torch.float64, capi.F64, 8),
}
_BITS = {"u8": (0, 255), "i16": (-2**15, 2**15 - 1), "i32": (-2**31, 2**31 - 1), "u32": (-2**31, 2**31 - 1),
         "i64": (-2**63, 2**63 - 1), "u64": (-2**63, 2**63 - 1)}


def listed():
    return [
        # thrust::sort of int32 keys, the first benchmark configuration
        dict(name="sort_i32_32m", op="sort", n=1 << 25, key="i32", val="none", dist="uniform", descending=False),
        # stable sort_by_key of 64-bit keys with 32-bit payload: the large benchmark configuration
        dict(name="sort_pairs_u64_256m", op="sort", n=1 << 28, key="u64", val="i32", dist="uniform", descending=False),
        # float keys with low entropy and heavy duplicates, index payload; an odd size
        dict(name="sort_pairs_f32_and3_64m", op="sort", n=67_000_003, key="f32", val="i32", dist="and3",
             descending=False),
        # ranking a million scores, highest first, with 64-bit row numbers
        dict(name="sort_pairs_f32_desc_1m", op="sort", n=1_000_003, key="f32", val="i64", dist="normal",
             descending=True),
        # the smallest sorts: a few thousand ids with an index, where launches and latency are the cost
        dict(name="sort_pairs_i32_4k", op="sort", n=4096, key="i32", val="i32", dist="uniform", descending=False),
        # streaming prefix sum
        dict(name="scan_f32_256m", op="scan", n=1 << 28, dtype="f32", exclusive=False, sync=True),
        # offsets of ragged rows: counts to start positions, enqueued without waiting
        dict(name="scan_i64_100k", op="scan", n=100_003, dtype="i64", exclusive=True, sync=False),
        # grouped sums, runs of mean length 16
        dict(name="reduce_by_key_64m", op="reduce_by_key", n=1 << 26, val="f32", run=16),
        # prefix sums that restart in every group
        dict(name="scan_by_key_10m", op="scan_by_key", n=10_000_019, val="f32", run=16, exclusive=True),
        # one representative per group of a small sorted table
        dict(name="unique_by_key_50k", op="unique_by_key", n=50_021, val="i32", run=5),
        # stream compaction with a byte mask, half selected
        dict(name="copy_flagged_32m", op="copy_flagged", n=33_554_467, val="f32", share=0.5),
        # the dense-histogram recipe: copy, sort, search, difference; 65536 bins, Zipf keys
        dict(name="histogram_zipf_16m", op="histogram", n=1 << 24, key="f32", bins=1 << 16, dist="zipf"),
    ]


def _size(rng, low, high):
    n = int(math.exp(rng.uniform(math.log(low), math.log(high))))
    # half of the sizes as they fall, a quarter odd, a quarter multiples of 1024
    pick = rng.random()
    if pick < 0.25:
        n |= 1
    elif pick < 0.5 and n > 2048:
        n -= n % 1024
    return n


def draw(rng):
    op = rng.choice(["sort", "sort", "sort", "sort", "scan", "reduce", "reduce_by_key", "scan_by_key",
                     "unique_by_key", "copy_flagged", "histogram"])
    if op == "sort":
        key = rng.choice(["i32", "u32", "f32", "u64", "i64", "f64", "i32", "u64", "f32", "i16", "u8"])
        dists = {"f32": ["uniform", "normal", "and3", "zipf"], "f64": ["uniform", "normal"],
                 "i16": ["uniform"], "u8": ["uniform"]}.get(key, ["uniform", "uniform", "and3", "ids", "zipf"])
        return dict(op=op, n=_size(rng, 1000, 1 << 27), key=key, val=rng.choice(["none", "i32", "i32", "i64"]),
                    dist=rng.choice(dists), descending=rng.random() < 0.3)
    if op == "scan":
        return dict(op=op, n=_size(rng, 1000, 1 << 28), dtype=rng.choice(["f32", "i32", "i64", "f64"]),
                    exclusive=rng.random() < 0.5, sync=rng.random() < 0.5)
    if op == "reduce":
        return dict(op=op, n=_size(rng, 1000, 1 << 28), dtype=rng.choice(["f32", "i32", "i64", "u8"]))
    if op == "reduce_by_key":
        return dict(op=op, n=_size(rng, 1000, 1 << 28), val=rng.choice(["f32", "i32", "f64"]),
                    run=rng.choice([2, 16, 16, 200]))
    if op == "scan_by_key":
        return dict(op=op, n=_size(rng, 1000, 1 << 28), val=rng.choice(["f32", "i32", "i64"]),
                    run=rng.choice([2, 16, 16, 200]), exclusive=rng.random() < 0.5)
    if op == "unique_by_key":
        return dict(op=op, n=_size(rng, 1000, 1 << 28), val=rng.choice(["none", "i32", "i64"]),
                    run=rng.choice([2, 5, 16]))
    if op == "copy_flagged":
        return dict(op=op, n=_size(rng, 1000, 1 << 28), val=rng.choice(["f32", "i64"]),
                    share=rng.choice([0.05, 0.5, 0.9]))
    return dict(op=op, n=_size(rng, 1000, 1 << 26), key="f32", bins=rng.choice([256, 4096, 1 << 16]), dist="zipf")


# ---- inputs ------------------------------------------------------------------------------------
def _generator(seed):
    g = torch.Generator(device=DEVICE)
    g.manual_seed(seed)
    return g


def _words(n, key, g):
    """Uniform bit patterns of an integer key type."""
    low, high = _BITS[key]
    return torch.randint(low, high, (n,), dtype=_KEYS[key][0], device=DEVICE, generator=g)


def _zipf(n, count, g):
    """Ranks 0..count-1 with probability proportional to 1 / (rank + 1)^1.2."""
    w = 1.0 / torch.arange(1, count + 1, dtype=torch.float64, device=DEVICE) ** 1.2
    cdf = torch.cumsum(w, 0)
    cdf /= cdf[-1].clone()
    u = torch.rand(n, dtype=torch.float64, device=DEVICE, generator=g)
    return torch.searchsorted(cdf, u).clamp_(max=count - 1)


def _table(count, seed):
    """Distinct ascending float32 values: the key values of a Zipf distribution and the bins of its histogram."""
    steps = 0.25 + np.random.default_rng(seed).random(count)
    return torch.from_numpy(np.cumsum(steps).astype(np.float32)).to(DEVICE)


def _keys(case, seed, g):
    n, key, dist = case["n"], case["key"], case["dist"]
    dtype = _KEYS[key][0]
    if dist == "zipf":  # frequent values lie anywhere in the value range
        count = case.get("bins", 1 << 16)
        ranks = torch.randperm(count, device=DEVICE, generator=g)[_zipf(n, count, g)]
        if key == "f32":
            return _table(count, seed)[ranks]
        return ranks.to(dtype)
    if dist == "ids":  # row numbers of a table with sixteen times fewer rows
        return torch.randint(0, max(2, n // 16), (n,), dtype=dtype, device=DEVICE, generator=g)
    if dist == "and3":
        word = {"f32": "u32"}.get(key, key)
        x = _words(n, word, g)
        x &= _words(n, word, g)
        x &= _words(n, word, g)
        if key != "f32":
            return x
        special = (x & 0x7F800000) == 0x7F800000  # infinity and NaN patterns
        return torch.where(special, x & ~0x00800000, x).view(torch.float32)
    if dist == "normal":
        return torch.randn(n, dtype=dtype, device=DEVICE, generator=g)
    if key in ("f32", "f64"):
        return torch.rand(n, dtype=dtype, device=DEVICE, generator=g)
    return _words(n, key, g)


def _numbers(n, dtype, g):
    if dtype in ("f32", "f64"):
        return torch.rand(n, dtype=_KEYS[dtype][0], device=DEVICE, generator=g).mul_(2).sub_(1)
    high = 255 if dtype == "u8" else (100 if dtype == "i32" else 1 << 20)
    return torch.randint(0, high, (n,), dtype=_KEYS[dtype][0], device=DEVICE, generator=g)


def _chosen(n, count, g):
    """A mask of n elements, each set independently, brought to exactly `count` set elements."""
    mask = torch.rand(n, device=DEVICE, generator=g) < count / n
    extra = int(mask.sum()) - count
    if extra:  # flip the surplus (or the deficit) at places spread over the whole mask
        at = torch.nonzero(mask if extra > 0 else ~mask).flatten()
        at = at[::max(1, at.numel() // abs(extra))][:abs(extra)]
        mask[at] = extra < 0
    return mask


def _groups(n, run, g):
    """int32 keys in n // run groups whose lengths are geometric with mean `run`."""
    heads = torch.zeros(n, dtype=torch.bool, device=DEVICE)
    heads[1:] = _chosen(n - 1, n // run - 1, g)
    return torch.cumsum(heads, 0, dtype=torch.int32)


def prepare(case, seed):
    g = _generator(seed)
    n, op = case["n"], case["op"]
    state = {"case": case}
    if op == "sort":
        state["keys"] = _keys(case, seed, g)
        if case["val"] != "none":  # the payload is the element's index
            state["values"] = torch.arange(n, dtype=_KEYS[case["val"]][0], device=DEVICE)
    elif op in ("scan", "reduce"):
        state["input"] = _numbers(n, case["dtype"], g)
    elif op in ("reduce_by_key", "scan_by_key", "unique_by_key"):
        state["keys"] = _groups(n, case["run"], g)
        state["values"] = None if case["val"] == "none" else _numbers(n, case["val"], g)
    elif op == "copy_flagged":
        state["data"] = _numbers(n, case["val"], g)
        state["flags"] = _chosen(n, int(n * case["share"]), g).to(torch.uint8)
    else:
        state["data"] = _keys(case, seed, g)
        state["bins"] = _table(case["bins"], seed)
    return state


# ---- one pass ----------------------------------------------------------------------------------
def run(state):
    case = state["case"]
    op = case["op"]
    if op == "sort":
        keys = state["keys"].clone()
        code = _KEYS[case["key"]][1]
        if "values" not in state:
            tb.sort(keys, descending=case["descending"], key_dtype=code)
            return (keys,)
        values = state["values"].clone()
        tb.sort_by_key(keys, values, descending=case["descending"], key_dtype=code)
        return keys, values
    if op == "scan":
        scan = tb.exclusive_scan if case["exclusive"] else tb.inclusive_scan
        return (scan(state["input"], sync=case["sync"]),)
    if op == "reduce":
        return (tb.reduce(state["input"]),)
    if op == "reduce_by_key":
        keys, sums, runs = tb.reduce_by_key(state["keys"], state["values"])
        return keys[:runs], sums[:runs]
    if op == "scan_by_key":
        scan = tb.exclusive_scan_by_key if case["exclusive"] else tb.inclusive_scan_by_key
        return (scan(state["keys"], state["values"]),)
    if op == "unique_by_key":
        keys, values, count = tb.unique_by_key(state["keys"], state["values"])
        return (keys[:count],) if values is None else (keys[:count], values[:count])
    if op == "copy_flagged":
        out, count = tb.copy_flagged(state["data"], state["flags"])
        return (out[:count],)
    return (tb.dense_histogram(state["data"], state["bins"]),)


# ---- what a pass cannot do without, and how its outputs are judged -----------------------------
def work(case):
    n, op = case["n"], case["op"]

    def width(name):
        return 0 if name == "none" else _KEYS[name][2]

    if op == "sort":
        moved = 2 * n * (width(case["key"]) + width(case["val"]))
    elif op == "scan":
        moved = 2 * n * width(case["dtype"])
    elif op == "reduce":
        moved = n * width(case["dtype"])
    elif op in ("reduce_by_key", "unique_by_key"):
        moved = (n + n // case["run"]) * (4 + width(case["val"]))
    elif op == "scan_by_key":
        moved = n * (4 + 2 * width(case["val"]))
    elif op == "copy_flagged":
        moved = n * (1 + width(case["val"])) + int(n * case["share"]) * width(case["val"])
    else:
        moved = n * width(case["key"]) + case["bins"] * 8
    return {"bytes": moved, "flops": 0}


def tolerance(case):
    op = case["op"]
    kind = case.get("dtype", case.get("val"))
    if op in ("scan", "reduce", "reduce_by_key", "scan_by_key") and kind in ("f32", "f64"):
        # sums of rounded terms in another order
        return {"rel": 1e-5 if kind == "f32" else 1e-13}
    return "exact"  # sorted, selected and counted values; integer sums


def exact(case, seed):
    op = case["op"]
    kind = case.get("dtype", case.get("val"))
    state = prepare(case, seed)
    if op == "sort":
        if case["key"] not in ("f32", "f64"):
            return None
        keys = torch.sort(state["keys"].double(), descending=case["descending"])[0]
        return (keys, None) if "values" in state else (keys,)
    if op in ("scan", "reduce"):
        if kind not in ("f32", "f64"):
            return None
        x = state["input"].double()
        if op == "reduce":
            return (float(x.sum()),)
        total = torch.cumsum(x, 0)
        return (total - x if case["exclusive"] else total,)
    if op in ("reduce_by_key", "scan_by_key"):
        if kind not in ("f32", "f64"):
            return None
        keys, x = state["keys"], state["values"].double()
        total = torch.cumsum(x, 0)
        head = torch.ones_like(keys, dtype=torch.bool)
        head[1:] = keys[1:] != keys[:-1]
        first = torch.nonzero(head).flatten()
        before = total[first] - x[first]  # sum of everything in front of the run
        if op == "scan_by_key":
            run_of = torch.cumsum(head, 0) - 1
            return ((total - x if case["exclusive"] else total) - before[run_of],)
        last = torch.cat([first[1:], first.new_tensor([keys.numel()])]) - 1
        return None, total[last] - before
    return None

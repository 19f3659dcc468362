"""What the framework is timed on: the work a user has it do, through its public entry points.

Each case is one of five operations of the path, over the sizes, element types and options that
programs use: sorting keys, sorting key/value pairs, reduce + scan, histogram, and removing the
duplicates of sorted data.  The listed cases are the benchmark configurations of this repository
(2^26 unsigned keys; 2^28 Zipf pairs; reduce + scan of 2^24 integers and of 2^30 floats; 256 bins
over 2^28 floats) with small, ordinary, ragged and many-bin cases of the same operations around
them; `draw` gives more of the same ranges.

Sorts and the removal of duplicates work in place, so a pass first brings the caller's data into
the working view, as a program does whose next batch arrives there.
"""
import math

import torch

import ilgpu_b200 as ib
from ilgpu_b200 import synthetic

TYPES = {
    "Int8": torch.int8, "UInt8": torch.uint8, "Int16": torch.int16, "UInt16": torch.uint16,
    "Int32": torch.int32, "UInt32": torch.uint32, "Int64": torch.int64, "UInt64": torch.uint64,
    "Half": torch.float16, "Float": torch.float32, "Double": torch.float64,
}
# unsigned types are filled through their signed counterparts
SIGNED = {torch.uint16: torch.int16, torch.uint32: torch.int32, torch.uint64: torch.int64}


def listed():
    return [
        # a few thousand keys: one of many small sorts of a program, where launches are what costs
        {"name": "sort_keys_small", "op": "sort_keys", "type": "UInt32", "n": 5_000, "descending": False, "values": "full"},
        # an ordinary ragged length, signed, largest first
        {"name": "sort_keys_mid", "op": "sort_keys", "type": "Int32", "n": 1_500_001, "descending": True, "values": "full"},
        # the headline benchmark
        {"name": "sort_keys_large", "op": "sort_keys", "type": "UInt32", "n": 1 << 26, "descending": False, "values": "full"},
        # argsort: float scores with the element index as payload
        {"name": "argsort_mid", "op": "sort_pairs", "type": "Float", "value_type": "Int32", "sequence": True, "n": 3_000_017,
         "descending": True, "values": "full"},
        # 64-bit identifiers with heavy duplicates and a payload index
        {"name": "sort_pairs_large", "op": "sort_pairs", "type": "UInt64", "value_type": "UInt32", "sequence": False, "n": 1 << 28,
         "descending": False, "values": "zipf"},
        # counts to offsets: a short list's total, which the host needs to size a buffer, and its prefix sums
        {"name": "reduce_scan_small", "op": "reduce_scan", "type": "Int32", "fold": "Add", "inclusive": False, "n": 10_000,
         "offset": 0, "to_host": True},
        {"name": "reduce_scan_mid", "op": "reduce_scan", "type": "Int32", "fold": "Add", "inclusive": False, "n": 1 << 24,
         "offset": 0, "to_host": False},
        # a sub-view that starts in the middle of its buffer: 64-bit counters, running totals
        {"name": "reduce_scan_subview", "op": "reduce_scan", "type": "Int64", "fold": "Add", "inclusive": True, "n": 5_000_011,
         "offset": 1, "to_host": False},
        {"name": "reduce_scan_large", "op": "reduce_scan", "type": "Float", "fold": "Add", "inclusive": True, "n": 1 << 30,
         "offset": 0, "to_host": False},
        {"name": "histogram_large", "op": "histogram", "type": "Float", "locator": "equal_width", "bins": 256, "n": 1 << 28},
        # one bin for each value of 16-bit samples
        {"name": "histogram_many_bins", "op": "histogram", "type": "Int32", "locator": "modulo", "bins": 65_536, "n": 30_000_001},
        # the step after a sort: each distinct key once
        {"name": "unique_large", "op": "unique", "type": "UInt32", "n": 50_000_017, "distinct": 0.25},
    ]


def _size(rng, least, most):
    return int(math.exp(rng.uniform(math.log(least), math.log(most))))


def draw(rng):
    op = rng.choice(["sort_keys", "sort_pairs", "reduce_scan", "reduce_scan", "histogram", "unique"])
    if op == "sort_keys":
        kind = rng.choice(["UInt32", "Int32", "Float", "UInt64", "Int64", "Double", "UInt16", "Int8", "Half"])
        return {"op": op, "type": kind, "n": _size(rng, 1_000, 1 << 26), "descending": rng.random() < 0.3, "values": _values(rng, kind)}
    if op == "sort_pairs":
        kind = rng.choice(["UInt32", "Int32", "Float", "UInt64", "Int64"])
        sequence = rng.random() < 0.4
        payload = "Int32" if sequence else rng.choice(["Int32", "Float", "Int64", "Double"])
        return {"op": op, "type": kind, "value_type": payload, "sequence": sequence, "n": _size(rng, 1_000, 1 << 26),
                "descending": rng.random() < 0.3, "values": _values(rng, kind)}
    if op == "reduce_scan":
        kind = rng.choice(["Int32", "Float", "Int64", "Double", "UInt32", "UInt64"])
        n = _size(rng, 1_000, 1 << (30 if TYPES[kind].itemsize == 4 else 29))
        return {"op": op, "type": kind, "fold": rng.choice(["Add", "Add", "Max", "Min"]), "inclusive": rng.random() < 0.5, "n": n,
                "offset": rng.choice([0, 0, 1, 3]), "to_host": rng.random() < 0.3}
    if op == "histogram":
        kind = rng.choice(["Float", "Float", "Int32", "UInt32", "Double"])
        locator = "equal_width" if kind in ("Float", "Double") else rng.choice(["equal_width", "modulo"])
        return {"op": op, "type": kind, "locator": locator, "bins": _size(rng, 16, 65_536), "n": _size(rng, 1_000, 1 << 28)}
    return {"op": op, "type": rng.choice(["UInt32", "Int32", "Int64", "Float"]), "n": _size(rng, 1_000, 1 << 27),
            "distinct": round(rng.uniform(0.02, 0.95), 3)}


def _values(rng, kind):
    """"full": over the type's whole range (floats: N(0, 1)); "narrow": identifiers below 2^20, whose upper bytes are
    all zero; "zipf": 64-bit identifiers with heavy duplicates."""
    if TYPES[kind].is_floating_point or TYPES[kind].itemsize < 4:
        return "full"
    return rng.choice(["full", "full", "narrow"] + (["zipf"] if kind == "UInt64" else []))


# ---- inputs --------------------------------------------------------------------------------------
def _keys(case, n, gen, seed):
    dtype = TYPES[case["type"]]
    if dtype.is_floating_point:
        return torch.randn(n, generator=gen, device="cuda", dtype=torch.float32 if dtype == torch.float16 else dtype).to(dtype)
    if case["values"] == "zipf":
        return synthetic.zipf_uint64_device(n, seed, torch.device("cuda"))
    signed = SIGNED.get(dtype, dtype)
    if case["values"] == "narrow":
        return torch.randint(0, 1 << 20, (n,), generator=gen, device="cuda", dtype=signed).view(dtype)
    if signed == torch.uint8:
        return torch.randint(0, 256, (n,), generator=gen, device="cuda", dtype=signed)
    info = torch.iinfo(signed)
    return torch.randint(info.min, info.max, (n,), generator=gen, device="cuda", dtype=signed).view(dtype)


def _numbers(case, n, gen):
    """What is folded: floats of [0, 1); small integers for sums, large ones for extremes."""
    dtype = TYPES[case["type"]]
    if dtype.is_floating_point:
        return torch.rand(n, generator=gen, device="cuda", dtype=dtype)
    return torch.randint(0, 16 if case["fold"] == "Add" else 1 << 30, (n,), generator=gen, device="cuda", dtype=SIGNED.get(dtype, dtype)).view(dtype)


def _samples(case, n, gen):
    """What is counted: N(0, 1), or bell-shaped 16-bit samples."""
    dtype = TYPES[case["type"]]
    if dtype.is_floating_point:
        return torch.randn(n, generator=gen, device="cuda", dtype=dtype)
    bell = torch.randn(n, generator=gen, device="cuda").mul_(8_000.0).add_(32_768.0).clamp_(0.0, 65_535.0)
    return bell.to(torch.int32).view(dtype)


def _distinct(case):
    return max(1, int(case["n"] * case["distinct"]))


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    acc = ib.Accelerator(0)
    n, dtype = case["n"], TYPES[case["type"]]
    state = {"case": case, "acc": acc}
    if case["op"] in ("sort_keys", "sort_pairs"):
        operation = getattr(ib.RadixSortOperations, ("Descending" if case["descending"] else "Ascending") + case["type"])
        total_order = dtype.is_floating_point  # by value, negative numbers first
        state["keys"] = _keys(case, n, gen, seed)
        state["sorted"] = torch.empty_like(state["keys"])
        if case["op"] == "sort_keys":
            state["temp"] = acc.Allocate1D(acc.ComputeRadixSortTempStorageSize(operation, n), torch.int32)
            state["sort"] = acc.CreateRadixSort(operation, total_order)
            return state
        payload = TYPES[case["value_type"]]
        state["temp"] = acc.Allocate1D(acc.ComputeRadixSortPairsTempStorageSize(operation, payload, n), torch.int32)
        state["sorted_values"] = acc.Allocate1D(n, payload)
        if case["sequence"]:
            state["sequencer"] = getattr(ib.Sequencers, case["value_type"] + "Sequencer")
            state["sort"] = acc.CreateRadixSortPairs(operation, total_order, sequencer=ib.Sequencers)
        else:
            state["values"] = torch.arange(n, device="cuda", dtype=SIGNED.get(payload, payload)).view(payload)
            state["sort"] = acc.CreateRadixSortPairs(operation, total_order)
    elif case["op"] == "reduce_scan":
        state["fold"] = getattr(ib.ScanReduceOperations, case["fold"] + case["type"])
        state["input"] = _numbers(case, n + case["offset"], gen)[case["offset"]:]
        state["output"] = acc.Allocate1D(n + case["offset"], dtype)[case["offset"]:]
        state["total"] = acc.Allocate1D(1, dtype)
        provider = acc.CreateScanProvider(dtype, n)
        state["scan"] = provider.CreateScan(state["fold"], ib.ScanKind.Inclusive if case["inclusive"] else ib.ScanKind.Exclusive)
    elif case["op"] == "histogram":
        state["input"] = _samples(case, n, gen)
        state["bins"] = acc.Allocate1D(case["bins"], torch.int32)
        state["overflow"] = acc.Allocate1D(1, torch.int32)
        if case["locator"] == "modulo":
            locator = ib.ModuloLocator()
        else:
            locator = ib.EqualWidthClampLocator(-4.0, 4.0) if dtype.is_floating_point else ib.EqualWidthClampLocator(0.0, 65_536.0)
        state["histogram"] = acc.CreateHistogram(locator)
    else:
        # runs of random lengths; a few starts more than wanted, so that the last wanted run takes in what is left
        wanted = _distinct(case)
        share = (wanted + 5.0 * math.sqrt(wanted)) / n
        starts = torch.rand(n, generator=gen, device="cuda").lt_(share).to(torch.int32)
        starts[0] = 1
        runs = torch.cumsum(starts, 0, dtype=torch.int32).clamp_(max=wanted)
        values = torch.randint(0, 8, (wanted + 1,), generator=gen, device="cuda", dtype=torch.int32)
        runs = 8 * runs + values[runs]
        if dtype == torch.float32:
            state["data"] = (runs + 0x3F800000).view(dtype)  # ascending bit patterns from 1.0 on: a value of its own for each run
        else:
            state["data"] = runs.to(SIGNED.get(dtype, dtype)).view(dtype)
        state["distinct"] = torch.empty_like(state["data"])
    return state


def _shown(view):
    """Unsigned results as the signed integers of the same bits, which more of torch can work with."""
    return view.view(SIGNED[view.dtype]) if view.dtype in SIGNED else view


# ---- one pass ------------------------------------------------------------------------------------
def run(state):
    case, acc = state["case"], state["acc"]
    if case["op"] == "sort_keys":
        state["sorted"].copy_(state["keys"])
        state["sort"](None, state["sorted"], state["temp"])
        return _shown(state["sorted"])
    if case["op"] == "sort_pairs":
        state["sorted"].copy_(state["keys"])
        if case["sequence"]:
            state["sort"](None, state["sorted"], state["sorted_values"], state["sequencer"], state["temp"])
        else:
            state["sorted_values"].copy_(state["values"])
            state["sort"](None, state["sorted"], state["sorted_values"], state["temp"])
        return _shown(state["sorted"]), _shown(state["sorted_values"])
    if case["op"] == "reduce_scan":
        if case["to_host"]:
            total = acc.Reduce(None, state["input"], state["fold"])
        else:
            total = state["total"]
            acc.Reduce(None, state["input"], state["fold"], total)
        state["scan"](None, state["input"], state["output"])
        return (total if case["to_host"] else _shown(total)), _shown(state["output"])
    if case["op"] == "histogram":
        acc.Initialize(None, state["bins"], 0)
        acc.Initialize(None, state["overflow"], 0)
        state["histogram"](None, state["input"], state["bins"], state["overflow"])
        return state["bins"], state["overflow"]
    state["distinct"].copy_(state["data"])
    count = acc.Unique(None, state["distinct"])
    return count, _shown(state["distinct"][:count])


# ---- what a pass cannot do without ---------------------------------------------------------------
def work(case):
    n, size = case["n"], TYPES[case["type"]].itemsize
    if case["op"] == "sort_keys":
        return {"bytes": 2 * n * size, "flops": 0}
    if case["op"] == "sort_pairs":
        payload = TYPES[case["value_type"]].itemsize
        return {"bytes": 2 * n * size + (1 if case["sequence"] else 2) * n * payload, "flops": 0}
    if case["op"] == "reduce_scan":
        return {"bytes": 3 * n * size, "flops": 2 * n}  # two calls, each reads its input
    if case["op"] == "histogram":
        return {"bytes": n * size + case["bins"] * 4, "flops": 0}
    return {"bytes": (n + _distinct(case)) * size, "flops": 0}


def tolerance(case):
    """Sorted data, counts and integer folds are exact; floating-point folds depend on the order of the additions."""
    if case["op"] == "reduce_scan" and case["type"] == "Float":
        return {"rel": 1e-5}
    if case["op"] == "reduce_scan" and case["type"] == "Double":
        return {"rel": 1e-12}
    return "exact"

"""Calls captured into a CUDA graph.  Most of them start as programmatic dependents of whatever comes before them on the
stream, so each is captured behind a copy, a memset, an event of another stream, a foreign kernel and another call
of the library that make its input, twice over the same views with a copy of the result behind each, and the graph is
replayed on new data: a call that started too early, or let its successor start too early, would read or leave
the data of the other round or replay."""
import ctypes

import numpy as np
import pytest
import torch

from ilgpu_b200 import ModuloLocator, RadixSortOperations, ScanKind, ScanReduceOperations
from ilgpu_b200 import _native as N

pytestmark = pytest.mark.gpu


def _sequence(vals):
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert N.lib().b200alg_sequence(stream, ctypes.c_void_p(vals.data_ptr()), vals.numel(), N.I32, 0, 1) == N.OK


def _sort(acc, name, n, values=False):
    op = getattr(RadixSortOperations, "Ascending" + name)
    dtype = {"Int32": torch.int32, "Int64": torch.int64, "Double": torch.float64}[name]
    view = torch.zeros(n, dtype=dtype, device="cuda")
    temp = acc.Allocate1D(acc.ComputeRadixSortPairsTempStorageSize(op, torch.int32, n), torch.int32)
    if not values:
        sort = acc.CreateRadixSort(op, True)
        return view, lambda: sort(None, view, temp), [view], lambda a: [np.sort(a)]
    vals = torch.zeros(n, dtype=torch.int32, device="cuda")
    sort = acc.CreateRadixSortPairs(op, True)

    def call():
        _sequence(vals)
        sort(None, view, vals, temp)
    return view, call, [view, vals], lambda a: [np.sort(a), np.argsort(a, kind="stable").astype(np.int32)]


def _reduce(acc, n):
    view, out = torch.zeros(n, dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    return view, lambda: acc.Reduce(None, view, ScanReduceOperations.AddInt32, out), [out], lambda a: [a.sum(dtype=np.int32, keepdims=True)]


def _scan(acc, n, kind):
    view, out = (torch.zeros(n, dtype=torch.int32, device="cuda") for _ in range(2))
    temp = acc.Allocate1D(acc.ComputeScanTempStorageSize(torch.int32, n), torch.int32)
    scan = acc.CreateScan(ScanReduceOperations.AddInt32, kind)
    inclusive = lambda a: np.cumsum(a, dtype=np.int32)
    return (view, lambda: scan(None, view, out, temp), [out],
            lambda a: [inclusive(a) if kind == ScanKind.Inclusive else np.concatenate([[0], inclusive(a)[:-1]]).astype(np.int32)])


def _histogram(acc, n, bins):
    view = torch.zeros(n, dtype=torch.int32, device="cuda")
    counts, overflow = torch.zeros(bins, dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    histogram = acc.CreateHistogram(ModuloLocator())

    def call():
        acc.Initialize(None, counts, 0)
        acc.Initialize(None, overflow, 0)
        histogram(None, view, counts, overflow)
    return view, call, [counts, overflow], lambda a: [np.bincount(a % bins, minlength=bins).astype(np.int32), np.zeros(1, np.int32)]


def _unique(acc, n):
    view, count = torch.zeros(n, dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.int64, device="cuda")
    need = ctypes.c_int64(0)
    assert N.lib().b200alg_unique_temp_bytes(N.I32, n, ctypes.byref(need)) == N.OK
    temp = torch.empty(need.value, dtype=torch.uint8, device="cuda")
    p = lambda t: ctypes.c_void_p(t.data_ptr())

    def call():
        stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        assert N.lib().b200alg_unique(stream, p(view), n, N.I32, p(count), p(temp), need.value) == N.OK
    return view, call, [count], lambda a: [np.array([1 + np.count_nonzero(np.diff(a))])]


CALLS = {
    "one block": lambda acc: _sort(acc, "Int32", 5_000),
    "a cluster": lambda acc: _sort(acc, "Int32", 30_000),
    "buckets in a cluster": lambda acc: _sort(acc, "Double", 20_000),
    "a grid": lambda acc: _sort(acc, "Int32", 300_000),
    "buckets": lambda acc: _sort(acc, "Int64", 200_001, True),
    "passes": lambda acc: _sort(acc, "Int32", 2_000_003, True),
    "short reduce": lambda acc: _reduce(acc, 10_000),
    "reduce": lambda acc: _reduce(acc, 3_000_001),
    "short scan": lambda acc: _scan(acc, 10_000, ScanKind.Exclusive),
    "scan in a cluster": lambda acc: _scan(acc, 60_000, ScanKind.Inclusive),
    "scan": lambda acc: _scan(acc, 3_000_001, ScanKind.Exclusive),
    "few bins": lambda acc: _histogram(acc, 400_001, 256),
    "many bins": lambda acc: _histogram(acc, 400_001, 65_536),
    "unique": lambda acc: _unique(acc, 1_000_003),
}


@pytest.mark.parametrize("behind", ["copy", "memset", "event", "kernel", "call"])
@pytest.mark.parametrize("name", list(CALLS))
def test_replays(accelerator, name, behind):
    view, call, outputs, expected = CALLS[name](accelerator)
    n, half = view.numel(), view.numel() // 2
    sources = [torch.empty_like(view) for _ in range(2)]
    results = [[torch.empty_like(o) for o in outputs] for _ in range(2)]

    def fill(source):   # what the call finds in its view, behind something else
        if behind == "event":
            here, side = torch.cuda.current_stream(), torch.cuda.Stream()
            side.wait_stream(here)
            with torch.cuda.stream(side):
                view.copy_(source)
            here.wait_stream(side)
        elif behind == "kernel":
            torch.add(source, source, out=view)
        else:
            view.copy_(source)
            if behind == "memset":
                view[half:].zero_()
            elif behind == "call":
                accelerator.Initialize(None, view[half:], 3)

    def rounds():
        for source, kept in zip(sources, results):
            fill(source)
            call()
            for k, o in zip(kept, outputs):
                k.copy_(o)

    def found(a):
        a = a.copy()
        if behind == "memset":
            a[half:] = 0
        elif behind == "call":
            a[half:] = 3
        return a + a if behind == "kernel" else a

    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        rounds()
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        rounds()
    rng = np.random.default_rng(n)
    for replay in range(3):
        inputs = []
        for source in sources:
            a = rng.integers(0, 1 << (60 if source.itemsize == 8 else 20), size=n).astype(source.cpu().numpy().dtype)
            source.copy_(torch.from_numpy(a))
            inputs.append(a)
        graph.replay()
        torch.cuda.synchronize()
        for a, kept in zip(inputs, results):
            for want, got in zip(expected(found(a)), kept):
                np.testing.assert_array_equal(got.cpu().numpy(), want)

"""The mirror's calls without their native host path (_host.so): the same results through algorithms.py."""
import numpy as np
import pytest
import torch

import ilgpu_b200 as ib
from ilgpu_b200 import _native as N

pytestmark = pytest.mark.gpu


@pytest.fixture
def plain(monkeypatch):
    monkeypatch.setattr(N, "_host", N._NoHostPath())
    return ib.Accelerator(0)


@pytest.mark.parametrize("n", [1, 5000, 300_001])
def test_every_call(plain, n):
    rng = np.random.default_rng(n)
    host = rng.integers(-1000, 1000, size=n).astype(np.int32)
    order = np.argsort(host, kind="stable")
    op = ib.RadixSortOperations.AscendingInt32

    keys = torch.from_numpy(host).cuda()
    temp = plain.Allocate1D(plain.ComputeRadixSortTempStorageSize(op, n), torch.int32)
    plain.CreateRadixSort(op)(None, keys, temp)
    np.testing.assert_array_equal(keys.cpu().numpy(), host[order])

    temp = plain.Allocate1D(plain.ComputeRadixSortPairsTempStorageSize(op, torch.int32, n), torch.int32)
    for sequencer in (None, ib.Sequencers):
        keys = torch.from_numpy(host).cuda()
        values = torch.arange(n, dtype=torch.int32, device="cuda")
        sort = plain.CreateRadixSortPairs(op, sequencer=sequencer)
        sort(None, keys, values, *([] if sequencer is None else [ib.Sequencers.Int32Sequencer]), temp)
        np.testing.assert_array_equal(values.cpu().numpy(), order)

    data = torch.from_numpy(host).cuda()
    add = ib.ScanReduceOperations.AddInt32
    out = torch.empty_like(data)
    plain.CreateScanProvider(torch.int32, n).CreateScan(add, ib.ScanKind.Inclusive)(None, data, out)
    np.testing.assert_array_equal(out.cpu().numpy(), np.cumsum(host, dtype=np.int32))
    assert plain.Reduce(None, data, add) == int(host.sum())
    total = torch.zeros(1, dtype=torch.int32, device="cuda")
    plain.Reduce(None, data, add, total)
    assert total.item() == int(host.sum())

    bins = torch.empty(16, dtype=torch.int32, device="cuda")
    overflow = torch.empty(1, dtype=torch.int32, device="cuda")
    plain.Initialize(None, bins, 0)
    plain.Initialize(None, overflow, 0)
    samples = np.abs(host)
    plain.Histogram(None, torch.from_numpy(samples).cuda(), bins, overflow, ib.ModuloLocator())
    np.testing.assert_array_equal(bins.cpu().numpy(), np.bincount(samples % 16, minlength=16))
    assert overflow.item() == 0

    ordered = torch.from_numpy(host[order]).cuda()
    count = plain.Unique(None, ordered)
    np.testing.assert_array_equal(ordered[:count].cpu().numpy(), np.unique(host))


def test_values_that_come_back_wait_for_their_stream(plain):
    data = torch.arange(100_001, dtype=torch.int64, device="cuda")
    add, side = ib.ScanReduceOperations.AddInt64, torch.cuda.Stream()
    torch.cuda.synchronize()
    for _ in range(3):
        marker = torch.full((1,), -1, dtype=torch.int64, device="cuda")   # what the result's memory holds before
        del marker
        torch.cuda.synchronize()
        with torch.cuda.stream(side):
            torch.cuda._sleep(20_000_000)   # some 10 ms in front of the call
        assert plain.Reduce(side, data, add) == 100_000 * 100_001 // 2
        with torch.cuda.stream(side):
            torch.cuda._sleep(20_000_000)
        assert plain.Unique(side, data) == 100_001
        with torch.cuda.stream(side):
            torch.cuda._sleep(20_000_000)
        assert plain.Unique(side, data[:0]) == 0

"""Sorts in one launch (a block, a cluster, a grid): lengths around the places where the number of
blocks or the way they meet changes, for every key and value size; keys that differ in few digits or
in none; strided and out-of-place sorts; against a stable host sort."""
import ctypes

import numpy as np
import pytest
import torch

from ilgpu_b200 import RadixSortOperations, Sequencers
from ilgpu_b200 import _native as N
from tests.helpers import NP

pytestmark = pytest.mark.gpu

LENGTHS = [1, 2, 511, 513, 4095, 4096, 4097, 6143, 6144, 6145, 8193, 16_385, 40_960, 40_961, 65_537, 131_073, 300_001]


def _keys(rng, dtype, n, kind):
    info = np.iinfo(dtype)
    if kind == "one":
        return np.full(n, 7, dtype)
    keys = rng.integers(info.min, info.max, size=n, dtype=dtype, endpoint=True)
    return keys if kind == "full" else (keys & dtype(0x70)).astype(dtype)   # four low bits and all bytes above the first agree


def _pairs(acc, name, keys, values, descending=False):
    op = getattr(RadixSortOperations, ("Descending" if descending else "Ascending") + name)
    dev, vals = torch.from_numpy(keys).cuda(), torch.from_numpy(values).cuda()
    temp = acc.Allocate1D(acc.ComputeRadixSortPairsTempStorageSize(op, vals.dtype, keys.size), torch.int32)
    acc.CreateRadixSortPairs(op)(None, dev, vals, temp)
    acc.CheckDeviceStatus(None, temp)
    return dev.cpu().numpy(), vals.cpu().numpy()


@pytest.mark.parametrize("n", LENGTHS + [786_432, 786_433, 1_048_576, 1_048_577])
@pytest.mark.parametrize("name", ["UInt8", "Int16", "UInt32", "Int64"])
@pytest.mark.parametrize("kind", ["full", "few", "one"])
def test_keys(accelerator, name, n, kind):
    keys = _keys(np.random.default_rng(n), NP[name], n, kind)
    for descending in (False, True):
        op = getattr(RadixSortOperations, ("Descending" if descending else "Ascending") + name)
        dev = torch.from_numpy(keys).cuda()
        temp = accelerator.Allocate1D(accelerator.ComputeRadixSortTempStorageSize(op, n), torch.int32)
        accelerator.CreateRadixSort(op)(None, dev, temp)
        accelerator.CheckDeviceStatus(None, temp)
        expected = np.sort(keys)
        np.testing.assert_array_equal(dev.cpu().numpy(), expected[::-1] if descending else expected)


@pytest.mark.parametrize("n", LENGTHS + [786_432])
@pytest.mark.parametrize("name,value", [("UInt8", np.uint8), ("UInt32", np.int32), ("UInt32", np.float64), ("Int64", np.int16),
                                        ("UInt64", np.uint32), ("UInt64", np.int64)])
@pytest.mark.parametrize("kind", ["full", "few", "one"])
def test_pairs_are_stable(accelerator, name, value, n, kind):
    keys = _keys(np.random.default_rng(n + 1), NP[name], n, kind)
    values = np.arange(n).astype(value)
    order = np.argsort(keys, kind="stable")
    got, got_values = _pairs(accelerator, name, keys, values)
    np.testing.assert_array_equal(got, keys[order])
    np.testing.assert_array_equal(got_values, values[order])


@pytest.mark.parametrize("n", [3000, 20_000, 100_000])
def test_sequenced_and_strided(accelerator, n):
    rng = np.random.default_rng(n)
    keys = rng.integers(0, 50, size=n, dtype=np.uint32)
    op = RadixSortOperations.DescendingUInt32
    dev, vals = torch.from_numpy(keys).cuda(), torch.zeros(n, dtype=torch.int32, device="cuda")
    temp = accelerator.Allocate1D(accelerator.ComputeRadixSortPairsTempStorageSize(op, vals.dtype, n), torch.int32)
    accelerator.CreateRadixSortPairs(op, sequencer=Sequencers)(None, dev, vals, Sequencers.Int32Sequencer, temp)
    np.testing.assert_array_equal(vals.cpu().numpy(), np.argsort(~keys, kind="stable"))

    storage = torch.from_numpy(np.repeat(keys, 3)).cuda()
    accelerator.CreateRadixSort(op)(None, storage[::3], temp)
    np.testing.assert_array_equal(storage.cpu().numpy()[::3], np.sort(keys)[::-1])
    np.testing.assert_array_equal(storage.cpu().numpy()[1::3], keys)   # what lies between stays


@pytest.mark.parametrize("n", [3000, 20_000, 100_000])
def test_out_of_place_with_a_count_on_the_device(n):
    L, rng = N.lib(), np.random.default_rng(n)
    keys, values = rng.integers(0, 1 << 40, size=n, dtype=np.uint64), np.arange(n, dtype=np.uint32)
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    need = ctypes.c_int64(0)
    assert L.b200alg_radix_sort_temp_bytes(N.U64, n, 4, ctypes.byref(need)) == N.OK
    temp = torch.empty(need.value, dtype=torch.uint8, device="cuda")
    k, v = torch.from_numpy(keys).cuda(), torch.from_numpy(values).cuda()
    for m in (n, n - 777, 5, 0):
        ok, ov = torch.full((n,), 9, dtype=torch.int64, device="cuda"), torch.full((n,), 9, dtype=torch.int32, device="cuda")
        count = torch.tensor([m], dtype=torch.int64, device="cuda")
        assert L.b200alg_radix_sort_out_of_place(None, p(k), p(v), p(ok), p(ov), n, p(count), N.U64, 4, 0, p(temp), need.value) == N.OK
        torch.cuda.synchronize()
        order = np.argsort(keys[:m], kind="stable")
        np.testing.assert_array_equal(ok.cpu().numpy()[:m].view(np.uint64), keys[:m][order])
        np.testing.assert_array_equal(ov.cpu().numpy()[:m], order)
        assert (ok.cpu().numpy()[m:] == 9).all() and (ov.cpu().numpy()[m:] == 9).all()
        np.testing.assert_array_equal(k.cpu().numpy().view(np.uint64), keys)

"""The sort that one block does alone: lengths around its thread counts and its largest, ranges of keys that
need no, one, two or three digits, keys that agree in the digits but not below them (few, many, all but one),
keys that agree in their lowest bits and whole numbers kept as floating-point, against a stable host sort."""
import numpy as np
import pytest
import torch

from ilgpu_b200 import RadixSortOperations
from tests.helpers import NP

pytestmark = pytest.mark.gpu


def _keys(rng, dtype, n, kind):
    bits = np.dtype(dtype).itemsize * 8
    keys = rng.integers(0, 1 << bits, size=n, dtype=f"u{bits // 8}")
    if kind == "ties":       # groups of a few neighbours, apart only in the lowest bits
        keys[1::3] = keys[: keys[1::3].size] ^ 1
    elif kind == "outlier":  # one distant key: all others agree in the upper bits
        keys &= 0x7F if bits == 8 else 0x3FF
        keys[n // 2] = (1 << bits) - 1
    elif kind != "full":     # that many bits, away from zero
        keys = (keys & ((1 << int(kind)) - 1)) + 3
    return keys.astype(f"u{bits // 8}").view(dtype)


@pytest.mark.parametrize("n", [1, 2, 33, 256, 257, 1024, 1025, 6144, 6145, 7680, 7681, 9728, 11_777, 12_288, 12_289])
@pytest.mark.parametrize("name,kind", [(name, kind) for name in ["UInt8", "Int16", "UInt32", "Int32", "UInt64", "Int64"]
                                       for kind in ["full", "ties", "outlier", "0", "1", "9", "10", "18", "19", "27", "28"]
                                       if not kind.isdigit() or int(kind) < np.dtype(NP[name]).itemsize * 8])
def test_against_a_stable_sort(accelerator, name, n, kind):
    dtype = NP[name]
    keys = _keys(np.random.default_rng(n), dtype, n, kind)
    order = np.argsort(keys, kind="stable")
    op = getattr(RadixSortOperations, "Ascending" + name)
    dev = torch.from_numpy(keys).cuda()
    temp = accelerator.Allocate1D(accelerator.ComputeRadixSortPairsTempStorageSize(op, torch.int64, n), torch.int32)
    accelerator.CreateRadixSort(op)(None, dev, temp)
    np.testing.assert_array_equal(dev.cpu().numpy(), keys[order])
    for value in (np.uint8, np.int32, np.int64):
        dev, vals = torch.from_numpy(keys).cuda(), torch.from_numpy(np.arange(n).astype(value)).cuda()
        accelerator.CreateRadixSortPairs(op)(None, dev, vals, temp)
        np.testing.assert_array_equal(dev.cpu().numpy(), keys[order])
        np.testing.assert_array_equal(vals.cpu().numpy(), order.astype(value))
    accelerator.CheckDeviceStatus(None, temp)


def _check(acc, keys, value, descending):
    name = {v: k for k, v in NP.items()}[keys.dtype.type]
    floating = keys.dtype.kind == "f"
    order = np.argsort((-keys if floating else ~keys) if descending else keys, kind="stable")
    op = getattr(RadixSortOperations, ("Descending" if descending else "Ascending") + name)
    dev = torch.from_numpy(keys).cuda()
    temp = acc.Allocate1D(acc.ComputeRadixSortPairsTempStorageSize(op, torch.int64, keys.size), torch.int32)
    if value is None:
        acc.CreateRadixSort(op, floating)(None, dev, temp)
    else:
        vals = torch.from_numpy(np.arange(keys.size).astype(value)).cuda()
        acc.CreateRadixSortPairs(op, floating)(None, dev, vals, temp)
        np.testing.assert_array_equal(vals.cpu().numpy(), order.astype(value))
    acc.CheckDeviceStatus(None, temp)
    np.testing.assert_array_equal(dev.cpu().numpy(), keys[order])


# bits that differ (the lowest and the highest among them) above `zeros` bits that are the same in all keys
@pytest.mark.parametrize("n", [2, 31, 513, 1500, 6001, 6656])
@pytest.mark.parametrize("name", ["UInt16", "UInt32", "UInt64", "Int64"])
@pytest.mark.parametrize("differing", [1, 9, 10, 27, 28, 40])
@pytest.mark.parametrize("zeros", [1, 4, 15, 31, 36, 63])
def test_lowest_bits_agree(accelerator, n, name, differing, zeros):
    dtype = np.dtype(NP[name])
    width = dtype.itemsize * 8
    zeros, differing = min(zeros, width - 1), min(differing, width - min(zeros, width - 1))
    unsigned = np.dtype(f"u{dtype.itemsize}").type
    rng = np.random.default_rng(n + zeros)
    top = rng.integers(0, 1 << differing, size=n, dtype=unsigned)
    top[0], top[n - 1] = 0, (1 << differing) - 1
    keys = ((top << unsigned(zeros)) ^ unsigned(0x5A5A5A5A5A5A5A5A & ((1 << width) - 1))).view(dtype)
    for value in (None, np.int32):
        _check(accelerator, keys, value, descending=n % 2 == 1)


@pytest.mark.parametrize("n", [33, 5000, 6656, 6657, 7168, 7169, 8704, 8705, 9216, 9217, 12_288])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("value", [None, np.int32, np.int64])
@pytest.mark.parametrize("least,most", [(0, 2), (0, 256), (-300, 300), (1, 1 << 16), (0, 1 << 21)])
def test_whole_numbers(accelerator, n, dtype, value, least, most):
    keys = np.random.default_rng(n).integers(least, most, size=n).astype(dtype)
    _check(accelerator, keys, value, descending=most == 256)

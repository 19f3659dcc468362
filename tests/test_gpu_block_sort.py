"""The sort that one block does alone: lengths around its thread counts and its largest, ranges of keys that
need no, one, two or three digits, keys that agree in the digits but not below them (few, many, all but one),
against a stable host sort."""
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

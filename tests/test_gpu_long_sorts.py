"""Sorts that are too long for one launch, so that the digit pass makes them: a count in device memory
that leaves it one to three tiles, more or less a key; keys that arrive in order, backwards, almost in
order, or with few values; views that do not start on 16 bytes and strided ones; against a stable host
sort."""
import ctypes

import numpy as np
import pytest
import torch

from ilgpu_b200 import RadixSortOperations
from ilgpu_b200 import _native as N
from ilgpu_b200.algorithms import dtype_code
from tests.helpers import NP, PASSES_WORD, to_device, to_host
from tests.test_gpu_digit_pass import TILES

pytestmark = pytest.mark.gpu

LONG = 1_600_003   # keys; one launch sorts up to 1.55 * 10^6 on 148 SMs


def _went_by_passes(temp):
    return int(temp.view(torch.int32)[PASSES_WORD]) != 0


@pytest.mark.parametrize("name,value", list(TILES))
@pytest.mark.parametrize("tiles,extra", [(0, 1), (1, -1), (1, 0), (1, 1), (2, 0), (2, 1), (3, 0)])
def test_few_tiles(name, value, tiles, extra):
    count = tiles * TILES[name, value] + extra
    rng = np.random.default_rng(count)
    info = np.iinfo(NP[name])
    keys = rng.integers(info.min, info.max, size=LONG, dtype=NP[name], endpoint=True)
    values = None if value is None else np.arange(LONG).astype(value)
    dk, ok, dn = to_device(keys), to_device(np.zeros_like(keys)), torch.tensor([count], device="cuda")
    dv, ov = (None, None) if value is None else (to_device(values), to_device(np.zeros_like(values)))
    vb = 0 if value is None else values.itemsize
    need = ctypes.c_int64(0)
    assert N.lib().b200alg_radix_sort_temp_bytes(dtype_code(dk.dtype), LONG, vb, ctypes.byref(need)) == N.OK
    temp = torch.zeros(need.value, dtype=torch.uint8, device="cuda")
    p = lambda t: ctypes.c_void_p(0 if t is None else t.data_ptr())
    assert N.lib().b200alg_radix_sort_out_of_place(None, p(dk), p(dv), p(ok), p(ov), LONG, p(dn), dtype_code(dk.dtype), vb, 0, p(temp),
                                                   need.value) == N.OK
    assert N.lib().b200alg_device_status(None, p(temp)) == N.OK and _went_by_passes(temp)
    order = np.argsort(keys[:count], kind="stable")
    got = to_host(ok)
    np.testing.assert_array_equal(got[:count], keys[:count][order])
    assert not got[count:].any()
    if value is not None:
        got = to_host(ov)
        np.testing.assert_array_equal(got[:count], values[:count][order])
        assert not got[count:].any()


def _arriving(kind, dtype, n):
    rng = np.random.default_rng(n)
    info = np.iinfo(dtype)
    keys = np.sort(rng.integers(info.min, info.max, size=n, dtype=dtype, endpoint=True))
    if kind == "backwards":
        return keys[::-1].copy()
    if kind == "almost":
        at = rng.integers(0, n, size=n // 100)
        keys[at] = rng.integers(info.min, info.max, size=at.size, dtype=dtype, endpoint=True)
    elif kind == "counting":
        keys = (np.arange(n) % info.max).astype(dtype)
    elif kind == "two":
        keys = rng.choice(np.array([info.min, info.max], dtype), size=n)
    elif kind == "one":
        keys[:] = 5
    return keys


@pytest.mark.parametrize("name", ["UInt16", "UInt32", "Int64"])
@pytest.mark.parametrize("kind", ["in order", "backwards", "almost", "counting", "two", "one"])
@pytest.mark.parametrize("descending", [False, True])
def test_arriving(accelerator, name, kind, descending):
    keys = _arriving(kind, NP[name], LONG)
    op = getattr(RadixSortOperations, ("Descending" if descending else "Ascending") + name)
    # a stable descending sort: the reverse of the stable ascending sort of the reverse
    order = LONG - 1 - np.argsort(keys[::-1], kind="stable")[::-1] if descending else np.argsort(keys, kind="stable")
    view = to_device(keys)
    temp = accelerator.Allocate1D(accelerator.ComputeRadixSortTempStorageSize(op, LONG), torch.int32).zero_()
    accelerator.CreateRadixSort(op)(None, view, temp)
    assert _went_by_passes(temp)
    np.testing.assert_array_equal(to_host(view), keys[order])
    view, values = to_device(keys), torch.arange(LONG, dtype=torch.int32, device="cuda")
    temp = accelerator.Allocate1D(accelerator.ComputeRadixSortPairsTempStorageSize(op, torch.int32, LONG), torch.int32).zero_()
    accelerator.CreateRadixSortPairs(op)(None, view, values, temp)
    accelerator.CheckDeviceStatus(None, temp)
    assert _went_by_passes(temp)
    np.testing.assert_array_equal(to_host(view), keys[order])
    np.testing.assert_array_equal(to_host(values), order)


@pytest.mark.parametrize("name", ["UInt8", "Int16", "UInt32", "Int64"])
@pytest.mark.parametrize("offset,stride", [(1, 1), (3, 1), (0, 2), (1, 3)])
def test_views(accelerator, name, offset, stride):
    info = np.iinfo(NP[name])
    storage = np.random.default_rng(offset + stride).integers(info.min, info.max, size=offset + LONG * stride, dtype=NP[name], endpoint=True)
    op = getattr(RadixSortOperations, "Ascending" + name)
    dev = to_device(storage)
    temp = accelerator.Allocate1D(accelerator.ComputeRadixSortTempStorageSize(op, LONG), torch.int32).zero_()
    accelerator.CreateRadixSort(op)(None, dev[offset::stride][:LONG], temp)
    accelerator.CheckDeviceStatus(None, temp)
    assert _went_by_passes(temp)
    expected = storage.copy()
    expected[offset::stride][:LONG] = np.sort(storage[offset::stride][:LONG])
    np.testing.assert_array_equal(to_host(dev), expected)   # what lies around and between stays
    if stride == 1:
        keys, values = to_device(storage), torch.arange(LONG + offset, dtype=torch.int32, device="cuda")
        temp = accelerator.Allocate1D(accelerator.ComputeRadixSortPairsTempStorageSize(op, torch.int32, LONG), torch.int32).zero_()
        accelerator.CreateRadixSortPairs(op)(None, keys[offset:], values[offset:], temp)
        assert _went_by_passes(temp)
        np.testing.assert_array_equal(to_host(keys), expected)
        np.testing.assert_array_equal(to_host(values)[offset:], np.argsort(storage[offset:], kind="stable") + offset)

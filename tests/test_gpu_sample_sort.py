"""The sort by buckets of a sample: lengths around the places where it begins, where it gets another bucket
or block and where it ends; distributions that put many equal keys into the sample; strided keys, sequenced
values; a count on the device; and data that mislead the sample, which are then sorted by digits instead.
Keys that differ in a few bytes only, which go by these from the start, and keys that only look as if they did.
Against a stable host sort."""
import ctypes

import numpy as np
import pytest
import torch

from ilgpu_b200 import RadixSortOperations, Sequencers
from ilgpu_b200 import _native as N

pytestmark = pytest.mark.gpu


def _keys(rng, dtype, n, kind):
    if dtype.kind == "f":
        keys = rng.standard_normal(n).astype(dtype)
        if kind == "same":
            keys[:] = 1.5
        elif kind == "few":
            keys = np.rint(keys * 2) + 0.0
        elif kind == "half":
            keys[rng.random(n) < 0.5] = 0.25
        elif kind == "sorted":
            keys.sort()
        return keys
    keys = rng.integers(0, 1 << (dtype.itemsize * 8), size=n, dtype=dtype)
    if kind == "same":
        keys[:] = 12345
    elif kind == "few":
        keys &= dtype.type(3)
    elif kind == "half":
        keys[rng.random(n) < 0.5] = 7
    elif kind == "sorted":
        keys.sort()
    return keys


MOVES = 58  # B200ALG_TESTING_SORT_MOVES_WORD


def _check(acc, keys, value, descending=False):
    """The number of times that the elements were moved by a digit."""
    name = {"f4": "Float", "f8": "Double", "u4": "UInt32", "u8": "UInt64"}[keys.dtype.str[1:]]
    floating = keys.dtype.kind == "f"
    op = getattr(RadixSortOperations, ("Descending" if descending else "Ascending") + name)
    order = np.argsort((-keys if floating else ~keys) if descending else keys, kind="stable")
    dev = torch.from_numpy(keys).cuda()
    temp = acc.Allocate1D(acc.ComputeRadixSortPairsTempStorageSize(op, torch.int64, keys.size), torch.int32)
    temp[MOVES] = -1
    if value is None:
        acc.CreateRadixSort(op, floating)(None, dev, temp)
    else:
        vals = torch.from_numpy(np.arange(keys.size).astype(value)).cuda()
        acc.CreateRadixSortPairs(op, floating)(None, dev, vals, temp)
        np.testing.assert_array_equal(vals.cpu().numpy(), order.astype(value))
    acc.CheckDeviceStatus(None, temp)
    np.testing.assert_array_equal(dev.cpu().numpy(), keys[order])
    return int(temp[MOVES])


@pytest.mark.parametrize("n", [9729, 12_289, 20_000, 99_999, 100_000, 227_327, 227_329, 400_001, 700_000, 1_091_200, 1_091_201, 1_159_000, 1_546_000])
@pytest.mark.parametrize("key,value", [(np.float64, None), (np.float64, np.int64), (np.float32, np.int32), (np.uint64, None), (np.uint64, np.uint8),
                                       (np.uint32, np.int32), (np.uint32, np.int16)])
@pytest.mark.parametrize("kind", ["full", "same", "few", "half", "sorted"])
def test_lengths_and_distributions(accelerator, n, key, value, kind):
    _check(accelerator, _keys(np.random.default_rng(n), np.dtype(key), n, kind), value, descending=kind == "half")


def _sampled(n, most=None):
    """Positions that the blocks look at in a view of n elements, launched for up to `most` (sample_sort.cu)."""
    most = most or n
    blocks = 16 if most <= 40_960 else min(-(-most // 1536), torch.cuda.get_device_properties(0).multi_processor_count)
    share = -(-n // blocks)
    at = []
    for b in range(blocks):
        lo = min(n, b * share)
        length = min(n - lo, share)
        t = np.arange(128)
        shift = (((b * 128 + t) * 2654435761 & 0xFFFFFFFF) >> 8) % max(1, length // 128)
        at.append(lo + t * length // 128 + (shift if length >= 128 else 0))
    return np.concatenate(at)


def _misleading(key, n, most=None):
    """Keys that are all in one bucket but for what is looked at."""
    rng, at, key = np.random.default_rng(5), _sampled(n, most), np.dtype(key)
    if key.kind == "f":
        keys = (2 + 30 * rng.random(n)).astype(key)   # (all bytes of a float differ)
        keys[at] = rng.random(at.size)
        return keys
    bits = key.itemsize * 8
    keys = (rng.integers(0, 1 << (bits - 1), size=n, dtype=key) >> key.type(4)) + key.type(1 << (bits - 1))
    keys[at] = rng.integers(0, 1 << 16, size=at.size)
    return keys


@pytest.mark.parametrize("key,value,n", [(np.uint64, np.int32, 300_007), (np.uint64, np.int16, 300_007), (np.uint32, np.int64, 300_007),
                                         (np.uint64, None, 800_003), (np.float64, None, 300_007), (np.float64, None, 30_001),
                                         (np.float64, np.int32, 40_960), (np.float32, np.int32, 40_001)])
@pytest.mark.parametrize("descending", [False, True])
def test_misled_sample(accelerator, key, value, n, descending):
    assert _check(accelerator, _misleading(key, n), value, descending) == np.dtype(key).itemsize   # by every digit


@pytest.mark.parametrize("n", [30_001, 300_007])
def test_misled_strided(accelerator, n):
    keys, op = _misleading(np.float64, n), RadixSortOperations.DescendingDouble
    storage = torch.from_numpy(np.repeat(keys, 3)).cuda()
    temp = accelerator.Allocate1D(accelerator.ComputeRadixSortTempStorageSize(op, n), torch.int32)
    temp[MOVES] = -1
    accelerator.CreateRadixSort(op, True)(None, storage[1::3], temp)
    assert int(temp[MOVES]) == 8
    got = storage.cpu().numpy()
    np.testing.assert_array_equal(got[1::3], np.sort(keys)[::-1])
    np.testing.assert_array_equal(got[::3], keys)     # what lies between stays
    np.testing.assert_array_equal(got[2::3], keys)


def test_misled_sequenced(accelerator):
    n = 300_007
    keys, op = _misleading(np.uint64, n), RadixSortOperations.AscendingUInt64
    dev, vals = torch.from_numpy(keys).cuda(), torch.zeros(n, dtype=torch.float32, device="cuda")
    temp = accelerator.Allocate1D(accelerator.ComputeRadixSortPairsTempStorageSize(op, vals.dtype, n), torch.int32)
    temp[MOVES] = -1
    accelerator.CreateRadixSortPairs(op, sequencer=Sequencers)(None, dev, vals, Sequencers.FloatSequencer, temp)
    assert int(temp[MOVES]) == 8
    order = np.argsort(keys, kind="stable")
    np.testing.assert_array_equal(dev.cpu().numpy(), keys[order])
    np.testing.assert_array_equal(vals.cpu().numpy(), order)


@pytest.mark.parametrize("value_bytes", [0, 4])
def test_misled_count_on_the_device(value_bytes):
    most, n = 800_000, 760_001
    L, keys = N.lib(), _misleading(np.uint64, 760_001, 800_000)
    p = lambda t: ctypes.c_void_p(t.data_ptr() if t is not None else 0)
    need = ctypes.c_int64(0)
    assert L.b200alg_radix_sort_temp_bytes(N.U64, most, value_bytes, ctypes.byref(need)) == N.OK
    temp = torch.full((need.value // 4,), -1, dtype=torch.int32, device="cuda")
    k = torch.from_numpy(np.concatenate([keys, np.zeros(most - n, np.uint64)])).cuda()
    ok, count = torch.full((most,), 9, dtype=torch.int64, device="cuda"), torch.tensor([n], dtype=torch.int64, device="cuda")
    v, ov = (torch.arange(most, dtype=torch.int32, device="cuda"), torch.full((most,), 9, dtype=torch.int32, device="cuda")) if value_bytes else (None, None)
    assert L.b200alg_radix_sort_out_of_place(None, p(k), p(v), p(ok), p(ov), most, p(count), N.U64, value_bytes, 0, p(temp), need.value) == N.OK
    assert int(temp[MOVES]) == 8
    order = np.argsort(keys, kind="stable")
    got = ok.cpu().numpy()
    np.testing.assert_array_equal(got[:n].view(np.uint64), keys[order])
    assert (got[n:] == 9).all()
    if value_bytes:
        got = ov.cpu().numpy()
        np.testing.assert_array_equal(got[:n], order)
        assert (got[n:] == 9).all()


def _looked(n):
    """Positions that every block looks at (sample_sort.cu)."""
    j = np.arange(64, dtype=np.uint64)
    return j * np.uint64(n) // np.uint64(64) + (np.uint64(n // 64) * (j * np.uint64(2654435761) & np.uint64(0xFFFFFFFF)) >> np.uint64(32))


def _with_bytes(rng, dtype, n, at):
    """Keys that differ in these bytes, also the first two; the other bytes are the same in all."""
    keys = np.full(n, 0x1122334455667788 & ((1 << 8 * np.dtype(dtype).itemsize) - 1), dtype=dtype)
    for p in at:
        digit = rng.integers(0, 256, size=n).astype(dtype)
        digit[:2] = 0, 255
        keys ^= digit << dtype(8 * p)
    return keys


@pytest.mark.parametrize("n", [100_000, 227_329, 800_000, 1_091_201])
@pytest.mark.parametrize("key,value,at", [(np.uint64, np.int32, a) for a in [(), (0,), (7,), (2, 5), (0, 1, 6), (0, 1, 2, 3), (1, 3, 4, 6, 7)]] +
                                         [(np.uint32, np.int64, a) for a in [(), (0,), (3,), (1, 2), (0, 1, 2), (0, 1, 2, 3)]])
def test_few_bytes(accelerator, n, key, value, at):
    for descending in (False, True):
        moves = _check(accelerator, _with_bytes(np.random.default_rng(n), key, n, at), value, descending)
        assert moves == (max(1, len(at)) if len(at) <= 3 else 0)


@pytest.mark.parametrize("n", [8705, 12_289, 16_384, 40_960, 40_961, 150_001])
@pytest.mark.parametrize("value", [None, np.int32, np.int64])
@pytest.mark.parametrize("most,moves", [(2, 2), (256, 3), (1 << 19, 0)])
def test_whole_numbers(accelerator, n, value, most, moves):
    keys = np.random.default_rng(n).integers(0, most, size=n).astype(np.float64)
    keys[0] = 0
    assert _check(accelerator, keys, value, descending=True) == moves


@pytest.mark.parametrize("n", [40_001, 150_001, 800_000])
@pytest.mark.parametrize("seen,odd,moves", [
    ((1, 2), (5,), 3), ((1, 2), (3, 5), 4), ((1, 2), (3, 5, 6), 5), ((1, 2), (3, 4, 5, 6), 0),   # higher bytes than the guess has
    ((1,), (0,), 2), ((1, 2), (0,), 3), ((1, 2), (0, 5), 0), ((), (3,), 1), ((), (2, 3, 4, 5), 0)])  # a lower one
def test_wrong_guess(accelerator, n, seen, odd, moves):
    rng = np.random.default_rng(n)
    raw = _with_bytes(rng, np.uint64, n, seen)
    one = next(p for p in range(n // 2, n) if p not in set(_looked(n).tolist()))
    for p in odd:
        raw[one] ^= np.uint64(0x81) << np.uint64(8 * p)
    if n < 100_000:
        keys = raw.view(np.float64)   # short views go this way with floating-point keys
        assert np.isfinite(keys).all()
        assert _check(accelerator, keys, None) == moves
    else:
        assert _check(accelerator, raw, np.int32) == moves


@pytest.mark.parametrize("n", [100_000, 250_001])
def test_sequenced_and_strided(accelerator, n):
    rng = np.random.default_rng(n)
    keys = rng.integers(0, 1 << 40, size=n, dtype=np.uint64) & 0xFFF0FF
    op = RadixSortOperations.DescendingUInt64
    dev, vals = torch.from_numpy(keys).cuda(), torch.zeros(n, dtype=torch.float32, device="cuda")
    temp = accelerator.Allocate1D(accelerator.ComputeRadixSortPairsTempStorageSize(op, vals.dtype, n), torch.int32)
    accelerator.CreateRadixSortPairs(op, sequencer=Sequencers)(None, dev, vals, Sequencers.FloatSequencer, temp)
    np.testing.assert_array_equal(vals.cpu().numpy(), np.argsort(~keys, kind="stable"))
    keys = rng.standard_normal(n)
    op = RadixSortOperations.DescendingDouble
    storage = torch.from_numpy(np.repeat(keys, 3)).cuda()
    accelerator.CreateRadixSort(op, True)(None, storage[1::3], temp)
    np.testing.assert_array_equal(storage.cpu().numpy()[1::3], np.sort(keys)[::-1])
    np.testing.assert_array_equal(storage.cpu().numpy()[::3], keys)


@pytest.mark.parametrize("few", [False, True])
def test_count_on_the_device(few):
    n = 300_000
    L, rng = N.lib(), np.random.default_rng(n)
    keys, values = rng.integers(0, 1 << 60, size=n, dtype=np.uint64), np.arange(n, dtype=np.uint32)
    if few:
        keys &= np.uint64(0xFF00FF00)
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    need = ctypes.c_int64(0)
    assert L.b200alg_radix_sort_temp_bytes(N.U64, n, 4, ctypes.byref(need)) == N.OK
    temp = torch.empty(need.value, dtype=torch.uint8, device="cuda")
    k, v = torch.from_numpy(keys).cuda(), torch.from_numpy(values).cuda()
    for m in (n, n - 777, 10_001, 147, 1, 0):
        ok, ov = torch.full((n,), 9, dtype=torch.int64, device="cuda"), torch.full((n,), 9, dtype=torch.int32, device="cuda")
        count = torch.tensor([m], dtype=torch.int64, device="cuda")
        assert L.b200alg_radix_sort_out_of_place(None, p(k), p(v), p(ok), p(ov), n, p(count), N.U64, 4, 0, p(temp), need.value) == N.OK
        torch.cuda.synchronize()
        order = np.argsort(keys[:m], kind="stable")
        np.testing.assert_array_equal(ok.cpu().numpy()[:m].view(np.uint64), keys[:m][order])
        np.testing.assert_array_equal(ov.cpu().numpy()[:m], order)
        assert (ok.cpu().numpy()[m:] == 9).all() and (ov.cpu().numpy()[m:] == 9).all()

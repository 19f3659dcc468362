"""The digit pass of the radix sort around its tiles: one key, the last key of a tile, of two tiles
(whose places are published together) and one more, for key and value sizes with different tiles;
keys that meet in few digits; against a stable host sort.  (The library sorts all but the longest of
these, the ones of many tiles, in one launch; test_gpu_long_sorts.py has the same edges in the digit pass itself.)"""
import numpy as np
import pytest
import torch

from ilgpu_b200 import RadixSortOperations
from tests.helpers import NP, PASSES_WORD

pytestmark = pytest.mark.gpu

# keys per tile: 512 threads, as many keys each as two blocks per SM leave room for
TILES = {("UInt8", None): 10240, ("UInt32", None): 10240, ("UInt64", None): 5632, ("UInt32", np.int32): 6144,
         ("UInt64", np.uint32): 4096, ("Int64", np.float64): 3072, ("UInt16", np.uint8): 8192}
NAMES = {v: k for k, v in NP.items()}
MANY = 1_600_000   # keys that many tiles hold: more than one launch sorts


def _sorts(acc, name, keys, values):
    """What the sort makes of keys and values, and whether it went by passes."""
    op = getattr(RadixSortOperations, "Ascending" + name)
    dev = torch.from_numpy(keys).cuda()
    if values is None:
        temp = acc.Allocate1D(acc.ComputeRadixSortTempStorageSize(op, keys.size), torch.int32).zero_()
        acc.CreateRadixSort(op)(None, dev, temp)
        acc.CheckDeviceStatus(None, temp)
        return dev.cpu().numpy(), None, int(temp[PASSES_WORD]) != 0
    vals = torch.from_numpy(values).cuda()
    temp = acc.Allocate1D(acc.ComputeRadixSortPairsTempStorageSize(op, vals.dtype, keys.size), torch.int32).zero_()
    acc.CreateRadixSortPairs(op)(None, dev, vals, temp)
    acc.CheckDeviceStatus(None, temp)
    return dev.cpu().numpy(), vals.cpu().numpy(), int(temp[PASSES_WORD]) != 0


@pytest.mark.parametrize("name,value", list(TILES))
@pytest.mark.parametrize("tiles,extra", [(0, 1), (1, -1), (1, 0), (1, 1), (2, 0), (2, 1), (3, 0), (131, 7), ("many", 7)])
def test_tile_edges(accelerator, name, value, tiles, extra):
    n = (-(-MANY // TILES[name, value]) if tiles == "many" else tiles) * TILES[name, value] + extra
    rng = np.random.default_rng(n)
    info = np.iinfo(NP[name])
    for few in (False, True):
        keys = rng.integers(info.min, info.max, size=n, dtype=NP[name], endpoint=True)
        if few:   # whole warps, and in later passes whole tiles, of one digit
            keys = rng.choice(keys[:3] if n > 3 else keys, size=n).astype(NP[name])
        values = None if value is None else np.arange(n).astype(value)
        got, got_values, by_passes = _sorts(accelerator, name, keys, values)
        assert by_passes or tiles != "many"
        order = np.argsort(keys, kind="stable")
        np.testing.assert_array_equal(got, keys[order])
        if values is not None:
            np.testing.assert_array_equal(got_values, values[order])

"""Unique in place and the run-length selection around the 32 KB tiles of the kernel: the last
element of a tile, one more and one less, for every element size, and views that do not start on
16 bytes, against the CPU oracle."""
import numpy as np
import pytest
import torch

from oracle import cpu_oracle as oracle
from tests.helpers import to_host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.uint8, np.int16, np.uint32, np.int64, np.float32, np.float64, np.float16])
@pytest.mark.parametrize("tiles,extra", [(1, -1), (1, 0), (1, 1), (2, 0), (300, 1)])
@pytest.mark.parametrize("offset", [0, 1])
def test_tile_edges(accelerator, dtype, tiles, extra, offset):
    n = tiles * (32768 // np.dtype(dtype).itemsize) + extra
    rng = np.random.default_rng(n + offset)
    for longest in (1, 4, 100_000):   # nothing to remove (almost), a quarter left, runs over several tiles
        runs = rng.integers(1, longest + 1, size=n // max(1, longest // 4) + 1)
        host = np.repeat(rng.integers(0, 100, size=runs.size), runs)[:n].astype(dtype)
        if host.size < n:
            host = np.concatenate([host, np.full(n - host.size, 3, dtype)])
        storage = torch.from_numpy(np.concatenate([np.zeros(offset, dtype), host, np.full(4, 77, dtype)])).cuda()
        view = storage[offset:offset + n]
        count = accelerator.Unique(None, view)
        expected = oracle.unique(host)
        np.testing.assert_array_equal(to_host(view)[:count], expected)
        assert to_host(storage)[offset + n:].tolist() == [77] * 4   # nothing behind the view is touched

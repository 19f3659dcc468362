"""Unique in place with one, three and seven tiles of 32 KB for every block, one element more or
less than that, and with survivors that go over the tiles right before their own, against numpy."""
import numpy as np
import pytest
import torch

from tests.helpers import to_host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.uint8, np.uint32, np.int64])
@pytest.mark.parametrize("turns", [1, 3, 7])
@pytest.mark.parametrize("extra", [-1, 1])
@pytest.mark.parametrize("kept", [0.02, 1.0])
def test_turns(accelerator, dtype, turns, extra, kept):
    blocks = 2 * torch.cuda.get_device_properties(0).multi_processor_count - 1
    n = turns * blocks * (32768 // np.dtype(dtype).itemsize) + extra
    new = np.random.default_rng(n).random(n) < kept
    new[0] = True
    host = (np.cumsum(new) & 0x7F).astype(dtype)
    view = torch.from_numpy(host).cuda()
    count = accelerator.Unique(None, view)
    np.testing.assert_array_equal(to_host(view)[:count], host[new])


@pytest.mark.parametrize("dtype", [np.uint32, np.int64])
@pytest.mark.parametrize("moved", [1, 3, 8191, 8192, 8193, 100_000])
@pytest.mark.parametrize("offset", [0, 1])
def test_stores_right_behind_the_reads(accelerator, dtype, moved, offset):
    """Duplicates at the start only: every tile goes over the tiles right before it."""
    n = 3_000_001
    host = np.maximum(np.arange(n), moved).astype(dtype)
    view = torch.from_numpy(np.concatenate([np.zeros(offset, dtype), host])).cuda()[offset:]
    count = accelerator.Unique(None, view)
    np.testing.assert_array_equal(to_host(view)[:count], np.arange(moved, n).astype(dtype))


def test_nothing_moves(accelerator):
    host = np.arange(3_000_001, dtype=np.uint32)
    view = torch.from_numpy(host).cuda()
    assert accelerator.Unique(None, view) == host.size
    np.testing.assert_array_equal(to_host(view), host)

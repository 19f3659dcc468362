"""The pipelined scan where its blocks have one, three and seven tiles to go round the ring, and one
element more or less than that, for aligned views and views that start off 16 bytes, against numpy."""
import numpy as np
import pytest
import torch

from ilgpu_b200 import ScanKind, ScanReduceOperations
from tests.helpers import NP

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["Int32", "Int64", "Float"])
@pytest.mark.parametrize("turns", [1, 3, 7])
@pytest.mark.parametrize("extra", [-1, 0, 1])
@pytest.mark.parametrize("offset", [0, 1])
def test_turns(accelerator, name, turns, extra, offset):
    blocks = 2 * torch.cuda.get_device_properties(0).multi_processor_count - 1
    n = turns * blocks * (32768 // np.dtype(NP[name]).itemsize) + extra
    rng = np.random.default_rng(n)
    host = rng.integers(0, 2, size=n).astype(NP[name])      # float sums are exact
    src = torch.from_numpy(np.concatenate([np.full(offset, 9, host.dtype), host])).cuda()[offset:]
    dst = torch.full((offset + n + 5,), 77, dtype=src.dtype, device="cuda")
    scan = accelerator.CreateScanProvider(src.dtype, n)
    scan.CreateScan(getattr(ScanReduceOperations, "Add" + name), ScanKind.Inclusive)(None, src, dst[offset:offset + n])
    accelerator.CheckDeviceStatus(None, scan.TempView)
    got = dst.cpu().numpy()
    np.testing.assert_array_equal(got[offset:offset + n], np.cumsum(host, dtype=host.dtype))
    assert (got[:offset] == 77).all() and (got[offset + n:] == 77).all()

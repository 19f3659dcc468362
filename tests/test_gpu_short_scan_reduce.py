"""Reduce and scan where one launch turns into two, one block into a cluster, and for views that start
off a 16-byte boundary (alike and not alike), against numpy."""
import numpy as np
import pytest
import torch

from ilgpu_b200 import ScanKind, ScanReduceOperations
from tests.helpers import NP

pytestmark = pytest.mark.gpu


def _numbers(name, n):
    rng = np.random.default_rng(n)
    if name in ("Float", "Double"):
        return rng.integers(0, 4, size=n).astype(NP[name])      # sums are exact
    return rng.integers(0, 1000, size=n).astype(NP[name])


@pytest.mark.parametrize("name", ["Int32", "UInt64", "Float", "Double"])
@pytest.mark.parametrize("n", [1, 7, 8191, 8192, 8193, 16_385, 65_533, 65_536, 65_537, 300_000, 1_000_003])
@pytest.mark.parametrize("offsets", [(0, 0), (1, 1), (3, 3), (0, 1), (2, 1)])
def test_scan(accelerator, name, n, offsets):
    host = _numbers(name, n)
    a, b = offsets
    src = torch.from_numpy(np.concatenate([np.full(a, 9, host.dtype), host, np.full(5, 9, host.dtype)])).cuda()[a:a + n]
    scan = accelerator.CreateScanProvider(src.dtype, n)
    for kind in (ScanKind.Inclusive, ScanKind.Exclusive):
        dst = torch.from_numpy(np.full(b + n + 5, 77, host.dtype)).cuda()
        scan.CreateScan(getattr(ScanReduceOperations, "Add" + name), kind)(None, src, dst[b:b + n])
        accelerator.CheckDeviceStatus(None, scan.TempView)
        want = np.cumsum(host, dtype=host.dtype)
        if kind == ScanKind.Exclusive:
            want = np.concatenate([[0], want[:-1]]).astype(host.dtype)
        got = dst.cpu().numpy()
        np.testing.assert_array_equal(got[b:b + n], want)
        assert (got[:b] == 77).all() and (got[b + n:] == 77).all()


@pytest.mark.parametrize("name", ["Int32", "Int64", "Float"])
@pytest.mark.parametrize("n", [1, 16_384, 16_385, 131_072, 131_073, 262_144, 262_145])
@pytest.mark.parametrize("stride", [1, 3])
def test_reduce(accelerator, name, n, stride):
    host = _numbers(name, n)
    view = torch.from_numpy(np.repeat(host, stride)).cuda()[::stride]
    for fold, want in (("Add", host.sum()), ("Max", host.max()), ("Min", host.min())):
        op = getattr(ScanReduceOperations, fold + name)
        out = torch.zeros(1, dtype=view.dtype, device="cuda")
        accelerator.Reduce(None, view, op, out)
        assert out.item() == want
        assert accelerator.Reduce(None, view, op) == want

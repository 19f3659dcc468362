"""Bins of elements at the edges of what a locator computes: remainders by an inverse (largest and smallest
integers, multiples of the bin count and their neighbours, powers of two and one bin), equal widths of integers
far outside the range; rounds of the table kernel that are whole, ragged and few.  Against exact host arithmetic."""
import numpy as np
import pytest
import torch

import ilgpu_b200 as ib

pytestmark = pytest.mark.gpu
BINS = [1, 2, 3, 7, 64, 641, 1000, 1025, 4096, 40_000, 65_535, 65_536, 100_000]


def _run(acc, data, bins, locator):
    out, overflow = torch.zeros(bins, dtype=torch.int64, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    acc.Histogram(None, torch.from_numpy(data).cuda(), out, overflow, locator)
    assert overflow.item() == 0
    return out.cpu().numpy()


def _edges(rng, dtype, bins, n):
    info = np.iinfo(dtype)
    data = rng.integers(info.min, info.max, size=n, dtype=dtype, endpoint=True)
    edge = [info.min, info.min + 1, -1, 0, 1, info.max - 1, info.max]
    for k in (1, 2, 3, info.max // bins, info.max // bins - 1, -(info.min // bins) if info.min else 5):
        edge += [k * bins - 1, k * bins, k * bins + 1, -k * bins, -k * bins + 1]
    edge = [e for e in edge if info.min <= e <= info.max]
    data[: len(edge)] = edge
    return data


@pytest.mark.parametrize("bins", BINS)
@pytest.mark.parametrize("dtype", [np.int32, np.uint32, np.int64, np.uint64])
@pytest.mark.parametrize("n", [1000, 606_207, 2_424_832, 5_000_011])
def test_modulo(accelerator, dtype, bins, n):
    data = _edges(np.random.default_rng(bins), dtype, bins, n)
    low = np.uint64(0) - data.astype(np.uint64) if data.dtype.kind == "i" else data.astype(np.uint64)
    size = np.where(data < 0, low, data.astype(np.uint64)) if data.dtype.kind == "i" else low
    expected = np.bincount((size % np.uint64(bins)).astype(np.int64), minlength=bins)
    np.testing.assert_array_equal(_run(accelerator, data, bins, ib.ModuloLocator()), expected)


@pytest.mark.parametrize("bins", BINS)
@pytest.mark.parametrize("dtype", [np.int32, np.uint32, np.int64, np.uint64])
def test_equal_width_of_integers(accelerator, dtype, bins):
    data = _edges(np.random.default_rng(bins), dtype, bins, 2_424_832)
    lo, hi = -1000.0, 70_000.0
    data[1000:2_000_000] %= np.array(80_000, dtype)
    t = (data.astype(np.float64) - lo) * (bins / (hi - lo))
    expected = np.bincount(np.minimum(np.trunc(np.clip(t, 0.0, float(bins))).astype(np.int64), bins - 1), minlength=bins)
    np.testing.assert_array_equal(_run(accelerator, data, bins, ib.EqualWidthClampLocator(lo, hi)), expected)

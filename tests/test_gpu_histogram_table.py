"""The histogram kernel with one table of all bins per SM, where its branches change: 1024 bins
and one more, the last count of 32-bit counters and the first of 16-bit ones, the last count the
table holds at all and one more; bell-shaped data and data that meets in few bins (16-bit counters
are then emptied on the way), unaligned and strided views, against the CPU oracle."""
import numpy as np
import pytest
import torch

from ilgpu_b200 import EqualWidthClampLocator, ModuloLocator
from oracle import cpu_oracle as oracle

pytestmark = pytest.mark.gpu


def _samples(rng, n, bins, shape):
    if shape == "bell":
        return np.clip(rng.normal(bins / 2, bins / 8, size=n), 0, bins - 1)
    return np.where(rng.random(n) < 0.9, 3, rng.integers(0, bins, size=n))


def _check(accelerator, host, view, bins, locator, name):
    counts = torch.full((bins,), 5, dtype=torch.int32, device="cuda")
    overflow = torch.zeros(1, dtype=torch.int32, device="cuda")
    accelerator.Histogram(None, view, counts, overflow, locator)
    expected, flag = oracle.histogram(host, np.full(bins, 5, np.int32), name, locator.lo, locator.hi)
    np.testing.assert_array_equal(counts.cpu().numpy(), expected)
    assert bool(overflow.item()) == bool(flag)


@pytest.mark.parametrize("bins", [1024, 1025, 12_288, 12_289, 57_344, 57_345, 114_688, 114_689])
@pytest.mark.parametrize("shape", ["bell", "few"])
def test_bin_counts_around_the_branches(accelerator, bins, shape):
    rng = np.random.default_rng(bins)
    n = max(16 * bins, 1 << 17) + 5
    host = _samples(rng, n, bins, shape).astype(np.int32)
    dev = torch.from_numpy(host).cuda()
    _check(accelerator, host[1:], dev[1:], bins, ModuloLocator(), "modulo")
    _check(accelerator, host[::3], dev[::3], bins, ModuloLocator(), "modulo")


@pytest.mark.parametrize("bins", [2000, 70_000])
@pytest.mark.parametrize("dtype", [np.float32, np.float64, np.int64])
def test_many_elements_of_one_bin(accelerator, bins, dtype):
    """Enough of them that a block's 16-bit counter is emptied several times."""
    host = _samples(np.random.default_rng(7), 24_000_001, bins, "few").astype(dtype)
    _check(accelerator, host, torch.from_numpy(host).cuda(), bins, EqualWidthClampLocator(0.0, float(bins)), "equal_width_clamp")


def test_input_beyond_the_cache(accelerator):
    rng = np.random.default_rng(3)
    host = rng.normal(size=(1 << 24) + 3)
    _check(accelerator, host, torch.from_numpy(host).cuda(), 256, EqualWidthClampLocator(-4.0, 4.0), "equal_width_clamp")

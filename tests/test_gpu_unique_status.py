"""Unique owns its temp, so a wait that ran out inside it has to come back as an exception from the call.
No wait is made to run out on the GPU: the native call, or the status query, is a fake that says so."""
import ctypes

import pytest
import torch

from ilgpu_b200 import _native as N
from ilgpu_b200.algorithms import B200AlgException

pytestmark = pytest.mark.gpu

UNIQUE_TO_HOST = ctypes.CFUNCTYPE(ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int64, ctypes.c_int,
                                  ctypes.POINTER(ctypes.c_int64), ctypes.c_void_p, ctypes.c_int64)


def _bind(replaced=None):
    names = N.host().ENTRY_POINTS
    addresses = [ctypes.cast(getattr(N.lib(), name), ctypes.c_void_p).value for name in names]
    if replaced is not None:
        addresses[names.index("b200alg_unique_to_host")] = ctypes.cast(replaced, ctypes.c_void_p).value
    N.host().bind(tuple(addresses))


def test_host_path_raises(accelerator):
    data = torch.arange(5000, dtype=torch.int32, device="cuda")
    assert accelerator.Unique(None, data) == 5000
    asked = []

    def gave_up(stream, view, n, code, out, temp, temp_bytes):
        asked.append((n, out[1]))
        out[0], out[1] = 4711, N.WAIT_LIMIT   # a count that is not valid, and that
        return N.OK

    fake = UNIQUE_TO_HOST(gave_up)
    _bind(fake)
    try:
        with pytest.raises(B200AlgException) as e:
            accelerator.Unique(None, data)
    finally:
        _bind()
    assert e.value.status == N.WAIT_LIMIT and asked == [(5000, N.OK)]   # asked once: the data may have changed
    assert accelerator.Unique(None, data) == 5000   # the status of one call is not the next one's


def test_long_way_raises(accelerator, monkeypatch):
    class NotCovered:
        def __getattr__(self, name):
            return lambda *a: None

    class GaveUp:
        def __getattr__(self, name):
            return (lambda *a: N.WAIT_LIMIT) if name == "b200alg_device_status" else getattr(N.lib(), name)

    data = torch.arange(5000, dtype=torch.int32, device="cuda")
    monkeypatch.setattr(accelerator, "_host", NotCovered())
    assert accelerator.Unique(None, data) == 5000
    assert accelerator.Unique(None, data[:0]) == 0
    monkeypatch.setattr(accelerator, "L", GaveUp())
    with pytest.raises(B200AlgException) as e:
        accelerator.Unique(None, data)
    assert e.value.status == N.WAIT_LIMIT


@pytest.mark.parametrize("n", [0, 1, 5000, 1_000_003])
def test_entry_point(n):
    """The length and the untouched status, in pinned memory; nothing in front of or behind them."""
    data = (torch.arange(n, device="cuda") // 3).to(torch.int32)
    need = ctypes.c_int64(0)
    assert N.lib().b200alg_unique_temp_bytes(N.I32, n, ctypes.byref(need)) == N.OK
    temp = torch.empty(need.value, dtype=torch.uint8, device="cuda")
    out = torch.tensor([-7, -7, 0, -7], dtype=torch.int64).pin_memory()
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert N.lib().b200alg_unique_to_host(stream, ctypes.c_void_p(data.data_ptr()), n, N.I32, ctypes.c_void_p(out.data_ptr() + 8),
                                          ctypes.c_void_p(temp.data_ptr()), need.value) == N.OK
    torch.cuda.synchronize()
    assert out.tolist() == [-7, (n + 2) // 3, 0, -7]
    assert N.lib().b200alg_unique_to_host(stream, ctypes.c_void_p(data.data_ptr()), n, N.I32, None, ctypes.c_void_p(temp.data_ptr()),
                                          need.value) == N.INVALID_ARGUMENT

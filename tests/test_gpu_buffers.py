"""Reuse of device buffers: a released buffer is handed out again only after every stream's work on it is over."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_a_released_result_that_another_stream_still_reads_is_not_overwritten(device):
    import torch
    import floneum_b200 as fb
    n = 1 << 22
    side = torch.cuda.Stream()
    a = fb.Tensor.from_slice(device, (n,), np.full(n, 1.0, np.float32))
    b = fb.Tensor.from_slice(device, (n,), np.full(n, 2.0, np.float32))
    for _ in range(12):  # more rounds than releases that may wait together
        x = a.cast(fb.BF16 if hasattr(fb, "BF16") else 1)
        device.synchronize()
        view = torch.empty(0)
        iface = {"data": (x.ptr, False), "shape": (n,), "typestr": "<i2", "strides": None, "version": 3}
        view = torch.as_tensor(type("V", (), {"__cuda_array_interface__": iface})(), device="cuda")
        with torch.cuda.stream(side):
            torch.cuda._sleep(2_000_000)  # about a millisecond before the copy starts
            copy = view.clone()
        del x
        y = b.cast(1)  # same size: must not land on the buffer that is still to be read
        side.synchronize()
        assert bool((copy == 0x3F80).all())
        del y


def test_buffers_come_back_and_a_second_free_is_refused(device):
    import floneum_b200 as fb
    from floneum_b200 import _lib
    L = _lib.load()
    seen = set()
    for _ in range(40):
        p = device.alloc(3000)
        assert p % 256 == 0
        seen.add(p)
        device.synchronize()
        device.free(p)
    assert len(seen) < 40
    with pytest.raises(fb.FusorCudaError):
        _lib.check(L.fusor_cuda_buffer_free(device.handle, ctypes.c_void_p(p)), device.handle)
    held = [device.alloc(1 + 700 * i) for i in range(50)]
    assert len(set(held)) == 50
    for q in held:
        device.free(q)

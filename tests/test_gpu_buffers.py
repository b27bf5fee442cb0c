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


@pytest.mark.parametrize("mode", ["thread_local", "relaxed"])
def test_buffers_while_another_thread_captures_a_graph(device, mode):
    """Allocation and release go on, and the other thread's capture survives them (both modes allow cudaMalloc and cudaFree)."""
    import threading
    import torch
    import floneum_b200 as fb
    x = torch.ones(1024, device="cuda")
    torch.cuda.synchronize()
    begun, done, got = threading.Event(), threading.Event(), []

    def capture():
        try:
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.stream(torch.cuda.Stream()):
                graph.capture_begin(capture_error_mode=mode)
                y = x * 2
                begun.set()
                done.wait(60)
                y = y + 1
                graph.capture_end()
            graph.replay()
            torch.cuda.synchronize()
            got.append(float(y[0]))
        except Exception as e:
            got.append(e)
            begun.set()

    t = threading.Thread(target=capture)
    t.start()
    begun.wait(60)
    try:
        for _ in range(600):  # enough releases for several rounds of reuse
            a, b = fb.Tensor.empty(device, (1 << 16,)), fb.Tensor.empty(device, (1 << 16,))
            del a, b
    finally:
        done.set()
        t.join()
    assert got == [3.0]

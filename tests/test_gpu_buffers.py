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


def _cudart():
    import glob
    import os
    import torch
    return ctypes.CDLL(sorted(glob.glob(os.path.join(os.path.dirname(torch.__file__), "..", "nvidia", "cuda_runtime", "lib", "libcudart.so*")))[0])


def _granted(cudart, p):
    """Bytes of the allocation that starts at p, as the driver knows it."""
    base, size = ctypes.c_uint64(), ctypes.c_size_t()
    cuda = ctypes.CDLL("libcuda.so.1")
    assert cuda.cuMemGetAddressRange_v2(ctypes.byref(base), ctypes.byref(size), ctypes.c_uint64(p)) == 0 and base.value == p
    return size.value


def test_a_buffer_freed_through_another_context_leaves_no_size_behind(device):
    """Its address may come back with fewer bytes; a release of that one must not enter the pool under the old size."""
    import torch
    import floneum_b200 as fb
    cudart, other = _cudart(), fb.Device.gpu(0)
    torch.cuda.synchronize()
    big = 48 << 20
    p = device.alloc(big)
    assert _granted(cudart, p) >= big
    other.free(p)
    held, got = [], ctypes.c_void_p()
    for _ in range(400):  # until the driver hands the address out again
        assert cudart.cudaMalloc(ctypes.byref(got), ctypes.c_size_t(3 << 20)) == 0
        held.append(got.value)
        if got.value == p:
            break
    for q in held:
        if q != p:
            assert cudart.cudaFree(ctypes.c_void_p(q)) == 0
    if held[-1] != p:
        pytest.skip("the driver did not hand the address out again")
    device.free(p)
    again = [device.alloc(big) for _ in range(12)]
    try:
        assert all(_granted(cudart, q) >= big for q in again)
    finally:
        for q in again:
            device.free(q)


def test_the_exchange_buffer_may_use_what_is_kept(device):
    """On a full GPU the bytes that the pool keeps are given back before an allocation of the library fails."""
    import gc
    import torch
    import floneum_b200 as fb
    from floneum_b200 import _lib
    L, ex = _lib.load(), ctypes.c_void_p()
    gc.collect()
    torch.cuda.empty_cache()
    mine = fb.Device.gpu(0)
    held = [mine.alloc(500 << 20) for _ in range(4)]
    for p in held:
        mine.free(p)
    rest = torch.empty(torch.cuda.mem_get_info()[0] - (400 << 20), dtype=torch.uint8, device="cuda")
    try:
        assert torch.cuda.mem_get_info()[0] < 900 << 20
        _lib.check(L.fusor_cuda_exchange_create(mine.handle, 1, 0, 1 << 27, ctypes.byref(ex)), mine.handle)  # two parities of 512 MB
        L.fusor_cuda_exchange_destroy(ex)
    finally:
        del rest
        torch.cuda.empty_cache()


def test_kept_buffers_can_be_asked_back(device):
    import torch
    import floneum_b200 as fb
    mine = fb.Device.gpu(0)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    held = [mine.alloc(500 << 20) for _ in range(4)]
    for p in held:
        mine.free(p)
    assert torch.cuda.mem_get_info()[0] < before - (1 << 30)  # kept
    mine.trim()
    assert torch.cuda.mem_get_info()[0] > before - (64 << 20)
    q = mine.alloc(500 << 20)
    mine.free(q)

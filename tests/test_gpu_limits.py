"""What the attention and projection entry points refuse, and the ends of what they take."""
import ctypes

import numpy as np
import pytest

from conftest import assert_close
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,D", [(0, 8), (1, 16), (0, 10)])
@pytest.mark.parametrize("axis", [0, 1])
def test_more_than_65535_batches_or_heads(device, dtype, D, axis):
    import floneum_b200 as fb
    shape = [1, 1, 1, D]
    shape[axis] = 65536
    x = fb.Tensor.zeros(device, tuple(shape), dtype)
    with pytest.raises(fb.FusorCudaError, match="65535"):
        x.flash_attention(x, x, 1.0)
    shape[axis] = 65535
    x = fb.Tensor.zeros(device, tuple(shape), dtype)
    assert not x.flash_attention(x, x, 1.0).as_slice().any()


def _t4(t, shape, stride, skip=0):
    from floneum_b200 import _lib
    x = _lib.Tensor4()
    x.data, x.dtype = t.ptr + skip * (4 if t.dtype == 0 else 2), t.dtype
    for i in range(4):
        x.shape[i], x.stride[i] = shape[i], stride[i]
    return x


@pytest.mark.parametrize("rows", [1, 16, 40, 3000])  # each of the projection's kernels
@pytest.mark.parametrize("which", ["weight", "out"])
def test_projection_rows_in_descending_order_are_refused(device, rows, which):
    import floneum_b200 as fb
    from floneum_b200 import _lib
    K, N = 128, 1024
    if rows == 1 and which == "out":
        pytest.skip("one row has no order")
    a, w, o = fb.Tensor.zeros(device, (rows, K), 1), fb.Tensor.zeros(device, (N, K), 1), fb.Tensor.zeros(device, (rows, N))
    ca = _t4(a, (1, 1, rows, K), (rows * K, rows * K, K, 1))
    up, down = which == "weight", which == "out"
    cw = _t4(w, (1, 1, N, K), (N * K, N * K, -K, 1), (N - 1) * K) if up else _t4(w, (1, 1, N, K), (N * K, N * K, K, 1))
    co = _t4(o, (1, 1, rows, N), (rows * N, rows * N, -N, 1), (rows - 1) * N) if down else _t4(o, (1, 1, rows, N), (rows * N, rows * N, N, 1))
    rc = _lib.load().fusor_cuda_attention_out_proj(device.handle, ctypes.byref(ca), ctypes.byref(cw), None, ctypes.byref(co))
    with pytest.raises(fb.FusorCudaError):
        _lib.check(rc, device.handle)
    device.synchronize()


@pytest.mark.parametrize("dtype,D", [(0, 64), (2, 64), (0, 136), (1, 128)])
def test_a_window_wider_than_the_keys_is_causal(device, dtype, D):
    import floneum_b200 as fb
    from floneum_b200 import _lib
    rng = np.random.default_rng(D)
    rnd = {0: lambda a: a, 1: O.bf16_round, 2: lambda a: a.astype(np.float16).astype(np.float32)}[dtype]
    q, k, v = (rnd(rng.standard_normal((1, 2, 200, D), dtype=np.float32)) for _ in range(3))
    tq, tk, tv = (fb.Tensor.from_slice(device, a.shape, a, dtype) for a in (q, k, v))
    out = fb.Tensor.empty(device, q.shape)
    c = [t._c4() for t in (tq, tk, tv, out)]
    for window in (200, 2 ** 31 - 1):
        _lib.check(_lib.load().fusor_cuda_flash_attention(device.handle, ctypes.byref(c[0]), ctypes.byref(c[1]), ctypes.byref(c[2]), ctypes.c_float(D ** -0.5),
                                                          None, _lib.MASK_SLIDING, window, ctypes.byref(c[3])), device.handle)
        want = O.flash_attention(q, k, v, D ** -0.5, mask_kind=O.MASK_CAUSAL)
        assert_close(out.as_slice(), want, *((2e-3, 2e-4) if dtype and D == 128 else (2e-5, 2e-6)), what=f"window {window}")

"""Attention on warp-level MMAs: 16-bit tensors the tcgen05 kernels do not take (head_dim other than 128, strided mask rows) and
f32 tensors, at the edges of their 64-query and 64- / 32-key tiles, against the CPU oracle.

Both kernels keep f32 accuracy (weights and f32 operands are sums of 16-bit terms), so they are held to the bounds of the
f32-arithmetic kernel, 2e-5 / 2e-6 on N(0, 1) data, plus half a unit in the last place of a 16-bit result (|out| < 8)."""
import numpy as np
import pytest

from conftest import assert_close
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _rounded(a, dtype):
    return O.bf16_round(a) if dtype == 1 else a.astype(np.float16).astype(np.float32) if dtype == 2 else a


def _case(device, dtype, out_dtype, B, Hq, Hkv, Sq, Skv, D, kind):
    import floneum_b200 as fb
    rng = np.random.default_rng(1000 * Sq + 10 * Skv + D)
    q, k, v = (_rounded(rng.standard_normal(s, dtype=np.float32), dtype) for s in ((B, Hq, Sq, D), (B, Hkv, Skv, D), (B, Hkv, Skv, D)))
    scale = np.float32(D ** -0.5)
    T = lambda a, dt=0: fb.Tensor.from_slice(device, a.shape, np.ascontiguousarray(a), dt)
    if kind == "none":
        mask, want = None, O.flash_attention(q, k, v, scale)
    elif kind == "causal":
        mask = (fb.MaskCache().get_mask(Sq, Skv - Sq, None, device), fb.MaskKind.QKMask)
        want = O.flash_attention(q, k, v, scale, mask_kind=O.MASK_CAUSAL)
    elif kind == "window":
        w = max(1, Sq // 3)
        assert Sq == Skv
        mask = (fb.MaskCache().get_mask(Sq, 0, w, device), fb.MaskKind.QKMask)
        want = O.flash_attention(q, k, v, scale, O.get_mask(Sq, 0, w), O.MASK_QK)
    elif kind == "key":
        m = np.where(np.arange(Skv)[None] < np.array([[max(1, Skv - 5 * b)] for b in range(B)]), 0.0, -np.inf).astype(np.float32)
        mask, want = (T(m), fb.MaskKind.BatchKeyMask), O.flash_attention(q, k, v, scale, m, O.MASK_BATCH_KEY)
    else:  # an additive [Sq, Skv] tensor whose rows are not contiguous (the transpose of a [Skv, Sq] one)
        m = np.where(rng.random((Sq, Skv)) < 0.2, -np.inf, rng.uniform(-1, 1, (Sq, Skv))).astype(np.float32)
        m[:, 0] = 0.0
        base = T(np.ascontiguousarray(m.T))
        mask, want = (fb.Tensor(device, base.ptr, (Sq, Skv), 0, (1, Sq), owner=base), fb.MaskKind.QKMask), O.flash_attention(q, k, v, scale, m, O.MASK_QK)
    before = device.launch_count()
    tq, tk, tv = T(q, dtype), T(k, dtype), T(v, dtype)
    got = tq.flash_attention(tk, tv, float(scale), mask, out_dtype)
    assert device.launch_count() - before == 1
    half_ulp = {0: 0.0, 1: 2.0 ** -7, 2: 2.0 ** -10}[out_dtype]
    assert_close(got.as_slice(), want, 2e-5 + half_ulp, 2e-6 + half_ulp / 4, f"{dtype}->{out_dtype} {B}x{Hq}/{Hkv}x{Sq}/{Skv}x{D} {kind}")


SHAPES = [
    (1, 2, 1, 1, 1, 64, "none"), (1, 1, 1, 63, 64, 64, "causal"), (2, 4, 2, 64, 64, 64, "causal"), (1, 2, 2, 65, 65, 64, "window"),
    (1, 2, 1, 129, 190, 64, "causal"), (3, 2, 2, 70, 70, 64, "key"), (1, 2, 1, 66, 129, 64, "strided"), (1, 2, 2, 40, 31, 32, "none"),
    (1, 2, 1, 33, 33, 24, "causal"), (1, 2, 2, 100, 100, 96, "window"), (2, 2, 1, 65, 127, 80, "causal"), (2, 2, 1, 65, 33, 104, "key"),
    (1, 3, 1, 130, 130, 128, "strided"),
]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("dtype,out_dtype", [(1, 0), (2, 2)])
def test_16_bit_tensors(device, dtype, out_dtype, shape):
    _case(device, dtype, out_dtype, *shape)


@pytest.mark.parametrize("shape", SHAPES + [(2, 2, 1, 64, 95, 128, "causal"), (1, 2, 2, 33, 33, 128, "window"), (2, 2, 1, 31, 32, 8, "key")])
def test_f32_tensors(device, shape):
    _case(device, 0, 0, *shape)

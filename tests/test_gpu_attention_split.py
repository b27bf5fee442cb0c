"""Tensor-core attention with few query tiles: the keys of a tile shared by a cluster of 2, 4 or 8 CTAs, parts with no tile and
rows that one part masks whole included, against the oracle (tolerances of the 11-bit softmax weights)."""
import numpy as np
import pytest

from conftest import assert_close
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,Hq,Hkv,Sq,Skv,kind", [
    (1, 2, 1, 1, 640, "none"), (1, 4, 2, 130, 700, "causal"), (1, 32, 8, 200, 1200, "causal"), (1, 8, 1, 300, 2700, "causal"), (1, 3, 3, 1100, 1100, "causal"),
    (2, 2, 2, 77, 3000, "key"), (1, 2, 2, 1500, 1500, "window"), (1, 2, 1, 150, 900, "tensor"), (1, 16, 4, 513, 2049, "none"), (1, 1, 1, 2600, 2600, "causal"),
])
@pytest.mark.parametrize("dtype,out_dtype", [(1, 0), (2, 2), (1, 1)])
def test_parts_of_the_keys(device, B, Hq, Hkv, Sq, Skv, kind, dtype, out_dtype):
    import floneum_b200 as fb
    rng = np.random.default_rng(Sq + Skv)
    rnd = O.bf16_round if dtype == 1 else lambda a: a.astype(np.float16).astype(np.float32)
    q, k, v = (rnd(rng.standard_normal(s, dtype=np.float32)) for s in ((B, Hq, Sq, 128), (B, Hkv, Skv, 128), (B, Hkv, Skv, 128)))
    scale = float(np.float32(128 ** -0.5))
    T = lambda a, dt=0: fb.Tensor.from_slice(device, a.shape, np.ascontiguousarray(a), dt)
    if kind == "none":
        mask, want = None, O.flash_attention(q, k, v, scale)
    elif kind == "causal":
        mask = (fb.MaskCache().get_mask(Sq, Skv - Sq, None, device), fb.MaskKind.QKMask)
        want = O.flash_attention(q, k, v, scale, mask_kind=O.MASK_CAUSAL)
    elif kind == "window":
        mask = (fb.MaskCache().get_mask(Sq, 0, 700, device), fb.MaskKind.QKMask)
        want = O.flash_attention(q, k, v, scale, O.get_mask(Sq, 0, 700), O.MASK_QK)
    elif kind == "key":  # the second sequence ends long before the last part begins
        m = np.where(np.arange(Skv)[None] < np.array([[Skv], [500]]), 0.0, -np.inf).astype(np.float32)
        mask, want = (T(m), fb.MaskKind.BatchKeyMask), O.flash_attention(q, k, v, scale, m, O.MASK_BATCH_KEY)
    else:
        m = np.where(rng.random((Sq, Skv)) < 0.3, -np.inf, rng.uniform(-1, 1, (Sq, Skv))).astype(np.float32)
        m[:, 400:] = np.where(np.arange(Sq)[:, None] % 2 == 0, -np.inf, m[:, 400:])  # every second row lives in the first part alone
        m[:, 0] = 0.0
        mask, want = (T(m), fb.MaskKind.QKMask), O.flash_attention(q, k, v, scale, m, O.MASK_QK)
    got = T(q, dtype).flash_attention(T(k, dtype), T(v, dtype), scale, mask, out_dtype).as_slice()
    half_ulp = {0: 0.0, 1: 2.0 ** -9, 2: 2.0 ** -12}[out_dtype] * 4.0  # |out| < 4
    assert_close(got, want, 2e-3 + half_ulp, 2e-4 + half_ulp / 4, f"{B}x{Hq}/{Hkv}x{Sq}/{Skv} {kind}")

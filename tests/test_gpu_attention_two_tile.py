"""The kernel with two query tiles per CTA, which takes calls with more 256-row items than SMs: each mask, key offsets, an idle
second tile and a nearly empty one, f16 tensors, values beyond f16, every output type.  That it is this kernel is asserted."""
import numpy as np
import pytest

from conftest import assert_close
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,Hq,Hkv,Sq,Skv,kind", [
    (1, 50, 10, 600, 600, "causal"),   # 150 items; the last of each head has an idle second tile
    (1, 75, 15, 385, 385, "causal"),   # one row in the second tile of the last item
    (1, 50, 10, 600, 1100, "causal"),  # keys before the first row
    (1, 50, 10, 513, 200, "none"),
    (2, 40, 8, 400, 777, "none"),
    (2, 40, 8, 500, 500, "window"),
    (1, 50, 10, 700, 700, "window"),
    (8, 10, 5, 450, 450, "key"),
    (8, 10, 2, 400, 1001, "key"),
])
@pytest.mark.parametrize("dtype,out_dtype", [(1, 0), (1, 1), (2, 0), (2, 2)])
def test_two_tiles(device, B, Hq, Hkv, Sq, Skv, kind, dtype, out_dtype):
    import floneum_b200 as fb
    rng = np.random.default_rng(Sq + Skv + Hq)
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
        mask = (fb.MaskCache().get_mask(Sq, 0, 150, device), fb.MaskKind.QKMask)
        want = O.flash_attention(q, k, v, scale, O.get_mask(Sq, 0, 150), O.MASK_QK)
    else:
        m = np.where(np.arange(Skv)[None] < np.linspace(Skv, 70, B).astype(int)[:, None], rng.uniform(-1, 1, (B, Skv)), -np.inf).astype(np.float32)
        mask, want = (T(m), fb.MaskKind.BatchKeyMask), O.flash_attention(q, k, v, scale, m, O.MASK_BATCH_KEY)
    got = T(q, dtype).flash_attention(T(k, dtype), T(v, dtype), scale, mask, out_dtype)
    assert device.last_kernel() == "prefill2_sm100_kernel"
    half_ulp = {0: 0.0, 1: 2.0 ** -9, 2: 2.0 ** -12}[out_dtype] * 4.0  # |out| < 4
    assert_close(got.as_slice(), want, 2e-3 + half_ulp, 2e-4 + half_ulp / 4, f"{B}x{Hq}/{Hkv}x{Sq}/{Skv} {kind}")


def test_values_beyond_f16(device):
    """|v| > 65504: bf16 weights and values (8 significant bits)."""
    import floneum_b200 as fb
    rng = np.random.default_rng(77)
    q, k, v = (O.bf16_round(rng.standard_normal((1, h, 600, 128), dtype=np.float32)) for h in (50, 10, 10))
    v[0, 3, 5, 7] = float(np.ravel(O.bf16_round(np.float32(1.0e5)))[0])
    scale = float(np.float32(128 ** -0.5))
    tq, tk, tv = (fb.Tensor.from_slice(device, a.shape, a, 1) for a in (q, k, v))
    got = tq.flash_attention(tk, tv, scale, (fb.MaskCache().get_mask(600, 0, None, device), fb.MaskKind.QKMask), 0)
    assert device.last_kernel() == "prefill2_sm100_kernel"
    want = O.flash_attention(q, k, v, scale, mask_kind=O.MASK_CAUSAL)
    rel = np.abs(got.as_slice() - want) / (1.0 + np.abs(want))
    assert np.isfinite(rel).all() and rel.max() < 8e-3, rel.max()

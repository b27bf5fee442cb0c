"""Infinities, NaN and values next to the largest float in the operands of the f32-accuracy attention kernels: what f32 arithmetic
gives.  An infinite V of positive weight gives its infinity in its own column and nothing else; a key whose score is -inf has
no weight; a NaN spoils the column (V) or the row (Q, K) it belongs to."""
import numpy as np
import pytest

from conftest import assert_close
from oracle import oracle as O

pytestmark = pytest.mark.gpu

FORMS = [(0, 64), (0, 128), (0, 24), (1, 64), (2, 64), (2, 96), (0, 136)]  # dtype, head_dim


def _case(device, dtype, D, change, causal, Sq=70, Skv=150):
    import floneum_b200 as fb
    rng = np.random.default_rng(D + Sq)
    rnd = {0: lambda a: a, 1: O.bf16_round, 2: lambda a: a.astype(np.float16).astype(np.float32)}[dtype]
    q, k, v = (rnd(rng.standard_normal(s, dtype=np.float32)) for s in ((1, 2, Sq, D), (1, 1, Skv, D), (1, 1, Skv, D)))
    q[..., 1] = np.maximum(np.abs(q[..., 1]), np.float32(0.25))  # so that the sign of an infinite product is known
    clean = [a.copy() for a in (q, k, v)]
    change(q, k, v)
    T = lambda a: fb.Tensor.from_slice(device, a.shape, np.ascontiguousarray(a), dtype)
    mask = (fb.MaskCache().get_mask(Sq, Skv - Sq, None, device), fb.MaskKind.QKMask) if causal else None
    got = T(q).flash_attention(T(k), T(v), float(D ** -0.5), mask, 0).as_slice()
    want = O.flash_attention(*clean, D ** -0.5, mask_kind=O.MASK_CAUSAL if causal else O.MASK_NONE)
    return got, want, clean


@pytest.mark.parametrize("dtype,D", FORMS)
def test_infinite_value(device, dtype, D):
    def change(q, k, v):
        v[0, 0, 100, 3], v[0, 0, 20, 7] = np.inf, -np.inf
    got, want, _ = _case(device, dtype, D, change, causal=True)  # row i sees keys 0 .. 80 + i, in whole tiles
    # (rows whose tile holds key 100 beyond their last key multiply it by a weight of zero: not looked at)
    assert np.isposinf(got[:, :, 20:, 3]).all() and np.isneginf(got[..., 7]).all()
    keep = np.ones(D, bool)
    keep[[3, 7]] = False
    assert_close(got[..., keep], want[..., keep], 2e-5, 2e-6)


@pytest.mark.parametrize("dtype,D", FORMS)
def test_key_whose_score_is_minus_infinity(device, dtype, D):
    def change(q, k, v):
        k[0, 0, 33, 1] = -np.inf
    got, _, (q, k, v) = _case(device, dtype, D, change, causal=False)
    m = np.zeros((1, k.shape[2]), np.float32)
    m[0, 33] = -np.inf
    assert_close(got, O.flash_attention(q, k, v, D ** -0.5, m, O.MASK_BATCH_KEY), 2e-5, 2e-6)


@pytest.mark.parametrize("dtype,D", FORMS)
def test_nan_stays_where_it_is(device, dtype, D):
    def change(q, k, v):
        v[0, 0, 9, 5] = np.nan
        q[0, 1, 41, 2] = np.nan
    got, want, _ = _case(device, dtype, D, change, causal=False)
    assert np.isnan(got[..., 5]).all() and np.isnan(got[0, 1, 41]).all()
    keep = np.ones(D, bool)
    keep[5] = False
    got[0, 1, 41], want[0, 1, 41] = 0.0, 0.0
    assert_close(got[..., keep], want[..., keep], 2e-5, 2e-6)


@pytest.mark.parametrize("D", [64, 128, 24, 136])
def test_values_next_to_the_largest_float(device, D):
    """3.4e38 has no 16-bit neighbour above it, 3.392e38 rounds up to one."""
    def change(q, k, v):
        v[0, 0, 40, 3], v[0, 0, 77, 4] = 3.4e38, -3.392e38
    got, want, (q, k, v) = _case(device, 0, D, change, causal=False)
    s = np.einsum("bhqd,bkd->bhqk", q.astype(np.float64), k[:, 0]) * D ** -0.5
    p = np.exp(s - s.max(-1, keepdims=True))
    p /= p.sum(-1, keepdims=True)
    # (the other keys' values lie far below)
    assert np.allclose(got[..., 3], p[..., 40] * 3.4e38, rtol=2e-5) and np.allclose(got[..., 4], p[..., 77] * -3.392e38, rtol=2e-5)
    keep = np.ones(D, bool)
    keep[[3, 4]] = False
    assert_close(got[..., keep], want[..., keep], 2e-5, 2e-6)

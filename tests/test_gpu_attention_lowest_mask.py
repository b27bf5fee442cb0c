"""Additive masks with finite values down to the lowest float (the usual value of padding masks) and -inf, mixed in every way a row
can hold them, against the CPU oracle: a row in which every key carries the lowest value is the mean of V, one that mixes it
with -inf the mean over its finite keys, and only a row of -inf alone is NaN.

Bounds: those of each path on N(0, 1) data (f32 arithmetic 2e-5 / 2e-6, the 11-bit weights of the tcgen05 kernels 2e-3 / 2e-4)."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

LOWEST = float(np.finfo(np.float32).min)


def _rows(rng, n, keys):
    """n mask rows over `keys` keys: all lowest, all -inf, lowest and -inf, lowest and 0, -2.4e38 (just below the overflow of a
    product with log2 e) alone, -1e4, lowest up to the last key, and mixtures of all of these."""
    m = np.zeros((n, keys), np.float32)
    for i in range(n):
        kind = i % 8
        if kind == 0: m[i] = LOWEST
        elif kind == 1: m[i] = -np.inf
        elif kind == 2: m[i] = np.where(rng.random(keys) < 0.5, LOWEST, -np.inf); m[i, keys // 2] = LOWEST
        elif kind == 3: m[i] = np.where(rng.random(keys) < 0.5, LOWEST, 0.0); m[i, keys // 3] = 0.0
        elif kind == 4: m[i] = -2.4e38 if i % 16 == 4 else -1e9
        elif kind == 5: m[i] = -1e4
        elif kind == 6: m[i] = LOWEST; m[i, -1] = 0.5
        else: m[i] = rng.choice(np.array([0.0, LOWEST, -np.inf, -1e4, 1.0], np.float32), keys); m[i, 0] = 0.0
    return m


def _check(device, dtype, D, kind, B, Hq, Hkv, Sq, Skv, max_tol, mean_tol):
    import floneum_b200 as fb
    rng = np.random.default_rng(D + Sq + Skv)
    rnd = {0: lambda a: a, 1: O.bf16_round, 2: lambda a: a.astype(np.float16).astype(np.float32)}[dtype]
    q, k, v = (rnd(rng.standard_normal(s, dtype=np.float32)) for s in ((B, Hq, Sq, D), (B, Hkv, Skv, D), (B, Hkv, Skv, D)))
    scale = float(np.float32(D ** -0.5))
    T = lambda a, dt=0: fb.Tensor.from_slice(device, a.shape, np.ascontiguousarray(a), dt)
    m = _rows(rng, Sq if kind == "tensor" else B, Skv)
    want = O.flash_attention(q, k, v, scale, m, O.MASK_QK if kind == "tensor" else O.MASK_BATCH_KEY)
    got = T(q, dtype).flash_attention(T(k, dtype), T(v, dtype), scale, (T(m), fb.MaskKind.QKMask if kind == "tensor" else fb.MaskKind.BatchKeyMask), 0).as_slice()
    assert np.array_equal(np.isnan(got), np.isnan(want)), f"{np.isnan(got).sum()} NaN, {np.isnan(want).sum()} expected"
    assert np.isnan(want).any() and not np.isnan(want).all()
    err = np.where(np.isnan(want), 0.0, np.abs(got.astype(np.float64) - want))
    assert err.mean() <= mean_tol, err.mean()
    # beside -1e4 a sum keeps multiples of 2^-10: scores that differ in their last place may round to neighbours, which moves a
    # weight (below a tenth) by 2^-10 of it
    alone = np.arange(Sq if kind == "tensor" else B) % 8 == 5
    rows = np.broadcast_to(alone[None, None, :, None] if kind == "tensor" else alone[:, None, None, None], err.shape)
    assert err[~rows].max() <= max_tol and err[rows].max() <= max_tol + 2.0 ** -10 / 10 * 8, (err[~rows].max(), err[rows].max())


@pytest.mark.parametrize("kind,B,Sq,Skv", [("tensor", 1, 72, 200), ("key", 8, 40, 131)])
@pytest.mark.parametrize("dtype,D", [(0, 64), (0, 128), (1, 64), (2, 64), (1, 96), (2, 32), (0, 192), (2, 136), (0, 30)])
def test_f32_accuracy_kernels(device, dtype, D, kind, B, Sq, Skv):
    """Warp MMAs on f32 and on 16-bit tensors, and the general kernel (head_dim above 128 or not a multiple of 8)."""
    _check(device, dtype, D, kind, B, 4, 2, Sq, Skv, 2e-5, 2e-6)


@pytest.mark.parametrize("kind,B,Hq,Hkv,Sq,Skv", [
    ("tensor", 1, 4, 2, 72, 200), ("key", 8, 4, 2, 40, 131), ("tensor", 1, 2, 1, 130, 1100), ("key", 8, 1, 1, 70, 1300),  # a tile's keys on one CTA, on several
    ("key", 8, 20, 4, 400, 400),                                                                                         # two query tiles per CTA
])
@pytest.mark.parametrize("dtype", [1, 2])
def test_tcgen05_kernels(device, dtype, kind, B, Hq, Hkv, Sq, Skv):
    _check(device, dtype, 128, kind, B, Hq, Hkv, Sq, Skv, 2e-3, 2e-4)

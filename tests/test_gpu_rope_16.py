"""RoPE (+ append) on tensors that all have one 16-bit type, at the edges of the head groups and of the smallest calls: equal to
the oracle's f32 result rounded once, bit for bit."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _rounded(a, dtype):
    return O.bf16_round(a) if dtype == 1 else a.astype(np.float16).astype(np.float32)


@pytest.mark.parametrize("interleaved", [False, True])
@pytest.mark.parametrize("dtype", [1, 2])
@pytest.mark.parametrize("B,Hq,Hkv,n,D,start", [(1, 1, 1, 1, 128, 0), (2, 5, 5, 3, 64, 7), (1, 9, 3, 17, 128, -1), (3, 32, 8, 40, 128, 2), (1, 8, 2, 3000, 64, 0),
                                                (2, 20, 10, 2500, 128, 0)])
def test_rope_append_16_bit(device, B, Hq, Hkv, n, D, start, dtype, interleaved):
    import floneum_b200 as fb
    rng = np.random.default_rng(100 * n + Hq)
    old = 5 if start < 0 else 0  # tokens already in the cache: with start < 0 they are the position
    rows = n + max(start, old)
    q, k, v = (_rounded(rng.standard_normal((B, h, n, D), dtype=np.float32), dtype) for h in (Hq, Hkv, Hkv))
    cos, sin = O.rope_tables(D, rows, 10000.0)
    T = lambda a, dt=dtype: fb.Tensor.from_slice(device, a.shape, np.ascontiguousarray(a), dt)
    pages = (n + old + 15) // 16
    cache = fb.PagedKvCache(device, B, Hkv, D, B * pages, pages)
    if old:
        cache.append(T(k[:, :, :old]), T(v[:, :, :old]))
    tc, ts = T(cos, 0), T(sin, 0)
    got = cache.rope_append(T(q), T(k), T(v), tc, ts, start, interleaved)
    at = start if start >= 0 else old
    assert np.array_equal(got.as_slice(), _rounded(O.rope(q, cos, sin, at, interleaved), dtype))
    gk, gv = cache.gather(B, n + old)
    assert np.array_equal(gk.as_slice()[:, :, old:], O.bf16_round(O.rope(k, cos, sin, at, interleaved)))
    assert np.array_equal(gv.as_slice()[:, :, old:], O.bf16_round(v))
    alone = T(k).rope_interleaved(tc, ts) if interleaved else T(k).rope(tc, ts)
    assert np.array_equal(alone.as_slice(), _rounded(O.rope(k, cos, sin, 0, interleaved), dtype))

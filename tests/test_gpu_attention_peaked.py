"""Attention at f32 accuracy where few weights carry a row: small weights that add up, scores of tens of nats, operands whose
mantissas are the worst for a split into 16-bit terms.  Against 64-bit softmax attention of the same inputs.

With V = 1 on every key but the peak, V = 0 there, a row is the sum of its n small weights over their total: what it may be off
by is the error of a score (the dot product's sums, below 6 x 2^-22 of a score of 20 nats, so 3e-5 of each weight) and, where
weights are two f16 terms under a scale of 2^14, 2^-39 per weight."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _attention64(q, k, v, scale):
    s = q.astype(np.float64) @ np.swapaxes(k.astype(np.float64), -1, -2) * scale
    p = np.exp(s - s.max(-1, keepdims=True))
    return p @ v.astype(np.float64) / p.sum(-1, keepdims=True)


def _run(device, q, k, v, scale, dtype):
    import floneum_b200 as fb
    T = lambda a: fb.Tensor.from_slice(device, a.shape, np.ascontiguousarray(a), dtype)
    return T(q).flash_attention(T(k), T(v), float(scale), None, 0).as_slice().astype(np.float64)


@pytest.mark.parametrize("nats", [8, 14, 17.4, 20])
@pytest.mark.parametrize("dtype,D,keys", [(2, 64, 2048), (2, 32, 300), (2, 96, 4099), (1, 64, 2048), (0, 64, 2048), (0, 128, 777), (0, 160, 777)])
def test_small_weights_that_add_up(device, dtype, D, keys, nats):
    rng = np.random.default_rng(int(10 * nats) + D)
    rnd = {0: lambda a: a, 1: O.bf16_round, 2: lambda a: a.astype(np.float16).astype(np.float32)}[dtype]
    u = rng.standard_normal(D).astype(np.float32)
    u *= np.float32(np.sqrt(nats) * D ** 0.25 / np.linalg.norm(u))
    q = rnd((u + 0.02 * rng.standard_normal((1, 1, 70, D))).astype(np.float32))
    k = rnd((0.02 * rng.standard_normal((1, 1, keys, D)) + u * (np.arange(keys) == keys // 3)[:, None]).astype(np.float32))
    v = np.ones((1, 1, keys, D), np.float32)
    v[:, :, keys // 3] = 0.0
    scale = np.float32(D ** -0.5)
    want = _attention64(q, k, v, float(scale))
    got = _run(device, q, k, v, scale, dtype)
    bound = 3e-5 * want + (keys * 2.0 ** -39 if dtype == 2 else 0.0)
    assert (np.abs(got - want) <= bound).all(), (np.abs(got - want) / want).max()


@pytest.mark.parametrize("D", [8, 64, 128, 192])
def test_products_of_f32_values_with_long_mantissas(device, D):
    """Two keys whose scores of 40 nats are one product each, of a value whose low 16 mantissa bits are set and of the next value,
    which has them clear.  In units of 2^-24 of 40 nats their difference may be off by 2 (what a split into three terms leaves out
    of the product) and by 2 for the cut at the end of each of the two sums."""
    rng = np.random.default_rng(D)
    bits = np.concatenate([[0x3F80FFFF], 0x3F80FFFF | (rng.integers(0, 128, 63) << 16)]).astype(np.uint32)
    x = bits.view(np.float32)
    q = np.zeros((1, 64, 64, D), np.float32)
    k = np.zeros((1, 64, 2, D), np.float32)
    q[0, :, :, 3] = x
    k[0, :, 0, 3], k[0, :, 1, 3] = x, (bits + 1).view(np.float32)
    v = np.zeros((1, 64, 2, D), np.float32)
    v[0, :, 0], v[0, :, 1] = 1.0, -1.0
    top = x[None, :] * x[:, None].astype(np.float64)  # [head, row]
    for scale in (40.0, 20.0, 10.0):
        want = _attention64(q, k, v, scale)
        got = _run(device, q, k, v, scale, 0)
        slope = (1.0 - want ** 2) / 2.0  # of the result in the difference of the scores
        assert (np.abs(got - want) <= slope * (scale * top[None, :, :, None]) * 6 * 2.0 ** -24 + 2.0 ** -22).all(), np.abs(got - want).max()


def test_values_are_carried_whole(device):
    """One key: the result is V itself, every bit of it."""
    rng = np.random.default_rng(5)
    for D in (64, 128):
        q, k = (rng.standard_normal((1, 2, n, D), dtype=np.float32) for n in (3, 1))
        v = (rng.standard_normal((1, 2, 1, D)) * 10.0 ** rng.integers(-20, 20, (1, 2, 1, D))).astype(np.float32)
        assert np.array_equal(_run(device, q, k, v, 0.1, 0), np.broadcast_to(v, (1, 2, 3, D)).astype(np.float64))


@pytest.mark.parametrize("dtype", [0, 1, 2])
@pytest.mark.parametrize("keys", [17, 100, 300])
def test_error_of_short_rows(device, dtype, keys):
    """Relative error of the whole result over ten inputs whose keys are 5 % outliers: no larger than that of f32 sums in order, which
    is what served these tensors first.  The sums of such a row: D products (a rounding of half a unit each, the running sum
    half the result on average), then one product per key: measured 0.7e-7 (bf16, 17 keys) to 4.6e-7 (f32, 300 keys)."""
    D, errs, refs = 64, [], []
    rnd = {0: lambda a: a, 1: O.bf16_round, 2: lambda a: a.astype(np.float16).astype(np.float32)}[dtype]
    for seed in range(10):
        rng = np.random.default_rng(seed)
        q, k, v = (rnd((0.5 * rng.standard_normal((2, 4, keys, D))).astype(np.float32)) for _ in range(3))
        k = rnd(np.where(rng.random((2, 4, keys, 1)) < 0.05, k * 8, k).astype(np.float32))
        scale = np.float32(D ** -0.5)
        want = _attention64(q, k, v, float(scale))
        errs.append(np.linalg.norm(_run(device, q, k, v, scale, dtype) - want) / np.linalg.norm(want))
        # the same in f32, every sum in order
        s = np.zeros((2, 4, keys, keys), np.float32)
        for d in range(D):
            s += q[..., d, None] * k[..., None, :, d]
        s *= scale
        p = np.exp(s - s.max(-1, keepdims=True))
        o, total = np.zeros(q.shape, np.float32), np.zeros(s.shape[:-1], np.float32)
        for j in range(keys):
            o += p[..., j, None] * v[..., j, None, :]
            total += p[..., j]
        refs.append(np.linalg.norm(o / total[..., None] - want) / np.linalg.norm(want))
    assert np.mean(errs) <= 1.05 * np.mean(refs), (np.mean(errs), np.mean(refs))

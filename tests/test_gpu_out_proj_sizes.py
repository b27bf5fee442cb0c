"""Output projection at the edges of its four kernels (a few rows, K split over a cluster, CTA pairs, single CTAs) against the oracle.
Which of them runs (for 148 SMs) is asserted.

The products are exact in f32 and the sums have up to 4096 terms of N(0, 1) x N(0, 1 / K): another order of summation moves a
result of size ~1 by a few units of sqrt(K) 2^-24 ~ 4e-6, well inside the bounds used here."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,Hq,S,D,N,kernel", [
    # a few rows: 1, 8, 9, 16; ragged N
    (1, 1, 1, 64, 8, "rows"), (1, 32, 1, 128, 4096, "rows"), (8, 4, 1, 64, 136, "rows"), (3, 5, 3, 64, 24, "rows"), (2, 8, 8, 128, 264, "rows"),
    # K split 4, 1, 8, 2 ways and not at all
    (1, 8, 17, 128, 40, "split"), (17, 2, 1, 64, 128, "split"), (1, 32, 129, 128, 384, "split"), (2, 16, 130, 128, 1032, "split"), (1, 8, 700, 128, 3000, "split"),
    # CTA pairs: ragged; an odd number of row tiles over three batches, two or three tiles for each pair (accumulators and ring come round)
    (3, 4, 1000, 128, 2056, "pair"), (3, 3, 600, 64, 6800, "pair"),
    # single CTAs: an odd number of row tiles, one wave; two or three tiles for each CTA
    (5, 2, 1100, 64, 512, "single"), (1, 16, 1300, 64, 2000, "single"), (3, 3, 600, 64, 7096, "single"),
])
@pytest.mark.parametrize("out_dtype", [0, 1])
def test_out_proj_sizes(device, B, Hq, S, D, N, kernel, out_dtype):
    import floneum_b200 as fb
    rng = np.random.default_rng(1000 * S + N)
    attn = O.bf16_round(rng.standard_normal((B, S, Hq, D)).astype(np.float32))
    w = O.bf16_round((rng.standard_normal((N, Hq * D)) / np.sqrt(Hq * D)).astype(np.float32))
    bias = rng.standard_normal(N).astype(np.float32)
    base = fb.Tensor.from_slice(device, attn.shape, attn, 1)  # rows of [B, S, Hq, D]: a strided [B, Hq, S, D] view
    view = fb.Tensor(device, base.ptr, (B, Hq, S, D), 1, (S * Hq * D, D, Hq * D, 1), owner=base)
    tw, tb = fb.Tensor.from_slice(device, w.shape, w, 1), fb.Tensor.from_slice(device, bias.shape, bias)
    for b in (None, bias):
        before = device.launch_count()
        got = view.out_proj(tw, tb if b is not None else None, out_dtype)
        assert device.launch_count() - before == 1 and device.last_kernel() == f"oproj_{kernel}_kernel"
        want = O.out_proj(np.ascontiguousarray(attn.transpose(0, 2, 1, 3)), w, b)
        err = np.abs(got.as_slice() - want)
        half_ulp = 2.0 ** -8 * np.abs(want) if out_dtype == 1 else 0.0  # rounding of a bf16 result
        assert (err <= 2e-5 + half_ulp * 1.01).all(), err.max()

"""Decode of short sequences by one cluster per (sequence, kv head): shares of no, one and many pages, more pages than the
ring holds, ragged batches, both head dimensions and every output, against the oracle and the two-launch form."""
import numpy as np
import pytest

from conftest import assert_close
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lens,Hq,Hkv,D", [
    ([128], 8, 8, 128), ([113], 8, 1, 128), ([1411], 32, 8, 128), ([2064], 6, 2, 64), ([4096, 4111], 8, 8, 64), ([1, 16, 17, 300], 12, 4, 128),
    ([600, 40, 129], 32, 16, 128), ([5000], 5, 5, 128), ([200] * 9, 16, 16, 64),
])
@pytest.mark.parametrize("q_dtype,out_dtype", [(1, 0), (0, 1)])
def test_cluster_decode(device, lens, Hq, Hkv, D, q_dtype, out_dtype):
    import floneum_b200 as fb
    rng = np.random.default_rng(sum(lens))
    B, n = len(lens), max(lens)
    k, v = (O.bf16_round(rng.standard_normal((B, Hkv, n, D), dtype=np.float32)) for _ in range(2))
    q = O.bf16_round(rng.standard_normal((B, Hq, 1, D), dtype=np.float32))
    pages = [(x + 15) // 16 for x in lens]
    order = rng.permutation(sum(pages)).astype(np.int32)
    table = np.zeros((B, max(pages)), np.int32)
    kp, vp = (np.zeros((sum(pages), Hkv, 16, D), np.float32) for _ in range(2))
    at = 0
    for b in range(B):
        table[b, :pages[b]] = order[at:at + pages[b]]
        for p in range(pages[b]):
            rows = slice(16 * p, min(16 * p + 16, lens[b]))
            kp[table[b, p], :, :rows.stop - rows.start] = k[b, :, rows]
            vp[table[b, p], :, :rows.stop - rows.start] = v[b, :, rows]
        at += pages[b]
    bits = lambda a: (a.view(np.uint32) >> 16).astype(np.uint16)
    cache = fb.PagedKvCache(device, B, Hkv, D, sum(pages), max(pages))
    cache.write_pages(0, bits(kp), bits(vp))
    cache.set_page_table(table, np.array(lens, np.int32))
    scale = float(D ** -0.5)
    want = np.concatenate([O.flash_attention(q[b:b + 1], k[b:b + 1, :, :lens[b]], v[b:b + 1, :, :lens[b]], scale) for b in range(B)])
    tq = fb.Tensor.from_slice(device, q.shape, q, q_dtype)
    before = device.launch_count()
    got = cache.decode(tq, scale, out_dtype=out_dtype).as_slice()
    assert device.launch_count() - before == 1
    half_ulp = 2.0 ** -8 * np.abs(want).max() if out_dtype == 1 else 0.0
    assert_close(got, want, 1e-4 + half_ulp, 1e-5 + half_ulp / 4, f"{lens}")  # bf16 hi + lo weights: 2^-17 of the values
    rec = cache.decode_partial(tq, scale).as_slice()
    assert_close(rec[:, :, 2:] / rec[:, :, 1:2], want[:, :, 0], 1e-4, 1e-5, "record")
    cache.set_decode_ctas(3)  # a grid of the caller's: the two-launch form
    before = device.launch_count()
    two = cache.decode_partial(tq, scale).as_slice()
    assert device.launch_count() - before == 2
    assert_close(rec[:, :, 0] + np.log(rec[:, :, 1]), two[:, :, 0] + np.log(two[:, :, 1]), 1e-4, 1e-5, "log-sum-exp")

"""Eviction that leaves the rows in place: windows that are full, at page edges and in pools with no page to spare."""
import numpy as np
import pytest

from conftest import assert_close
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _fb():
    import floneum_b200 as fb
    return fb


@pytest.mark.parametrize("D,window,first", [(128, 1, 1), (64, 16, 16), (128, 17, 9), (128, 40, 40), (64, 300, 300)])
def test_full_window(device, D, window, first):
    fb = _fb()
    rng = np.random.default_rng(window)
    B, Hq, Hkv = 2, 4, 2
    steps = [first] + [1] * 18 + [3, 1]
    n = sum(steps)
    k, v = (O.bf16_round(rng.standard_normal((B, Hkv, n, D), dtype=np.float32)) for _ in range(2))
    q = O.bf16_round(rng.standard_normal((B, Hq, n, D), dtype=np.float32))
    T = lambda a: fb.Tensor.from_slice(device, a.shape, np.ascontiguousarray(a))
    cache, at, scale = fb.KvCache.new(2, window), 0, float(D ** -0.5)
    for s in steps:
        ck, cv = cache.append(device, T(k[:, :, at:at + s]), T(v[:, :, at:at + s]))
        at += s
        lo = max(0, at - window)
        assert cache.current_seq_len() == at - lo
        assert np.array_equal(ck.as_slice(), k[:, :, lo:at]) and np.array_equal(cv.as_slice(), v[:, :, lo:at])
        got = T(q[:, :, at - 1:at]).flash_attention(ck, cv, scale).as_slice()
        assert_close(got, O.flash_attention(q[:, :, at - 1:at], k[:, :, lo:at], v[:, :, lo:at], scale), what=f"{at} tokens")


def test_rope_positions_and_partial_records_skip_the_evicted_rows(device):
    fb = _fb()
    rng = np.random.default_rng(2)
    Hq, Hkv, D = 4, 2, 128
    k, v = (O.bf16_round(rng.standard_normal((1, Hkv, 50, D), dtype=np.float32)) for _ in range(2))
    T = lambda a: fb.Tensor.from_slice(device, a.shape, np.ascontiguousarray(a))
    cache = fb.PagedKvCache(device, 1, Hkv, D, num_pages=5, max_pages_per_seq=5)
    cache.append(T(k[:, :, :40]), T(v[:, :, :40]))
    cache.drop_front(0, 30)
    rope = fb.RopeCache.new(D, 64, 10000.0, device)
    cos, sin = O.rope_tables(D, 64, 10000.0)
    q = rng.standard_normal((1, Hq, 10, D), dtype=np.float32)
    rot = cache.rope_append(T(q), T(k[:, :, 40:]), T(v[:, :, 40:]), rope.cos, rope.sin, start_pos=-1)
    assert np.array_equal(rot.as_slice(), O.rope(q, cos, sin, 30, False))  # the position is the cache length, 30
    want_k = np.concatenate([k[:, :, 10:40], O.bf16_round(O.rope(k[:, :, 40:], cos, sin, 30, False))], 2)
    assert np.array_equal(cache.gather(1, 40)[0].as_slice(), want_k)
    q1 = O.bf16_round(q[:, :, :1])
    part = cache.decode_partial(T(q1), float(D ** -0.5)).as_slice()
    assert_close(part[:, :, 2:] / part[:, :, 1:2], O.flash_attention(q1, want_k, v[:, :, 10:], float(D ** -0.5))[:, :, 0], what="record")


def test_a_pool_with_no_page_to_spare_takes_what_fits(device):
    """64 rows in 4 pages: after a drop of 10 the next 10 only fit once the kept rows have moved to the page's start."""
    fb = _fb()
    rng = np.random.default_rng(3)
    T = lambda a: fb.Tensor.from_slice(device, a.shape, np.ascontiguousarray(a))
    k = O.bf16_round(rng.standard_normal((2, 2, 74, 64), dtype=np.float32))
    for pages, per_seq in ((8, 4), (8, 5)):  # the sequence's own limit, then the pool's
        cache = fb.PagedKvCache(device, 2, 2, 64, pages, per_seq)
        cache.append(T(k[:, :, :64]), T(k[:, :, :64]))
        for b in range(2):
            cache.drop_front(b, 54)
        cache.append(T(k[:, :, 64:]), T(k[:, :, 64:]))
        assert np.array_equal(cache.gather(2, 64)[0].as_slice(), k[:, :, 10:])
        with pytest.raises(fb.FusorCudaError, match="pages"):
            cache.append(T(k[:, :, :1]), T(k[:, :, :1]))
        cache.truncate_front(0, 20)
        cache.drop_front(1, 0)
        assert [cache.seq_len(b) for b in range(2)] == [20, 0]
        got = cache.gather(2, 20)[0].as_slice()
        assert np.array_equal(got[0], k[0, :, 54:]) and not got[1].any()


@pytest.mark.parametrize("keep", [0, 20, 33, 38, 1000])
def test_truncate_front_moves_what_drop_front_left(device, keep):
    """After truncate_front the first row of the first page is the oldest row kept, also where the call itself evicts nothing."""
    fb = _fb()
    rng = np.random.default_rng(keep)
    T = lambda a: fb.Tensor.from_slice(device, a.shape, np.ascontiguousarray(a))
    k = O.bf16_round(rng.standard_normal((1, 2, 40, 64), dtype=np.float32))
    cache = fb.PagedKvCache(device, 1, 2, 64, 6, 4)
    cache.append(T(k), T(k))
    cache.drop_front(0, 33)
    cache.truncate_front(0, keep)
    n = min(keep, 33)
    assert cache.seq_len(0) == n
    pages = cache.read_pages(0, 6)[0].reshape(6, 2, 16, 64)
    if n:
        rows = O.bf16_bits(np.ascontiguousarray(k[0, :, 40 - n:40 - n + min(n, 16)]))
        assert any(np.array_equal(pages[p][:, :min(n, 16)], rows) for p in range(6))
        assert np.array_equal(cache.gather(1, n)[0].as_slice(), k[:, :, 40 - n:])


@pytest.mark.parametrize("B", [1, 32, 33])
def test_lengths_reach_the_device_with_and_without_a_launch_that_carries_them(device, B):
    """Appends that map no page bring the lengths in their launch (up to 32 sequences); a drop with no append after it, and the
    plain append kernel, are seen by the next read all the same."""
    fb = _fb()
    rng = np.random.default_rng(B)
    T = lambda a: fb.Tensor.from_slice(device, a.shape, np.ascontiguousarray(a))
    k = O.bf16_round(rng.standard_normal((B, 1, 40, 64), dtype=np.float32))
    q = O.bf16_round(rng.standard_normal((B, 2, 1, 64), dtype=np.float32))
    cache = fb.PagedKvCache(device, B, 1, 64, 4 * B, 4)
    lo = at = 0
    for n, drop in ((20, 0), (3, 0), (1, 5), (0, 2), (9, 0), (2, 17), (1, 0), (0, 1)):
        if n:
            cache.append(T(k[:, :, at:at + n]), T(k[:, :, at:at + n]))
            at += n
        lo += drop
        for b in range(B):
            cache.drop_front(b, at - lo)
        got = cache.decode(T(q), 0.125).as_slice()
        assert_close(got, O.flash_attention(q, k[:, :, lo:at], k[:, :, lo:at], 0.125), what=f"{lo}..{at}")
        assert np.array_equal(cache.gather(B, at - lo)[0].as_slice(), k[:, :, lo:at])


@pytest.mark.parametrize("D,window", [(128, 40), (64, 40), (128, 200), (64, 200)])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_an_evicted_row_has_no_part_in_the_result(device, D, window, bad):
    """A value that is not finite leaves with its row, whether the decode runs in one cluster per head or on the even deal."""
    fb = _fb()
    rng = np.random.default_rng(D + window)
    B, Hq, Hkv, n = 1, 4, 2, window + 20
    k, v = (O.bf16_round(rng.standard_normal((B, Hkv, n, D), dtype=np.float32)) for _ in range(2))
    q = O.bf16_round(rng.standard_normal((B, Hq, 1, D), dtype=np.float32))
    v[0, 0, 3, 1], v[0, 1, 17, 2] = bad, bad
    T = lambda a: fb.Tensor.from_slice(device, a.shape, np.ascontiguousarray(a))
    cache, scale = fb.KvCache.new(2, window), float(D ** -0.5)
    cache.append(device, T(k[:, :, :window]), T(v[:, :, :window]))
    for at in range(window + 1, n + 1):
        ck, cv = cache.append(device, T(k[:, :, at - 1:at]), T(v[:, :, at - 1:at]))
        lo = at - window
        got = T(q).flash_attention(ck, cv, scale).as_slice()
        assert np.isfinite(got[:, :2]).all() == (lo > 3) and np.isfinite(got[:, 2:]).all() == (lo > 17), lo
        if lo > 17:
            assert_close(got, O.flash_attention(q, k[:, :, lo:at], v[:, :, lo:at], scale), what=f"{at} tokens")

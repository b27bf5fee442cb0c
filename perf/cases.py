"""The work a program has this package do, as cases that can be timed and compared: dense attention, paged decode, a
layer's part of a chat session, a sliding-window layer at its limit, the output projection, and RoPE with the append.

Every pass goes through the package's public objects (`Tensor`, `KvCache`, `PagedKvCache`, `RopeCache`, `MaskCache`) on
inputs that torch made on the GPU.  A case is a dict of plain values; `kind` says which of the paths it takes."""
import math

import torch

import floneum_b200 as fb

F32, BF16, F16 = 0, 1, 2
CODE = {"f32": F32, "bf16": BF16, "f16": F16}
TORCH = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}
SIZE = {"f32": 4, "bf16": 2, "f16": 2}
PAGE = 16

_dev = None


def _device():
    """One library context for the life of the process, on a stream of its own (as a server would hold it)."""
    global _dev
    if _dev is None:
        _dev = fb.Device.gpu(0)
    return _dev


class _Borrowed:
    """A library tensor (or a raw device pointer) in the form torch can wrap without a copy."""

    def __init__(self, owner, ptr, shape, code):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": "<f4" if code == F32 else "<i2",
                                         "strides": None, "version": 3}


def _torch(t):
    """The library's result as a torch tensor on the same memory."""
    x = torch.as_tensor(_Borrowed(t, t.ptr, t.shape(), t.dtype), device="cuda")
    return x if t.dtype == F32 else x.view(torch.bfloat16 if t.dtype == BF16 else torch.float16)


def _pools(cache):
    """The page pools of a paged cache as two bf16 torch tensors [pages, kv heads, 16, head_dim]."""
    shape = (cache.num_pages, cache.num_kv_heads, PAGE, cache.head_dim)
    return tuple(torch.as_tensor(_Borrowed(cache, p, shape, BF16), device="cuda").view(torch.bfloat16) for p in cache.pools())


# ------------------------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # A long document through a 70B-shaped layer: 64 query heads on 8 kv heads, 5 % of the keys eight times as large.
        {"name": "prefill_document", "kind": "attention", "B": 1, "Hq": 64, "Hkv": 8, "Sq": 16384, "past": 0, "D": 128, "dtype": "bf16",
         "out": "f32", "mask": "causal", "window": 0, "outliers": True},
        # A batch of full prompts through an 8B-shaped layer: the benchmark's own configuration.
        {"name": "prefill_batch", "kind": "attention", "B": 4, "Hq": 32, "Hkv": 8, "Sq": 4096, "past": 0, "D": 128, "dtype": "bf16",
         "out": "f32", "mask": "causal", "window": 0, "outliers": False},
        # One chat prompt of an odd length: a call of some ten microseconds, where launches and the host count.
        {"name": "prefill_prompt", "kind": "attention", "B": 1, "Hq": 32, "Hkv": 8, "Sq": 777, "past": 0, "D": 128, "dtype": "bf16",
         "out": "bf16", "mask": "causal", "window": 0, "outliers": False},
        # The CPU reference's configuration: f32 tensors of head_dim 64, as the layer passes them when nothing is cast.
        {"name": "attention_f32", "kind": "attention", "B": 1, "Hq": 32, "Hkv": 8, "Sq": 512, "past": 0, "D": 64, "dtype": "f32",
         "out": "f32", "mask": "causal", "window": 0, "outliers": False},
        # A padded batch of an encoder: every row sees every key, a [batch, keys] mask takes the padding out, head_dim 64.
        {"name": "encoder_padded", "kind": "attention", "B": 8, "Hq": 16, "Hkv": 16, "Sq": 300, "past": 0, "D": 64, "dtype": "f16",
         "out": "f16", "mask": "key", "window": 0, "outliers": False},
        # A server's decode step: 64 sequences of 1024 to 8192 tokens in permuted 16-token pages.
        {"name": "decode_batch", "kind": "decode", "B": 64, "Hq": 32, "Hkv": 8, "D": 128, "lo": 1024, "hi": 8192, "dtype": "bf16", "out": "f32"},
        # One sequence of 131072 tokens, 64 query heads.
        {"name": "decode_long", "kind": "decode", "B": 1, "Hq": 64, "Hkv": 8, "D": 128, "lo": 131072, "hi": 131072, "dtype": "bf16", "out": "f32"},
        # One user's next token over a short conversation: the smallest call of all.
        {"name": "decode_chat", "kind": "decode", "B": 1, "Hq": 32, "Hkv": 8, "D": 128, "lo": 1411, "hi": 1411, "dtype": "bf16", "out": "bf16"},
        # A layer's share of a chat: a prompt, a follow-up on the warm cache, eight generated tokens; RoPE + append,
        # attention over the cache and the output projection each time, from f32 activations.
        {"name": "chat_session", "kind": "session", "B": 1, "Hq": 32, "Hkv": 8, "D": 128, "prompt": 1000, "follow": 200, "tokens": 8,
         "N": 4096, "dtype": "f32"},
        # A sliding-window layer that is full: each new token pushes the oldest one out.
        {"name": "window_step", "kind": "window", "B": 2, "Hq": 32, "Hkv": 8, "D": 128, "window": 4096, "dtype": "bf16"},
        # The output projection behind the prefill batch.
        {"name": "project_batch", "kind": "project", "B": 4, "Hq": 32, "S": 4096, "D": 128, "N": 4096, "bias": False, "out": "f32"},
        # RoPE of q and k with the append of k and v to the pages, for the prefill batch.
        {"name": "rotate_append", "kind": "rotate", "B": 4, "Hq": 32, "Hkv": 8, "S": 4096, "D": 128, "dtype": "bf16", "interleaved": False},
    ]


def _log(rng, lo, hi):
    """A whole number from lo to hi, spread over the logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _heads(rng, most=64):
    while True:
        hkv, g = rng.choice((1, 2, 4, 8, 16)), rng.choice((1, 2, 4, 4, 8))
        if hkv * g <= most:
            return hkv * g, hkv


def draw(rng):
    kind = rng.choice(("attention", "attention", "attention", "attention", "decode", "decode", "session", "window", "project", "rotate"))
    D = rng.choice((128, 128, 64))
    if kind == "attention":
        dtype = rng.choice(("bf16", "bf16", "f16", "f32"))
        # f32 tensors and head_dim 64 come from smaller models and shorter inputs
        small = dtype == "f32" or D == 64
        S = _log(rng, 16, 2048 if small else 16384)
        Hq, Hkv = _heads(rng)
        past = _log(rng, 16, 2 * S + 64) if rng.random() < 0.3 else 0
        most = (1 << 31 if small else 1 << 40) // (D * S * (S + past))  # (batch, head) pairs
        while Hq > max(1, most) and Hkv > 1:
            Hq, Hkv = Hq // 2, Hkv // 2
        Hq = min(Hq, max(1, most)) if Hkv == 1 else Hq
        mask = rng.choice(("causal", "causal", "causal", "none", "window", "key"))
        return {"kind": kind, "B": _log(rng, 1, max(1, min(16, most // Hq))), "Hq": Hq, "Hkv": Hkv, "Sq": S, "past": 0 if mask == "window" else past,
                "D": D, "dtype": dtype, "out": rng.choice(("f32", dtype)), "mask": mask,
                "window": _log(rng, 8, S) if mask == "window" else 0, "outliers": rng.random() < 0.2}
    if kind == "decode":
        Hq, Hkv = _heads(rng)
        hi = _log(rng, 16, 131072)
        B = _log(rng, 1, max(1, min(128, (1 << 29) // (2 * Hkv * D * hi))))
        return {"kind": kind, "B": B, "Hq": Hq, "Hkv": Hkv, "D": D, "lo": max(1, int(hi * rng.uniform(0.1, 1.0))), "hi": hi,
                "dtype": rng.choice(("bf16", "f32")), "out": rng.choice(("f32", "bf16"))}
    if kind == "session":
        Hq, Hkv = _heads(rng, 32)
        return {"kind": kind, "B": rng.choice((1, 1, 2, 4)), "Hq": Hq, "Hkv": Hkv, "D": D, "prompt": _log(rng, 16, 2048), "follow": _log(rng, 2, 512),
                "tokens": rng.randint(4, 12), "N": Hq * D, "dtype": rng.choice(("f32", "bf16"))}
    if kind == "window":
        Hq, Hkv = _heads(rng)
        return {"kind": kind, "B": rng.randint(1, 4), "Hq": Hq, "Hkv": Hkv, "D": D, "window": _log(rng, 64, 8192), "dtype": rng.choice(("f32", "bf16"))}
    if kind == "project":
        Hq = rng.choice((4, 8, 16, 32, 64))
        rows = _log(rng, 1, 16384)
        B = min(rows, rng.choice((1, 1, 2, 4, 16, 64)))
        return {"kind": kind, "B": B, "Hq": Hq, "S": rows // B, "D": D, "N": 8 * _log(rng, 32, 1024), "bias": rng.random() < 0.5,
                "out": rng.choice(("f32", "bf16"))}
    Hq, Hkv = _heads(rng)
    B = rng.choice((1, 1, 2, 4, 16))
    return {"kind": kind, "B": B, "Hq": Hq, "Hkv": Hkv, "S": _log(rng, 1, 32768 // B), "D": D, "dtype": rng.choice(("f32", "bf16")),
            "interleaved": rng.random() < 0.5}


# ------------------------------------------------------------------------------------------------------------ inputs
def _spread(c):
    """The sequence lengths of a decode batch: evenly from lo to hi."""
    B, lo, hi = c["B"], c["lo"], c["hi"]
    return [hi if B == 1 else lo + (hi - lo) * i // (B - 1) for i in range(B)]


def prepare(case, seed):
    c, dev = dict(case), _device()
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))

    def normal(*shape, dtype="f32", sigma=1.0):
        x = torch.randn(shape, generator=gen, device="cuda", dtype=torch.float32)
        return (x if sigma == 1.0 else x.mul_(sigma)).to(TORCH[dtype])

    def tensor(x):
        return fb.Tensor.from_torch(dev, x)

    def rope_tables(rows):
        inv = 1.0 / (10000.0 ** (torch.arange(0, c["D"], 2, device="cuda", dtype=torch.float32) / c["D"]))
        ang = torch.arange(rows, device="cuda", dtype=torch.float32)[:, None] * inv[None]
        return fb.RopeCache.from_parts(tensor(ang.cos()), tensor(ang.sin()))

    s = {"case": c, "kind": c["kind"]}
    if c["kind"] == "attention":
        B, Sq, Skv, D, dt = c["B"], c["Sq"], c["Sq"] + c["past"], c["D"], c["dtype"]
        sigma = 0.5 if c["outliers"] else 1.0
        q, k, v = normal(B, c["Hq"], Sq, D, sigma=sigma), normal(B, c["Hkv"], Skv, D, sigma=sigma), normal(B, c["Hkv"], Skv, D, sigma=sigma)
        if c["outliers"]:
            k = torch.where(torch.rand((B, c["Hkv"], Skv, 1), generator=gen, device="cuda") < 0.05, k * 8.0, k)
        s.update(q=tensor(q.to(TORCH[dt])), k=tensor(k.to(TORCH[dt])), v=tensor(v.to(TORCH[dt])), scale=D ** -0.5, out=CODE[c["out"]], mask=None)
        if c["mask"] == "key":
            # each sequence of the batch has its own length, from half of the keys to all of them
            n = torch.tensor([Skv - (Skv // 2) * b // B for b in range(B)], device="cuda")
            m = torch.where(torch.arange(Skv, device="cuda")[None] < n[:, None], 0.0, float("-inf")).to(torch.float32)
            s["mask"] = (tensor(m), fb.MaskKind.BatchKeyMask)
        elif c["mask"] != "none":
            masks = fb.MaskCache()
            s["mask"] = (masks.get_mask(Sq, c["past"], c["window"] or None, dev), fb.MaskKind.QKMask)
    elif c["kind"] == "decode":
        lens = torch.tensor(_spread(c))
        host = torch.Generator().manual_seed(int(seed))
        lens = lens[torch.randperm(c["B"], generator=host)]
        pages = (lens + PAGE - 1) // PAGE
        total, widest = int(pages.sum()), int(pages.max())
        order = torch.randperm(total, generator=host).to(torch.int32)
        table = torch.zeros((c["B"], widest), dtype=torch.int32)
        at = 0
        for b in range(c["B"]):
            n = int(pages[b])
            table[b, :n] = order[at:at + n]
            at += n
        cache = fb.PagedKvCache(dev, c["B"], c["Hkv"], c["D"], total, widest)
        dev.synchronize()  # the new pools have been cleared
        for pool in _pools(cache):
            for i in range(0, total, 4096):
                pool[i:i + 4096] = normal(*pool[i:i + 4096].shape, dtype="bf16")
        cache.set_page_table(table.numpy(), lens.to(torch.int32).numpy())
        out = torch.empty((c["B"], c["Hq"], 1, c["D"]), device="cuda", dtype=TORCH[c["out"]])
        s.update(cache=cache, q=tensor(normal(c["B"], c["Hq"], 1, c["D"], dtype=c["dtype"])), out=tensor(out), out_torch=out, scale=c["D"] ** -0.5)
    elif c["kind"] == "session":
        B, D, dt = c["B"], c["D"], c["dtype"]
        turns = [c["prompt"], c["follow"]] + [1] * c["tokens"]
        s.update(turns=[tuple(tensor(normal(B, h, n, D, dtype=dt)) for h in (c["Hq"], c["Hkv"], c["Hkv"])) for n in turns],
                 rope=rope_tables(sum(turns)), cache=fb.KvCache.new(2, sum(turns)), masks=fb.MaskCache(), scale=D ** -0.5,
                 weight=tensor(normal(c["N"], c["Hq"] * D, dtype="bf16", sigma=(c["Hq"] * D) ** -0.5)))
    elif c["kind"] == "window":
        B, D, dt, w = c["B"], c["D"], c["dtype"], c["window"]
        cache = fb.KvCache.new(2, w)
        cache.append(dev, *(tensor(normal(B, c["Hkv"], w, D, dtype=dt)) for _ in range(2)))
        s.update(cache=cache, q=tensor(normal(B, c["Hq"], 1, D, dtype=dt)), k=tensor(normal(B, c["Hkv"], 1, D, dtype=dt)),
                 v=tensor(normal(B, c["Hkv"], 1, D, dtype=dt)), scale=D ** -0.5)
    elif c["kind"] == "project":
        K = c["Hq"] * c["D"]
        out = torch.empty((c["B"], c["S"], c["N"]), device="cuda", dtype=TORCH[c["out"]])
        s.update(x=tensor(normal(c["B"], c["Hq"], c["S"], c["D"], dtype="bf16")), weight=tensor(normal(c["N"], K, dtype="bf16", sigma=K ** -0.5)),
                 bias=tensor(normal(c["N"])) if c["bias"] else None, out=tensor(out), out_torch=out)
    else:
        B, S, D, dt = c["B"], c["S"], c["D"], c["dtype"]
        pages = (S + PAGE - 1) // PAGE
        cache = fb.PagedKvCache(dev, B, c["Hkv"], D, B * pages, pages)
        s.update(cache=cache, pools=_pools(cache), rope=rope_tables(S),
                 qkv=tuple(tensor(normal(B, h, S, D, dtype=dt)) for h in (c["Hq"], c["Hkv"], c["Hkv"])))
    dev.synchronize()
    return s


# ------------------------------------------------------------------------------------------------------------ one pass
def run(s):
    kind = s["kind"]
    if kind == "attention":
        return _torch(s["q"].flash_attention(s["k"], s["v"], s["scale"], s["mask"], s["out"]))
    if kind == "decode":
        s["cache"].decode(s["q"], s["scale"], s["out"])
        return s["out_torch"]
    if kind == "session":
        cache, pos, got = s["cache"], 0, []
        cache.reset()
        for q, k, v in s["turns"]:
            n = q.shape()[2]
            q, k, v = s["rope"].forward_append(q, k, v, cache, pos)
            mask = s["masks"].get_mask(n, pos, None, q.device)
            attn = q.flash_attention(k, v, s["scale"], (mask, fb.MaskKind.QKMask), BF16)
            got.append(_torch(attn.out_proj(s["weight"])))
            pos += n
        return got
    if kind == "window":
        k, v = s["cache"].append(s["q"].device, s["k"], s["v"])
        return _torch(s["q"].flash_attention(k, v, s["scale"]))
    if kind == "project":
        s["x"].out_proj(s["weight"], s["bias"], out=s["out"])
        return s["out_torch"]
    s["cache"].reset()
    q = s["rope"].forward_append(*s["qkv"], s["cache"], 0, s["case"]["interleaved"])
    return (_torch(q),) + s["pools"]


# ------------------------------------------------------------------------------------------------------------ what it takes
def _pairs(c):
    """(query, key) pairs of one head that the mask leaves, over the batch."""
    B, Sq, past, w = c["B"], c["Sq"], c["past"], c["window"]
    Skv = Sq + past
    if c["mask"] == "causal":
        return B * (Sq * past + Sq * (Sq + 1) // 2)
    if c["mask"] == "window":
        return B * sum(min(i + 1, w) for i in range(Sq))
    if c["mask"] == "key":
        return sum(Sq * (Skv - (Skv // 2) * b // B) for b in range(B))
    return B * Sq * Skv


def _decode_work(B, Hq, Hkv, D, tokens):
    return {"bytes": 4.0 * Hkv * D * tokens + 6.0 * B * Hq * D, "flops": 4.0 * Hq * D * tokens}


def work(case):
    c = case
    if c["kind"] == "attention":
        kv = 2 * c["B"] * c["Hkv"] * (c["Sq"] + c["past"]) * c["D"] * SIZE[c["dtype"]]
        q = c["B"] * c["Hq"] * c["Sq"] * c["D"]
        return {"bytes": float(kv + q * (SIZE[c["dtype"]] + SIZE[c["out"]])), "flops": 4.0 * c["Hq"] * c["D"] * _pairs(c)}
    if c["kind"] == "decode":
        return _decode_work(c["B"], c["Hq"], c["Hkv"], c["D"], sum(_spread(c)))
    if c["kind"] == "session":
        B, Hq, Hkv, D, N, pos = c["B"], c["Hq"], c["Hkv"], c["D"], c["N"], 0
        total = {"bytes": 0.0, "flops": 0.0}
        for n in [c["prompt"], c["follow"]] + [1] * c["tokens"]:
            total["bytes"] += B * n * D * (Hq + 2 * Hkv) * SIZE[c["dtype"]] + 4.0 * B * Hkv * D * (pos + n) + 2.0 * N * Hq * D + 4.0 * B * n * N
            total["flops"] += 4.0 * B * Hq * D * (n * pos + n * (n + 1) // 2) + 2.0 * B * n * N * Hq * D
            pos += n
        return total
    if c["kind"] == "window":
        return _decode_work(c["B"], c["Hq"], c["Hkv"], c["D"], c["B"] * c["window"])
    if c["kind"] == "project":
        K, rows = c["Hq"] * c["D"], c["B"] * c["S"]
        return {"bytes": 2.0 * K * (rows + c["N"]) + rows * c["N"] * float(SIZE[c["out"]]), "flops": 2.0 * rows * K * c["N"]}
    rows, e = c["B"] * c["S"] * c["D"], SIZE[c["dtype"]]
    return {"bytes": rows * (2.0 * c["Hq"] * e + 2.0 * c["Hkv"] * (e + 2)) + 4.0 * c["S"] * c["D"], "flops": 3.0 * rows * (c["Hq"] + c["Hkv"])}


def tolerance(case):
    """About four times what each path is off by against the same computation in 64 bits (on the listed cases and forty drawn
    ones)."""
    c = case
    if c["kind"] == "attention":
        if c["out"] == "bf16":
            return {"rel": 7e-3, "max": 1.8e-2}  # the rounding of the result: 1.7e-3 and 4.4e-3
        if c["dtype"] != "f32" and c["D"] == 128:
            return {"rel": 1e-3, "max": 1.7e-2}  # 11-bit softmax weights: 2.8e-4 and 4.2e-3
        if c["out"] == "f16":
            return {"rel": 8e-4, "max": 2e-3}    # the rounding of the result: 2.1e-4 and 4.9e-4
        return {"rel": 2e-6, "max": 4e-5}        # f32 arithmetic: 4.5e-7 and 8.6e-6
    if c["kind"] == "session":
        return {"rel": 3.5e-3, "max": 4e-2}      # the attention output is rounded to bf16 before the projection: 8.6e-4 and 1.1e-2
    if c["kind"] == "project":
        return {"rel": 7e-3, "max": 1.8e-2} if c["out"] == "bf16" else {"rel": 2.5e-5, "max": 7e-5}  # f32 sums over up to 8192: 6.4e-6 and 1.7e-5
    if c["kind"] == "rotate":
        return "exact"                           # each product is rounded before the sum, and the pages hold rounded values
    if c.get("out") == "bf16":
        return {"rel": 7e-3, "max": 1.8e-2}      # decode: the rounding of the result
    return {"rel": 1.2e-5, "max": 8e-5}          # decode: 16-bit softmax weights: 2.9e-6 and 1.9e-5

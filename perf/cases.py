"""The attention calls whose speed this repository is judged by, as data: sizes, inputs, one pass each.

Every case is one call (for training: forward and backward) of the public functions of `flash_attention_b200`, at
the sizes of this repository's benchmark and tests and between them.  Dropout is 0 throughout, as in every workload
of the benchmark: its result depends on the state of torch's generator and not on the inputs alone.
"""
import math
import random

import torch

import flash_attention_b200 as fa

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}


def _case(name, kind, **kw):
    """kind: forward (no gradients), train (forward + backward), varlen (packed sequences, forward + backward),
    cache (new tokens against a KV cache).  pack: how q, k, v are handed over (separate / kv / qkv).  new: tokens per
    sequence.  len_lo, len_hi: range of the sequence lengths (varlen) or of the filled part of the cache (cache).
    page: rows of a page of the cache, 0 for one slab per sequence."""
    c = dict(kind=kind, batch=1, sq=0, sk=0, heads=16, heads_k=16, dim=128, dtype="bf16", causal=True, left=-1, right=-1,
             pack="separate", new=0, len_lo=0, len_hi=0, page=0, rotary=False)
    c.update(kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest calls: a short prompt or a test model; launches and host time are what a user waits for
        _case("forward_small", "forward", batch=2, sq=512, sk=512, heads=8, heads_k=8, dim=64),
        # small training step on odd lengths with grouped-query heads (the lengths of the parity tests)
        _case("train_small_odd", "train", batch=4, sq=113, sk=203, heads=6, heads_k=3, dim=64, causal=False),
        # prefill of one prompt on a grouped-query model
        _case("prefill_gqa", "forward", sq=4096, sk=4096, heads=32, heads_k=8),
        # the benchmark's training shapes: 32768 tokens, hidden size 2048, packed qkv
        _case("train_d128_causal", "train", batch=16, sq=2048, sk=2048, pack="qkv"),
        _case("train_d64_full", "train", batch=16, sq=2048, sk=2048, heads=32, heads_k=32, dim=64, causal=False, pack="qkv"),
        _case("train_d256_causal", "train", batch=16, sq=2048, sk=2048, heads=8, heads_k=8, dim=256, pack="qkv"),
        # cross attention on ragged lengths, a head dim between the kernels' own, packed kv
        _case("train_cross_ragged_d96", "train", batch=8, sq=1023, sk=1795, heads=12, heads_k=12, dim=96, dtype="fp16",
              causal=False, pack="kv"),
        # packed batch of sequences of 128 to 4096 tokens
        _case("train_varlen_fp16", "varlen", sq=65536, dtype="fp16", len_lo=128, len_hi=4096),
        # long context, grouped-query, full causal and sliding window: the largest calls
        _case("train_long_causal", "train", sq=32768, sk=32768, heads=32, heads_k=8),
        _case("train_long_window", "train", sq=32768, sk=32768, heads=32, heads_k=8, causal=False, left=4096, right=0),
        # one token per sequence on a full serving batch, appended with rotary in the same call
        _case("decode_batch64", "cache", batch=64, sk=32768, heads=32, heads_k=8, new=1, len_lo=1024, len_hi=32767, rotary=True),
        # a chunk of a prompt (or a draft to verify) appended to a paged cache
        _case("append_chunk_paged", "cache", batch=4, sk=8192, heads=32, heads_k=8, new=128, len_lo=512, len_hi=8000, page=256,
              rotary=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


_DIMS = [32, 40, 64, 64, 64, 80, 96, 128, 128, 128, 128, 160, 192, 256]


def draw(rng):
    kind = rng.choice(["forward", "forward", "train", "train", "train", "varlen", "cache", "cache"])
    heads_k = rng.choice([1, 2, 4, 8, 8, 16])
    heads = heads_k * rng.choice([1, 1, 1, 2, 4])
    dtype = rng.choice(["bf16", "bf16", "fp16"])
    dim = rng.choice(_DIMS)
    if kind == "cache":
        batch = _log(rng, 1, 64)
        page = rng.choice([0, 0, 64, 256])
        cap = _log(rng, 1024, max(2048, min(32768, (1 << 23) // (batch * heads_k) * 2))) // 256 * 256
        new = rng.choice([1, 1, 1, 2, 5, 16, _log(rng, 17, 512)])
        hi = cap - new - rng.randrange(8)
        return _case("", "cache", batch=batch, sk=cap, heads=heads_k * rng.choice([1, 4, 8]), heads_k=heads_k,
                     dim=rng.choice([64, 128, 128, 128]), dtype=dtype, new=new, len_lo=max(1, hi // rng.choice([1, 4, 32])),
                     len_hi=hi, page=page, rotary=rng.random() < 0.7)
    if kind == "varlen":
        total = _log(rng, 1024, 65536)
        hi = _log(rng, 128, min(4096, total))
        return _case("", "varlen", sq=total, heads=heads, heads_k=heads_k, dim=dim, dtype=dtype, causal=rng.random() < 0.7,
                     len_lo=max(1, hi // 32), len_hi=hi)
    sq = _log(rng, 64, 16384)
    sk = sq if rng.random() < 0.7 else _log(rng, 64, 16384)
    tokens = _log(rng, max(sq, 256), 32768)
    batch = max(1, tokens // max(sq, sk))
    if sq == sk and heads == heads_k:
        pack = rng.choice(["qkv", "separate"])
    else:
        pack = rng.choice(["kv", "separate", "separate"])
    mask = rng.choice(["causal", "causal", "full", "window"])
    left = _log(rng, 16, 4096) if mask == "window" else -1
    return _case("", kind, batch=batch, sq=sq, sk=sk, heads=heads, heads_k=heads_k, dim=dim, dtype=dtype,
                 causal=mask == "causal", left=left, right=0 if mask == "window" else -1, pack=pack)


def _spread(lo, hi, n):
    """n whole numbers spread evenly over [lo, hi]."""
    return [lo + (hi - lo) * (2 * i + 1) // (2 * n) for i in range(n)]


def _varlen_lengths(case):
    """Lengths of a packed batch: uniform over the range until the tokens are used up.  The same for every seed (the
    order is not), so that the work of a case is a number."""
    r, lens, left = random.Random(case["sq"]), [], case["sq"]
    while left > 0:
        lens.append(min(left, r.randint(case["len_lo"], case["len_hi"])))
        left -= lens[-1]
    return lens


def _pairs(sq, sk, causal, left, right):
    """How many (query, key) pairs the mask leaves (aligned to the bottom right corner)."""
    if causal:
        right = 0
    if left < 0 and right < 0:
        return sq * sk
    n, shift = 0, sk - sq
    for i in range(sq):
        lo = max(0, i + shift - left) if left >= 0 else 0
        hi = min(sk - 1, i + shift + right) if right >= 0 else sk - 1
        n += max(0, hi - lo + 1)
    return n


def prepare(case, seed):
    dev, dt = torch.device("cuda"), DTYPES[case["dtype"]]
    g = torch.Generator(device=dev).manual_seed(seed)
    order = random.Random(seed)
    B, H, Hk, D = case["batch"], case["heads"], case["heads_k"], case["dim"]

    def randn(*shape):
        return torch.randn(*shape, device=dev, dtype=dt, generator=g)

    s = {"case": case, "causal": case["causal"], "window": (case["left"], case["right"])}
    if case["kind"] == "cache":
        cap, new, page = case["sk"], case["new"], case["page"]
        lens = _spread(case["len_lo"], case["len_hi"], B)
        order.shuffle(lens)
        s["lens"] = torch.tensor(lens, dtype=torch.int32, device=dev)
        s["q"], s["k"], s["v"] = randn(B, new, H, D), randn(B, new, Hk, D), randn(B, new, Hk, D)
        s["table"] = None
        if page:
            n = cap // page
            ids = list(range(B * n))
            order.shuffle(ids)
            s["table"] = torch.tensor(ids, dtype=torch.int32, device=dev).view(B, n)
            s["kc"], s["vc"] = randn(B * n, page, Hk, D), randn(B * n, page, Hk, D)
        else:
            s["kc"], s["vc"] = randn(B, cap, Hk, D), randn(B, cap, Hk, D)
        s["cos"] = s["sin"] = None
        if case["rotary"]:
            inv = 1.0 / (10000 ** (torch.arange(0, D, 2, device=dev).float() / D))
            angle = torch.outer(torch.arange(cap, device=dev).float(), inv)
            s["cos"], s["sin"] = torch.cos(angle).to(dt), torch.sin(angle).to(dt)
        return s
    if case["kind"] == "varlen":
        lens = _varlen_lengths(case)
        order.shuffle(lens)
        ends = [0]
        for n in lens:
            ends.append(ends[-1] + n)
        s["cu"], s["max"] = torch.tensor(ends, dtype=torch.int32, device=dev), max(lens)
        s["in"] = [randn(case["sq"], h, D).requires_grad_() for h in (H, Hk, Hk)]
        s["dout"] = randn(case["sq"], H, D)
        return s
    sq, sk = case["sq"], case["sk"]
    if case["pack"] == "qkv":
        s["in"] = [randn(B, sq, 3, H, D)]
    elif case["pack"] == "kv":
        s["in"] = [randn(B, sq, H, D), randn(B, sk, 2, Hk, D)]
    else:
        s["in"] = [randn(B, sq, H, D), randn(B, sk, Hk, D), randn(B, sk, Hk, D)]
    if case["kind"] == "train":
        for t in s["in"]:
            t.requires_grad_()
        s["dout"] = randn(B, sq, H, D)
    return s


_CALL = {"qkv": fa.flash_attn_qkvpacked_func, "kv": fa.flash_attn_kvpacked_func, "separate": fa.flash_attn_func}


def run(state):
    case = state["case"]
    if case["kind"] == "cache":
        out = fa.flash_attn_with_kvcache(state["q"], state["kc"], state["vc"], state["k"], state["v"], state["cos"], state["sin"],
                                         cache_seqlens=state["lens"], causal=state["causal"], rotary_interleaved=False,
                                         block_table=state["table"])
        return out, state["kc"], state["vc"]
    if case["kind"] == "varlen":
        out = fa.flash_attn_varlen_func(*state["in"], state["cu"], state["cu"], state["max"], state["max"], causal=state["causal"])
    else:
        out = _CALL[case["pack"]](*state["in"], causal=state["causal"], window_size=state["window"])
    if case["kind"] == "forward":
        return out
    return (out,) + torch.autograd.grad(out, state["in"], state["dout"])


def work(case):
    B, H, Hk, D = case["batch"], case["heads"], case["heads_k"], case["dim"]
    if case["kind"] == "cache":
        lens = [n + case["new"] for n in _spread(case["len_lo"], case["len_hi"], B)]
        pairs = sum(_pairs(case["new"], n, case["causal"], -1, -1) for n in lens)
        # keys and values attended to, read once; new tokens in, their cache rows and the output out
        return {"bytes": 2 * D * (2 * Hk * sum(lens) + B * case["new"] * (2 * H + 2 * Hk)), "flops": 4 * pairs * H * D}
    if case["kind"] == "varlen":
        pairs = sum(_pairs(n, n, case["causal"], -1, -1) for n in _varlen_lengths(case))
        q, k = case["sq"] * H * D, case["sq"] * Hk * D
    else:
        pairs = B * _pairs(case["sq"], case["sk"], case["causal"], case["left"], case["right"])
        q, k = B * case["sq"] * H * D, B * case["sk"] * Hk * D
    if case["kind"] == "forward":
        return {"bytes": 2 * (2 * q + 2 * k), "flops": 4 * pairs * H * D}
    # in: q, k, v, dout; out: out, dq, dk, dv.  The backward needs 2.5 times the forward's products.
    return {"bytes": 2 * (4 * q + 4 * k), "flops": 14 * pairs * H * D}


def tolerance(case):
    """Of another correct implementation that keeps its sums in 32 bits and the operands of its products (P, dS, the
    rotated tokens) in the input type: four times what these kernels are off from the same call in 64 bits.  Seen over
    the listed cases (batch reduced to 2, lengths to 8192): bf16 2.0e-3 to 2.8e-3 relative and at most 0.087 in one
    element, fp16 2.5e-4 to 3.1e-4 and at most 0.012."""
    return {"rel": 0.011, "max": 0.35} if case["dtype"] == "bf16" else {"rel": 0.00125, "max": 0.047}


def _attend(q, k, v, causal, left, right, dout=None):
    """One sequence in 64 bits, heads first: q (H, sq, D), k, v (Hk, sk, D).  out, and with dout also dq, dk, dv."""
    H, sq, D = q.shape
    Hk, sk, _ = k.shape
    out, dq = torch.empty_like(q), torch.empty_like(q)
    dk, dv = torch.zeros_like(k), torch.zeros_like(v)
    cols, scale = torch.arange(sk, device=q.device), 1 / math.sqrt(D)
    right = 0 if causal else right
    step = max(1, (1 << 26) // max(1, sk))
    for h in range(H):
        g = h // (H // Hk)
        for i in range(0, sq, step):
            at = torch.arange(i, min(sq, i + step), device=q.device) + (sk - sq)
            e = slice(i, i + len(at))
            s = (q[h, e] @ k[g].T) * scale
            if right >= 0:
                s.masked_fill_(cols > at[:, None] + right, -math.inf)
            if left >= 0:
                s.masked_fill_(cols < at[:, None] - left, -math.inf)
            p = torch.softmax(s, -1).nan_to_num_(0.0)  # a row without a key gives zero
            del s
            out[h, e] = p @ v[g]
            if dout is not None:
                dv[g] += p.T @ dout[h, e]
                ds = dout[h, e] @ v[g].T
                ds -= (dout[h, e] * out[h, e]).sum(-1, keepdim=True)
                ds *= p
                dq[h, e] = (ds @ k[g]) * scale
                dk[g] += (ds.T @ q[h, e]) * scale
                del ds
            del p
    return (out,) if dout is None else (out, dq, dk, dv)


def _turn(x, cos, sin, pos):
    """Rows of x (n, h, D) turned to the positions pos (n): the first half of a row against the second."""
    c, s = cos[pos].double()[:, None], sin[pos].double()[:, None]
    a, b = x.chunk(2, -1)
    return torch.cat([a * c - b * s, a * s + b * c], -1)


def exact(case, seed):
    """What run() returns for these inputs, in 64 bits with plain torch.  The caches are left out where they are large:
    all but their new rows is input."""
    s = prepare(case, seed)
    heads_first = lambda t: t.detach().double().transpose(0, 1)  # noqa: E731
    left, right = s["window"]
    if case["kind"] == "cache":
        out, new, cap = torch.empty(s["q"].shape, dtype=torch.float64, device="cuda"), case["new"], case["sk"]
        whole = s["kc"].numel() <= 1 << 26
        kc, vc = (s["kc"].double(), s["vc"].double()) if whole else (None, None)
        for b, n in enumerate(s["lens"].tolist()):
            pos = torch.arange(n, n + new, device="cuda")
            q, k, v = s["q"][b].double(), s["k"][b].double(), s["v"][b].double()
            if s["cos"] is not None:
                q, k = _turn(q, s["cos"], s["sin"], pos), _turn(k, s["cos"], s["sin"], pos)
            if s["table"] is None:
                old_k, old_v = s["kc"][b, :n], s["vc"][b, :n]
            else:
                pages = s["table"][b].long()
                old_k, old_v = s["kc"][pages].flatten(0, 1)[:n], s["vc"][pages].flatten(0, 1)[:n]
            if whole:
                at = (b, pos) if s["table"] is None else (pages[pos // case["page"]], pos % case["page"])
                kc[at], vc[at] = k, v
            k, v = torch.cat([old_k.double(), k]), torch.cat([old_v.double(), v])
            out[b] = _attend(q.transpose(0, 1), k.transpose(0, 1), v.transpose(0, 1), case["causal"], left, right)[0].transpose(0, 1)
        return out, kc, vc
    if case["kind"] == "varlen":
        parts, ends = [], s["cu"].tolist()
        for i, j in zip(ends, ends[1:]):
            q, k, v, d = (heads_first(t[i:j]) for t in s["in"] + [s["dout"]])
            parts.append([t.transpose(0, 1) for t in _attend(q, k, v, case["causal"], left, right, d)])
        return tuple(torch.cat(t) for t in zip(*parts))
    if case["pack"] == "qkv":
        q, k, v = s["in"][0].unbind(2)
    elif case["pack"] == "kv":
        q, (k, v) = s["in"][0], s["in"][1].unbind(2)
    else:
        q, k, v = s["in"]
    dout = s.get("dout")
    parts = []
    for b in range(case["batch"]):
        d = None if dout is None else heads_first(dout[b])
        parts.append([t.transpose(0, 1) for t in _attend(heads_first(q[b]), heads_first(k[b]), heads_first(v[b]), case["causal"], left, right, d)])
    got = [torch.stack(t) for t in zip(*parts)]
    if dout is None:
        return got[0]
    out, dq, dk, dv = got
    if case["pack"] == "qkv":
        return out, torch.stack([dq, dk, dv], 2)
    if case["pack"] == "kv":
        return out, dq, torch.stack([dk, dv], 2)
    return out, dq, dk, dv

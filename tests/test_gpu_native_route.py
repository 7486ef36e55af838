"""Plain calls are checked and launched by csrc/torch_glue.cpp, all others by the python code of flash_attn_2_cuda.  The two take
the same calls, refuse the same ones and give the same bits."""
import pytest
import torch

from gpu_util import make_qkv

pytestmark = pytest.mark.gpu

if torch.cuda.is_available():
    import flash_attn_2_cuda as ext
    from flash_attention_b200 import _lib

    _lib.lib()
    from flash_attention_b200.csrc import _torch_glue


def test_packed_calls_need_their_offsets():
    """4-D operands and no cu_seqlens: an error of the packed entry points, not a padded batch."""
    q, k, v, dout = make_qkv(2, 130, 130, 4, 2, 64, torch.bfloat16)
    out, *_, lse, _, rng = ext.fwd(q, k, v, None, 0.0, 0.125, False, -1, -1, False, None)
    cu = torch.tensor([0, 130, 260], dtype=torch.int32, device="cuda")
    grads = [torch.empty_like(t) for t in (q, k, v)]
    flat = [t.flatten(0, 1) for t in (q, k, v, dout, out)]
    for a, b in ((None, None), (None, cu), (cu, None)):
        for ts in ((q, k, v, dout, out), flat):
            with pytest.raises((RuntimeError, AttributeError)):
                ext.varlen_fwd(*ts[:3], None, a, b, 130, 130, 0.0, 0.125, False, False, -1, -1, False, None)
            with pytest.raises((RuntimeError, AttributeError)):
                ext.varlen_bwd(ts[3], *ts[:3], ts[4], lse, *grads, a, b, 130, 130, 0.0, 0.125, False, False, -1, -1, None, rng)
    packed = ext.varlen_fwd(*flat[:3], None, cu, cu, 130, 130, 0.0, 0.125, False, False, -1, -1, False, None)
    assert torch.equal(packed[0].view_as(out), out)


def test_out_of_memory_keeps_its_type():
    q = torch.zeros(1, 65536, 16, 128, dtype=torch.bfloat16, device="cuda")
    k, v = (torch.zeros(1, 128, 16, 128, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    try:  # room for 64 MiB more, the output takes 256
        torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (64 << 20)) / total)
        with pytest.raises(torch.OutOfMemoryError):
            ext.fwd(q, k, v, None, 0.0, 0.1, False, -1, -1, False, None)
        with pytest.raises(torch.OutOfMemoryError):
            ext.fwd_kvcache(q, k, v, None, None, None, None, None, None, None, 0.1, False, -1, -1, False, 1)
        grads = [torch.empty_like(k) for _ in range(2)]
        lse = torch.zeros(1, 16, 65536, device="cuda")
        with pytest.raises(torch.OutOfMemoryError):
            ext.bwd(q, q, k, v, q, lse, q, *grads, 0.0, 0.1, False, -1, -1, None, None)
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)


# ---- the native route against the python one ------------------------------------------------------------------------------
class _Native:
    """The native functions, and which of their calls they took."""

    def __init__(self):
        self.taken = []
        for name in ("fwd", "bwd", "fwd_kvcache"):
            setattr(self, name, self._wrap(getattr(_torch_glue, name)))

    def _wrap(self, f):
        def call(*args):
            r = f(*args)
            self.taken.append(r is not None)
            return r

        return call


class _Python:
    fwd = bwd = fwd_kvcache = staticmethod(lambda *args: None)


def _both(monkeypatch, run, native=True):
    """run() on the two routes: the same bits in the same layout, or the same error.  native: which route the call takes by itself
    (None: either)."""
    got = []
    for route in (_Native(), _Python()):
        monkeypatch.setattr(ext, "_glue", route)
        try:
            got.append([t for t in run()])
        except Exception as e:
            got.append((type(e), str(e)))
        if isinstance(route, _Native) and native is not None:
            assert route.taken and all(t == native for t in route.taken)
    a, b = got
    if isinstance(a, tuple) or isinstance(b, tuple):
        assert a == b
        return a
    for x, y in zip(a, b, strict=True):
        assert (x is None) == (y is None)
        if x is not None:
            assert x.shape == y.shape and x.dtype == y.dtype and x.stride() == y.stride() and torch.equal(x, y)
    return None


def _refused(monkeypatch, run):
    error = _both(monkeypatch, run, native=False)
    assert error is not None and error[0] is RuntimeError, error


def _fwd(q, k, v, causal=False, wl=-1, wr=-1):
    return ext.fwd(q, k, v, None, 0.0, 0.11, causal, wl, wr, False, None)[:6]


def _views(kind, sq, sk, heads, heads_k, d, dtype):
    """q, k, v of a case: which route a layout takes."""
    g = torch.Generator().manual_seed(sq + sk + d)
    r = lambda *shape: torch.randn(*shape, generator=g).to(dtype).cuda()
    if kind == "packed":  # slices of one tensor
        return tuple(r(2, sq, 3, heads, d).unbind(2)) if sq == sk and heads == heads_k else (r(2, sq, heads, d), *r(2, sk, 2, heads_k, d).unbind(2))
    if kind == "heads_first":
        return r(2, heads, sq, d).transpose(1, 2), r(2, heads_k, sk, d).transpose(1, 2), r(2, heads_k, sk, d).transpose(1, 2)
    if kind == "wide":  # rows longer than the head dim
        return r(2, sq, heads, d + 8)[..., :d], r(2, sk, heads_k, d + 24)[..., 8:d + 8], r(2, sk, heads_k, d)
    if kind == "odd_base":
        n = 2 * sk * heads_k * d
        return r(2, sq, heads, d), r(n + 1)[1:].view(2, sk, heads_k, d), r(2, sk, heads_k, d)
    if kind == "odd_rows":
        return r(2, sq, heads, d), r(2, sk, heads_k, d + 4)[..., :d], r(2, sk, heads_k, d)
    if kind == "expanded":
        return r(2, sq, heads, d), r(1, sk, heads_k, d).expand(2, sk, heads_k, d), r(2, sk, 1, d).expand(2, sk, heads_k, d)
    return r(2, sq, heads, d), r(2, sk, heads_k, d), r(2, sk, heads_k, d)


_KINDS = {"plain": True, "packed": True, "heads_first": True, "wide": True, "odd_base": False, "odd_rows": False, "expanded": False}


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("kind", list(_KINDS))
@pytest.mark.parametrize("sq,sk,heads,heads_k,d", [(130, 130, 4, 4, 64), (37, 700, 8, 2, 128), (257, 100, 6, 3, 96), (64, 64, 2, 1, 256), (2, 5000, 2, 2, 40)])
def test_padded_batches(sq, sk, heads, heads_k, d, kind, dtype, monkeypatch):
    q, k, v = _views(kind, sq, sk, heads, heads_k, d, dtype)
    for kw in ({}, {"causal": True}, {"wl": 20}, {"wr": 3}, {"wl": 9, "wr": 0}, {"causal": True, "wl": 50}):
        error = _both(monkeypatch, lambda: _fwd(q, k, v, **kw), _KINDS[kind])
        assert error is None or (kind == "odd_base" and error[0] is RuntimeError)  # (a contiguous tensor cannot be copied to a better base)
    if kind == "odd_base":
        return
    out, *_, lse = _fwd(q, k, v, causal=True)
    dout = torch.randn_like(out)
    for layout, native in (("plain", True), ("odd", False), ("given", False)):
        def run():
            new = lambda t: torch.empty(*t.shape[:-1], d + (4 if layout == "odd" else 0), dtype=dtype, device="cuda")[..., :d]
            grads = [None] * 3 if layout == "given" else [new(t) for t in (q, k, v)]
            dq, dk, dv, sd = ext.bwd(dout, q, k, v, out, lse, *grads, 0.0, 0.11, True, -1, -1, None, None, deterministic=True)
            return dq, dk, dv, sd[..., :sq]

        assert _both(monkeypatch, run, native and _KINDS[kind]) is None
    assert _both(monkeypatch, lambda: ext.bwd(dout[:1, :1, :1, :1].expand(dout.shape), q, k, v, out, lse, None, None, None, 0.0, 0.11, False, -1, -1, None, None)[:3],
                 False) is not None  # (a stride of 0 in the last dim is refused)


def test_shapes_that_python_does(monkeypatch):
    for sq, sk, d in ((1, 300, 64), (5, 0, 64), (64, 64, 60)):
        q, k, v = _views("plain", sq, sk, 4, 2, d, torch.float16)
        assert _both(monkeypatch, lambda: _fwd(q, k, v), False) is None


def test_padded_refusals(monkeypatch):
    q, k, v = _views("plain", 64, 96, 4, 2, 64, torch.float16)
    out, *_, lse = _fwd(q, k, v)
    for bad in ((q.float(), k.float(), v.float()), (q, k.bfloat16(), v), (q, k, v.bfloat16()), (q, k.cpu(), v), (q, k, v[:, :90]), (q, k[:1], v[:1]), (q[:, :, :3], k, v),
                (q, k[..., :56], v), (q, k[..., :56], v[..., :56]), (q.transpose(1, 3), k, v), (q[:0], k[:0], v[:0]),
                tuple(torch.zeros(2, 8, 2, 264, dtype=torch.float16, device="cuda") for _ in range(3))):
        _refused(monkeypatch, lambda: _fwd(*bad))
    good = dict(dout=out, q=q, k=k, v=v, out=out)
    grads = [torch.empty_like(t) for t in (q, k, v)]
    for name, t in (("dout", out.bfloat16()), ("k", k[:, :90]), ("out", out[:, :60]), ("v", v.bfloat16()), ("dout", out.transpose(1, 3)), ("dout", out[:, :60])):
        a = {**good, name: t}
        _refused(monkeypatch, lambda: ext.bwd(a["dout"], a["q"], a["k"], a["v"], a["out"], lse, *grads, 0.0, 0.1, False, -1, -1, None, None))
    for i, t in ((0, grads[0].float()), (1, grads[1][:, :90]), (2, grads[2].cpu()), (0, grads[0][:, :, :3])):
        g = [*grads[:i], t, *grads[i + 1:]]
        _refused(monkeypatch, lambda: ext.bwd(out, q, k, v, out, lse, *g, 0.0, 0.1, False, -1, -1, None, None))


@pytest.mark.parametrize("heads,heads_k,d", [(4, 4, 64), (6, 2, 128), (2, 1, 192)])
def test_packed_batches(heads, heads_k, d, monkeypatch):
    q, k, v = (t.flatten(0, 1) for t in _views("plain", 150, 210, heads, heads_k, d, torch.bfloat16))
    cu_q, cu_k = (torch.tensor(t, dtype=torch.int32, device="cuda") for t in ((0, 100, 100, 300), (0, 200, 333, 420)))

    def fwd(q=q, k=k, v=v, a=cu_q, b=cu_k, max_q=200, max_k=200, causal=True):
        return ext.varlen_fwd(q, k, v, None, a, b, max_q, max_k, 0.0, 0.11, False, causal, -1, -1, False, None)[:5]  # (lse: rows behind a sequence's end are not written)

    for causal in (False, True):
        assert _both(monkeypatch, lambda: fwd(causal=causal)) is None
    out, lse = fwd()[0], ext.varlen_fwd(q, k, v, None, cu_q, cu_k, 200, 200, 0.0, 0.11, False, True, -1, -1, False, None)[5]
    dout = torch.randn_like(out)

    def bwd(dout=dout, a=cu_q, b=cu_k, grads=None):
        grads = grads or [torch.empty_like(t) for t in (q, k, v)]
        return ext.varlen_bwd(dout, q, k, v, out, lse, *grads, a, b, 200, 200, 0.0, 0.11, False, True, -1, -1, None, None)[:3]

    assert _both(monkeypatch, bwd) is None
    assert _both(monkeypatch, lambda: bwd(dout=dout[:, :1].expand(dout.shape)), False) is None
    wide = torch.stack([cu_q, cu_q], 1)[:, 0]
    for bad in (dict(a=cu_q.long()), dict(b=cu_k.long()), dict(a=cu_q.cpu()), dict(b=cu_k[:3]), dict(a=wide)):
        _refused(monkeypatch, lambda: fwd(**bad))
        _refused(monkeypatch, lambda: bwd(**bad))


@pytest.mark.parametrize("heads,heads_k,d,dtype", [(4, 4, 64, torch.float16), (8, 2, 128, torch.bfloat16), (6, 2, 96, torch.float16)])
@pytest.mark.parametrize("new", [1, 3, 40])
def test_caches(new, heads, heads_k, d, dtype, monkeypatch):
    g = torch.Generator().manual_seed(new + d)
    r = lambda *shape: torch.randn(*shape, generator=g).to(dtype).cuda()
    q, k, v, kc, vc = r(3, new, heads, d), r(3, new, heads_k, d), r(3, new, heads_k, d), r(4, 512, heads_k, d), r(4, 512, heads_k, d)
    lens, idx = torch.tensor([0, 77, 400], dtype=torch.int32, device="cuda"), torch.tensor([2, 0, 3], dtype=torch.int32, device="cuda")
    angle = torch.rand(512, d // 2, generator=g)
    cos, sin = torch.cos(angle).to(dtype).cuda(), torch.sin(angle).to(dtype).cuda()
    table = torch.randperm(32, generator=g)[:24].view(3, 8).int().cuda()

    def call(q=q, k=None, v=None, lens=lens, cos=None, sin=None, idx=None, causal=True, wl=-1, wr=-1, splits=0, table=None, kc=kc, vc=vc):
        kc, vc = kc.clone(), vc.clone()
        if table is not None:
            kc, vc = (t.flatten(0, 1).view(32, 64, heads_k, d) for t in (kc, vc))
        out, lse = ext.fwd_kvcache(q, kc, vc, k, v, lens, cos, sin, idx, None, 0.11, causal, wl, wr, False, splits, block_table=table)
        return out, lse, kc, vc

    for kw in (dict(lens=torch.full_like(lens, 512)), dict(lens=None, causal=False), dict(k=k, v=v), dict(k=k, v=v, cos=cos, sin=sin), dict(k=k, v=v, idx=idx),
               dict(k=k, v=v, cos=cos, sin=sin, table=table), dict(wl=30, k=k, v=v), dict(wl=100, wr=2), dict(splits=3, k=k, v=v), dict(causal=False, k=k, v=v, cos=cos, sin=sin)):
        if kw.get("k") is None and new > 1 and kw.get("lens", 0) is not None and "lens" not in kw:
            kw["lens"] = lens + new
        assert _both(monkeypatch, lambda: call(**kw)) is None
    spread = r(3, new, 2, heads, d)[:, :, 0]
    # one token's heads are rows of a call: spread heads are copied first; a batch of one more head in between is not
    assert _both(monkeypatch, lambda: call(q=spread, k=k, v=v), None) is None
    for bad in (dict(k=k), dict(k=k, v=v, lens=None), dict(cos=cos, sin=sin), dict(k=k, v=v, cos=cos[:500], sin=sin[:500]), dict(k=k, v=v.float()), dict(lens=lens.long()),
                dict(lens=lens[:2]), dict(idx=idx, table=table), dict(idx=idx.long()), dict(splits=200), dict(splits=-1), dict(kc=kc[:2], vc=vc[:2]), dict(kc=kc, vc=vc[:3]),
                dict(k=k[:2], v=v[:2]), dict(k=k, v=v, cos=cos, sin=sin[:, :8]), dict(k=k.cpu(), v=v), dict(table=table.long()), dict(table=table[:2])):
        if not ("k" in bad and new > 400):
            _refused(monkeypatch, lambda: call(**bad))

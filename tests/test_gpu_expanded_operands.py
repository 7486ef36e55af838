"""Operands that repeat their elements (a stride of 0 on an extent above 1): the gradient of a sum, k and v expanded over the
batch or to more heads, a prefix that all sequences of a cache share.  A tensor map cannot describe them; every call must give
what it gives for the contiguous copy."""
import pytest
import torch

from gpu_util import assert_within, make_qkv
from oracle import attention_oracle as O

pytestmark = pytest.mark.gpu

if torch.cuda.is_available():
    import flash_attention_b200 as fa
    from flash_attention_b200 import _lib
    from flash_attention_b200.ring import CudaBlockOps


def _leaf(t):
    return t.detach().requires_grad_(True)


@pytest.mark.parametrize("d", [64, 128, 256])
@pytest.mark.parametrize("dims", [(1,), (2,), (0, 1, 2)])
def test_gradient_of_a_sum(d, dims):
    q, k, v, _ = (_leaf(t) for t in make_qkv(2, 200, 333, 4, 2, d, torch.bfloat16, seed=d))
    weight = torch.randn(d, device="cuda", dtype=torch.bfloat16)
    out = fa.flash_attn_func(q, k, v, causal=True)
    got = torch.autograd.grad((out.sum(dims) * weight).sum(), (q, k, v))
    assert "bwd_generic" not in _lib.last_path()
    dout = weight.expand(out.shape).contiguous()
    want = torch.autograd.grad(fa.flash_attn_func(q, k, v, causal=True), (q, k, v), dout)
    assert all(torch.equal(x, y) for x, y in zip(got, want))  # the kernels are deterministic


@pytest.mark.parametrize("d", [64, 128, 256])
def test_gradient_of_a_sum_packed_sequences(d):
    q, k, v = (_leaf(t.flatten(0, 1)) for t in make_qkv(1, 300, 300, 4, 2, d, torch.float16, seed=d)[:3])
    cu = torch.tensor([0, 100, 101, 300], dtype=torch.int32, device="cuda")
    run = lambda: fa.flash_attn_varlen_func(q, k, v, cu, cu, 199, 199, causal=True)
    weight = torch.randn(4, d, device="cuda", dtype=torch.float16)
    got = torch.autograd.grad((run().sum(0) * weight).sum(), (q, k, v))
    want = torch.autograd.grad(run(), (q, k, v), weight.expand(300, 4, d).contiguous())
    assert all(torch.equal(x, y) for x, y in zip(got, want))


@pytest.mark.parametrize("d", [64, 128, 256])
@pytest.mark.parametrize("what,base", [("kv", (1, 257, 4)), ("kv", (3, 257, 1)), ("kv", (3, 1, 4)), ("q", (1, 257, 4)), ("q", (3, 257, 1)), ("q", (3, 1, 4))])
def test_expanded_inputs(what, base, d):
    q, k, v, dout = make_qkv(3, 257, 257, 4, 4, d, torch.bfloat16, seed=d)
    small = [torch.randn(*base, d, device="cuda", dtype=torch.bfloat16) for _ in range(2)]
    big = [t.expand(3, 257, 4, d) for t in small]
    ins = (q, *big) if what == "kv" else (big[0], k, v)
    run = lambda ts: (lambda ls: (lambda o: (o, *torch.autograd.grad(o, ls, dout)))(fa.flash_attn_func(*ls, causal=True)))([_leaf(t) for t in ts])
    got, want = run(ins), run([t.contiguous() for t in ins])
    assert all(torch.equal(x, y) for x, y in zip(got, want))


@pytest.mark.parametrize("d", [64, 128, 256])
@pytest.mark.parametrize("over", ["batch", "heads"])
@pytest.mark.parametrize("sq", [1, 4, 40])  # the decode kernel's two uses, the tensor-core forward
def test_cache_that_repeats(sq, over, d):
    base = (1, 300, 2) if over == "batch" else (3, 300, 1)
    kc, vc = (torch.randn(*base, d, device="cuda", dtype=torch.bfloat16).expand(3, 300, 2, d) for _ in range(2))
    q = torch.randn(3, sq, 4, d, device="cuda", dtype=torch.bfloat16)
    lens = torch.tensor([300, 64, 129], dtype=torch.int32, device="cuda")
    out = fa.flash_attn_with_kvcache(q, kc, vc, cache_seqlens=lens, causal=True)
    assert _lib.last_path().startswith("kvcache_prep+fwd_generic"), _lib.last_path()  # reads by address, copies nothing
    kw = dict(cache_seqlens=lens, causal=True)
    ref, _, _ = O.kvcache_oracle(q, kc, vc, None, None, None, None, **kw)
    low, _, _ = O.kvcache_oracle(q, kc, vc, None, None, None, None, upcast=False, reorder_ops=True, **kw)
    assert_within(out, ref, low, mult=3, what="out")


def test_ring_block_with_an_expanded_query():
    q, k, v, _ = make_qkv(2, 256, 256, 4, 2, 128, torch.bfloat16)
    big = q[:, :, :1].expand(2, 256, 4, 128)
    got = CudaBlockOps.fwd(big, k, v, 0.1, (-1, 0), 0)
    assert _lib.last_path() == "fwd_generic"
    want = CudaBlockOps.fwd(big.contiguous(), k, v, 0.1, (-1, 0), 0)
    # another kernel: both round P to 16 bits before P V
    assert torch.allclose(got[0].float(), want[0].float(), atol=2e-2, rtol=2e-2) and torch.allclose(got[1], want[1], atol=1e-3)

"""The backward kernels in their two forms: one CTA per SM with wide blocks where the grid leaves every CTA an SM of its own, two
CTAs per SM with narrow ones (dQ, and dK / dV at head dim 64) where it does not.  The same sequences in a small and in a large
batch take one form each; both must match the oracle, and each other: the products are added up in the same order."""
import pytest
import torch

from gpu_util import assert_within, make_qkv, oracle_fwd_bwd

pytestmark = pytest.mark.gpu

if torch.cuda.is_available():
    import flash_attention_b200 as fa
    from flash_attention_b200 import _lib


def _grads(q, k, v, dout, **kw):
    ls = [t.detach().requires_grad_(True) for t in (q, k, v)]
    grads = torch.autograd.grad(fa.flash_attn_func(*ls, **kw), ls, dout)
    assert _lib.last_path() == "bwd_tc+bwd_dq_tc"
    return grads


@pytest.mark.parametrize("causal,window", [(True, (-1, -1)), (False, (-1, -1)), (False, (70, 40))])
@pytest.mark.parametrize("sq,sk,heads,heads_k,d,dtype", [
    (130, 130, 4, 4, 64, torch.bfloat16), (1, 257, 6, 2, 64, torch.float16), (300, 65, 4, 1, 64, torch.bfloat16),
    (129, 400, 4, 2, 128, torch.float16), (200, 128, 6, 6, 96, torch.bfloat16), (64, 64, 2, 2, 40, torch.bfloat16),
])
def test_both_forms(sq, sk, heads, heads_k, d, dtype, causal, window, monkeypatch):
    monkeypatch.setenv("FA_B200_FWD_SPLITS", "1")  # the same out and LSE: a small batch's forward may be split
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    ctas = min(-(-sq // 128) * heads, -(-sk // 128) * heads_k)  # of one sequence, in the smaller of the two grids
    small, large = 2, sms // ctas + 1
    assert max(-(-sq // 128) * heads, -(-sk // 128) * heads_k) * small <= sms < ctas * large
    q, k, v, dout = make_qkv(small, sq, sk, heads, heads_k, d, dtype, seed=sq + d)
    got = _grads(q, k, v, dout, causal=causal, window_size=window)
    (_, *ref), (_, *low) = oracle_fwd_bwd(q, k, v, dout, causal=causal, window_size=window)
    for x, t, l, name in zip(got, ref, low, ("dq", "dk", "dv")):
        assert_within(x, t, l, mult=3, what=name)
    many = [t.repeat(-(-large // small), 1, 1, 1) for t in (q, k, v, dout)]
    other = _grads(*many, causal=causal, window_size=window)
    for x, y in zip(got, other):
        assert torch.equal(x, y[:small]) and torch.equal(x, y[-small:])


@pytest.mark.parametrize("d", [64, 128])
def test_packed_sequences(d):
    lens = [0, 1, 129, 300, 64]
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    run = []
    for times in (1, sms // (3 * len(lens)) + 1):  # grid: 3 blocks x heads x sequences
        cu = torch.tensor([0] + lens * times, dtype=torch.int32).cumsum(0).int().cuda()
        q, k, v, dout = (t[0].repeat(times, 1, 1) for t in make_qkv(1, sum(lens), sum(lens), 2, 1, d, torch.bfloat16, seed=d))
        ls = [t.detach().requires_grad_(True) for t in (q, k, v)]
        out = fa.flash_attn_varlen_func(*ls, cu, cu, 300, 300, causal=True)
        run.append(torch.autograd.grad(out, ls, dout))
    n = sum(lens)
    assert 3 * 2 * len(lens) <= sms
    for x, y in zip(*run):
        assert torch.equal(x, y[:n]) and torch.equal(x, y[-n:])
    q, k, v, dout = make_qkv(1, n, n, 2, 1, d, torch.bfloat16, seed=d)
    first = 0
    for length in lens:
        s = slice(first, first + length)
        first += length
        if length:
            (_, *ref), (_, *low) = oracle_fwd_bwd(q[:, s], k[:, s], v[:, s], dout[:, s], causal=True)
            for x, t, l in zip(run[0], ref, low):
                assert_within(x[s], t[0], l[0], mult=3, what="length %d" % length)

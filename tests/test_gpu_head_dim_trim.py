"""Head dims between the tensor-core kernels' own (64, 128, 256), on both sides of every number of k-steps and chunks that the
kernels take.  A call whose tiles were full of NaN runs first: what a kernel read behind the head dim would show."""
import pytest
import torch

from gpu_util import assert_within, make_qkv, oracle_fwd_bwd

pytestmark = pytest.mark.gpu

if torch.cuda.is_available():
    import flash_attention_b200 as fa
    from flash_attention_b200 import _lib


def _run(q, k, v, dout, **kw):
    ls = [t.detach().requires_grad_(True) for t in (q, k, v)]
    out = fa.flash_attn_func(*ls, **kw)
    assert _lib.last_path() == "fwd_tc"
    return (out,) + torch.autograd.grad(out, ls, dout)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("d", [8, 32, 40, 48, 56, 72, 80, 88, 96, 104, 136, 160, 168, 192, 200])
@pytest.mark.parametrize("batch", [2, 40])  # 40: more CTAs than SMs, the other form of the backward
def test_nothing_behind_the_head_dim(d, dtype, batch, monkeypatch):
    monkeypatch.setenv("FA_B200_FWD_SPLITS", "1")
    full = 64 if d <= 64 else 128 if d <= 128 else 256
    _run(*(torch.full_like(t, float("nan")) for t in make_qkv(batch, 200, 200, 4, 2, full, dtype)))
    q, k, v, dout = make_qkv(2, 200, 200, 4, 2, d, dtype, seed=d)
    ref, low = oracle_fwd_bwd(q, k, v, dout, causal=True)
    got = _run(*(t.repeat(batch // 2, 1, 1, 1) for t in (q, k, v, dout)), causal=True)
    assert _lib.last_path() == ("bwd_wide_tc" if d > 128 else "bwd_tc+bwd_dq_tc")
    for x, t, l, name in zip(got, ref, low, ("out", "dq", "dk", "dv")):
        assert_within(x[:2], t, l, mult=3, what=name)
        assert torch.equal(x[:2], x[-2:])

"""The order of CTAs is worked out with multiplications the host prepares: grids whose sizes are 1, powers of two and their
neighbours, with whole and smaller last groups of heads, must visit every row block of every head once."""
import pytest
import torch

from gpu_util import assert_within, make_qkv, oracle_fwd_bwd

pytestmark = pytest.mark.gpu

if torch.cuda.is_available():
    import flash_attention_b200 as fa


@pytest.mark.parametrize("batch,heads,heads_k,d", [(1, 1, 1, 64), (3, 7, 7, 64), (17, 5, 5, 128), (2, 31, 31, 32), (5, 33, 11, 64), (2, 12, 1, 128),
                                                   (1, 63, 7, 160), (129, 1, 1, 40)])
@pytest.mark.parametrize("sq,sk", [(1, 70), (257, 257), (130, 1025)])
def test_every_row_once(batch, heads, heads_k, d, sq, sk):
    q, k, v, dout = make_qkv(batch, sq, sk, heads, heads_k, d, torch.bfloat16, seed=batch + heads)
    ls = [t.requires_grad_(True) for t in (q, k, v)]
    out = fa.flash_attn_func(*ls, causal=True)
    got = (out,) + torch.autograd.grad(out, ls, dout)
    ref, low = oracle_fwd_bwd(q, k, v, dout, causal=True)
    for x, t, l, name in zip(got, ref, low, ("out", "dq", "dk", "dv")):
        assert_within(x, t, l, mult=3, what=name)

"""The forward with one query tile per CTA and with two: lengths on both sides of the line between them, and tiles that are
full, ragged or a single row."""
import pytest
import torch

from gpu_util import assert_within, make_qkv, oracle_fwd_bwd

pytestmark = pytest.mark.gpu

if torch.cuda.is_available():
    import flash_attention_b200 as fa
    from flash_attention_b200 import _lib


@pytest.mark.parametrize("heads,heads_k,d,dtype", [(4, 4, 64, torch.bfloat16), (4, 4, 128, torch.float16), (8, 2, 128, torch.bfloat16),
                                                   (6, 1, 96, torch.bfloat16), (2, 2, 256, torch.float16)])
@pytest.mark.parametrize("sq,sk,causal,window", [
    (128, 128, False, (-1, -1)), (129, 640, False, (-1, -1)), (300, 576, False, (-1, -1)), (300, 577, False, (-1, -1)), (257, 1, False, (-1, -1)),
    (600, 1300, True, (-1, -1)), (128, 2300, True, (-1, -1)), (400, 129, True, (-1, -1)), (700, 700, False, (500, 0)), (700, 900, False, (900, 300)),
])
def test_both_sides(heads, heads_k, d, dtype, sq, sk, causal, window, monkeypatch):
    monkeypatch.setenv("FA_B200_FWD_SPLITS", "1")
    q, k, v, _ = make_qkv(2, sq, sk, heads, heads_k, d, dtype, seed=sq + sk)
    out = fa.flash_attn_func(q, k, v, causal=causal, window_size=window)
    assert _lib.last_path() == "fwd_tc"
    ref, low = oracle_fwd_bwd(q, k, v, None, causal=causal, window_size=window)
    assert_within(out, ref[0], low[0], what="out")
    # a longer batch takes the same form: the same bits
    more = fa.flash_attn_func(*(t.repeat(40, 1, 1, 1) for t in (q, k, v)), causal=causal, window_size=window)
    assert torch.equal(more[:2], out) and torch.equal(more[-2:], out)

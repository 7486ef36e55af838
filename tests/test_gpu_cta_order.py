"""Under a mask the CTAs of the tensor-core kernels take the row blocks of a group of (batch, head) pairs in turn, and the last
group may be smaller than the others.  Shapes whose pairs are not a multiple of the group (16 MB / bytes of a pair's streamed
rows); every output starts as NaN, so that a block nobody computes shows."""
import pytest
import torch

import flash_attn_2_cuda as ext
from gpu_util import assert_within, make_qkv, oracle_fwd_bwd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,S,H,Hk,d", [
    (1, 1500, 32, 32, 128),   # groups of 21 and 11 pairs
    (4, 1500, 32, 8, 128),    # the forward: 4 heads share a tile, 21 and 11 of 32 pairs
    (1, 1500, 48, 48, 64),    # 43 and 5
    (2, 1100, 9, 9, 256),     # 14 and 4, and the three passes of the wide backward
    (1, 4097, 5, 5, 256),     # 3 and 2, ragged
])
def test_last_group_is_smaller(B, S, H, Hk, d):
    q, k, v, dout = make_qkv(B, S, S, H, Hk, d, torch.bfloat16, seed=S + d)
    nan = lambda t: torch.full_like(t, float("nan"))
    out = nan(q)
    lse = ext.fwd(q, k, v, out, 0.0, d ** -0.5, True, -1, -1, False, None)[5]
    dq, dk, dv = ext.bwd(dout, q, k, v, out, lse, nan(q), nan(k), nan(v), 0.0, d ** -0.5, True, -1, -1, None, None)[:3]
    assert torch.isfinite(lse).all()
    step = max(1, Hk // 4)  # the oracle takes a few KV heads at a time
    for h in range(0, Hk, step):
        hs, hq = slice(h, h + step), slice(h * (H // Hk), min(Hk, h + step) * (H // Hk))
        (o_t, *ref), (o_l, *low) = oracle_fwd_bwd(q[:, :, hq], k[:, :, hs], v[:, :, hs], dout[:, :, hq], causal=True)
        for x, t, l, name in zip((out[:, :, hq], dq[:, :, hq], dk[:, :, hs], dv[:, :, hs]), (o_t, *ref), (o_l, *low), ("out", "dq", "dk", "dv")):
            assert_within(x, t, l, mult=3, what="%s of KV heads from %d" % (name, h))

"""Long streams through the backward of head dims above 128: thousands of blocks per CTA hand their operand over to the issuing warp, in every pass and
both widths of the tiles.  No wait may give up, and every run gives the same bits."""
import pytest
import torch

from gpu_util import make_qkv

pytestmark = pytest.mark.gpu

if torch.cuda.is_available():
    import flash_attention_b200 as fa
    from flash_attention_b200 import _lib


@pytest.mark.parametrize("d", [136, 160, 168, 192, 200, 256])
@pytest.mark.parametrize("sq,sk,heads,heads_k,causal", [(1568, 10332, 16, 16, False), (10332, 1568, 16, 16, False), (2048, 2048, 32, 8, True), (512, 512, 64, 1, False)])
def test_long_streams(d, sq, sk, heads, heads_k, causal):
    q, k, v, dout = make_qkv(1, sq, sk, heads, heads_k, d, torch.bfloat16, seed=d)
    ls = [t.requires_grad_(True) for t in (q, k, v)]
    out = fa.flash_attn_func(*ls, causal=causal)
    first = torch.autograd.grad(out, ls, dout, retain_graph=True)
    assert _lib.last_path() == "bwd_wide_tc"
    for _ in range(10):
        again = torch.autograd.grad(out, ls, dout, retain_graph=True)
        assert all(torch.equal(x, y) for x, y in zip(first, again))
    assert _lib.lib().fa_device_status() == 0

"""The decode kernel gives the same bits on every run: a slot of its ring is refilled only after all of it has been read.  Many CTAs per
SM and few keys each, one and several tokens, both head dims, one part and two."""
import pytest
import torch

pytestmark = pytest.mark.gpu

if torch.cuda.is_available():
    import flash_attention_b200 as fa
    from flash_attention_b200 import _lib


@pytest.mark.parametrize("splits", [1, 2])
@pytest.mark.parametrize("new", [1, 2, 4])
@pytest.mark.parametrize("batch,cap,heads,heads_k,d", [(45, 2560, 16, 4, 64), (64, 1536, 8, 8, 64), (40, 2048, 16, 4, 128)])
def test_same_bits(batch, cap, heads, heads_k, d, new, splits):
    g = torch.Generator(device="cuda").manual_seed(cap + new)
    r = lambda *shape: torch.randn(*shape, device="cuda", dtype=torch.bfloat16, generator=g)
    q, kc, vc = r(batch, new, heads, d), r(batch, cap, heads_k, d), r(batch, cap, heads_k, d)
    lens = torch.randint(cap // 4, cap + 1, (batch,), device="cuda", dtype=torch.int32, generator=g)
    first = None
    for i in range(80):
        if i % 2 == 0:  # (the caches partly out of the L2, as in a program that does other things between two steps)
            kc.copy_(kc.clone())
        out = fa.flash_attn_with_kvcache(q, kc, vc, cache_seqlens=lens, causal=True, num_splits=splits)
        assert "decode" in _lib.last_path()
        first = out if first is None else first
        assert torch.equal(out, first), "run %d" % i

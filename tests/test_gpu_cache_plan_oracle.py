"""Parts that the library plans for several tokens against a KV cache, against the oracle: the tolerance is that of the 16-bit oracle, not of the
kernel's own result in one part.  Which calls are split is asserted."""
import pytest
import torch

from gpu_util import assert_within
from oracle import attention_oracle as O

pytestmark = pytest.mark.gpu

if torch.cuda.is_available():
    import flash_attention_b200 as fa
    from flash_attention_b200 import _lib


@pytest.mark.parametrize("batch,new,heads,heads_k,cap,d,split", [
    (1, 17, 2, 2, 128, 128, False), (40, 20, 4, 4, 700, 128, False), (1, 33, 8, 1, 5000, 128, True), (2, 129, 8, 2, 2200, 64, True), (1, 64, 2, 1, 16500, 64, True),
    (3, 40, 6, 6, 1300, 160, True), (1, 20, 4, 4, 3000, 40, True), (2, 300, 4, 4, 4100, 96, True), (1, 300, 8, 8, 6000, 128, True), (5, 50, 16, 2, 1500, 256, True),
])
@pytest.mark.parametrize("fill", ["full", "ragged", "few"])
def test_planned_parts(batch, new, heads, heads_k, cap, d, split, fill):
    g = torch.Generator().manual_seed(cap)
    q = torch.randn(batch, new, heads, d, generator=g).bfloat16().cuda()
    kc, vc = (torch.randn(batch, cap, heads_k, d, generator=g).bfloat16().cuda() for _ in range(2))
    lo, hi = {"full": (cap, cap), "ragged": (new, cap), "few": (new, min(cap, new + 100))}[fill]
    lens = torch.randint(lo, hi + 1, (batch,), generator=g).int().cuda()
    truth, low = (O.kvcache_oracle(q, kc, vc, cache_seqlens=lens, causal=True, upcast=u, reorder_ops=not u)[0] for u in (True, False))
    behind = torch.arange(cap, device="cuda")[None] >= lens[:, None]
    kc[behind], vc[behind] = float("nan"), float("nan")
    for parts in (0, 1):
        out = fa.flash_attn_with_kvcache(q, kc, vc, cache_seqlens=lens, causal=True, num_splits=parts)
        assert _lib.last_path() == ("kvcache_prep+fwd_tc+combine" if split and not parts else "kvcache_prep+fwd_tc")
        assert_within(out, truth, low, mult=3, what="%d parts" % parts)

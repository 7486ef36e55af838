"""Parts of a multi-token call against a KV cache: whatever count the plan finds for small and large batches, row counts and capacities,
the result is that of one part."""
import pytest
import torch

from gpu_util import assert_within

pytestmark = pytest.mark.gpu

if torch.cuda.is_available():
    import flash_attention_b200 as fa


@pytest.mark.parametrize("batch,new,heads,heads_k,cap,d", [(1, 17, 4, 4, 1, 64), (1, 17, 2, 2, 128, 128), (1, 33, 8, 1, 5000, 128), (2, 129, 8, 2, 2200, 64),
                                                           (40, 20, 4, 4, 700, 128), (1, 64, 2, 1, 16500, 64), (3, 40, 6, 6, 1300, 160)])
def test_planned_parts(batch, new, heads, heads_k, cap, d):
    new = min(new, cap)
    g = torch.Generator().manual_seed(cap)
    q = torch.randn(batch, new, heads, d, generator=g).bfloat16().cuda()
    kc, vc = (torch.randn(batch, cap, heads_k, d, generator=g).bfloat16().cuda() for _ in range(2))
    lens = torch.randint(new, cap + 1, (batch,), generator=g).int().cuda()
    got = fa.flash_attn_with_kvcache(q, kc, vc, cache_seqlens=lens, causal=True)
    one = fa.flash_attn_with_kvcache(q, kc, vc, cache_seqlens=lens, causal=True, num_splits=1)
    f32 = []
    for b, n in enumerate(lens.tolist()):
        k, v = (t[b, :n].float().repeat_interleave(heads // heads_k, 1) for t in (kc, vc))
        s = torch.einsum("qhd,khd->hqk", q[b].float(), k) / d**0.5
        i, j = torch.arange(new, device="cuda")[:, None] + n - new, torch.arange(n, device="cuda")
        f32.append(torch.einsum("hqk,khd->qhd", s.masked_fill(j > i, float("-inf")).softmax(-1), v))
    assert_within(got, torch.stack(f32), one, mult=3, what="planned parts")

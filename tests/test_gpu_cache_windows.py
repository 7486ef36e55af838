"""Chunks against a KV cache on the tensor-core forward where the walk over the keys starts in the middle of the page table (a
window that cuts keys off), and shared query tiles read from a slice of a fused projection."""
import pytest
import torch

from gpu_util import assert_within
from oracle import attention_oracle as O

pytestmark = pytest.mark.gpu

if torch.cuda.is_available():
    import flash_attention_b200 as fa
    from flash_attention_b200 import _lib


@pytest.mark.parametrize("num_splits", [0, 1, 5])
@pytest.mark.parametrize("page", [0, 64, 128, 256])
@pytest.mark.parametrize("sq,heads,heads_k,d,window,dtype", [
    (33, 2, 2, 64, (100, 0), torch.bfloat16),     # one row more than the any-shape kernel keeps
    (130, 4, 2, 128, (200, 17), torch.float16),   # two tiles that start at different blocks
    (9, 8, 2, 128, (64, 0), torch.bfloat16),      # 36 rows: 9 positions x 4 heads
    (64, 3, 1, 96, (0, 0), torch.bfloat16),       # a row sees one key
    (40, 2, 2, 256, (129, 5), torch.bfloat16),
])
def test_window_that_cuts_keys_off(sq, heads, heads_k, d, window, dtype, page, num_splits):
    g = torch.Generator().manual_seed(sq + d)
    cap, lens = 1024, [0, 127, 128, 700, 1024 - sq]
    B = len(lens)
    q = torch.randn(B, sq, heads, d, generator=g).to(dtype).cuda()
    kn, vn = (torch.randn(B, sq, heads_k, d, generator=g).to(dtype).cuda() for _ in range(2))
    kc, vc = (torch.randn(B, cap, heads_k, d, generator=g).to(dtype).cuda() for _ in range(2))
    lens_t = torch.tensor(lens, dtype=torch.int32, device="cuda")
    kw = dict(cache_seqlens=lens_t, window_size=window)
    ref, _, _ = O.kvcache_oracle(q, kc, vc, kn, vn, None, None, **kw)
    low, _, _ = O.kvcache_oracle(q, kc, vc, kn, vn, None, None, upcast=False, reorder_ops=True, **kw)
    end = lens_t + sq
    kc[torch.arange(cap, device="cuda")[None] >= end[:, None]] = float("nan")
    vc[torch.arange(cap, device="cuda")[None] >= end[:, None]] = float("nan")
    if page:
        perm = torch.randperm(B * cap // page, generator=g).cuda()
        kp, vp = torch.empty_like(kc).view(-1, page, heads_k, d), torch.empty_like(vc).view(-1, page, heads_k, d)
        kp[perm], vp[perm] = kc.view(-1, page, heads_k, d), vc.view(-1, page, heads_k, d)
        # Pages whose keys no row sees are named by nothing that a kernel may follow.  The first key that is loaded starts the
        # 128-key block of the first row's first key.
        table = perm.view(B, cap // page).int()
        page_end = (torch.arange(cap // page, device="cuda")[None] + 1) * page
        first = (lens_t - window[0]).clamp(min=0) // 128 * 128
        seen = (page_end > first[:, None]) & (page_end - page < end[:, None])
        kw["block_table"] = torch.where(seen, table, torch.full_like(table, -1))
        kc, vc = kp, vp
    out = fa.flash_attn_with_kvcache(q, kc, vc, kn, vn, num_splits=num_splits, **kw)
    assert _lib.last_path().startswith("kvcache_prep+fwd_tc"), _lib.last_path()
    assert_within(out, ref, low, mult=3, what="out")


@pytest.mark.parametrize("d", [64, 128, 256])
@pytest.mark.parametrize("heads,heads_k,sq", [(8, 2, 130), (6, 2, 300), (5, 1, 77)])
def test_shared_tiles_of_a_strided_query(heads, heads_k, sq, d):
    """q, k and v as slices of one projection (batch, seq, (heads + 2 heads_k) * d), and with the heads in front of the positions"""
    g = torch.Generator().manual_seed(sq + d)
    proj = torch.randn(2, sq, (heads + 2 * heads_k) * d, generator=g).bfloat16().cuda()
    q = proj[..., :heads * d].unflatten(-1, (heads, d))
    k, v = proj[..., heads * d:].unflatten(-1, (2, heads_k, d)).unbind(2)
    want = fa.flash_attn_func(q.contiguous(), k.contiguous(), v.contiguous(), causal=True)
    assert torch.equal(fa.flash_attn_func(q, k, v, causal=True), want)
    front = [t.transpose(1, 2).contiguous().transpose(1, 2) for t in (q, k, v)]
    assert torch.equal(fa.flash_attn_func(*front, causal=True), want)
    ref, _ = O.attention_oracle(q, k, v, causal=True)
    low, _ = O.attention_oracle(q, k, v, causal=True, upcast=False, reorder_ops=True)
    assert_within(want, ref, low, what="out")
    # the chunk of a cache call: 40 new tokens
    kc, vc = (torch.zeros(2, 512, heads_k, d, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    lens = torch.tensor([200, 3], dtype=torch.int32, device="cuda")
    qs, ks, vs = q[:, :40], k[:, :40], v[:, :40]
    got = fa.flash_attn_with_kvcache(qs, kc.clone(), vc.clone(), ks, vs, cache_seqlens=lens, causal=True)
    assert _lib.last_path().startswith("kvcache_prep+fwd_tc")
    assert torch.equal(got, fa.flash_attn_with_kvcache(qs.contiguous(), kc, vc, ks.contiguous(), vs.contiguous(), cache_seqlens=lens, causal=True))

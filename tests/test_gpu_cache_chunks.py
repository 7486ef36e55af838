"""Several new tokens per sequence against a KV cache on the tensor-core forward, and its shared query tiles (128 rows =
positions x heads of a group): sizes at the edges of key blocks, pages and tiles, lengths 0 and full, group sizes that do
and do not divide 128.  Everything behind a sequence's last key is NaN: none of it may reach the result."""
import pytest
import torch

from gpu_util import assert_within, kvcache_truth, make_qkv
from oracle import attention_oracle as O

pytestmark = pytest.mark.gpu

if torch.cuda.is_available():
    import flash_attention_b200 as fa
    from flash_attention_b200 import _lib


@pytest.mark.parametrize("num_splits", [0, 1, 3])
@pytest.mark.parametrize("page", [0, 64, 256])
@pytest.mark.parametrize("sq,heads,heads_k,d,dtype,interleaved", [
    (33, 4, 4, 64, torch.bfloat16, False),
    (128, 8, 2, 128, torch.bfloat16, False),
    (129, 6, 2, 128, torch.float16, True),   # a tile of 42 positions x 3 heads leaves two rows unused
    (17, 14, 2, 96, torch.bfloat16, False),
    (40, 48, 1, 64, torch.float16, False),   # 48 heads on one KV head: tiles of 8 positions x 16 heads
    (70, 2, 1, 256, torch.bfloat16, True),
    (5, 8, 2, 128, torch.bfloat16, False),   # 20 rows
    (17, 3, 3, 80, torch.float16, False),    # 17 rows: one more than the decode kernel takes
])
def test_chunk_against_a_cache_with_nan_behind_the_keys(sq, heads, heads_k, d, dtype, interleaved, page, num_splits):
    g = torch.Generator().manual_seed(sq + d)
    lens, cap = [0, 1, 128 - sq % 128, 255 - sq % 100, 768 - sq], 768  # ends before, on and behind block and page edges
    B = len(lens)
    q = torch.randn(B, sq, heads, d, generator=g).to(dtype).cuda()
    kn = torch.randn(B, sq, heads_k, d, generator=g).to(dtype).cuda()
    vn = torch.randn(B, sq, heads_k, d, generator=g).to(dtype).cuda()
    kc = torch.randn(B, cap, heads_k, d, generator=g).to(dtype).cuda()
    vc = torch.randn(B, cap, heads_k, d, generator=g).to(dtype).cuda()
    angle = torch.rand(cap, d // 2, generator=g) * 6.3
    # the tables start 2 bytes into their storage in one case: no 16-byte loads from them then
    odd = 1 if sq == 33 else 0
    cos, sin = (torch.cat([torch.zeros(odd), f(angle).flatten()]).to(dtype).cuda()[odd:].view(cap, d // 2) for f in (torch.cos, torch.sin))
    lens_t = torch.tensor(lens, dtype=torch.int32, device="cuda")
    out_t, out_l, kc_t, vc_t = kvcache_truth(q, kc, vc, kn, vn, cos, sin, lens_t, interleaved)
    used = torch.arange(cap, device="cuda")[None] < lens_t[:, None] + sq
    kc[~used], vc[~used] = float("nan"), float("nan")
    kw = {}
    kp, vp = kc.clone(), vc.clone()
    if page:
        perm = torch.randperm(B * cap // page, generator=g).cuda()
        table = perm.view(B, cap // page).int()
        kp[:], vp[:] = float("nan"), float("nan")
        kp, vp = kp.view(-1, page, heads_k, d), vp.view(-1, page, heads_k, d)
        kp[perm], vp[perm] = kc.view(-1, page, heads_k, d), vc.view(-1, page, heads_k, d)
        # pages without a key are named by nothing that a kernel may follow
        first = torch.arange(cap // page, device="cuda")[None] * page
        kw["block_table"] = torch.where(first < lens_t[:, None] + sq, table, torch.full_like(table, -1))
    out, lse = fa.flash_attn_with_kvcache(q, kp, vp, kn, vn, cos, sin, lens_t, causal=True, rotary_interleaved=interleaved,
                                          num_splits=num_splits, return_softmax_lse=True, **kw)
    assert _lib.last_path().startswith("kvcache_prep+fwd_tc"), _lib.last_path()
    assert_within(out, out_t, out_l, mult=3, what="out")
    assert torch.isfinite(lse).all()
    if page:
        kp, vp = (t[perm].view(B, cap, heads_k, d) for t in (kp, vp))
    assert torch.allclose(kp[used].float(), kc_t[used].float(), rtol=1e-3, atol=1e-3) and torch.equal(vp[used], vc_t[used])
    assert torch.isnan(kp[~used]).all() and torch.isnan(vp[~used]).all()


@pytest.mark.parametrize("causal,window", [(True, (-1, -1)), (False, (-1, -1)), (False, (70, 9))])
@pytest.mark.parametrize("sq,sk,heads,heads_k,d", [
    (64, 64, 8, 2, 128), (65, 130, 8, 2, 64), (85, 257, 9, 3, 128), (300, 300, 10, 2, 64), (256, 384, 16, 1, 256),
    (127, 513, 48, 1, 64), (50, 128, 67, 1, 64),
])
def test_tiles_shared_by_the_heads_of_a_group(sq, sk, heads, heads_k, d, causal, window):
    q, k, v, _ = make_qkv(2, sq, sk, heads, heads_k, d, torch.bfloat16, seed=sq + sk)
    out, lse, _ = fa.flash_attn_func(q, k, v, causal=causal, window_size=window, return_attn_probs=True)
    assert _lib.last_path().startswith("fwd_tc")
    ref, _ = O.attention_oracle(q, k, v, causal=causal, window_size=window)
    low, _ = O.attention_oracle(q, k, v, causal=causal, window_size=window, upcast=False, reorder_ops=True)
    assert_within(out, ref, low, what="out")
    s = torch.einsum("bqhd,bkhd->bhqk", q.float(), k.float().repeat_interleave(heads // heads_k, 2)) * d ** -0.5
    i, j = torch.arange(sq, device="cuda")[:, None] + sk - sq, torch.arange(sk, device="cuda")[None]
    hidden = (j > i + (0 if causal else window[1])) if causal or window[1] >= 0 else torch.zeros_like(j > i)
    if window[0] >= 0:
        hidden = hidden | (j < i - window[0])
    want = torch.logsumexp(s.masked_fill(hidden, float("-inf")), -1)
    assert torch.allclose(lse, want.masked_fill(want == float("-inf"), float("inf")), atol=1e-3)


@pytest.mark.parametrize("num_splits", [0, 1, 5])
@pytest.mark.parametrize("page", [0, 64])
@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("sq,new,heads,heads_k,d,dtype", [
    (2, 2, 8, 1, 128, torch.bfloat16),   # all 16 rows of the tile
    (5, 5, 6, 2, 64, torch.float16),     # 15 rows
    (16, 16, 2, 2, 128, torch.bfloat16),
    (1, 3, 4, 2, 64, torch.bfloat16),    # more new tokens than queries
    (4, 0, 4, 2, 128, torch.float16),    # queries against what the cache holds
])
def test_a_few_tokens_per_sequence(sq, new, heads, heads_k, d, dtype, causal, page, num_splits):
    g = torch.Generator().manual_seed(sq + d)
    cap, B = 512, 5
    lens = [max(0, sq - new), 64 - new if new else 64, 65, 200, cap - new]
    q = torch.randn(B, sq, heads, d, generator=g).to(dtype).cuda()
    kn, vn = (torch.randn(B, new, heads_k, d, generator=g).to(dtype).cuda() if new else None for _ in range(2))
    kc = torch.randn(B, cap, heads_k, d, generator=g).to(dtype).cuda()
    vc = torch.randn(B, cap, heads_k, d, generator=g).to(dtype).cuda()
    lens_t = torch.tensor(lens, dtype=torch.int32, device="cuda")
    kw = dict(cache_seqlens=lens_t, causal=causal)
    out_t, kc_t, vc_t = O.kvcache_oracle(q, kc, vc, kn, vn, None, None, **kw)
    out_l, _, _ = O.kvcache_oracle(q, kc, vc, kn, vn, None, None, upcast=False, reorder_ops=True, **kw)
    used = torch.arange(cap, device="cuda")[None] < lens_t[:, None] + new
    kc[~used], vc[~used] = float("nan"), float("nan")
    kp, vp = kc.clone(), vc.clone()
    if page:
        perm = torch.randperm(B * cap // page, generator=g).cuda()
        kp, vp = torch.empty_like(kc).view(-1, page, heads_k, d), torch.empty_like(vc).view(-1, page, heads_k, d)
        kp[perm], vp[perm] = kc.view(-1, page, heads_k, d), vc.view(-1, page, heads_k, d)
        kw["block_table"] = perm.view(B, cap // page).int()
    out = fa.flash_attn_with_kvcache(q, kp, vp, kn, vn, num_splits=num_splits, **kw)
    assert "decode" in _lib.last_path(), _lib.last_path()
    assert_within(out, out_t, out_l, mult=3, what="out")
    if page:
        kp, vp = (t[perm].view(B, cap, heads_k, d) for t in (kp, vp))
    assert torch.equal(kp[used], kc_t[used]) and torch.equal(vp[used], vc_t[used])

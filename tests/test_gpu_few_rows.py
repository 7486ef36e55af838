"""Rows that fill one query tile at most, in parts: CTAs that share an SM, and CTAs that have one each and then walk many key blocks,
which take the two-tile form for its longer ring.  KV caches on both sides of their line."""
import pytest
import torch

from gpu_util import assert_within, make_qkv, oracle_fwd_bwd
from oracle import attention_oracle as O

pytestmark = pytest.mark.gpu

if torch.cuda.is_available():
    import flash_attention_b200 as fa
    from flash_attention_b200 import _lib


@pytest.mark.parametrize("batch,sq,heads,heads_k,d,parts,sk,tiles", [
    (4, 18, 16, 8, 96, 4, 8300, 2), (4, 18, 16, 8, 96, 9, 10240, 1), (4, 18, 16, 8, 128, 4, 5000, 1), (1, 128, 8, 8, 128, 12, 17000, 2),
    (2, 31, 8, 4, 128, 1, 1409, 2), (2, 31, 8, 4, 128, 1, 1280, 1), (2, 31, 8, 4, 80, 3, 4300, 2), (1, 20, 4, 2, 64, 2, 4500, 2),
    (1, 20, 4, 2, 40, 2, 4500, 2), (1, 20, 4, 2, 64, 2, 4000, 1), (1, 128, 2, 2, 128, 1, 1, 1), (2, 31, 8, 4, 88, 2, 1100, 2), (2, 31, 8, 4, 104, 2, 896, 1), (2, 33, 6, 6, 192, 2, 5000, 1),
])
@pytest.mark.parametrize("causal", [False, True])
def test_parts(batch, sq, heads, heads_k, d, parts, sk, tiles, causal, monkeypatch):
    monkeypatch.setenv("FA_B200_FWD_SPLITS", str(parts))
    q, k, v, _ = make_qkv(batch, sq, sk, heads, heads_k, d, torch.bfloat16, seed=sk)
    out = fa.flash_attn_func(q, k, v, causal=causal)
    assert _lib.last_path() == ("fwd_tc+combine" if parts > 1 else "fwd_tc")
    if not causal or tiles == 2:
        assert _lib.last_forward_tiles() == tiles
    ref, low = oracle_fwd_bwd(q, k, v, None, causal=causal)
    assert_within(out, ref[0], low[0], what="out")


@pytest.mark.parametrize("batch,new,heads,heads_k,d,parts,cap,tiles", [
    (4, 40, 8, 8, 128, 1, 1400, 2), (4, 40, 8, 8, 128, 1, 1280, 1), (40, 40, 8, 8, 128, 1, 1400, 1), (4, 40, 4, 4, 64, 1, 2200, 2),
    (2, 129, 8, 8, 128, 1, 1250, 2), (2, 129, 8, 8, 128, 1, 1000, 1), (2, 120, 8, 2, 64, 2, 2300, 2), (2, 140, 4, 4, 64, 2, 2300, 1),
    (2, 140, 4, 4, 96, 1, 2300, 2), (2, 140, 4, 4, 96, 2, 3000, 1), (2, 300, 8, 8, 128, 1, 1500, 1), (2, 300, 8, 8, 128, 1, 1900, 2), (2, 140, 4, 4, 104, 1, 900, 2), (2, 140, 4, 4, 72, 1, 700, 1), (2, 140, 8, 2, 120, 1, 500, 2),
])
@pytest.mark.parametrize("page", [0, 64])
def test_cache(batch, new, heads, heads_k, d, parts, cap, tiles, page):
    cap = (cap + 63) // 64 * 64 if page else cap
    g = torch.Generator().manual_seed(cap)
    q = torch.randn(batch, new, heads, d, generator=g).bfloat16().cuda()
    kc, vc = (torch.randn(batch, cap, heads_k, d, generator=g).bfloat16().cuda() for _ in range(2))
    lens = torch.randint(new, cap + 1, (batch,), generator=g).int().cuda()
    truth, low = (O.kvcache_oracle(q, kc, vc, cache_seqlens=lens, causal=True, upcast=u, reorder_ops=not u)[0] for u in (True, False))
    behind = torch.arange(cap, device="cuda")[None] >= lens[:, None]
    kc[behind], vc[behind] = float("nan"), float("nan")
    kw = {}
    if page:
        perm = torch.randperm(batch * cap // page, generator=g).cuda()
        kp, vp = (torch.empty_like(t).view(-1, page, heads_k, d) for t in (kc, vc))
        kp[perm], vp[perm] = kc.view(-1, page, heads_k, d), vc.view(-1, page, heads_k, d)
        kc, vc, kw = kp, vp, {"block_table": perm.view(batch, -1).int()}
    out = fa.flash_attn_with_kvcache(q, kc, vc, cache_seqlens=lens, causal=True, num_splits=parts, **kw)
    assert _lib.last_path() == "kvcache_prep+fwd_tc" + ("+combine" if parts > 1 else "")
    assert _lib.last_forward_tiles() == tiles
    assert_within(out, truth, low, mult=3, what="out")

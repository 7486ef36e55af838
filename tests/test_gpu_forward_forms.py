"""The forward with two query tiles per CTA and with one, each where the rule of the library takes it: the form that ran is asserted.
Head dims that fill the kernel's own and ones that are trimmed, masks, packed batches, tiles of one head and shared ones."""
import pytest
import torch

from gpu_util import assert_within, make_qkv, oracle_fwd_bwd

pytestmark = pytest.mark.gpu

if torch.cuda.is_available():
    import flash_attention_b200 as fa
    from flash_attention_b200 import _lib


def _check(q, k, v, tiles, **kw):
    out = fa.flash_attn_func(q, k, v, **kw)
    assert _lib.last_path() == "fwd_tc" and _lib.last_forward_tiles() == tiles
    ref, low = oracle_fwd_bwd(q, k, v, None, **kw)
    assert_within(out, ref[0], low[0], what="out")


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("heads,heads_k", [(60, 60), (80, 10)])  # enough heads for one part; own tiles and shared ones
@pytest.mark.parametrize("d", [8, 32, 48, 56, 64, 72, 80, 96, 104, 128])
@pytest.mark.parametrize("blocks,more", [(4.5, 0), (4.5, 1), (4.5, 200)])  # the line without a mask; 2.5 where rows are not whole sectors
def test_no_mask(d, heads, heads_k, blocks, more, dtype):
    sk, tiles = int((2.5 if d in (72, 104) else blocks) * 128) + more, 2 if more else 1
    q, k, v, _ = make_qkv(2, 300, sk, heads, heads_k, d, dtype, seed=d)
    _check(q, k, v, tiles)


@pytest.mark.parametrize("sk,tiles", [(320, 1), (321, 2)])  # 240 one-tile CTAs, two to an SM: 2.5 blocks
@pytest.mark.parametrize("d", [64, 80, 128])
def test_no_mask_two_to_an_sm(d, sk, tiles):
    q, k, v, _ = make_qkv(2, 300, sk, 40, 40, d, torch.bfloat16, seed=d)
    _check(q, k, v, tiles)


@pytest.mark.parametrize("sq,sk,d,tiles,causal,window", [
    (300, 2600, 64, 2, True, (-1, -1)), (300, 2600, 40, 2, True, (-1, -1)), (300, 1900, 64, 1, True, (-1, -1)), (300, 1900, 32, 1, True, (-1, -1)), (300, 2000, 64, 2, True, (-1, -1)),
    (300, 2600, 64, 2, False, (2300, 0)), (300, 2600, 48, 2, False, (2200, 100)), (300, 2600, 64, 1, False, (1500, 0)),
    (300, 1400, 128, 2, True, (-1, -1)), (300, 1400, 80, 2, True, (-1, -1)), (300, 1200, 128, 1, True, (-1, -1)), (300, 1200, 96, 1, True, (-1, -1)),
    (300, 1400, 128, 2, False, (1000, 200)), (300, 1400, 72, 2, False, (1200, 0)), (300, 1400, 128, 1, False, (900, 0)),
    (300, 900, 104, 2, True, (-1, -1)), (300, 800, 88, 1, True, (-1, -1)), (300, 900, 120, 2, False, (700, 20)), (300, 900, 112, 1, True, (-1, -1)),
    (1111, 2500, 96, 2, True, (-1, -1)), (257, 4100, 56, 2, True, (-1, -1)),
])
def test_masked(sq, sk, d, tiles, causal, window):
    q, k, v, _ = make_qkv(1, sq, sk, 60, 60, d, torch.bfloat16, seed=sk + d)
    _check(q, k, v, tiles, causal=causal, window_size=window)


@pytest.mark.parametrize("s,heads,d,dtype", [(4300, 8, 64, torch.float16), (4300, 8, 40, torch.bfloat16), (2300, 14, 128, torch.bfloat16), (2300, 14, 80, torch.float16)])
def test_long_causal(s, heads, d, dtype):
    q, k, v, _ = make_qkv(1, s, s, heads, heads, d, dtype, seed=d)
    _check(q, k, v, 2, causal=True)


@pytest.mark.parametrize("heads,heads_k,d,tiles,lens_q,lens_k", [
    (4, 4, 64, 2, (1, 300, 128, 257), (2300, 2701, 3000, 2049)), (4, 4, 40, 2, (200, 130, 0, 300), (3000, 2500, 2600, 2100)),
    (4, 4, 128, 2, (1, 300, 128, 257), (1300, 1401, 1700, 1025)), (4, 4, 80, 2, (255, 256, 300, 0), (1300, 1401, 1700, 1025)),
    (8, 2, 128, 2, (300, 129, 65, 31), (700, 900, 641, 1000)), (4, 4, 64, 1, (1, 300, 128, 257), (300, 500, 900, 257)),
    (4, 4, 96, 1, (255, 256, 300, 0), (300, 500, 900, 257)),
])
@pytest.mark.parametrize("causal", [True, False])
def test_packed(heads, heads_k, d, tiles, lens_q, lens_k, causal):
    g = torch.Generator().manual_seed(d)
    q = torch.randn(sum(lens_q), heads, d, generator=g).bfloat16().cuda()
    k, v = (torch.randn(sum(lens_k), heads_k, d, generator=g).bfloat16().cuda() for _ in range(2))
    cu_q, cu_k = (torch.tensor([0, *t], dtype=torch.int32).cumsum(0).int().cuda() for t in (lens_q, lens_k))
    out = fa.flash_attn_varlen_func(q, k, v, cu_q, cu_k, max(lens_q), max(lens_k), causal=causal)
    assert _lib.last_path() == "fwd_tc"
    if causal or tiles == 2:
        assert _lib.last_forward_tiles() == tiles
    qs, ks, vs = q.split(lens_q), k.split(lens_k), v.split(lens_k)
    for i, o in enumerate(out.split(lens_q)):
        if lens_q[i]:
            ref, low = oracle_fwd_bwd(qs[i][None], ks[i][None], vs[i][None], None, causal=causal)
            assert_within(o[None], ref[0], low[0], what="sequence %d" % i)


@pytest.mark.parametrize("heads,heads_k,d,tiles,lens", [
    (4, 4, 64, 2, (4200, 60, 40, 33)), (4, 4, 64, 2, (33, 60, 4200, 1, 0)), (4, 4, 128, 2, (70, 4000, 200)), (4, 4, 80, 1, (2600, 60, 50, 40)), (8, 2, 128, 2, (900, 20, 30)),
    (8, 2, 64, 1, (600, 500, 550)), (4, 4, 128, 1, (2600, 60, 50, 40)), (4, 4, 128, 2, (2300, 2300)),
])
def test_packed_unequal(heads, heads_k, d, tiles, lens):
    """Few long sequences among short ones go by the long ones."""
    g = torch.Generator().manual_seed(d)
    q = torch.randn(sum(lens), heads, d, generator=g).half().cuda()
    k, v = (torch.randn(sum(lens), heads_k, d, generator=g).half().cuda() for _ in range(2))
    cu = torch.tensor([0, *lens], dtype=torch.int32).cumsum(0).int().cuda()
    out = fa.flash_attn_varlen_func(q, k, v, cu, cu, max(lens), max(lens), causal=True)
    assert _lib.last_path() == "fwd_tc" and _lib.last_forward_tiles() == tiles
    for i, (o, qs, ks, vs) in enumerate(zip(out.split(lens), q.split(lens), k.split(lens), v.split(lens))):
        if lens[i]:
            ref, low = oracle_fwd_bwd(qs[None], ks[None], vs[None], None, causal=True)
            assert_within(o[None], ref[0], low[0], what="sequence %d" % i)

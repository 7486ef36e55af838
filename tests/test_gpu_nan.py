"""A NaN in q or in a key must reach every row that sees it, whatever the number of splits: with parts that are merged the
result is what one pass gives (O = NaN, LSE = +inf), and rows that do not see the NaN are not touched."""
import pytest
import torch

from gpu_util import make_qkv
from oracle import attention_oracle as O

pytestmark = pytest.mark.gpu

if torch.cuda.is_available():
    import flash_attention_b200 as fa
    from flash_attention_b200 import _lib

NAN = float("nan")


def _check(out, lse, ref, sees):
    """out (B, S, H, D), lse (B, H, S); sees (B, S, H) says which rows see a NaN"""
    assert torch.isnan(out[sees]).all()
    assert torch.isfinite(out[~sees]).all()
    # P and O are rounded to 16 bits, each to 2^-9 of a value of at most about 4
    assert torch.allclose(out[~sees].float(), ref[~sees].float(), rtol=2 ** -6, atol=1e-2)
    assert torch.equal(torch.isinf(lse).transpose(1, 2), sees) and (lse[torch.isinf(lse)] > 0).all()


@pytest.mark.parametrize("generic", [False, True])
@pytest.mark.parametrize("splits", [1, 2, 3, 5, 6])
@pytest.mark.parametrize("d", [64, 128, 256])
def test_forward(d, splits, generic, monkeypatch):
    monkeypatch.setenv("FA_B200_FWD_SPLITS", str(splits))
    if generic:
        monkeypatch.setenv("FA_B200_FORCE_GENERIC", "1")
    B, S, H = 2, 700, 2
    q, k, v, _ = make_qkv(B, S, S, H, H, d, torch.bfloat16, seed=d)
    ref, _ = O.attention_oracle(q, k, v, causal=True)
    sees = torch.zeros(B, S, H, dtype=torch.bool, device="cuda")
    q[0, 300, 1, 5], sees[0, 300, 1] = NAN, True
    k[1, 400, 0, 7], sees[1, 400:, 0] = NAN, True
    out, lse, _ = fa.flash_attn_func(q, k, v, causal=True, return_attn_probs=True)
    assert _lib.last_path() == ("fwd_generic" if generic else "fwd_tc") + ("+combine" if splits > 1 else "")
    _check(out, lse, ref, sees)


@pytest.mark.parametrize("num_splits", [1, 2, 3, 6])
@pytest.mark.parametrize("d,sq,path", [(128, 40, "kvcache_prep+fwd_tc"), (64, 4, "kvcache_prep+decode"), (128, 1, "decode"), (96, 4, "kvcache_prep+fwd_generic")])
def test_cache(d, sq, path, num_splits):
    B, cap, H = 3, 700, 2
    q, k, v, _ = make_qkv(B, sq, cap, H, H, d, torch.bfloat16, seed=d)
    lens = torch.tensor([700, 650, 500], dtype=torch.int32, device="cuda")
    ref, _, _ = O.kvcache_oracle(q, k, v, None, None, None, None, cache_seqlens=lens, causal=True)
    sees = torch.zeros(B, sq, H, dtype=torch.bool, device="cuda")
    q[0, sq - 1, 1, 5], sees[0, sq - 1, 1] = NAN, True
    k[1, 200, 0, 7], sees[1, :, 0] = NAN, True
    k[2, 600, 0, 7] = NAN  # behind the last key
    out, lse = fa.flash_attn_with_kvcache(q, k, v, cache_seqlens=lens, causal=True, num_splits=num_splits, return_softmax_lse=True)
    assert _lib.last_path() == path + ("+combine" if num_splits > 1 else "")
    _check(out, lse, ref, sees)


@pytest.mark.parametrize("splits", [1, 3, 6])
def test_a_value_that_is_nan_or_infinite_stays_in_its_column(splits, monkeypatch):
    monkeypatch.setenv("FA_B200_FWD_SPLITS", str(splits))
    q, k, v, _ = make_qkv(1, 130, 700, 1, 1, 128, torch.bfloat16)
    ref, _ = O.attention_oracle(q, k, v)
    v[0, 650, 0, 3], v[0, 20, 0, 9] = NAN, float("inf")
    k[0, 20] = -60 * q.mean(1)  # weights that may be 0 in the merge: 0 * inf is NaN in one pass as well
    out = fa.flash_attn_func(q, k, v)
    assert torch.isnan(out[..., 3]).all() and not torch.isfinite(out[..., 9]).any()
    rest = [c for c in range(128) if c not in (3, 9)]
    assert torch.isfinite(out[..., rest]).all()

"""The merge of split parts at the edges of its groups of 32 parts: empty parts (LSE -inf, rows that nobody wrote) in front, in the
middle and at the end, rows without any key, a part with a NaN score; against the sum in 64 bits."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu

if torch.cuda.is_available():
    from flash_attention_b200._lib import check, lib, ptr


@pytest.mark.parametrize("n_parts", [1, 2, 3, 8, 9, 31, 32, 33, 64, 65, 127, 128])
@pytest.mark.parametrize("rows,d,dtype", [(1, 64, torch.bfloat16), (5, 40, torch.float16), (129, 128, torch.bfloat16), (66, 256, torch.float16)])
def test_merge(rows, d, dtype, n_parts):
    g = torch.Generator().manual_seed(rows + n_parts)
    parts = torch.randn(n_parts, rows, d, generator=g).cuda()
    lse = (torch.randn(n_parts, rows, generator=g) * 3).cuda()
    kind = torch.arange(rows, device="cuda") % 6  # 0: all parts, 1: every third empty, 2: only the first, 3: only the last, 4: none, 5: NaN
    part = torch.arange(n_parts, device="cuda")[:, None]
    empty = ((kind == 1) & (part % 3 == 1)) | ((kind == 2) & (part > 0)) | ((kind == 3) & (part < n_parts - 1)) | (kind == 4)
    lse[empty] = float("-inf")
    parts[empty] = float("nan")  # never written
    bad = kind == 5
    lse[n_parts // 2, bad], parts[n_parts // 2, bad] = float("nan"), float("nan")
    out = torch.full((rows, d), 7.0, dtype=dtype, device="cuda")
    got_lse = torch.full((rows,), 7.0, device="cuda")
    check(lib().fa_combine(ptr(parts), ptr(lse), ptr(out), ptr(got_lse), n_parts, rows, d, d, 1 if dtype == torch.bfloat16 else 0,
                           ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)), "fa_combine")
    want_lse = torch.logsumexp(lse.double(), 0)
    none = kind == 4
    weight = torch.exp(lse.double() - torch.where(none, torch.zeros_like(want_lse), want_lse)).masked_fill(empty, 0)
    want = (weight[..., None] * parts.double().masked_fill(empty[..., None], 0)).sum(0)
    assert torch.isnan(out[bad]).all() and (got_lse[bad | none] == float("inf")).all()
    assert (out[none] == 0).all()
    ok = ~bad & ~none
    # fp32 sums of at most 128 terms below 5 with __expf weights, then one rounding to 16 bits
    assert torch.allclose(out[ok].double(), want[ok], rtol=2 ** -8, atol=1e-4)
    assert torch.allclose(got_lse[ok].double(), want_lse[ok], rtol=1e-5, atol=1e-4)

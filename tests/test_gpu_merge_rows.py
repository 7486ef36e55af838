"""The merge of one to five parts with more rows than are loaded before their weights are known (4096), and just as many: an instance of the
kernel of its own below four parts.  Empty parts whose rows nobody wrote, rows without any key, NaN scores."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu

if torch.cuda.is_available():
    from flash_attention_b200._lib import check, lib, ptr


@pytest.mark.parametrize("n_parts", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("rows,d,dtype", [(4096, 128, torch.bfloat16), (4097, 64, torch.float16), (4100, 128, torch.bfloat16), (4103, 40, torch.float16), (4100, 256, torch.bfloat16)])
def test_many_rows(rows, d, dtype, n_parts):
    g = torch.Generator().manual_seed(rows + n_parts)
    parts = torch.randn(n_parts, rows, d, generator=g).cuda()
    lse = (torch.randn(n_parts, rows, generator=g) * 3).cuda()
    # which parts of a row are empty: every subset in turn; every 37th row has a NaN part
    row, part = torch.arange(rows, device="cuda"), torch.arange(n_parts, device="cuda")[:, None]
    empty = ((row % (1 << n_parts)) >> part & 1) == 1
    lse[empty], parts[empty] = float("-inf"), float("nan")
    bad = row % 37 == 36
    lse[row[bad] % n_parts, row[bad]] = float("nan")
    parts[row[bad] % n_parts, row[bad]] = float("nan")
    none = empty.all(0) & ~bad
    out = torch.full((rows, d), 7.0, dtype=dtype, device="cuda")
    got_lse = torch.full((rows,), 7.0, device="cuda")
    check(lib().fa_combine(ptr(parts), ptr(lse), ptr(out), ptr(got_lse), n_parts, rows, d, d, 1 if dtype == torch.bfloat16 else 0,
                           ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)), "fa_combine")
    assert torch.isnan(out[bad]).all() and (got_lse[bad | none] == float("inf")).all()
    assert (out[none] == 0).all()
    ok = ~bad & ~none
    want_lse = torch.logsumexp(lse.double(), 0)
    weight = torch.exp(lse.double() - want_lse).masked_fill(empty, 0)
    want = (weight[..., None] * parts.double().masked_fill(empty[..., None], 0)).sum(0)
    # fp32 sums of at most 5 terms below 6 with __expf weights, then one rounding to 16 bits
    assert torch.allclose(out[ok].double(), want[ok], rtol=2 ** -8, atol=1e-4)
    assert torch.allclose(got_lse[ok].double(), want_lse[ok], rtol=1e-5, atol=1e-4)

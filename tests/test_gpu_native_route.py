"""Plain calls are checked and launched by csrc/torch_glue.cpp, all others by the python code of flash_attn_2_cuda.  The two take
the same calls, refuse the same ones and give the same bits."""
import pytest
import torch

from gpu_util import make_qkv

pytestmark = pytest.mark.gpu

if torch.cuda.is_available():
    import flash_attn_2_cuda as ext


def test_packed_calls_need_their_offsets():
    """4-D operands and no cu_seqlens: an error of the packed entry points, not a padded batch."""
    q, k, v, dout = make_qkv(2, 130, 130, 4, 2, 64, torch.bfloat16)
    out, *_, lse, _, rng = ext.fwd(q, k, v, None, 0.0, 0.125, False, -1, -1, False, None)
    cu = torch.tensor([0, 130, 260], dtype=torch.int32, device="cuda")
    grads = [torch.empty_like(t) for t in (q, k, v)]
    flat = [t.flatten(0, 1) for t in (q, k, v, dout, out)]
    for a, b in ((None, None), (None, cu), (cu, None)):
        for ts in ((q, k, v, dout, out), flat):
            with pytest.raises((RuntimeError, AttributeError)):
                ext.varlen_fwd(*ts[:3], None, a, b, 130, 130, 0.0, 0.125, False, False, -1, -1, False, None)
            with pytest.raises((RuntimeError, AttributeError)):
                ext.varlen_bwd(ts[3], *ts[:3], ts[4], lse, *grads, a, b, 130, 130, 0.0, 0.125, False, False, -1, -1, None, rng)
    packed = ext.varlen_fwd(*flat[:3], None, cu, cu, 130, 130, 0.0, 0.125, False, False, -1, -1, False, None)
    assert torch.equal(packed[0].view_as(out), out)

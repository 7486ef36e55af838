"""The first call of a process inside a stream capture: what the kernels keep on the device and on the host (status word,
mirror, shared-memory limits) is set up there and then, without breaking the capture."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CALL = """
import sys, torch
sys.path.insert(0, {root!r})
import flash_attention_b200 as fa
from flash_attention_b200 import _lib
new = {new}
q, kn, vn = (torch.randn(2, new or 300, 4, 128, device="cuda", dtype=torch.bfloat16) for _ in range(3))
kc, vc = (torch.randn(2, 1024, 4, 128, device="cuda", dtype=torch.bfloat16) for _ in range(2))
lens = torch.tensor([100, 300], dtype=torch.int32, device="cuda")
call = lambda: (fa.flash_attn_with_kvcache(q, kc, vc, kn, vn, cache_seqlens=lens, causal=True) if new else
                fa.flash_attn_func(q, kn, vn, causal=True))
torch.cuda.synchronize()
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph):
    out = call()
path = _lib.last_path()
graph.replay()
torch.cuda.synchronize()
assert torch.equal(out, call())
print("path", path)
"""


@pytest.mark.parametrize("new,path", [(0, "fwd_tc"), (1, "decode"), (4, "kvcache_prep+decode"), (40, "kvcache_prep+fwd_tc")])
def test_first_call_of_a_process_is_captured(new, path):
    r = subprocess.run([sys.executable, "-c", CALL.format(root=ROOT, new=new)], capture_output=True, text=True, timeout=240)
    assert r.returncode == 0, r.stderr[-2000:]
    assert "path " + path in r.stdout

"""The first call of a process, where the library sets up what it keeps per device."""

import pytest

from tests.test_operator_errors import run_python

CAPTURE_AT_ONCE = """
import torch
from trifast_b200 import triangle_attention
n, d, dtype = %d, %d, torch.%s
q, k, v = (torch.randn(1, 2, n, n, d, device="cuda").to(dtype) for _ in range(3))
b = torch.randn(1, 2, n, n, device="cuda").to(dtype)
m = torch.zeros(1, n, n, dtype=torch.bool, device="cuda")
torch.cuda.synchronize()
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph):
    o = triangle_attention(q, k, v, b, m)
graph.replay()
torch.cuda.synchronize()
assert torch.equal(o, triangle_attention(q, k, v, b, m))
print("replayed")
"""


@pytest.mark.gpu
@pytest.mark.parametrize("n,d,dtype", [(32, 32, "float32"), (64, 32, "bfloat16"), (192, 128, "float16")])
def test_first_call_may_be_captured(n, d, dtype):
    """CUDA-core kernels, one tile without a prepare kernel, and with one: the set-up of the
    status word used calls that end a capture."""
    r = run_python(CAPTURE_AT_ONCE % (n, d, dtype))
    assert r.returncode == 0 and "replayed" in r.stdout, (r.returncode, r.stderr[-2000:])

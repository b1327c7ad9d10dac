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


TIME_OUT_THEN_CAPTURE = """
import ctypes as C
import torch
from trifast_b200 import _lib, triangle_attention
q, k, v = (torch.randn(1, 2, 136, 136, 32, device="cuda").bfloat16() for _ in range(3))
b = torch.randn(1, 2, 136, 136, device="cuda").bfloat16()
m = torch.zeros(1, 136, 136, dtype=torch.bool, device="cuda")
good = triangle_attention(q, k, v, b, m)
assert _lib.load().trifast_debug_wait_probe(200, C.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
triangle_attention(q, k, v, b, m)          # its prepare kernel repeats the status on the host word
torch.cuda.synchronize()
try:
    with torch.cuda.graph(torch.cuda.CUDAGraph()):
        triangle_attention(q, k, v, b, m)
    raise SystemExit("the capture went through")
except RuntimeError as e:
    print("in the capture:", str(e).splitlines()[0])
try:
    triangle_attention(q, k, v, b, m)
    raise SystemExit("the time-out was forgotten")
except RuntimeError as e:
    assert "bounded wait" in str(e) and "status cleared" in str(e), e
assert torch.equal(triangle_attention(q, k, v, b, m), good)
print("reported")
"""


@pytest.mark.gpu
def test_a_time_out_met_during_a_capture_is_reported_again_after_it():
    """The status word on the device cannot be read there; clearing the host word all the same let
    the next call return memory that was never written."""
    r = run_python(TIME_OUT_THEN_CAPTURE)
    assert r.returncode == 0 and "reported" in r.stdout, (r.returncode, r.stdout, r.stderr[-2000:])

"""What the native operators (csrc/torch_ops.cpp) say about arguments and overrides they
refuse: an exception that names the offending value, never a crash."""

import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def run_python(code, **env):
    """In a process of its own, so that a crash is a failure of this test alone."""
    return subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True,
                          timeout=300, env=dict(os.environ, **env))


# The CUDA implementation itself, called with host tensors: it checks shapes before anything else.
CALL_CUDA_KERNEL = """
import torch
import trifast_b200.torch
op = torch.ops.trifast_b200.triangle_attention.default
q = torch.zeros(1, 2, 16, 16, 32)
args = dict(q=q, k=q, v=q, b=torch.zeros(1, 2, 16, 16), mask=torch.zeros(1, 16, 16, dtype=torch.bool))
args[%r] = %s
try:
    op.redispatch(torch._C.DispatchKeySet(torch._C.DispatchKey.CUDA), *args.values())
except Exception as e:
    print(type(e).__name__, str(e).splitlines()[0])
"""


@pytest.mark.parametrize("name,value,want", [
    ("b", "torch.zeros(1, 2, 16, 15)", "ValueError bias must be [1, 2, 16, 16]; got [1, 2, 16, 15]"),
    ("mask", "torch.zeros(1, 15, 16, dtype=torch.bool)", "ValueError mask must be [1, 16, 16]; got [1, 15, 16]"),
    ("q", "torch.zeros(16, 16, 32)", "ValueError q must be (batch, heads, rows, n, d); got [16, 16, 32]"),
])
def test_messages_with_numbers(name, value, want):
    """A second C++ runtime in the operator library made these end the process."""
    r = run_python(CALL_CUDA_KERNEL % (name, value))
    assert r.returncode == 0, (r.returncode, r.stderr[-2000:])
    assert r.stdout.strip() == want


def small(dtype="float32"):
    import torch
    q, k, v = (torch.randn(1, 2, 16, 16, 32, device="cuda", dtype=getattr(torch, dtype)) for _ in range(3))
    return q, k, v, torch.zeros(1, 2, 16, 16, device="cuda", dtype=q.dtype), \
        torch.zeros(1, 16, 16, dtype=torch.bool, device="cuda")


@pytest.mark.gpu
@pytest.mark.parametrize("value", ["abc", "1x", "0x1", " "])
def test_flags_override_must_be_a_decimal_integer(monkeypatch, value):
    from trifast_b200 import triangle_attention
    monkeypatch.setenv("TRIFAST_B200_FLAGS", value)
    with pytest.raises(ValueError):
        triangle_attention(*small())
    with pytest.raises(ValueError):       # the same rule in the Python layer
        from trifast_b200 import _lib
        _lib.flags_choice()
    monkeypatch.setenv("TRIFAST_B200_FLAGS", "1")
    assert triangle_attention(*small()).shape == (1, 2, 16, 16, 32)

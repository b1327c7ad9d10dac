"""A bias shared by all heads or all batches, passed as an expanded view (stride 0): no tensor map
can describe it, so the operators hand it over as a strided one and the C ABI keeps it off TMA."""

import pytest
import torch

from tests.helpers import abi_backward, abi_forward
from trifast_b200 import _lib, triangle_attention
from trifast_b200.torch import _prep4

DEV = "cuda"


def test_python_layer_materialises_an_expanded_bias():
    b = torch.randn(1, 1, 16, 16)
    for e in (b.expand(1, 4, 16, 16), b.expand(3, 1, 16, 16)):
        assert _prep4(e).is_contiguous() and torch.equal(_prep4(e), e)
    assert _prep4(b.expand(1, 1, 16, 16)).data_ptr() == b.data_ptr()
    wide = torch.randn(2, 3, 16, 20)[..., :16]
    assert _prep4(wide).data_ptr() == wide.data_ptr()


def _problem(n, d, dtype, over):
    g = torch.Generator(device=DEV).manual_seed(n + d)
    bs, h = 2, 3
    draw = lambda *s: torch.randn(*s, generator=g, device=DEV).to(dtype)
    q, k, v, do = (draw(bs, h, n, n, d) for _ in range(4))
    m = torch.rand(bs, n, n, generator=g, device=DEV) < 0.3
    m[:, n // 2] = True
    small = {"heads": (bs, 1), "batch": (1, h), "both": (1, 1)}[over]
    return q, k, v, draw(*small, n, n).expand(bs, h, n, n), m, do


# one tile (no prepare kernel in the forward), several tiles, head dim 128, CUDA cores, ragged, fp32
SIZES = [(64, 32, torch.bfloat16), (136, 64, torch.float16), (264, 16, torch.bfloat16), (72, 128, torch.bfloat16),
         (40, 32, torch.float16), (65, 32, torch.bfloat16), (48, 32, torch.float32)]


@pytest.mark.gpu
@pytest.mark.parametrize("n,d,dtype", SIZES)
@pytest.mark.parametrize("over", ["heads", "batch", "both"])
def test_operator_takes_an_expanded_bias(n, d, dtype, over):
    """Bit for bit the results of a dense copy: the copies that the kernels read hold the same."""
    q, k, v, b, m, do = _problem(n, d, dtype, over)
    res = []
    for bias in (b, b.contiguous()):
        leaves = [t.detach().requires_grad_(True) for t in (q, k, v, bias)]
        o = triangle_attention(*leaves, m)
        res.append((o.detach(),) + torch.autograd.grad(o, leaves, do))
    for name, x, y in zip(("o", "dq", "dk", "dv", "db"), *res):
        assert torch.equal(x, y), name


@pytest.mark.gpu
@pytest.mark.parametrize("n,d,dtype", SIZES)
def test_c_abi_takes_an_expanded_bias(n, d, dtype):
    """Without TRIFAST_FLAG_STRIDED: the CUDA-core kernels where TMA would have to read it, so
    their results on a dense copy are the same to the bit.  (db may be split into another number
    of row groups: fp32 sums in another order, below n 2^-24 sum|dS| < 2e-4 apart, then rounded.)"""
    q, k, v, b, m, do = _problem(n, d, dtype, "heads")
    packed = n % 8 != 0        # (the workspace holds a padded copy: the usual kernels)
    res = []
    for bias, kernel in ((b, None), (b.contiguous(), None if packed else _lib.KERNEL_SIMT)):
        o, lse = torch.empty_like(q), torch.empty(q.shape[:4], dtype=torch.float32, device=DEV)
        abi_forward(q, k, v, bias, m, o, lse, kernel=kernel)
        grads = [torch.empty_like(q) for _ in range(3)] + [torch.empty(b.shape, dtype=dtype, device=DEV)]
        abi_backward(do, q, k, v, bias, m, o, lse, *grads, kernel=kernel)
        res.append([o, lse] + grads)
    torch.cuda.synchronize()
    for name, x, y in zip(("o", "lse", "dq", "dk", "dv"), *res):
        assert torch.equal(x, y), name
    torch.testing.assert_close(res[0][-1], res[1][-1], rtol=torch.finfo(dtype).eps, atol=2e-4)

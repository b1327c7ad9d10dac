"""Values that are not finite: they reach the results that depend on them and no others."""

import pytest
import torch

from trifast_b200 import triangle_attention

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("n,d,dtype", [
    (40, 32, torch.float32), (72, 128, torch.float32), (48, 64, torch.bfloat16),   # CUDA cores
    (136, 128, torch.bfloat16), (200, 128, torch.float16),                         # head dim 128
])
@pytest.mark.parametrize("what", ["dO nan", "dO inf", "v inf"])
def test_dropped_keys_keep_zero_gradients(n, d, dtype, what):
    """dk and dv of a dropped key are exactly zero whatever the row's other operands hold (0 times
    NaN is not), and the other pair rows stay finite."""
    g = torch.Generator(device=DEV).manual_seed(n)
    h = 2
    q, k, v, do = (torch.randn(1, h, n, n, d, generator=g, device=DEV).to(dtype) for _ in range(4))
    b = torch.randn(1, h, n, n, generator=g, device=DEV).to(dtype)
    m = torch.rand(1, n, n, generator=g, device=DEV) < 0.3
    row = 3
    m[0, row, 7] = False
    if what == "v inf":
        v[0, 0, row, 7, 1] = float("inf")
    else:
        do[0, 0, row, 5, 1] = float(what.split()[1])
    leaves = [t.requires_grad_(True) for t in (q, k, v, b)]
    o = triangle_attention(*leaves, m)
    dq, dk, dv, _ = torch.autograd.grad(o, leaves, do)
    dropped = (m & ~m.all(-1, keepdim=True))[:, None, :, :, None].expand_as(k)
    assert dropped[:, :, row].any()
    assert not dk[dropped].any() and not dv[dropped].any()     # (NaN counts as true)
    assert not torch.isfinite(dk[0, 0, row]).all()              # open keys: as the mathematics has it
    if what == "dO inf":   # P times infinity is one, unless P has no second 16-bit part (below 2^-12 of them)
        assert torch.isinf(dv[0, 0, row, :, 1][~m[0, row]]).float().mean() > 0.95
    others = [i for i in range(n) if i != row]
    assert all(torch.isfinite(t[:, :, others]).all() for t in (dq, dk, dv))

"""The forward at head dims up to 64 where its walk changes: key steps of 64 and their remainders, pair
rows in groups of four with a group cut short, a last round of half items, rows without a dropped key
beside rows with some and rows without an open one (finished by the prepare kernel, or inside the
kernel where none runs), masks as bytes and as packed words."""

import pytest
import torch

from tests.helpers import abi_forward

pytestmark = pytest.mark.gpu
DEV = "cuda"

SHAPES = [  # n, heads, rows, d, dtype
    (64, 3, 64, 32, torch.bfloat16),      # one step; 48 items, all halves
    (72, 2, 5, 16, torch.float16),        # a step and a remainder, no prepare kernel
    (128, 5, 128, 64, torch.bfloat16),    # 160 items: a round of whole ones, then 24 halves
    (129, 1, 3, 32, torch.float16),       # two query tiles, a last key step of one key
    (136, 2, 7, 64, torch.float16),
    (200, 4, 150, 32, torch.bfloat16),    # 304 items: two rounds and halves
    (257, 1, 21, 16, torch.bfloat16),
    (520, 1, 6, 32, torch.bfloat16),
    (1100, 1, 2, 64, torch.float16),      # the second half of the one group is beyond the rows
    (136, 20, 9, 64, torch.float16),      # few rows, many heads: a block for each in rows without an open key
    (200, 33, 130, 32, torch.bfloat16),   # four blocks with eight or nine heads
    (136, 70, 136, 64, torch.float16),    # more than 1024 columns a block: several passes
]


def _mask(n, rows, g):
    m = torch.rand(1, rows, n, generator=g) < 0.2
    kind = torch.arange(rows) % 7
    m[0, kind == 1] = False                         # nothing dropped
    m[0, kind == 3] = True                          # nothing open
    m[0, kind == 4, : min(n - 1, 70)] = True        # the first step(s) without an open key
    m[0, kind == 5, 1:] = True                      # one open key
    if rows >= 16:
        m[0, 8:12] = True                           # a whole group
    return m


def _ranges(n, rows, g):
    """Rows of a group that walk different key tiles: one tile each, all but the first or the last
    ones, every tile, none."""
    tile, m = torch.arange(n) // 128, torch.rand(1, rows, n, generator=g) < 0.1
    for i in range(rows):
        kind, at = (i + i // 4) % 6, i % int(tile[-1] + 1)
        m[0, i] |= [tile != at, tile < at, tile > at, tile < 0, tile >= 0, tile != 0][kind]
        if kind != 4 and i % 3 == 0:
            m[0, i] = ~(~m[0, i] | (torch.arange(n) == n - 1))      # and the last key
    return m


@pytest.mark.parametrize("n,h,rows,d,dtype", SHAPES)
def test_forward_and_lse_against_float64(n, h, rows, d, dtype):
    _check(n, h, rows, d, dtype, _mask)


@pytest.mark.parametrize("n,h,rows,d,dtype", [
    (257, 2, 50, 32, torch.bfloat16),
    (384, 2, 13, 64, torch.float16),
    (640, 3, 65, 32, torch.float16),
    (700, 1, 30, 64, torch.bfloat16),
    (520, 2, 26, 16, torch.bfloat16),
])
def test_rows_of_a_group_with_different_steps(n, h, rows, d, dtype):
    _check(n, h, rows, d, dtype, _ranges)


def _check(n, h, rows, d, dtype, make_mask):
    g = torch.Generator().manual_seed(n + d)
    q, k, v = (torch.randn(1, h, rows, n, d, generator=g).to(dtype).to(DEV) for _ in range(3))
    bias = torch.randn(1, h, n, n, generator=g).to(dtype).to(DEV)
    mask = make_mask(n, rows, g).to(DEV)
    o = torch.full_like(q, float("nan"))
    lse = torch.full(q.shape[:4], float("nan"), device=DEV)
    abi_forward(q, k, v, bias, mask, o, lse)
    again, lse2 = torch.empty_like(o), torch.empty_like(lse)
    abi_forward(q, k, v, bias, mask, again, lse2)
    assert torch.equal(o, again) and torch.equal(lse, lse2)

    s = torch.einsum("bhijd,bhikd->bhijk", q.double(), k.double()) * d ** -0.5 + bias.double()[:, :, None]
    s = s.masked_fill(mask[:, None, :, None], float("-inf"))
    full = mask.all(-1)[0]
    s[:, :, full] = 0.0
    ref = torch.einsum("bhijk,bhikd->bhijd", s.softmax(-1), v.double())
    # weights and outputs rounded to the type, 2^-9 (2^-12) at most each; four times that
    unit = 2.0 ** -9 if dtype == torch.bfloat16 else 2.0 ** -12
    for i in range(rows):
        err, size = (o[0, :, i].double() - ref[0, :, i]).norm(), ref[0, :, i].norm()
        assert float(err) <= 4 * unit * float(size), f"row {i}"
    want = s.logsumexp(-1)[:, :, ~full]
    assert float((lse[:, :, ~full].double() - want).abs().max()) < 1e-4      # fp32 scores of size 10
    assert bool((lse[:, :, full] == torch.finfo(dtype).min).all())

"""The one-pass dq / dk / dv kernel where its walk changes: steps per key tile odd and even, one
step per tile, the row lengths at which a TMEM buffer goes (dQ takes its columns) and at which a
row is split into query chunks, with several rows per CTA and, in the second test, rows of one CTA
that walk different key tiles."""

import pytest
import torch

from tests.test_backward_gpu import NAMES, _inputs, _run_abi
from trifast_b200 import _lib

pytestmark = pytest.mark.gpu

SHAPES = [  # n, heads, d, dtype, rows; buffers of S, dP, (dK, dV); chunks
    (64, 5, 32, torch.bfloat16, 64),      # one step per key tile
    (129, 4, 32, torch.float16, 90),      # three steps, the last key tile with one key
    (256, 2, 32, torch.bfloat16, 160),    # 3, 2, 2
    (257, 2, 32, torch.bfloat16, 90),     # 3, 2, 1
    (512, 1, 32, torch.float16, 160),
    (513, 1, 32, torch.bfloat16, 150),    # 3, 1, 1
    (768, 1, 16, torch.bfloat16, 20),
    (769, 1, 32, torch.bfloat16, 150),    # 2, 1, 1
    (1100, 1, 32, torch.float16, 12),     # chunks of five and four query tiles: 3, 1, 1
    (2000, 1, 32, torch.bfloat16, 5),     # chunks of eight: 2, 1, 1
    (128, 4, 64, torch.float16, 90),      # 2, 2, 1
    (257, 1, 64, torch.bfloat16, 150),    # 2, 1, 1
    (385, 1, 64, torch.bfloat16, 40),     # two chunks of two: 2, 2, 1
    (900, 1, 64, torch.float16, 8),       # three chunks, the last one short
]


@pytest.mark.parametrize("n,h,d,dtype,rows", SHAPES)
def test_every_walk_gives_the_two_kernel_results(n, h, d, dtype, rows):
    args = _inputs(n, h, d, dtype, "random", rows, seed=n)
    one = _run_abi(args)
    for x, y in zip(one, _run_abi(args)):
        assert torch.equal(x, y)
    # head dim 16 has no two-kernel backward: the CUDA-core kernels, whose P and dS stay in fp32
    two = _run_abi(args, kernel=_lib.KERNEL_SIMT) if d == 16 else _run_abi(args, flags=_lib.FLAG_SPLIT_BWD)
    chunks = _lib.pick_plan(1, h, n, rows, d, dtype)["bwd_chunks"]
    for name, x, y in zip(NAMES, one, two):
        x, y = x.float(), y.float()
        assert not torch.isnan(x).any(), name
        if d == 16:
            # P and dS rounded to 8 bits: 2^-9 each, uncorrelated over the sums; four times that
            assert float((x - y).norm()) <= 4 * 2.0 ** -9 * float(y.norm()), name
        elif chunks > 1 and name in ("dk", "dv"):
            # summed per chunk, the fp32 partials added: last places of a few elements
            assert float((x - y).abs().max()) <= 2.0 ** -7 * float(y.abs().max()), name
            assert float((x != y).float().mean()) < 0.02, name
        else:
            assert torch.equal(x, y), name


def _ranges(n, rows):
    """Rows next to each other that walk different key tiles."""
    keys, m = torch.arange(n), torch.zeros(1, rows, n, dtype=torch.bool)
    for i in range(rows):
        kind = i % 7
        if kind == 0:
            m[0, i] = keys < n // 3 + i % 90                    # head dropped
        elif kind == 1:
            m[0, i] = keys >= n // 2 - i % 90                   # tail dropped
        elif kind == 2:
            m[0, i] = keys // 128 != (i // 7) % ((n + 127) // 128)   # a single tile
        elif kind == 3:
            m[0, i] = keys != 77 * i % n                        # a single key
        elif kind == 4:
            m[0, i] = True                                      # all dropped: every tile
        elif kind == 5:
            m[0, i] = keys % 256 < 130                          # every other tile, within the range
    return m


@pytest.mark.parametrize("n,h,d,dtype,rows", [   # at least 400 items: two or three rows per CTA
    (257, 4, 32, torch.bfloat16, 110),    # 3, 2, 1
    (800, 4, 32, torch.bfloat16, 110),    # 2, 1, 1
    (1024, 4, 16, torch.float16, 110),
    (1100, 4, 32, torch.float16, 101),    # chunks of five and four: 3, 1, 1
    (2000, 4, 32, torch.bfloat16, 101),   # chunks of eight: 2, 1, 1
    (257, 4, 64, torch.float16, 110),     # 2, 1, 1
    (385, 4, 64, torch.bfloat16, 110),    # chunks of two: 2, 2, 1
    (700, 4, 64, torch.bfloat16, 110),    # chunks of three: 2, 1, 1
])
def test_rows_of_a_cta_with_different_ranges(n, h, d, dtype, rows):
    q, k, v, b, _, do = _inputs(n, h, d, dtype, "none", rows, seed=n)
    m = _ranges(n, rows)
    args = (q, k, v, b, m, do)
    one = _run_abi(args)
    for x, y in zip(one, _run_abi(args)):
        assert torch.equal(x, y)
    dropped = (m & ~m.all(-1, keepdim=True))[:, None, :, :, None].to(one[2].device).expand_as(one[2])
    assert not bool(one[2][dropped].any()) and not bool(one[3][dropped].any())
    two = _run_abi(args, kernel=_lib.KERNEL_SIMT) if d == 16 else _run_abi(args, flags=_lib.FLAG_SPLIT_BWD)
    chunks = _lib.pick_plan(1, h, n, rows, d, dtype)["bwd_chunks"]
    for name, x, y in zip(NAMES, one, two):
        x, y = x.float(), y.float()
        assert not torch.isnan(x).any(), name
        if d == 16:   # (as above, with the 11 bits of fp16)
            assert float((x - y).norm()) <= 4 * 2.0 ** -12 * float(y.norm()), name
        elif chunks > 1 and name in ("dk", "dv"):   # (as above)
            assert float((x - y).abs().max()) <= 2.0 ** -7 * float(y.abs().max()), name
            assert float((x != y).float().mean()) < 0.02, name
        else:
            assert torch.equal(x, y), name

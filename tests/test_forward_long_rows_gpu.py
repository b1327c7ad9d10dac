"""The tensor-core forward on long rows: key steps beyond 12 bits, and rows longer than a shared-memory
copy of their key masks would allow, with the masks read as bytes and as packed words."""

import pytest
import torch

from tests.helpers import abi_forward
from trifast_b200 import _lib

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _check(n, rows, d, dtype, bias, queries):
    """Against float64 at some queries; everything else written and finite."""
    g = torch.Generator(device=DEV).manual_seed(n + d)
    q, k, v = (torch.randn(1, 1, rows, n, d, generator=g, device=DEV).to(dtype) for _ in range(3))
    for j in queries:
        bias[0, 0, j] = torch.randn(n, generator=g, device=DEV).to(dtype)
    mask = torch.rand(1, rows, n, generator=g, device=DEV) < 0.1
    if rows > 1:
        mask[0, 1, : n // 2] = True      # the row's first key tiles hold no open key
    o = torch.full_like(q, float("nan"))
    lse = torch.full(q.shape[:4], float("nan"), device=DEV)
    # (the family asked for by name: refused instead of run on the CUDA cores)
    abi_forward(q, k, v, bias, mask, o, lse, kernel=_lib.KERNEL_TCGEN05)
    assert bool(o.isfinite().all()) and bool(lse.isfinite().all())

    unit = 2.0 ** -9 if dtype == torch.bfloat16 else 2.0 ** -12
    for i in range(rows):
        s = q[0, 0, i, queries].double() @ k[0, 0, i].double().T * d ** -0.5 + bias[0, 0, queries].double()
        s = s.masked_fill(mask[0, i], float("-inf"))
        ref = s.softmax(-1) @ v[0, 0, i].double()
        # weights and outputs rounded to the type, at most a unit each; four times that
        assert float((o[0, 0, i, queries].double() - ref).norm()) <= 4 * unit * float(ref.norm()), f"row {i}"
        # scores of size 10 in fp32, n weights added in fp32: n / 4 terms to a partial sum at most
        assert float((lse[0, 0, i, queries].double() - s.logsumexp(-1)).abs().max()) < 1e-4 + n / 4 * 2.0 ** -24


@pytest.mark.parametrize("n,rows,d,dtype", [
    (6016, 5, 64, torch.float16),
    (6001, 3, 64, torch.bfloat16),
    (12296, 2, 32, torch.bfloat16),
])
def test_rows_of_thousands_of_keys(n, rows, d, dtype):
    bias = torch.zeros(1, 1, n, n, dtype=dtype, device=DEV)
    _check(n, rows, d, dtype, bias, [0, 1, 127, 128, n // 2, n - 1])


def test_key_steps_beyond_twelve_bits():
    """262,208 keys are 4097 steps of 64; the bias map takes 128 GiB."""
    n = 262208
    torch.cuda.empty_cache()
    if torch.cuda.mem_get_info()[0] < 2 * n * n + (4 << 30):
        pytest.skip("needs 142 GB of free device memory")
    bias = torch.empty(1, 1, n, n, dtype=torch.bfloat16, device=DEV).zero_()
    try:
        _check(n, 1, 16, torch.bfloat16, bias, [0, 12345, n // 2, n - 1])
    finally:
        del bias
        torch.cuda.empty_cache()

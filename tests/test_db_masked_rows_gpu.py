"""db in fp32, as trifast_backward_db returns it, over many rows without an open key."""

import ctypes as C
import math

import pytest
import torch

from tests.helpers import abi_forward
from trifast_b200 import _lib

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("n,h,d,dtype,share", [
    (512, 2, 32, torch.bfloat16, 1.0),
    (512, 2, 64, torch.float16, 0.9),
    (1024, 1, 16, torch.float16, 1.0),
    (200, 3, 32, torch.float16, 0.6),
    (97, 2, 16, torch.bfloat16, 0.3),
])
def test_sums_over_masked_rows_keep_fp32(n, h, d, dtype, share):
    g = torch.Generator(device=DEV).manual_seed(n + d)
    q, k, v, do = (torch.randn(1, h, n, n, d, generator=g, device=DEV).to(dtype) for _ in range(4))
    v = v + 2            # dP and delta of a row are much of a size
    bias = torch.randn(1, h, n, n, generator=g, device=DEV).to(dtype)
    full = torch.rand(n, generator=g, device=DEV) < share
    mask = full[None, :, None].expand(1, n, n).contiguous()
    o, lse = torch.empty_like(q), torch.empty(1, h, n, n, device=DEV)
    abi_forward(q, k, v, bias, mask, o, lse)

    lib, shape = _lib.load(), _lib.make_shape(1, h, n, n, d, dtype)
    size = lib.trifast_backward_workspace_bytes(C.byref(shape))
    ws = torch.empty(size, dtype=torch.uint8, device=DEV)
    db = torch.full((1, h, n, n), float("nan"), device=DEV)
    _lib.check(lib.trifast_backward_db(
        C.byref(shape), C.byref(_lib.t5(do)), C.byref(_lib.t5(q)), C.byref(_lib.t5(k)), C.byref(_lib.t5(v)),
        C.byref(_lib.t4(bias)), C.byref(_lib.mask_view(mask.view(torch.uint8))), C.byref(_lib.t5(o)),
        C.c_void_p(lse.data_ptr()), C.c_void_p(db.data_ptr()), C.c_void_p(ws.data_ptr()), C.c_size_t(size),
        C.c_void_p(torch.cuda.current_stream().cuda_stream)), "trifast_backward_db")

    ref = torch.zeros(h, n, n, dtype=torch.float64, device=DEV)
    for i in range(n):
        gi, vi = do[0, :, i].double(), v[0, :, i].double()
        if bool(full[i]):
            p = torch.full((h, n, n), 1 / n, dtype=torch.float64, device=DEV)
        else:
            p = (q[0, :, i].double() @ k[0, :, i].double().mT * d ** -0.5 + bias[0].double()).softmax(-1)
        # (the delta that the stored o gives is what the kernel is asked for)
        ref += p * (gi @ vi.mT - (gi * o[0, :, i].double()).sum(-1, keepdim=True))
    # a split's rows added one after the other: 2^-24 at most each, uncorrelated; the other rows'
    # weights by way of scores of size 10 in fp32: 10 * 2^-24
    rows = n / lib.trifast_backward_db_partials(C.byref(shape))
    assert float((db[0].double() - ref).norm() / ref.norm()) < (math.sqrt(rows) + 10) * 2.0 ** -24

"""Head dim 128, backward on the tensor cores: weights and score gradients enter the products as
two 16-bit parts each, so dq, dk and dv carry the rounding of the result and no more."""

import pytest
import torch

from tests.helpers import abi_backward, abi_forward
from trifast_b200 import _lib

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("n,dtype,mask,do_scale,bias_std", [
    (64, torch.bfloat16, "none", 1.0, 1.0),        # one step
    (200, torch.bfloat16, "random", 1.0, 1.0),     # ragged steps and tiles
    (520, torch.bfloat16, "padding", 1e-6, 1.0),
    (200, torch.float16, "random", 1.0, 1.0),
    (333, torch.float16, "padding", 1.0, 1.0),     # padded bias copy
    (264, torch.float16, "none", 2e-3, 1.0),       # dS among the subnormals of fp16
    (264, torch.float16, "random", 4e3, 3.0),      # dS beyond the range of fp16
    (136, torch.float16, "outlier", 1.0, 1.0),     # a dropped key's large values do not count
])
def test_gradients_as_precise_as_fp32_products(n, dtype, mask, do_scale, bias_std):
    """Against the CUDA-core kernels (fp32 throughout).  If the values before the last rounding are
    a relative `e` apart, about e / u of the results (u: one unit in the last place) round to
    a neighbour, so the 2-norms differ by sqrt(e / u) u.  The split leaves e < 2^-16 (bf16) and
    2^-18 (fp16): 2.4e-4 and 4.3e-5, an eighth of u allowed.  P and dS in one 16-bit part each
    give 1.7e-3 and 2.1e-4."""
    g = torch.Generator(device=DEV).manual_seed(n)
    h, d = 2, 128
    rows = n if n < 300 else 40
    draw = lambda *s: torch.randn(*s, generator=g, device=DEV)
    q, k, v = (draw(1, h, rows, n, d).to(dtype) for _ in range(3))
    do = (draw(1, h, rows, n, d) * do_scale).to(dtype)
    b = (draw(1, h, n, n) * bias_std).to(dtype)
    m = torch.zeros(1, rows, n, dtype=torch.bool, device=DEV)
    if mask == "random":
        m = torch.rand(1, rows, n, generator=g, device=DEV) < 0.2
        m[0, 1] = True
    elif mask == "padding":
        m[:, :, n * 8 // 10:] = True
        m[:, rows - 3:] = True
    elif mask == "outlier":
        m[:, :, 5] = True
        v[:, :, :, 5] = 6e4
    o, lse = torch.empty_like(q), torch.empty(q.shape[:4], dtype=torch.float32, device=DEV)
    abi_forward(q, k, v, b, m, o, lse)

    def grads(kernel):
        out = [torch.empty_like(q) for _ in range(3)] + [torch.empty_like(b)]
        abi_backward(do, q, k, v, b, m, o, lse, *out, kernel=kernel)
        return [t.double() for t in out]

    u = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}[dtype]
    for name, x, y in zip(("dq", "dk", "dv", "db"), grads(None), grads(_lib.KERNEL_SIMT)):
        held = torch.isfinite(y)      # (db of the largest dO leaves fp16's own range here and there)
        assert torch.equal(torch.isfinite(x), held) and (held.all() or name == "db"), name
        err = float((x - y)[held].norm() / y[held].norm())
        assert err <= u / 8, f"{name}: {err:.2e}"


def test_separate_calls_equal_the_whole_backward():
    """trifast_backward_db, then trifast_backward_dqkv (the row-sharded order): the scales that the
    first leaves in the workspace serve the second."""
    from trifast_b200.dist import CudaKernels
    g = torch.Generator(device=DEV).manual_seed(0)
    q, k, v, do = (torch.randn(1, 2, 40, 136, 128, generator=g, device=DEV).half() for _ in range(4))
    b = torch.randn(1, 2, 136, 136, generator=g, device=DEV).half()
    m = torch.rand(1, 40, 136, generator=g, device=DEV) < 0.2
    do[0, 0, 3] *= 1e-4
    kern = CudaKernels()
    o, lse = kern.forward(q, k, v, b, m)
    db32, ws = kern.backward_db(do, q, k, v, b, m, o, lse)
    got = kern.backward_dqkv(do, q, k, v, b, m, lse, ws) + (kern.db_finalize(db32, b.dtype),)
    want = [torch.empty_like(q) for _ in range(3)] + [torch.empty_like(b)]
    abi_backward(do, q, k, v, b, m, o, lse, *want)
    for name, x, y in zip(("dq", "dk", "dv", "db"), got, want):
        assert torch.equal(x, y), name


def test_static_scratch_and_graph_replay_with_row_scales():
    """fp16: the scales share the scratch with db, and follow the values of a replay."""
    import ctypes as C
    lib = _lib.load()
    g = torch.Generator(device=DEV).manual_seed(1)
    q, k, v, do = (torch.randn(1, 2, 104, 104, 128, generator=g, device=DEV).half() for _ in range(4))
    b = torch.randn(1, 2, 104, 104, generator=g, device=DEV).half()
    m = torch.rand(1, 104, 104, generator=g, device=DEV) < 0.2
    o, lse = torch.empty_like(q), torch.empty(q.shape[:4], dtype=torch.float32, device=DEV)
    abi_forward(q, k, v, b, m, o, lse)

    def step(static):
        out = [torch.full_like(q, float("nan")) for _ in range(3)] + [torch.full_like(b, float("nan"))]
        if not static:
            abi_backward(do, q, k, v, b, m, o, lse, *out)
            return out
        t5 = lambda t: C.byref(_lib.t5(t))
        rc = lib.trifast_backward_static_scratch(
            C.byref(_lib.make_shape(1, 2, 104, 104, 128, q.dtype)), t5(do), t5(q), t5(k), t5(v), C.byref(_lib.t4(b)),
            C.byref(_lib.mask_view(m.view(torch.uint8))), t5(o), C.c_void_p(lse.data_ptr()), t5(out[0]), t5(out[1]),
            t5(out[2]), C.byref(_lib.t4(out[3])), C.c_void_p(torch.cuda.current_stream().cuda_stream))
        _lib.check(rc, "trifast_backward_static_scratch")
        return out

    for scale in (1.0, 1e-3):
        do.mul_(scale)
        for x, y in zip(step(True), step(False)):
            assert torch.equal(x, y)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        step(False)
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        captured = step(False)
    do.mul_(3e3)
    graph.replay()
    for x, y in zip(captured, step(False)):
        assert torch.isfinite(x).all() and torch.equal(x, y)

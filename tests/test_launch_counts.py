"""The launches that ``bench.py`` and the host-resident pipeline report are those that run."""

import ctypes as C

import pytest
import torch

from trifast_b200 import _lib


@pytest.mark.parametrize("n,h,d,dtype,partials", [
    (1024, 4, 32, torch.bfloat16, 4),      # 256 tiles in 7 rounds of 256 rows, not 2 of 1024
    (733, 4, 32, torch.bfloat16, 1),
    (384, 4, 32, torch.bfloat16, 4),       # 36 tiles x 4 row groups: one round
    (256, 4, 128, torch.bfloat16, 1),      # row groups summed in a cluster
    (32, 4, 32, torch.float32, 16),        # CUDA cores: what the plan says
])
def test_db_partials_that_run(n, h, d, dtype, partials):
    shp = _lib.make_shape(1, h, n, n, d, dtype)
    got = _lib.load().trifast_backward_db_partials(C.byref(shp))
    assert got == partials <= max(1, _lib.pick_plan(1, h, n, n, d, dtype)["db_row_splits"])


def test_db_partials_of_an_invalid_shape():
    bad = _lib.Shape(1, 4, 64, 64, 48, 1, 0, 0)
    assert _lib.load().trifast_backward_db_partials(C.byref(bad)) == -3


@pytest.mark.gpu
@pytest.mark.parametrize("n,d,dtype", [(136, 32, torch.bfloat16), (264, 64, torch.float16), (733, 32, torch.bfloat16),
                                       (200, 128, torch.float16), (48, 32, torch.bfloat16), (72, 16, torch.float32)])
def test_host_pipeline_counts_its_launches(n, d, dtype):
    """Against the kernels that the profiler saw, the library's alone."""
    from trifast_b200.host import HostPipeline
    rows = min(n, 72)
    draw = lambda *s: torch.randn(*s).to(dtype).pin_memory()
    q, k, v, do = (draw(1, 2, rows, n, d) for _ in range(4))
    b, m = draw(1, 2, n, n), torch.zeros(1, rows, n, dtype=torch.bool).pin_memory()
    pipe = HostPipeline(1, 2, n, d, dtype, torch.device("cuda", 0), rows=rows, chunk_rows=32)
    pipe.run(q, k, v, b, m, do=do)
    torch.cuda.synchronize()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        pipe.run(q, k, v, b, m, do=do)
        torch.cuda.synchronize()
    ours = sum(e.count for e in prof.key_averages() if "trifast::" in e.key)
    assert ours == pipe.kernel_launches

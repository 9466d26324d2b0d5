"""Device memory that FP32 runs keep for their coherence records."""
import numpy as np
import pytest

from fringe_gb300 import synth
from tests.parity import assert_parity, compare

pytestmark = pytest.mark.gpu


def test_records_kept_by_a_context(gpu_lib):
    """FP32 runs keep 4 GiB of records at most, however large the frame."""
    torch = pytest.importorskip("torch")
    from fringe_gb300 import _lib, phase_link
    n, rows, cols = 64, 1024, 1024
    stack = torch.ones((n, rows, cols), dtype=torch.complex64, device="cuda")
    nmap = torch.zeros((rows, cols, 8), dtype=torch.int32, device="cuda")      # every pixel is skipped
    out = {"phase": torch.zeros_like(stack), "tcorr": torch.zeros((rows, cols), device="cuda"),
           "comp": torch.zeros((rows, cols), dtype=torch.complex64, device="cuda")}
    ctx = _lib.Context(0)
    phase_link(stack[:, :8, :8].contiguous(), nmap[:8, :8].contiguous(), (5, 10), ctx=ctx)   # modules loaded
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    before = torch.cuda.mem_get_info()[0]
    phase_link(stack, nmap, (5, 10), ctx=ctx, out=out)
    torch.cuda.synchronize()
    assert before - torch.cuda.mem_get_info()[0] < 4.4e9
    ctx.set_record_limit(0)                           # releases them
    assert before - torch.cuda.mem_get_info()[0] < 1e8
    phase_link(stack, nmap, (5, 10), ctx=ctx, out=out)
    torch.cuda.synchronize()
    assert before - torch.cuda.mem_get_info()[0] < 1e8
    ctx.close()


@pytest.mark.parametrize("rows", [None, (5, 71)])
@pytest.mark.parametrize("precision", ["fp32", "mixed"])
def test_results_under_a_limit(gpu_lib, rows, precision):
    """Chunks of any number of rows give the same bits; a limit that does not
    hold a row of tiles gives the plain kernel's, and does not bind mixed runs."""
    from fringe_gb300 import _lib, phase_link
    stack, nmap = synth.scene("voronoi", 77, 83, 20, 3, 5, seed=20)
    ctx = _lib.Context(0)
    row = 83 * (4 * 8 * 55 + 8)                       # 55 blocks of 8 floats a pixel
    want = phase_link(stack, nmap, (3, 5), precision=precision, rows=rows, ctx=ctx)
    for limit in (-1, 1 << 40, 30 * row, 16 * row, 8 * row, 8 * row - 1, 0):
        ctx.set_record_limit(limit)
        got = phase_link(stack, nmap, (3, 5), precision=precision, rows=rows, ctx=ctx)
        same = all(np.array_equal(got[k], want[k], equal_nan=True) for k in want)
        assert same == (precision == "mixed" or limit < 0 or limit >= 8 * row), limit
        m = compare(got, want)
        assert m["valid_both"] > 4000, m
        assert_parity(m)
    ctx.close()

"""Out-of-range samples at the end of a Gamma tile's sample list: the last union
row of every 8 x 16 pixel tile holds a NaN, tile counts beyond the SMs, chunk
counts odd and even, shallow stacks (short chunks).  A pixel whose window holds
one must get the FP64 form's code, every time."""
import numpy as np
import pytest

from fringe_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [4, 7, 10])
@pytest.mark.parametrize("ny,nx", [(4, 4), (2, 4), (1, 8)])       # 12, 9 and 10 chunks of 32 samples
@pytest.mark.parametrize("precision", ["mixed", "fp32"])
def test_last_samples_of_a_tile(gpu_lib, n, ny, nx, precision):
    from fringe_gb300 import _lib, phase_link
    rows, cols = 250, 213
    stack, nmap = synth.scene("voronoi", rows, cols, n, ny, nx, seed=n)
    rng = np.random.default_rng(n)
    for r0 in range(0, rows, 8):
        for c0 in range(0, cols, 16):
            if r0 + 7 + ny < rows and rng.random() < 0.5:
                stack[rng.integers(n), r0 + 7 + ny, min(cols - 1, c0 + rng.integers(16))] = np.nan
    ctx = _lib.Context(0)
    ctx.set_tuning(force_fp64=True)
    ref = phase_link(stack, nmap, (ny, nx), ctx=ctx, want_status=True)
    assert 1000 < (ref["status"] == -1).sum() < rows * cols // 2
    ctx.set_tuning(force_fp64=False)
    for _ in range(5):
        got = phase_link(stack, nmap, (ny, nx), precision=precision, ctx=ctx, want_status=True)
        assert np.array_equal(got["status"], ref["status"])
        assert np.array_equal(got["tcorr"][ref["status"] < 0], ref["tcorr"][ref["status"] < 0])
    ctx.close()

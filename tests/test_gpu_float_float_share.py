"""The float-float form settles the pixels that FP32 leaves open: of the listed
pixels it hands few on to FP64, and their outputs are no longer FP32's."""
import numpy as np
import pytest

from fringe_gb300 import synth
from tests.test_gpu_float_float import _both

pytestmark = pytest.mark.gpu


def _stats(stack, nmap, ny, nx, **kw):
    from fringe_gb300 import _lib, phase_link
    ctx = _lib.Context(0)
    ctx.set_tuning(amb_scale=1.0 / (stack.shape[0] * 2.0 ** -23))      # nearly every pixel is listed
    phase_link(stack, nmap, (ny, nx), ctx=ctx, **kw)
    s = ctx.stats()
    ctx.close()
    return s


@pytest.mark.parametrize("n", [2, 7, 16, 17, 30, 32, 33, 45, 64])
@pytest.mark.parametrize("precision", ["mixed", "fp32"])
def test_listed_pixels_are_settled_in_float_float(gpu_lib, n, precision):
    stack, nmap = synth.scene("illcond", 13, 17, n, 5, 7, seed=400 + n)
    s = _stats(stack, nmap, 5, 7, method="MLE", precision=precision)
    assert s["fp64_pixels"] > 60
    assert s["mixed_fp64_inverse"] <= s["fp64_pixels"] // 10, s
    _, got, plain, listed = _both(stack, nmap, 5, 7, method="MLE", precision=precision)
    moved = (got["phase"] != plain["phase"]).any(axis=0) | (got["tcorr"] != plain["tcorr"])
    assert moved.sum() >= (1 if n == 2 else listed // 2), (int(moved.sum()), listed)


@pytest.mark.parametrize("exp,beyond", [(-50, True), (-45, True), (-34, False), (40, False), (48, True)])
def test_amplitudes_beyond_its_range_go_to_fp64(gpu_lib, exp, beyond):
    """A window's power is 2^(2 exp) times 1e2 to 1e4; float-float takes 1e-20 to 1e30."""
    stack, nmap = synth.scene("voronoi", 13, 17, 12, 5, 7, seed=77)
    stack = (stack * np.float32(2.0) ** np.float32(exp)).astype(np.complex64)
    s = _stats(stack, nmap, 5, 7, method="MLE", precision="mixed")
    assert s["fp64_pixels"] > 60 and s["mixed_fp64_inverse"] == (s["fp64_pixels"] if beyond else 0), s

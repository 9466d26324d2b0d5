"""The float-float settling of undecided pixels against FP64 for every pixel.  A
wide FP32 band sends most pixels to the list; float-float's own band (2^-46 for
2^-23) stays narrow.  A listed pixel is known by an output that differs from the one the
usual band gives: FP32's own results do not depend on the band."""
import numpy as np
import pytest

from fringe_gb300 import synth

pytestmark = pytest.mark.gpu

# Both forms round the same number to FP32 once it is accurate to well under an ulp: a
# component then differs by at most one ulp (6e-8), the angle of a unit phasor by
# sqrt(2) of it; two ulps leave room for the FP32 phase reference both go through.
PHASE_TOL, TCORR_TOL = 4 * 6e-8, 2 * 6e-8


def _both(stack, nmap, ny, nx, **kw):
    from fringe_gb300 import _lib, phase_link
    out = []
    # a band of |C|_F, which no eigenvalue of C exceeds
    wide = 1.0 / (stack.shape[0] * 2.0 ** -23)
    for tuning in ({"force_fp64": True}, {"amb_scale": wide}, {}):
        ctx = _lib.Context(0)
        ctx.set_tuning(**tuning)
        out.append(phase_link(stack, nmap, (ny, nx), ctx=ctx, want_status=True, **kw))
        if "amb_scale" in tuning:
            listed = ctx.stats()["fp64_pixels"]
        ctx.close()
    return *out, listed


def _compare(ref, got, plain):
    assert np.array_equal(ref["status"], got["status"])
    ok = ref["tcorr"] > 0
    assert np.array_equal(ok, got["tcorr"] > 0)
    assert np.array_equal(ref["tcorr"][~ok], got["tcorr"][~ok])
    moved = ok & ((got["phase"] != plain["phase"]).any(axis=0) | (got["tcorr"] != plain["tcorr"]))
    d = np.abs(np.angle(ref["phase"].astype(np.complex128) * np.conj(got["phase"].astype(np.complex128))))[:, moved]
    assert d.max(initial=0.0) <= PHASE_TOL
    assert np.abs(ref["tcorr"] - got["tcorr"])[moved].max(initial=0.0) <= TCORR_TOL
    return int(ok.sum())


@pytest.mark.parametrize("n", [2, 7, 16, 17, 30, 32, 33, 45, 64])
@pytest.mark.parametrize("precision", ["mixed", "fp32"])
def test_settled_pixels(gpu_lib, n, precision):
    stack, nmap = synth.scene("illcond", 13, 17, n, 5, 7, seed=400 + n)
    ref, got, plain, listed = _both(stack, nmap, 5, 7, method="MLE", precision=precision)
    assert _compare(ref, got, plain) > 60
    assert listed > 60


@pytest.mark.parametrize("exp", [-50, -34, 40])
def test_amplitudes_beyond_its_range(gpu_lib, exp):
    """Powers under 1e-20 and over 1e30, whose low parts FP32 cannot hold, go on to FP64."""
    stack, nmap = synth.scene("voronoi", 13, 17, 12, 5, 7, seed=77)
    stack = (stack * np.float32(2.0) ** np.float32(exp)).astype(np.complex64)
    ref, got, plain, listed = _both(stack, nmap, 5, 7, method="MLE", precision="mixed")
    assert _compare(ref, got, plain) > 60
    assert listed > 60

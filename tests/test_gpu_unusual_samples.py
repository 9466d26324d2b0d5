"""Samples that are not finite, or lie outside the range of the bf16 parts, do
not take their pixels to the FP64 list where FP32 settles them: a window with a non-finite
sample has a known outcome, and the FP32 form solves windows of very small or large
samples in FP32."""
import numpy as np
import pytest

import oracle
from fringe_gb300 import synth
from tests.parity import assert_parity, compare

pytestmark = pytest.mark.gpu

RUNS = [dict(method="MLE"), dict(method="EVD"), dict(method="MLE", semantics="phase_link"),
        dict(method="STBAS", band_width=1), dict(method="STBAS", band_width=4)]


def _listed(stack, nmap, half, **kw):
    from fringe_gb300 import _lib, phase_link
    ctx = _lib.Context(0)
    out = phase_link(stack, nmap, half, ctx=ctx, want_status=True, **kw)
    n = ctx.stats()["fp64_pixels"]
    ctx.close()
    return out, n


@pytest.mark.parametrize("n", [9, 30, 45])
@pytest.mark.parametrize("precision", ["mixed", "fp32"])
def test_non_finite_samples_are_coded(gpu_lib, n, precision):
    from fringe_gb300 import _lib, phase_link
    stack, nmap = synth.scene("voronoi", 41, 53, n, 3, 5, seed=n)
    hurt = stack.copy()
    hurt[:, :, :9] = np.nan                           # a border
    hurt[2, 20, 30] = np.inf
    hurt[n - 1, 33, 44] = -np.inf * 1j
    ctx = _lib.Context(0)
    ctx.set_tuning(force_fp64=True)
    for kw in RUNS:
        ref = phase_link(hurt, nmap, (3, 5), ctx=ctx, want_status=True, **kw)
        assert (ref["status"] < 0).sum() > 400
        _, clean = _listed(stack, nmap, (3, 5), precision=precision, **kw)
        got, listed = _listed(hurt, nmap, (3, 5), precision=precision, **kw)
        assert np.array_equal(got["status"], ref["status"]), kw
        assert listed <= clean, (kw, listed, clean)
        off = (ref["status"] != 0) & (ref["status"] != 3)      # 3: solved by EVD
        assert np.array_equal(got["tcorr"][off], ref["tcorr"][off])
        assert not got["phase"][:, off].any() and not got["comp"][off].any()
    ctx.close()


@pytest.mark.parametrize("n", [5, 16, 30, 45, 64])
def test_amplitudes_outside_the_split_stay_in_fp32(gpu_lib, n):
    """Dates scaled by powers of two that the split cannot hold: the coherence
    is the unscaled scene's."""
    stack, nmap = synth.scene("uniform", 37, 43, n, 4, 6, seed=n)
    scaled = stack.copy()
    scaled[1] *= np.float32(2.0 ** 52)
    scaled[n - 2] *= np.float32(2.0 ** -56)
    for kw in [r for r in RUNS if r.get("band_width", 0) < n - 1]:
        _, clean = _listed(stack, nmap, (4, 6), precision="fp32", **kw)
        got, listed = _listed(scaled, nmap, (4, 6), precision="fp32", **kw)
        assert listed <= clean + stack.shape[1] * stack.shape[2] // 50, (kw, listed, clean)
        o = oracle.run(scaled, nmap, 4, 6, **kw)
        got["comp"] = o["comp"]                       # dominated by the scaled date
        m = compare(got, o)
        assert m["valid_both"] > 1000, (kw, m)
        assert_parity(m)

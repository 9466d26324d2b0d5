"""The register eigen-solve of the Gamma records at the edges of its grids
(16 lanes per pixel up to 16, 24 and 32 dates, 32 lanes up to 48 and 64), odd
depths and odd pixel counts, against the FP64 oracle."""
import numpy as np
import pytest

import oracle
from fringe_gb300 import synth
from tests.parity import assert_parity, compare

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 3, 7, 8, 9, 15, 16, 17, 23, 24, 25, 31, 32, 33, 39, 40, 41, 47, 48, 49, 63, 64])
@pytest.mark.parametrize("semantics", ["evd", "phase_link"])
def test_depths(gpu_lib, n, semantics):
    from fringe_gb300 import phase_link
    stack, nmap = synth.scene("uniform", 9, 13, n, 6, 7, seed=100 + n)
    kw = dict(method="MLE", semantics=semantics, mini_stack_count=min(n, 3))
    g = phase_link(stack, nmap, (6, 7), precision="mixed", **kw)
    o = oracle.run(stack, nmap, 6, 7, **kw)
    m = compare(g, o)
    assert m["valid_both"] > 60, m                     # the corners' windows hold 56 samples
    assert_parity(m, phase_tol=1e-3, tcorr_tol=2e-4)


@pytest.mark.parametrize("n", [5, 12, 20, 30, 45, 60])
def test_every_outcome_beside_another(gpu_lib, n):
    """Pixels skipped, with too few SHPs, with fewer SHPs than dates, without
    power at a date, and with dates that duplicate each other (C singular),
    next to ordinary ones, which share their warp."""
    from fringe_gb300 import phase_link
    rng = np.random.default_rng(n)
    stack, nmap = synth.scene("uniform", 15, 17, n, 4, 8, seed=n)
    words = nmap.shape[2]
    centre = 4 * 17 + 8
    for r, c in zip(rng.integers(0, 15, 30), rng.integers(0, 17, 30)):
        keep = rng.choice([0, 1, n // 2 + 1])
        bits = np.zeros(words, np.uint32)
        if keep:
            for f in [centre] + list(rng.permutation(17 * 9)[: keep - 1]):
                bits[f // 32] |= np.uint32(1) << np.uint32(f % 32)
        nmap[r, c] = bits
    stack[:, 0:3, 0:3] = 0
    stack[1, 9:, 10:] = stack[0, 9:, 10:]
    for semantics in ("evd", "phase_link"):
        g = phase_link(stack, nmap, (4, 8), semantics=semantics, precision="mixed")
        o = oracle.run(stack, nmap, 4, 8, semantics=semantics)
        assert_parity(compare(g, o), phase_tol=1e-3, tcorr_tol=2e-4)


@pytest.mark.parametrize("n", [1, 2, 4, 8, 15, 16, 17, 24, 25, 31, 32, 33, 45, 48, 49, 64])
@pytest.mark.parametrize("precision", ["mixed", "fp32"])
def test_evd_and_stbas(gpu_lib, n, precision):
    """Largest eigenvectors: power iteration, and the shifted inverse
    iteration that banded coherences need."""
    from fringe_gb300 import phase_link
    stack, nmap = synth.scene("voronoi", 11, 19, n, 6, 7, seed=300 + n)
    runs = [dict(method="EVD")]
    if n >= 4:
        runs += [dict(method="STBAS", band_width=b) for b in sorted({1, n // 3 + 1, n - 2})]
        runs += [dict(method="STBAS", band_width=2, semantics="phase_link", mini_stack_count=2)]
    for kw in runs:
        g = phase_link(stack, nmap, (6, 7), precision=precision, **kw)
        o = oracle.run(stack, nmap, 6, 7, **kw)
        m = compare(g, o)
        assert m["valid_both"] > 100, (kw, m)
        assert_parity(m, phase_tol=1e-3, tcorr_tol=2e-4)

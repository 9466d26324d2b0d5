"""Counts that a run reports."""
import numpy as np
import pytest

from fringe_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["mixed", "fp32"])
def test_slow_path_counts_a_pixel_once(gpu_lib, precision):
    """Two groups of dates that never share a sample and whose coherences' largest
    eigenvalues differ by 0.06 to 0.07%: the power iteration cannot tell the
    eigenvectors apart, nor can the shifted iteration."""
    from fringe_gb300 import _lib, phase_link
    rows, cols, g, half = 24, 26, 6, (3, 4)
    k = np.arange(g)

    def coherence(step, p):
        v = np.exp(1j * step * k)
        return p + (1 - p) * np.outer(v, v.conj())
    steps = (0.5, 0.501)
    for up in range(half[0] + 1):                      # even and odd rows in a window
        for down in range(half[0] + 1):
            for first in (0, 1):
                par = (np.arange(-up, down + 1) + first) % 2
                a, b = (np.linalg.eigvalsh(coherence(s, np.mean(par == 0))) for s in steps)
                if np.mean(par == 0) in (0.0, 1.0):
                    continue
                assert 3e-4 < abs(a[-1] - b[-1]) / a[-1] < 1e-3, (up, down, a[-1], b[-1])
    x = np.zeros((2 * g, rows, cols), np.complex64)
    for r in range(rows):
        for q, s in enumerate(steps):
            x[q * g:(q + 1) * g, r, q::2] = (np.ones(g) if r % 2 == 0 else np.exp(1j * s * k))[:, None]
    nmap = synth.nmap_all_ones(rows, cols, *half)
    ctx = _lib.Context(0)
    phase_link(x, nmap, half, method="EVD", precision=precision, ctx=ctx)
    s = ctx.stats()
    ctx.close()
    assert s["pixels"] == rows * cols
    assert rows * cols // 2 < s["slow_path_pixels"] <= rows * cols, s

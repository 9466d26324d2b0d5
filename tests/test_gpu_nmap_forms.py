"""The SHP map kernels at the edges of their forms -- stack depths around the
register groups (8 dates) and padded depths (16, 32, 64), windows wider than a
32-column group, tiles that only fit packed, shared and infinite amplitudes,
calibrated amplitudes -- bit for bit against the oracle."""
import numpy as np
import pytest

import oracle
from fringe_gb300 import synth

pytestmark = pytest.mark.gpu


def _check(stack, ny, nx, **kw):
    from fringe_gb300 import nmap
    g = nmap(stack, (ny, nx), **kw)
    o_map, o_cnt = oracle.nmap(stack, ny, nx, kw.pop("prob", 0.05), **kw)
    assert np.array_equal(g["count"], o_cnt), int((g["count"] != o_cnt).sum())
    assert np.array_equal(g["nmap"], o_map)


def _scene(rows, cols, n, seed, tied):
    stack, _ = synth.scene("voronoi", rows, cols, n, 1, 1, seed=seed)
    if tied:
        stack = (np.round(np.abs(stack) * 4) / 4 + 0.25).astype(np.complex64)
        stack[n // 2, 3, 4] = np.inf                  # a valid amplitude to the reference
    return stack


@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 15, 16, 17, 24, 31, 32, 33, 57, 63, 64])
@pytest.mark.parametrize("method", ["KS2", "AD2"])
@pytest.mark.parametrize("tied", [False, True])
def test_depths(gpu_lib, n, method, tied):
    _check(_scene(13, 37, n, n, tied), 2, 3, method=method, prob=0.2)


@pytest.mark.parametrize("rows,cols,ny,nx", [(1, 1, 0, 0), (1, 70, 0, 3), (70, 1, 3, 0), (9, 33, 0, 40), (5, 129, 2, 35),
                                             (41, 64, 12, 1), (3, 5, 6, 6)])
@pytest.mark.parametrize("method", ["KS2", "AD2"])
def test_windows(gpu_lib, rows, cols, ny, nx, method):
    _check(_scene(rows, cols, 12, rows + cols, False), ny, nx, method=method)


@pytest.mark.parametrize("method,ny,nx", [("KS2", 27, 0), ("AD2", 24, 2)])
def test_tile_that_fits_only_packed(gpu_lib, method, ny, nx):
    _check(_scene(34, 40, 64, 6, True), ny, nx, method=method)


@pytest.mark.parametrize("method", ["KS2", "AD2"])
def test_calibrated_moduli_near_rounding_midpoints(gpu_lib, method):
    """Integer samples make many moduli exact or shared, and constants that
    are not powers of two put the quotients anywhere between floats."""
    rng = np.random.default_rng(3)
    stack = (rng.integers(1, 60, (18, 20, 50)) + 1j * rng.integers(0, 60, (18, 20, 50))).astype(np.complex64)
    stack[:, 4, 5] *= np.float32(1e-22)               # outside the float-float range of the modulus
    stack[:, 4, 6] *= np.float32(1e19)
    _check(stack, 2, 4, method=method, amp_const=rng.uniform(0.3, 3.0, 18))
    _check(stack, 2, 4, method=method, prob=0.5)

"""Module runs give the same bits however the file is cut into blocks of rows."""
import os

import numpy as np
import pytest

from fringe_gb300 import stackio, synth
from fringe_gb300.evdlib import Evd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32", "mixed"])
@pytest.mark.parametrize("ny,nx", [(3, 5), (5, 2)])
def test_block_size_does_not_change_the_results(gpu_lib, tmp_path, precision, ny, nx):
    rows, cols, n = 173, 61, 14
    stack, nmap = synth.scene("voronoi", rows, cols, n, ny, nx, seed=31)
    vrt = stackio.write_stack(str(tmp_path / "stack"), stack)
    wts = stackio.write_nmap(str(tmp_path / "nmap"), nmap, ny, nx)
    files = [d + ".slc" for d in stackio.dates_for(n)] + ["tcorr.bin", "compslc.bin"]
    want = None
    for memsize, blocksize in ((4000, 64), (1, 17), (1, 30), (1, 41)):
        out = str(tmp_path / ("out%d" % blocksize))
        m = Evd()
        m.inputDS, m.weightsDS, m.outputFolder = vrt, wts, out
        m.halfWindowX, m.halfWindowY, m.verbose, m.precision = nx, ny, 0, precision
        m.memsize, m.blocksize = memsize, blocksize
        assert m.run() == 0
        got = [np.fromfile(os.path.join(out, f), np.uint8) for f in files]
        want = want or got
        for f, a, b in zip(files, got, want):
            assert np.array_equal(a, b), (blocksize, f)

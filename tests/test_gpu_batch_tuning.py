"""Autotuning a batch times candidate shapes only of launches that take them."""
import time

import numpy as np
import pytest

from fringe_gb300 import synth

pytestmark = pytest.mark.gpu


def test_pieces_with_launches_of_their_own_are_not_tuned(gpu_lib):
    """Pieces of 65,536 pixels and more take no shape from the tuner: creating a
    batch of them runs the batch at most once, not once per candidate."""
    torch = pytest.importorskip("torch")
    from fringe_gb300 import _lib
    from fringe_gb300.linker import PhaseLinkBatch
    stack, nmap = synth.scene("uniform", 64, 64, 30, 5, 10, seed=9)
    stack = torch.from_numpy(np.tile(stack, (1, 16, 16))).cuda()
    nmap = torch.from_numpy(np.tile(nmap, (16, 16, 1)).view(np.int32)).cuda()
    job = {"stack": stack, "nmap": nmap, "half_window": (5, 10), "precision": "mixed"}

    def create(autotune):
        ctx = _lib.Context(0)                         # tuned shapes are kept in the context
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        b = PhaseLinkBatch([job], graph=False, autotune=autotune, ctx=ctx)
        torch.cuda.synchronize()
        return time.perf_counter() - t0, b, ctx
    extra = []
    for _ in range(3):
        plain, b, ctx = create(False)
        b.run()
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        b.run()
        torch.cuda.synchronize()
        run = time.perf_counter() - t0
        b.close(), ctx.close()
        tuned, b, ctx = create(True)
        b.close(), ctx.close()
        extra.append((tuned - plain) / run)
    assert min(extra) < 2.0, extra

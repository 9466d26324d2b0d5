"""FP32 batches under the context's limit on record memory."""
import numpy as np
import pytest

from fringe_gb300 import synth
from tests.parity import assert_parity, compare

pytestmark = pytest.mark.gpu

JOBS = [(61, 83, 20, "fp32", None), (96, 64, 33, "fp32", (3, 90)), (40, 120, 12, "mixed", None), (5, 7, 9, "fp32", None)]


@pytest.mark.parametrize("graph", [False, True])
def test_waves_under_a_limit(gpu_lib, graph):
    """Waves of any size give the single runs' bits; jobs that a limit leaves
    without records get the plain kernel's results, beside jobs that keep theirs."""
    torch = pytest.importorskip("torch")
    from fringe_gb300 import _lib
    from fringe_gb300.linker import PhaseLinkBatch, phase_link
    jobs, ref = [], []
    for rows, cols, n, precision, span in JOBS:
        stack, nmap = synth.scene("voronoi", rows, cols, n, 3, 5, seed=n)
        jobs.append({"stack": torch.from_numpy(stack).cuda(), "nmap": torch.from_numpy(nmap.view(np.int32)).cuda(),
                     "half_window": (3, 5), "precision": precision, "rows": span})
        r = phase_link(jobs[-1]["stack"], jobs[-1]["nmap"], (3, 5), precision=precision, rows=span)
        ref.append({k: v.cpu().numpy() for k, v in r.items()})
    torch.cuda.synchronize()
    row = [c * (8 * 4 * (p * (p + 1) // 2) + 8) for _, c, n, *_ in JOBS for p in [(n + 1) // 2]]
    ctx = _lib.Context(0)
    for limit in (-1, 2 * 8 * max(row), 8 * row[0], 0):
        ctx.set_record_limit(limit)
        b = PhaseLinkBatch(jobs, graph=graph, ctx=ctx)
        for _ in range(2):
            b.run()
        torch.cuda.synchronize()
        for (rows, cols, n, precision, span), o, r, w in zip(JOBS, b.outputs, ref, row):
            o = {k: v.cpu().numpy() for k, v in o.items()}
            same = all(np.array_equal(o[k], r[k], equal_nan=True) for k in r)
            tiled = precision == "mixed" or limit < 0 or limit >= w * min(8, rows)
            assert same or not tiled, (limit, n)
            assert_parity(compare(o, r))
        b.close()
    ctx.close()

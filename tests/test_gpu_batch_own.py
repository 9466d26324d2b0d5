"""Batch pieces on both sides of the size from which a piece gets solve launches
of its own (65,536 pixels) give exactly the results of running each job alone."""
import numpy as np
import pytest

from fringe_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["mixed", "fp32"])
@pytest.mark.parametrize("n,method", [(9, "MLE"), (20, "EVD"), (33, "MLE")])
def test_both_sides_of_the_line(gpu_lib, n, method, precision):
    torch = pytest.importorskip("torch")
    from fringe_gb300.linker import PhaseLinkBatch, phase_link
    stack, nmap = synth.scene("voronoi", 256, 257, n, 2, 3, seed=500 + n)
    jobs = []
    for rows, cols in ((256, 256), (255, 257), (256, 255), (64, 64), (256, 257)):
        jobs.append({"stack": torch.from_numpy(np.ascontiguousarray(stack[:, :rows, :cols])).cuda(),
                     "nmap": torch.from_numpy(np.ascontiguousarray(nmap[:rows, :cols]).view(np.int32)).cuda(),
                     "half_window": (2, 3), "method": method, "precision": precision})
    b = PhaseLinkBatch(jobs, graph=True)
    out = b.run()
    torch.cuda.synchronize()
    for j, o in zip(jobs, out):
        r = phase_link(j["stack"], j["nmap"], j["half_window"], method=method, precision=precision)
        torch.cuda.synchronize()
        for k in ("phase", "tcorr", "comp"):
            assert np.array_equal(o[k].cpu().numpy(), r[k].cpu().numpy(), equal_nan=True), (k, j["stack"].shape)
    b.close()

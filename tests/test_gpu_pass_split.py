"""Small launches, where several CTAs share a tile's passes: the same bits as a
launch whose CTAs take whole tiles, and no slower than the plain kernel that the
FP32 form used for them before."""
import numpy as np
import pytest

from fringe_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [17, 33, 64])            # 2 to 12 passes
@pytest.mark.parametrize("precision", ["mixed", "fp32"])
def test_rows_of_a_scene(gpu_lib, n, precision):
    """416 tiles as a whole; 13 to 104 in the row ranges."""
    from fringe_gb300 import phase_link
    stack, nmap = synth.scene("voronoi", 256, 200, n, 3, 6, seed=n)
    stack[1, 5, 7] = stack[n - 1, 100, 150] = np.nan
    stack[2, 40, 60] *= np.float32(1e-20)
    whole = phase_link(stack, nmap, (3, 6), precision=precision, want_status=True)
    assert (whole["status"] < 0).sum() >= 2
    for r0, r1 in ((0, 8), (3, 29), (96, 104), (192, 256)):
        part = phase_link(stack, nmap, (3, 6), precision=precision, rows=(r0, r1), want_status=True)
        for k in whole:
            assert np.array_equal(part[k][..., r0:r1, :], whole[k][..., r0:r1, :], equal_nan=True), (k, r0, r1)


@pytest.mark.parametrize("n", [48, 64])
def test_small_frames_are_no_slower_than_the_plain_kernel(gpu_lib, n):
    torch = pytest.importorskip("torch")
    from fringe_gb300 import _lib, phase_link
    stack, nmap = synth.scene("voronoi", 32, 32, n, 5, 10, seed=n)
    stack, nmap = torch.from_numpy(stack).cuda(), torch.from_numpy(nmap.view(np.int32)).cuda()
    ctx, best = _lib.Context(0), {}
    ctx.set_profiling()
    for limit in (-1, 0):                             # records; the plain kernel
        ctx.set_record_limit(limit)
        for _ in range(6):
            phase_link(stack, nmap, (5, 10), method="EVD", ctx=ctx)
            torch.cuda.synchronize()
            best[limit] = min(best.get(limit, 1e9), ctx.profile()[0])
    ctx.close()
    assert best[-1] <= best[0], best

"""The plain FP32 kernel, which windows wider than 63 columns or of more than
2,048 union samples take: every padded depth and method against the oracle, through
runs, batches and servers, and beside jobs with records."""
import numpy as np
import pytest

import oracle
from fringe_gb300 import synth
from tests.parity import assert_parity, compare

pytestmark = pytest.mark.gpu

WINDOWS = [(0, 32), (80, 2)]                          # 65 columns; 168 x 20 union samples
RUNS = [dict(method="MLE"), dict(method="EVD"), dict(method="STBAS"), dict(method="MLE", semantics="phase_link")]


def _scene(n, half, seed):
    rows, cols = (19, 90) if half[0] == 0 else (70, 23)
    return synth.scene("uniform", rows, cols, n, *half, seed=seed)


@pytest.mark.parametrize("n", [5, 15, 16, 17, 30, 32, 33, 45, 64])
@pytest.mark.parametrize("half", WINDOWS)
def test_runs(gpu_lib, n, half):
    from fringe_gb300 import _lib, phase_link
    stack, nmap = _scene(n, half, n)
    ctx = _lib.Context(0)
    ctx.set_profiling()
    for kw in RUNS:
        if half[0] == 0 and n > 30 and kw["method"] == "MLE":
            continue                                  # fewer samples than dates at the borders
        if kw["method"] == "STBAS":                   # bandwidths that FP32 tells eigenvectors apart at
            kw = dict(kw, band_width=max(2, n // 8))
        g = phase_link(stack, nmap, half, ctx=ctx, **kw)
        fp32, _, _ = ctx.profile()
        ms = ctx.profile_kernels()
        assert ms["fp32"] > 0 and ms["gram"] == 0     # the plain kernel it was
        o = oracle.run(stack, nmap, *half, **kw)
        m = compare(g, o)
        assert m["valid_both"] > 1000, (kw, m)
        assert_parity(m)
    ctx.close()


@pytest.mark.parametrize("graph,autotune", [(False, False), (True, True)])
def test_batches(gpu_lib, graph, autotune):
    torch = pytest.importorskip("torch")
    from fringe_gb300.linker import PhaseLinkBatch, phase_link
    jobs = []
    for k, (n, half) in enumerate([(9, WINDOWS[0]), (30, WINDOWS[1]), (20, (3, 5)), (50, WINDOWS[1]), (24, WINDOWS[0])]):
        stack, nmap = _scene(n, half, 60 + k)
        jobs.append({"stack": torch.from_numpy(stack).cuda(), "nmap": torch.from_numpy(nmap.view(np.int32)).cuda(),
                     "half_window": half, "method": "EVD" if k == 1 else "MLE", "precision": "mixed" if k == 3 else "fp32"})
    b = PhaseLinkBatch(jobs, graph=graph, autotune=autotune)
    for _ in range(2):
        out = b.run()
    torch.cuda.synchronize()
    for j, o in zip(jobs, out):
        r = phase_link(j["stack"], j["nmap"], j["half_window"], method=j["method"], precision=j["precision"])
        torch.cuda.synchronize()
        for k in ("phase", "tcorr", "comp"):
            assert np.array_equal(o[k].cpu().numpy(), r[k].cpu().numpy(), equal_nan=True), (k, j["stack"].shape)
    b.close()


def test_server(gpu_lib):
    from fringe_gb300 import phase_link
    from fringe_gb300.serve import Server
    scenes = [(_scene(n, half, 80 + n), half) for n, half in ((12, WINDOWS[0]), (28, WINDOWS[1]), (40, WINDOWS[1]), (18, (3, 5)))]
    srv = Server(wave_pixels=1500)
    tickets = [srv.submit(st, nm, half) for (st, nm), half in scenes]
    for t, ((st, nm), half) in zip(tickets, scenes):
        srv.wait(t)
        got, ref = srv.result(t), phase_link(st, nm, half)
        for k in ref:
            assert np.array_equal(got[k], ref[k], equal_nan=True), k
    srv.close()

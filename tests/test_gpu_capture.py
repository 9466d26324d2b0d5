"""Runs captured into a CUDA graph: the graph's replays stay valid whatever the
context does later, and a capture needs no earlier run of its size."""
import numpy as np
import pytest

from fringe_gb300 import synth

pytestmark = pytest.mark.gpu

HALF = (3, 5)


def _job(torch, n, rows=96, cols=88):
    stack, nmap = synth.scene("voronoi", rows, cols, n, *HALF, seed=n)
    out = {"phase": torch.zeros((n, rows, cols), dtype=torch.complex64, device="cuda"),
           "tcorr": torch.zeros((rows, cols), dtype=torch.float32, device="cuda"),
           "comp": torch.zeros((rows, cols), dtype=torch.complex64, device="cuda")}
    return torch.from_numpy(stack).cuda(), torch.from_numpy(nmap.view(np.int32)).cuda(), out


def _host(out):
    return {k: v.cpu().numpy().copy() for k, v in out.items()}


@pytest.mark.parametrize("precision", ["fp32", "mixed"])
@pytest.mark.parametrize("warm", [True, False])
@pytest.mark.parametrize("rows", [96, 400])
def test_replay_after_a_deeper_and_a_larger_run(gpu_lib, precision, warm, rows):
    torch = pytest.importorskip("torch")
    from fringe_gb300 import _lib, phase_link
    ctx = _lib.Context(0)
    stack, nmap, out = _job(torch, 15)
    phase_link(stack, nmap, HALF, precision=precision, ctx=_lib.context(0), out=out)
    torch.cuda.synchronize()
    want = _host(out)
    if warm:
        phase_link(stack, nmap, HALF, precision=precision, ctx=ctx, out=out)
    g = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(g):
        phase_link(stack, nmap, HALF, precision=precision, ctx=ctx, out=out)
    for v in out.values():
        v.zero_()
    g.replay()
    torch.cuda.synchronize()
    for k, v in _host(out).items():
        assert np.array_equal(v, want[k], equal_nan=True), k
    # the context outgrows the scratch that the graph refers to
    big = _job(torch, 40, rows)
    phase_link(*big[:2], HALF, precision=precision, ctx=ctx, out=big[2])
    torch.cuda.synchronize()
    after = _host(big[2])
    # whatever is allocated now must be safe from the replay
    guard = [torch.full((1 << 22,), 7, dtype=torch.uint8, device="cuda") for _ in range(64)]
    for v in out.values():
        v.zero_()
    for _ in range(3):
        g.replay()
    torch.cuda.synchronize()
    for k, v in _host(out).items():
        assert np.array_equal(v, want[k], equal_nan=True), k
    assert all(bool((t == 7).all()) for t in guard)
    phase_link(*big[:2], HALF, precision=precision, ctx=ctx, out=big[2])
    torch.cuda.synchronize()
    for k, v in _host(big[2]).items():
        assert np.array_equal(v, after[k], equal_nan=True), k
    del g
    ctx.close()


def test_capture_of_a_deeper_run(gpu_lib):
    """An FP32 run whose records are larger than any before it."""
    torch = pytest.importorskip("torch")
    from fringe_gb300 import _lib, phase_link
    ctx = _lib.Context(0)
    small, deep = _job(torch, 9), _job(torch, 33)
    phase_link(*deep[:2], HALF, ctx=_lib.context(0), out=deep[2])
    torch.cuda.synchronize()
    want = _host(deep[2])
    phase_link(*small[:2], HALF, ctx=ctx, out=small[2])
    g = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(g):
        phase_link(*deep[:2], HALF, ctx=ctx, out=deep[2])
    for v in deep[2].values():
        v.zero_()
    g.replay()
    torch.cuda.synchronize()
    for k, v in _host(deep[2]).items():
        assert np.array_equal(v, want[k], equal_nan=True), k
    del g
    ctx.close()

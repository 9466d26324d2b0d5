"""FP32 jobs need no Gamma records: where the device has no room for them, runs,
batches and servers fall back to the plain FP32 kernel, and only jobs of the mixed form
are refused.  A preloaded cudaMalloc that refuses large requests stands in for
the full device."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SHIM = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stdlib.h>
int cudaMalloc(void **p, size_t n)
{
    static int (*real)(void **, size_t);
    const char *m = getenv("TEST_MALLOC_MAX");
    if (!real) real = (int (*)(void **, size_t))dlsym(RTLD_NEXT, "cudaMalloc");
    if (m && n > strtoull(m, 0, 10)) return 2;          /* cudaErrorMemoryAllocation */
    return real(p, n);
}
"""

SCRIPT = r"""
import ctypes, os, sys
import numpy as np
from fringe_gb300 import _lib, synth
from fringe_gb300.linker import _make_job, phase_link
from fringe_gb300.serve import Server
from tests.parity import assert_parity, compare

MAX = str(16 << 20)                  # the records below take 22 to 80 MB, every other buffer less than 16
N, R, C, W = 33, 128, 128, (3, 5)
stack, nmap = synth.scene("voronoi", R, C, N, *W, seed=5)
ref = phase_link(stack, nmap, W)
lib = _lib.load()
cudart = ctypes.CDLL("libcudart.so.13")


def check(got):
    m = compare(got, ref)
    assert m["valid_both"] > 15000, m
    assert_parity(m, phase_tol=1e-4, tcorr_tol=1e-5)


def run():
    ctx = _lib.Context(0)
    os.environ["TEST_MALLOC_MAX"] = MAX
    check(phase_link(stack, nmap, W, ctx=ctx))


def batch(precision):
    def up(a):
        p = ctypes.c_void_p()
        assert cudart.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(a.nbytes)) == 0
        assert cudart.cudaMemcpy(p, a.ctypes.data_as(ctypes.c_void_p), ctypes.c_size_t(a.nbytes), 1) == 0
        return p.value
    outs = {"phase": np.zeros((N, R, C), np.complex64), "tcorr": np.zeros((R, C), np.float32),
            "comp": np.zeros((R, C), np.complex64)}
    dev = {k: up(v) for k, v in outs.items()}
    job = _make_job(N, R, C, *W, "MLE", "evd", 1, -1, 2, precision, None, _lib.FPL_MEM_DEVICE, up(stack),
                    up(np.ascontiguousarray(nmap)), dev["phase"], dev["tcorr"], dev["comp"], None)
    ctx, h = _lib.Context(0), ctypes.c_void_p()
    os.environ["TEST_MALLOC_MAX"] = MAX
    for flags in (0, _lib.FPL_BATCH_GRAPH | _lib.FPL_BATCH_AUTOTUNE):
        rc = lib.fpl_batch_create(ctx.handle, ctypes.byref(job), 1, flags, ctypes.byref(h))
        if precision == "mixed":
            assert rc == _lib.header_defines()["FPL_ERR_NOMEM"], rc
            continue
        assert rc == 0, rc
        assert lib.fpl_batch_run(h, None) == 0
        assert cudart.cudaDeviceSynchronize() == 0
        for k, v in outs.items():
            assert cudart.cudaMemcpy(v.ctypes.data_as(ctypes.c_void_p), ctypes.c_void_p(dev[k]),
                                     ctypes.c_size_t(v.nbytes), 2) == 0
        check(outs)
        lib.fpl_batch_destroy(h)


def serve(wave_pixels):
    srv = Server(wave_pixels=wave_pixels)
    os.environ["TEST_MALLOC_MAX"] = MAX
    tickets = [srv.submit(stack, nmap, W) for _ in range(3)]
    for t in tickets:
        srv.wait(t)
        check(srv.result(t))
    srv.close()


eval(sys.argv[1])
print("short memory ok")
"""


@pytest.mark.parametrize("call", ["run()", "batch('fp32')", "batch('mixed')", "serve(1 << 20)", "serve(8192)"])
def test_without_room_for_records(gpu_lib, tmp_path, call):
    src, so = tmp_path / "shim.c", tmp_path / "shim.so"
    src.write_text(SHIM)
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.check_call(["gcc", "-shared", "-fPIC", str(src), "-o", str(so), "-ldl", "-Wl,--no-as-needed",
                           "-L", cuda + "/lib64", "-lcudart", "-Wl,-rpath," + cuda + "/lib64"])
    env = dict(os.environ, LD_PRELOAD=str(so), PYTHONPATH=ROOT)
    env.pop("TEST_MALLOC_MAX", None)
    r = subprocess.run([sys.executable, "-c", SCRIPT, call], cwd=ROOT, env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "short memory ok" in r.stdout, r.stdout + r.stderr

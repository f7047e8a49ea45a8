"""Kernel limits belong to a CUDA context: after a device reset, and in a further context on the
same device, the transforms still run. Each case is a process of its own that drives the C ABI
without torch's allocator, since the reset takes the process's context away."""

import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

COMMON = """
import ctypes
import numpy as np
import torch
from s2fft_b200 import _lib

lib = _lib.lib()
rt = ctypes.CDLL("libcudart.so.12")
L = 256
flm = np.random.default_rng(1).standard_normal((L, 2 * L - 1, 2))


def ok(rc):
    assert rc == 0, (rc, lib.s2b_last_error())


def alloc(n):
    p = ctypes.c_void_p()
    ok(rt.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(n)))
    return p


def round_trip():
    plan = ctypes.c_void_p()
    d = _lib.Desc(L=L, spin=0, nside=0, sampling=0, reality=0, L_lower=0, precision=0, batch=1,
                  iter=0, N=0)
    ok(lib.s2b_plan_create(ctypes.byref(d), ctypes.byref(plan)))
    need = ctypes.c_size_t()
    sizes = []
    for way in (0, 1):
        ok(lib.s2b_workspace_size(plan, way, ctypes.byref(need)))
        sizes.append(need.value)
    x, f, ws = alloc(flm.nbytes), alloc(flm.nbytes), alloc(max(sizes))
    ok(rt.cudaMemcpy(x, flm.ctypes.data_as(ctypes.c_void_p), ctypes.c_size_t(flm.nbytes), 1))
    ok(lib.s2b_inverse(plan, x, f, ws, sizes[0], None))
    ok(lib.s2b_forward(plan, f, x, ws, sizes[1], None))
    out = np.empty_like(flm)
    ok(rt.cudaMemcpy(out.ctypes.data_as(ctypes.c_void_p), x, ctypes.c_size_t(out.nbytes), 2))
    for p in (x, f, ws):
        ok(rt.cudaFree(p))
    ok(lib.s2b_plan_destroy(plan))
    return out


def same(a, b):  # sums by atomics: equal to rounding
    assert np.abs(a - b).max() < 1e-12 * np.abs(a).max()


ok(rt.cudaSetDevice(0))
first = round_trip()
"""

RESET = """
ok(rt.cudaDeviceReset())
ok(rt.cudaSetDevice(0))
same(first, round_trip())
print("done")
"""

SECOND = """
cu = ctypes.CDLL("libcuda.so.1")
main, other = ctypes.c_void_p(), ctypes.c_void_p()
ok(cu.cuCtxGetCurrent(ctypes.byref(main)))
ok(cu.cuCtxCreate_v2(ctypes.byref(other), 0, 0))  # becomes current
same(first, round_trip())
ok(cu.cuCtxSetCurrent(main))
same(first, round_trip())
ok(cu.cuCtxDestroy_v2(other))
print("done")
"""


@pytest.mark.parametrize("body", [RESET, SECOND], ids=["reset", "second context"])
def test_limits_follow_the_context(body):
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    r = subprocess.run([sys.executable, "-c", COMMON + body], capture_output=True, text=True,
                       timeout=300, cwd=ROOT)
    assert r.returncode == 0 and "done" in r.stdout, r.stdout + r.stderr

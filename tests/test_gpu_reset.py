"""A context made after cudaDeviceReset asks the new CUDA context for what it needs:
a run whose grid takes a cluster of 16 CTAs gives the same forces as before."""
from __future__ import annotations

import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

_CHILD = r'''
import ctypes as C, glob, os, sys
sys.path.insert(0, sys.argv[1])
import numpy as np
import gi
gi.lib()
home = os.environ.get("CUDA_HOME", "/usr/local/cuda")
rt = C.CDLL(sorted(glob.glob(os.path.join(home, "lib64", "libcudart.so*")))[0])

def ok(e):
    assert e == 0, f"CUDA runtime error {e}"

p = gi.params_from_material(1.0, 1.0, 1.0, 0.4, 5.0, 1.5, 0.02, 0.01, 0.002, 0.001)
n = 70000
pos, vel, nfe = gi.ic_uniform_ball(5, n, 30.0)

def force():
    ok(rt.cudaSetDevice(0))
    ptr = []
    for host in (pos, vel, np.zeros_like(pos)):
        d = C.c_void_p()
        ok(rt.cudaMalloc(C.byref(d), C.c_size_t(host.nbytes)))
        ok(rt.cudaMemcpy(d, host.ctypes.data_as(C.c_void_p), C.c_size_t(host.nbytes), 1))
        ptr.append(d.value)
    ctx = gi.Context(0)
    ctx.forces(*ptr, [gi.Run(0, n, nfe, 0, 0, 0, 0, 0)], p)
    ok(rt.cudaDeviceSynchronize())
    f = np.zeros((n, 4), np.float32)
    ok(rt.cudaMemcpy(f.ctypes.data_as(C.c_void_p), C.c_void_p(ptr[2]), C.c_size_t(f.nbytes), 2))
    ctx.close()
    return f

before = force()
ok(rt.cudaDeviceReset())
assert np.array_equal(before, force()) and before.any()
print("done")
'''


def test_forces_after_a_device_reset(gi, torch_cuda, tmp_path):
    from conftest import PKG
    script = tmp_path / "reset.py"
    script.write_text(_CHILD)
    out = subprocess.run([sys.executable, str(script), PKG], capture_output=True, text=True, timeout=300,
                         env=dict(os.environ))
    assert out.returncode == 0 and "done" in out.stdout, out.stderr[-3000:]

"""The pinned memory that small results come back through belongs to the CUDA
context it was made in: after a cudaDeviceReset its address may be a caller's own
allocation, which the library must leave alone.  In a process of its own."""
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

PROGRAM = """
import ctypes, os, sys
import imexlbm_gb300 as m
try:
    rt = ctypes.CDLL("libcudart.so.13")
except OSError:
    rt = ctypes.CDLL("/usr/local/cuda/lib64/libcudart.so.13")

def report(prec):
    with m.LBM(12, 10, 16, 0.05, 1.0, 0.05, precision=prec) as lat:
        lat.Initialize()
        lat.step(5)
        return lat.Conserved()

kept = m.LBM(8, 8, 8, 0.05, 1.0, 0.05)      # never closed: it holds what the library has for its context
want = [report(p) for p in (m.IMEX_F64, m.IMEX_F32, m.IMEX_F16DEV)]
assert rt.cudaDeviceReset() == 0
blocks = []
for _ in range(64):                          # one of them likely lies where the library's page lay
    p = ctypes.c_void_p()
    assert rt.cudaHostAlloc(ctypes.byref(p), ctypes.c_size_t(4096), 0) == 0
    ctypes.memset(p, 0x5a, 4096)
    blocks.append(p.value)
got = [report(p) for p in (m.IMEX_F64, m.IMEX_F32, m.IMEX_F16DEV)]
assert got == want, (got, want)
for p in blocks:
    assert ctypes.string_at(p, 4096) == b"\\x5a" * 4096, "the caller's memory was written"
print("ok", flush=True)
os._exit(0)                                  # `kept` is of a context that is gone
"""


def test_reset_leaves_a_callers_pinned_memory_alone(imex):
    r = subprocess.run([sys.executable, "-c", PROGRAM], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "ok" in r.stdout, r.stdout + r.stderr

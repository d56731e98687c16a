"""The C entry points in contexts that the caller made itself, one after another on one device (in a process of their own: the
tests' process has torch's context)."""

import os
import subprocess
import sys

import pytest

from gdn_qsa_sm80_b200 import _lib

pytestmark = pytest.mark.gpu

SCRIPT = """
import ctypes, sys
lib, cu = ctypes.CDLL(sys.argv[1]), ctypes.CDLL("libcuda.so.1")
lib.gdn_chunk_scratch_bytes.restype = ctypes.c_size_t

def ok(status):
    assert status == 0, status

dev = ctypes.c_int()
ok(cu.cuInit(0))
ok(cu.cuDeviceGet(ctypes.byref(dev), 0))
for _ in range(2):
    ctx = ctypes.c_void_p()
    ok(cu.cuCtxCreate_v2(ctypes.byref(ctx), 0, dev))

    def zeros(n):
        p = ctypes.c_uint64()
        ok(cu.cuMemAlloc_v2(ctypes.byref(p), ctypes.c_size_t(n)))
        ok(cu.cuMemsetD8_v2(p, 0, ctypes.c_size_t(n)))
        return ctypes.c_void_p(p.value)

    S, Hq, Hv = 256, 1, 2
    q, k, v, out, g, beta = [zeros(S * h * w) for h, w in ((Hq, 256), (Hq, 256), (Hv, 256), (Hv, 256), (Hv, 4), (Hv, 4))]
    n = lib.gdn_chunk_scratch_bytes(1, S, Hq, Hv, 0)
    scratch = zeros(n)
    for tokens in (S, 4):
        ok(lib.gdn_chunk_fwd_sm100(q, k, v, g, beta, None, out, None, scratch, ctypes.c_size_t(n), 1, tokens, Hq, Hv, 1, 0, None))
        word = ctypes.c_int(-1)
        ok(lib.gdn_chunk_read_status(scratch, None, ctypes.byref(word)))
    ok(cu.cuCtxSynchronize())
    ok(cu.cuCtxDestroy_v2(ctx))
"""


def test_a_second_context():
    r = subprocess.run([sys.executable, "-c", SCRIPT, os.path.abspath(_lib.LIB_PATH)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr

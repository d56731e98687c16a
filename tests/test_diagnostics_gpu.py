"""A library built with the kernels' cycle accounting writes both kernels' phases (the production build has none of it)."""

import os
import subprocess
import sys

import pytest

from gdn_qsa_sm80_b200 import build

pytestmark = pytest.mark.gpu

SCRIPT = """
import ctypes, sys, torch
from gdn_qsa_sm80 import gdn_chunk
from gdn_qsa_sm80_b200 import _lib
from gdn_qsa_sm80_b200.synthetic import make_inputs
_lib.LIB_PATH, _lib.FRONTEND_PATH = sys.argv[1:]
d = [t.cuda() for t in make_inputs("default", seed=1, B=1, S=1000, Hq=16, Hv=32)[:5]]
prof = torch.zeros(128, dtype=torch.int64, device="cuda")
_lib.load().gdn_chunk_set_phase_profile(prof.data_ptr())
gdn_chunk(*d)
p = prof.tolist()
# 256 items of two heads on 3 CTAs per SM, 16 chunk steps at most in the first CTA of the chain
assert p[15] == 1 and 1 <= p[14] <= 16, p[:16]
assert all(0 < x < 10 ** 8 for x in p[8:14]) and sum(p[:8]) > 0, p[:16]
"""


def test_both_kernels_account_for_their_phases(tmp_path, monkeypatch):
    monkeypatch.setattr(build, "LIB_DIR", str(tmp_path))
    monkeypatch.setattr(build, "OBJ_DIR", str(tmp_path))
    monkeypatch.setattr(build, "LIB_PATH", str(tmp_path / "libgdn_chunk_sm100.so"))
    monkeypatch.setattr(build, "FRONTEND_PATH", str(tmp_path / "_gdn_frontend.so"))
    monkeypatch.setattr(build, "TORCH_STAMP", str(tmp_path / "torch"))
    build.build(force=True, diagnostics=True)
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-W", "error", "-c", SCRIPT, build.LIB_PATH, build.FRONTEND_PATH], cwd=root, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr

"""The chain stages a chunk's outputs in shared memory; a whole tile leaves by TMA, which drops the rows behind a regular sequence's end,
and the last tile of a packed sequence row by row, because the rows below are the next sequence's."""

import ctypes

import numpy as np
import pytest
import torch

from gdn_qsa_sm80 import gdn_chunk, gdn_chunk_varlen
from gdn_qsa_sm80_b200 import _lib
from gdn_qsa_sm80_b200.gdn_chunk_interface import check_device_status
from gdn_qsa_sm80_b200.synthetic import make_inputs

from helpers import assert_close, oracle_f32

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S", [9, 31, 63, 64, 65, 96, 127, 129])
@pytest.mark.parametrize("Hq,Hv", [(1, 2), (3, 3)])
def test_both_ways_out_write_every_row_and_no_other(S, Hq, Hv):
    B = 3
    q, k, v, g, beta, _ = make_inputs("default", seed=S, B=B, S=S, Hq=Hq, Hv=Hv)
    dev = torch.device("cuda")
    d = [t.to(dev) for t in (q, k, v, g, beta)]
    out, st = gdn_chunk(*d)
    packed, st2 = gdn_chunk_varlen(*[t.flatten(0, 1)[None] for t in d], [S * i for i in range(B + 1)])
    check_device_status(dev)
    assert torch.equal(out.flatten(0, 1), packed[0]) and torch.equal(st, st2)
    ro, rs = oracle_f32(q, k, v, g, beta)
    assert_close(out.float().cpu().numpy(), ro, "out")
    assert_close(st.cpu().numpy(), rs, "state")


SENTINEL, GUARD = -12345.0, 128    # what lies around the output, and for how many tokens on either side


def run_guarded(d, T, Hq, Hv, cu=None, B=1):
    """The call through the C entry with the output inside a larger buffer; returns (out, state)."""
    lib, vp = _lib.load(), lambda t: ctypes.c_void_p(t.data_ptr())
    n = B if cu is None else len(cu) - 1
    buf = torch.full((T + 2 * GUARD, Hv, 128), SENTINEL, dtype=torch.bfloat16, device="cuda")
    out, st = buf[GUARD:GUARD + T], torch.empty(n, Hv, 128, 128, device="cuda")
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    ptrs = [vp(t) for t in d]
    if cu is None:
        size = lib.gdn_chunk_scratch_bytes(B, T // B, Hq, Hv, _lib.PATHS["auto"])
        scratch = torch.empty(size, dtype=torch.uint8, device="cuda")
        rc = lib.gdn_chunk_fwd_sm100(*ptrs, None, vp(out), vp(st), vp(scratch), size, B, T // B, Hq, Hv, _lib.GATE_F32, _lib.PATHS["auto"], stream)
    else:
        bounds = (ctypes.c_int * len(cu))(*cu)
        size = lib.gdn_chunk_varlen_scratch_bytes(bounds, n, Hv)
        scratch = torch.empty(size, dtype=torch.uint8, device="cuda")
        rc = lib.gdn_chunk_fwd_varlen_sm100(*ptrs, None, vp(out), vp(st), vp(scratch), size, bounds, n, Hq, Hv, _lib.GATE_F32, 0, stream)
    _lib.check(rc, "guarded call")
    word = ctypes.c_int(0)
    _lib.check(lib.gdn_chunk_read_status(vp(scratch), stream, ctypes.byref(word)), "status")
    assert bool((buf[:GUARD] == SENTINEL).all()) and bool((buf[GUARD + T:] == SENTINEL).all())
    return out.clone(), st


@pytest.mark.parametrize("B,S", [(2, 9), (1, 63), (2, 64), (1, 65), (1, 2005), (2, 1990)])   # the last two are split and warm up
@pytest.mark.parametrize("Hq,Hv", [(1, 2), (3, 3)])
def test_nothing_around_the_output_is_written(B, S, Hq, Hv):
    q, k, v, g, beta, _ = make_inputs("default", seed=S, B=B, S=S, Hq=Hq, Hv=Hv)
    out, st = run_guarded([t.cuda() for t in (q, k, v, g, beta)], B * S, Hq, Hv, B=B)
    ro, rs = oracle_f32(q, k, v, g, beta)
    assert_close(out.view(B, S, Hv, 128).float().cpu().numpy(), ro, "out")
    assert_close(st.cpu().numpy(), rs, "state")


@pytest.mark.parametrize("lens", [[581, 700, 9], [9, 65, 640, 63], [2005, 33, 1990]])
@pytest.mark.parametrize("scale", [1.0, 0.001])   # of the log gates: with the second nothing is split
def test_a_packed_tail_leaves_the_next_sequence_alone(lens, scale):
    """A tail that comes several steps behind the first tile of the next sequence (nothing split): an overrun would stay there.  And
    sequences that are split, whose tails are formed by segments that warm up."""
    T, cu = sum(lens), np.concatenate([[0], np.cumsum(lens)]).tolist()
    q, k, v, g, beta, _ = make_inputs("default", seed=T, B=1, S=T, Hq=1, Hv=2)
    g = g * scale
    out, st = run_guarded([t.cuda() for t in (q, k, v, g, beta)], T, 1, 2, cu=cu)
    for i, (a, b) in enumerate(zip(cu, cu[1:])):
        ro, rs = oracle_f32(*(x[:, a:b] for x in (q, k, v, g, beta)))
        assert_close(out[a:b].float().cpu().numpy(), ro[0], f"out {i}")
        assert_close(st[i:i + 1].cpu().numpy(), rs, f"state {i}")

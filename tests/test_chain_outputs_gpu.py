"""The chain stages a chunk's outputs in shared memory; a whole tile leaves by TMA, which drops the rows behind a regular sequence's end,
and the last tile of a packed sequence row by row, because the rows below are the next sequence's."""

import pytest
import torch

from gdn_qsa_sm80 import gdn_chunk, gdn_chunk_varlen
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

"""Decode of four to eight tokens with four CTAs per SM: three stages of four tokens' vectors, or a ring of two.  A batch gives the bits that its sequences give
alone (one round of tiles, the ring of three), with every stage used again and with states in, out, both or neither."""

import pytest
import torch

from gdn_qsa_sm80 import gdn_chunk
from gdn_qsa_sm80_b200.gdn_chunk_interface import check_device_status

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("state_in,state_out", [(True, True), (False, True), (True, False), (False, False)])
@pytest.mark.parametrize("S,B,Hq,Hv", [(4, 8, 16, 32), (4, 37, 16, 32), (5, 4, 16, 32), (5, 5, 16, 32), (6, 13, 16, 32), (8, 8, 16, 32), (7, 32, 16, 32), (8, 101, 3, 3)])
def test_a_batch_gives_the_bits_of_its_sequences(S, B, Hq, Hv, state_in, state_out):
    gen = torch.Generator(device="cuda").manual_seed(S * B)
    r = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    q, k = (torch.nn.functional.normalize(r(B, S, Hq, 128), dim=-1).bfloat16() for _ in range(2))
    v, g, beta, h0 = r(B, S, Hv, 128).bfloat16(), -torch.rand(B, S, Hv, device="cuda"), torch.rand(B, S, Hv, device="cuda"), 0.1 * r(B, Hv, 128, 128)
    call = lambda i: gdn_chunk(*(t[i] for t in (q, k, v, g, beta)), initial_state=h0[i] if state_in else None, output_final_state=state_out)
    out, st = call(slice(None))
    check_device_status()
    for b in {0, 1, B // 2, B - 1}:
        o1, s1 = call(slice(b, b + 1))
        assert torch.equal(out[b:b + 1], o1)
        assert not state_out or torch.equal(st[b:b + 1], s1)

"""The chain fetches its first tiles of K and V and the initial state, and the normalisation its first rows of z, before the kernel in front of them has ended.  Whatever
made those had ended by then, however late: inputs written on the stream just before the call, and states handed from call to call without a wait of the host."""

import pytest
import torch

from gdn_qsa_sm80 import gdn_chunk
from gdn_qsa_sm80_b200 import _lib
from gdn_qsa_sm80_b200.gdn_chunk_interface import check_device_status

pytestmark = pytest.mark.gpu


def make(B, S, Hq, Hv):
    gen = torch.Generator(device="cuda").manual_seed(S)
    r = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    q, k = (torch.nn.functional.normalize(r(B, S, Hq, 128), dim=-1).bfloat16() for _ in range(2))
    x = [q, k, r(B, S, Hv, 128).bfloat16(), -torch.rand(B, S, Hv, generator=gen, device="cuda"), torch.rand(B, S, Hv, generator=gen, device="cuda"), 0.1 * r(B, Hv, 128, 128)]
    return x, r(B, S, Hv, 128).bfloat16(), torch.ones(128, device="cuda").bfloat16()


@pytest.mark.parametrize("B,S,Hq,Hv", [(1, 9, 4, 8), (1, 333, 16, 32), (4, 200, 4, 8), (2, 300, 3, 3), (2, 1500, 4, 8)])   # the last in segments
@pytest.mark.parametrize("captured", [False, True])
def test_inputs_made_just_before_the_call(B, S, Hq, Hv, captured):
    x, z, w = make(B, S, Hq, Hv)
    call = lambda x, z: gdn_chunk(*x[:5], initial_state=x[5], output_gate=(z, w))
    want, want_st = call(x, z)
    check_device_status()
    buf = [torch.empty_like(t) for t in x + [z]]

    def late():
        for t in buf:
            t.zero_()
        torch.cuda._sleep(20000)
        for t, src in zip(buf, x + [z]):
            t.copy_(src)
        return call(buf[:6], buf[6])

    step = late
    if captured:
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            late()
        torch.cuda.current_stream().wait_stream(side)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            got = late()

        def step():
            graph.replay()
            return got

    for _ in range(20):
        out, st = step()
        assert torch.equal(out, want) and torch.equal(st, want_st)
    check_device_status()


@pytest.mark.parametrize("B,S,Hq,Hv", [(1, 9, 16, 32), (2, 100, 16, 32), (1, 65, 3, 3)])
def test_states_from_call_to_call(B, S, Hq, Hv):
    x, _, _ = make(B, S, Hq, Hv)
    calls, states = 40, []
    st = x[5]
    for _ in range(calls):               # the host waits for every call
        out, st = gdn_chunk(*x[:5], initial_state=st)
        torch.cuda.synchronize()
        states.append((out, st))
    for _ in range(3):
        a, b = x[5].clone(), torch.empty_like(x[5])     # two buffers in turn, and one in place, through the C entry
        one, out = x[5].clone(), torch.empty_like(states[0][0])
        lib = _lib.load()
        n = lib.gdn_chunk_scratch_bytes(B, S, Hq, Hv, 0)
        scratch = torch.empty(n, dtype=torch.uint8, device="cuda")
        stream = torch.cuda.current_stream().cuda_stream
        run = lambda src, dst: lib.gdn_chunk_fwd_sm100(*[t.data_ptr() for t in x[:5]], src.data_ptr(), out.data_ptr(), dst.data_ptr(), scratch.data_ptr(), n, B, S, Hq, Hv,
                                                       _lib.GATE_F32, 0, stream)
        for i in range(calls):
            assert run(a, b) == 0
            a, b = b, a
        assert torch.equal(a, states[-1][1]) and torch.equal(out, states[-1][0])
        for i in range(calls):
            assert run(one, one) == 0
        assert torch.equal(one, states[-1][1]) and torch.equal(out, states[-1][0])
    check_device_status()

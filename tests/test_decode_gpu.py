"""Decode shapes: one or a few new tokens on top of a stored state.  The decode kernel is the exact fp32 recurrence,
so it is held to a tighter bound than the chunked paths (only the bf16 rounding of the output separates it from
the fp32 oracle), and the automatic path must pick it for S <= 8."""

import numpy as np
import pytest
import torch

from gdn_qsa_sm80 import gdn_chunk, rmsnorm_gated
from gdn_qsa_sm80_b200.gdn_chunk_interface import check_device_status
from gdn_qsa_sm80_b200.synthetic import make_inputs
from oracle import gdn_chunk_oracle as O

from helpers import oracle_f32

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,S,Hq,Hv", [(1, 1, 2, 4), (3, 1, 16, 32), (2, 2, 2, 4), (5, 4, 1, 4), (1, 17, 2, 2), (64, 1, 16, 32)])
@pytest.mark.parametrize("gates", ["fp32", "bf16"])
def test_decode_matches_recurrent_oracle(B, S, Hq, Hv, gates):
    q, k, v, g, beta, _ = make_inputs("default", seed=B * 100 + S, B=B, S=S, Hq=Hq, Hv=Hv)
    if gates == "bf16":
        g, beta = g.bfloat16(), beta.bfloat16()
    h0 = torch.randn(B, Hv, 128, 128, generator=torch.Generator().manual_seed(9))
    dev = "cuda"
    d = [t.to(dev) for t in (q, k, v, g, beta)]
    out, st = gdn_chunk(*d, initial_state=h0.to(dev), path="decode")
    check_device_status()
    ro, rs = oracle_f32(q, k, v, g, beta, h0, form="recurrent")
    assert O.rel_l2(st.cpu().numpy(), rs) < 1e-5
    assert O.rel_l2(out.float().cpu().numpy(), ro) < 3e-3          # bf16 rounding of the output only
    assert np.all(np.abs(out.float().cpu().numpy() - ro) <= 2.0 ** -7 * np.abs(ro) + 1e-6)
    if S <= 8:   # the automatic choice for these shapes
        o2, s2 = gdn_chunk(*d, initial_state=h0.to(dev))
        assert torch.equal(o2, out) and torch.equal(s2, st)
    # token-by-token calls chained through the state give the same bits as one call
    s_run = h0.to(dev)
    pieces = []
    for t in range(S):
        o1, s_run = gdn_chunk(*[x[:, t:t + 1] for x in d], initial_state=s_run, path="decode")
        pieces.append(o1)
    assert torch.equal(torch.cat(pieces, 1), out) and torch.equal(s_run, st)


def test_decode_without_initial_or_final_state():
    q, k, v, g, beta, _ = make_inputs("default", seed=4, B=2, S=3, Hq=2, Hv=4)
    dev = "cuda"
    out, st = gdn_chunk(*[t.to(dev) for t in (q, k, v, g, beta)], output_final_state=False, path="decode")
    assert st is None
    ro, _ = oracle_f32(q, k, v, g, beta, None, form="recurrent")
    assert O.rel_l2(out.float().cpu().numpy(), ro) < 3e-3


def test_decode_updates_the_state_in_place_through_the_c_abi():
    """h0 and hT may be the same buffer for the decode kernel (a CTA reads its whole state before it writes it)."""
    from gdn_qsa_sm80_b200 import _lib
    B, S, Hq, Hv = 4, 1, 2, 4
    q, k, v, g, beta, _ = make_inputs("default", seed=21, B=B, S=S, Hq=Hq, Hv=Hv)
    dev = "cuda"
    d = [t.to(dev).contiguous() for t in (q, k, v, g.float(), beta.float())]
    h0 = torch.randn(B, Hv, 128, 128, device=dev)
    ref_o, ref_s = gdn_chunk(*d, initial_state=h0, path="decode")
    state = h0.clone()
    out = torch.empty_like(d[2])
    scratch = torch.empty(256, dtype=torch.uint8, device=dev)
    st = _lib.load().gdn_chunk_fwd_sm100(d[0].data_ptr(), d[1].data_ptr(), d[2].data_ptr(), d[3].data_ptr(),
                                         d[4].data_ptr(), state.data_ptr(), out.data_ptr(), state.data_ptr(),
                                         scratch.data_ptr(), 256, B, S, Hq, Hv, _lib.GATE_F32, _lib.PATHS["decode"],
                                         torch.cuda.current_stream().cuda_stream)
    assert st == _lib.GDN_OK
    torch.cuda.synchronize()
    assert torch.equal(out, ref_o) and torch.equal(state, ref_s)


@pytest.mark.parametrize("B,S,Hq,Hv", [(1, 1, 2, 4), (64, 1, 16, 32), (40, 3, 8, 16), (5, 4, 1, 4), (75, 5, 4, 8), (40, 8, 8, 16)])
@pytest.mark.parametrize("gates", ["fp32", "bf16"])
@pytest.mark.parametrize("stored", [True, False])
def test_gated_decode(B, S, Hq, Hv, gates, stored):
    """Normalisation fused into the decode kernel: fewer states than SMs and up to 14 per CTA (148 SMs), more tokens than travel
    with the tile (4), with and without states.  The row that is normalised is the ungated call's; what may differ from the separate
    normalisation is the order of its fp32 sums: one bf16 rounding, 2^-8 relative at most on either side."""
    q, k, v, g, beta, _ = make_inputs("default", seed=B + S, B=B, S=S, Hq=Hq, Hv=Hv)
    if gates == "bf16":
        g, beta = g.bfloat16(), beta.bfloat16()
    gen = torch.Generator().manual_seed(S)
    z = (1.5 * torch.randn(B, S, Hv, 128, generator=gen)).bfloat16().cuda()
    w = (1 + 0.1 * torch.randn(128, generator=gen)).bfloat16().cuda()
    h0 = torch.randn(B, Hv, 128, 128, generator=gen).cuda() if stored else None
    d = [t.cuda() for t in (q, k, v, g, beta)]
    plain, st = gdn_chunk(*d, output_final_state=stored, initial_state=h0)
    ref = rmsnorm_gated(plain, z, w).float()
    for _ in range(20):   # the same bits every time: the partial sums of a row meet no other row's
        out, st2 = gdn_chunk(*d, output_final_state=stored, initial_state=h0, output_gate=(z, w))
        first = out if _ == 0 else first
        assert torch.equal(out, first)
    check_device_status()
    assert (st is None and st2 is None) or torch.equal(st, st2)
    assert ((first.float() - ref).abs() <= 2.0 ** -7 * ref.abs() + 1e-6).all()
    if B * S * Hv <= 2048:
        ro, _ = oracle_f32(q, k, v, g, beta, None if h0 is None else h0.cpu(), form="recurrent")
        ro = O.rmsnorm_gated(ro, z.float().cpu().numpy(), w.float().cpu().numpy())
        assert O.rel_l2(first.float().cpu().numpy(), ro) < 6e-3   # two bf16 roundings: the row, then the result


def test_more_rows_than_a_state_map_could_address():
    """Without states the decode kernel's range is that of its inputs: more than 2^24 (sequence, head) pairs."""
    B, Hv, tail = (1 << 21) + 3, 8, 1000
    gen = torch.Generator(device="cuda").manual_seed(5)
    q, k = (torch.randn(B, 1, 1, 128, generator=gen, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    v = torch.randn(B, 1, Hv, 128, generator=gen, device="cuda", dtype=torch.bfloat16)
    g, beta = -torch.rand(B, 1, Hv, generator=gen, device="cuda"), torch.rand(B, 1, Hv, generator=gen, device="cuda")
    out, _ = gdn_chunk(q, k, v, g, beta, output_final_state=False, path="decode")
    check_device_status()
    for part in (slice(0, tail), slice(B - tail, B)):
        ref, _ = gdn_chunk(*[x[part].contiguous() for x in (q, k, v, g, beta)], output_final_state=False)
        assert torch.equal(out[part], ref)


@pytest.mark.parametrize("S", [2, 7, 8, 9])
@pytest.mark.parametrize("Hq,Hv", [(1, 2), (3, 3)])
def test_several_tokens_over_a_ring_that_wraps(S, Hq, Hv):
    """Vectors of several tokens come as boxes of up to eight rows of a sequence.  Of four tiles a state, a CTA (at most four per SM)
    gets at least seven: each of its three stages is used twice and the first a third time.  fp32 throughout: bounds as above."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    B = -(-7 * sms // Hv)
    q, k, v, g, beta, _ = make_inputs("default", seed=S, B=B, S=S, Hq=Hq, Hv=Hv)
    h0 = torch.randn(B, Hv, 128, 128, generator=torch.Generator().manual_seed(S))
    out, st = gdn_chunk(*[t.cuda() for t in (q, k, v, g, beta)], initial_state=h0.cuda(), path="decode")
    check_device_status()
    ro, rs = oracle_f32(q, k, v, g, beta, h0, form="recurrent")
    assert O.rel_l2(st.cpu().numpy(), rs) < 1e-5
    assert np.all(np.abs(out.float().cpu().numpy() - ro) <= 2.0 ** -7 * np.abs(ro) + 1e-6)


@pytest.mark.parametrize("S", [2, 3, 4])
@pytest.mark.parametrize("Hq,Hv", [(1, 4), (4, 4)])
@pytest.mark.parametrize("stored", [True, False])
def test_vectors_by_rows_and_by_boxes(S, Hq, Hv, stored):
    """Calls of few tiles (four a state) fetch several tokens' vectors row by row, larger ones as boxes: the same bits on either side
    of the line, which lies at a tile per CTA (four per SM, at four tokens three)."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    line = sms * (4 if S < 4 else 3) // (4 * Hv)
    B = line + 1
    q, k, v, g, beta, _ = make_inputs("default", seed=S, B=B, S=S, Hq=Hq, Hv=Hv)
    h0 = torch.randn(B, Hv, 128, 128, generator=torch.Generator().manual_seed(S)).cuda() if stored else None
    d = [t.cuda() for t in (q, k, v, g, beta)]
    out, st = gdn_chunk(*d, initial_state=h0, output_final_state=stored, path="decode")
    for n in (1, line):
        o1, s1 = gdn_chunk(*[t[:n].contiguous() for t in d], initial_state=None if h0 is None else h0[:n].contiguous(),
                           output_final_state=stored, path="decode")
        assert torch.equal(o1, out[:n]) and (st is None or torch.equal(s1, st[:n])), n
    check_device_status()


def layer_inputs(seed, B, S, Hq, Hv):
    """Raw projections as a layer hands them over: q and k of any length, gates before their activations; z and the norm's weight."""
    gen = torch.Generator().manual_seed(seed)
    q, k = (3 * torch.randn(B, S, Hq, 128, generator=gen)).bfloat16(), (3 * torch.randn(B, S, Hq, 128, generator=gen)).bfloat16()
    v = torch.randn(B, S, Hv, 128, generator=gen).bfloat16()
    g, beta = 1.5 * torch.randn(B, S, Hv, generator=gen), 1.5 * torch.randn(B, S, Hv, generator=gen)
    z, w = (1.5 * torch.randn(B, S, Hv, 128, generator=gen)).bfloat16(), (1 + 0.1 * torch.randn(128, generator=gen)).bfloat16()
    return (q, k, v, g, beta), z, w


@pytest.mark.parametrize("S", [2, 3, 4, 5, 9])
@pytest.mark.parametrize("rounds", [1, 2, 3, 4, 40])
@pytest.mark.parametrize("h_in,h_out", [(True, True), (True, False), (False, False)])
def test_gated_decode_of_a_layer(S, rounds, h_in, h_out):
    """Both gated forms of several tokens with all that a layer adds, one to four states per SM and many: a stage used once and again,
    either side of the lines between the forms.  The row that is normalised is the ungated call's (bounds as in test_gated_decode); the first
    and last sequences against the oracle."""
    Hq, Hv = 2, 4
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    B = rounds * sms // Hv
    x, z, w = layer_inputs(10 * S + rounds, B, S, Hq, Hv)
    h0 = 0.1 * torch.randn(B, Hv, 128, 128, generator=torch.Generator().manual_seed(S)).cuda() if h_in else None
    d, opts = [t.cuda() for t in x], {"use_qk_l2norm_in_kernel": True, "gate_activations": True, "path": "decode"}
    plain, st = gdn_chunk(*d, initial_state=h0, output_final_state=h_out, **opts)
    out, st2 = gdn_chunk(*d, initial_state=h0, output_final_state=h_out, output_gate=(z.cuda(), w.cuda()), **opts)
    check_device_status()
    assert (st is None and st2 is None) or torch.equal(st, st2)
    ref = rmsnorm_gated(plain, z.cuda(), w.cuda()).float()
    assert ((out.float() - ref).abs() <= 2.0 ** -7 * ref.abs() + 1e-6).all()
    for part in (slice(0, 2), slice(B - 2, B)):
        q, k, v, g, beta = (t[part] for t in x)
        ro, rs = oracle_f32(q, k, v, -torch.nn.functional.softplus(g), torch.sigmoid(beta), None if h0 is None else h0[part].cpu(),
                            form="recurrent", l2norm=True)
        ro = O.rmsnorm_gated(ro, z[part].float().numpy(), w.float().numpy())
        assert O.rel_l2(out[part].float().cpu().numpy(), ro) < 6e-3
        assert st is None or O.rel_l2(st[part].cpu().numpy(), rs) < 1e-5


@pytest.mark.parametrize("S", [2, 3])
def test_gated_decode_of_three_states_per_sm(S):
    """Three states per SM take about half as long again as two, and not as long as four: times of graphs of 20 calls."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    times = []
    for rounds in (2, 3):
        B = rounds * sms // 4
        x, z, w = layer_inputs(S, B, S, 2, 4)
        d, gate = [t.cuda() for t in x], (z.cuda(), w.cuda())
        h0 = torch.zeros(B, 4, 128, 128, device="cuda")
        def call():
            gdn_chunk(*d, initial_state=h0, use_qk_l2norm_in_kernel=True, gate_activations=True, output_gate=gate)
        call()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            for _ in range(20):
                call()
        best = float("inf")
        for _ in range(20):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            graph.replay()
            b.record()
            b.synchronize()
            best = min(best, a.elapsed_time(b))
        times.append(best)
    assert times[1] < 1.56 * times[0], times

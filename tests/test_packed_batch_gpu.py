"""A packed batch in one pass of the kernels: lengths around the chunk and decode limits, split sequences, the table kernel's
piece limit, and tiles shared by two sequences, where one's values (infinities included) must not reach the other.

The kernels' arithmetic does not depend on where a sequence lies, so every sequence has the bits it has on its own."""

import numpy as np
import pytest
import torch

from gdn_qsa_sm80 import gdn_chunk, gdn_chunk_varlen
from gdn_qsa_sm80_b200 import _lib
from gdn_qsa_sm80_b200.gdn_chunk_interface import check_device_status
from gdn_qsa_sm80_b200.synthetic import make_inputs

from helpers import assert_close, oracle_f32

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lens", [[9], [63, 65, 8, 128, 1, 10], [129] * 3 + [64], [700, 30, 2048, 257], [9, 10] * 520])
@pytest.mark.parametrize("Hq,Hv,layer", [(1, 2, False), (2, 2, True)])
def test_every_sequence_as_on_its_own(lens, Hq, Hv, layer):
    T = sum(lens)
    q, k, v, g, beta, _ = make_inputs("default", seed=T, B=1, S=T, Hq=Hq, Hv=Hv)
    if layer:
        gen = torch.Generator().manual_seed(T)
        g, beta = (1.5 * torch.randn(1, T, Hv, generator=gen)).bfloat16(), (1.5 * torch.randn(1, T, Hv, generator=gen)).bfloat16()
        q, k = (3 * q.float()).bfloat16(), (3 * k.float()).bfloat16()
    h0 = 0.1 * torch.randn(len(lens), Hv, 128, 128, generator=torch.Generator().manual_seed(T + 1))
    cu = np.concatenate([[0], np.cumsum(lens)]).tolist()
    opts = {"use_qk_l2norm_in_kernel": True, "gate_activations": True} if layer else {}
    d = [t.cuda() for t in (q, k, v, g, beta)]
    h = h0.cuda()
    out, st = gdn_chunk_varlen(*d, cu, initial_state=h, strategy="packed", **opts)
    check_device_status()
    for i in range(0, len(lens), max(1, len(lens) // 6)):
        a, b = cu[i], cu[i + 1]
        o1, s1 = gdn_chunk(*[x[:, a:b].contiguous() for x in d], initial_state=h[i:i + 1], **opts)
        assert torch.equal(o1, out[:, a:b]) and torch.equal(s1, st[i:i + 1]), i
    i = len(lens) - 1
    a = cu[i]
    gr = -torch.nn.functional.softplus(g.float()) if layer else g
    br = torch.sigmoid(beta.float()) if layer else beta
    ro, rs = oracle_f32(q[:, a:], k[:, a:], v[:, a:], gr[:, a:], br[:, a:], h0[i:], l2norm=layer)
    assert_close(out[:, a:].float().cpu().numpy(), ro, "last sequence out")
    assert_close(st[i:].cpu().numpy(), rs, "last sequence state")


@pytest.mark.parametrize("layer", [False, True])
def test_infinities_stay_in_their_sequence(layer):
    lens = [70, 40, 200]
    T, cu = sum(lens), [0, 70, 110, 310]
    q, k, v, g, beta, _ = make_inputs("default", seed=1, B=1, S=T, Hq=1, Hv=2)
    opts = {"use_qk_l2norm_in_kernel": True, "gate_activations": True} if layer else {}
    d = [t.cuda() for t in (q, k, v, g, beta)]
    clean_o, clean_s = gdn_chunk_varlen(*d, cu, strategy="packed", **opts)
    for x in (d[0], d[1], d[2]):
        x[:, 70:110] = float("inf")
    out, st = gdn_chunk_varlen(*d, cu, strategy="packed", **opts)
    check_device_status()
    keep = list(range(70)) + list(range(110, 310))
    assert torch.equal(out[:, keep], clean_o[:, keep]) and torch.equal(st[[0, 2]], clean_s[[0, 2]])


def test_views_at_odd_offsets_are_gathered():
    """More than eight lengths and little padding: such a batch ran before the packed route existed, by gathering."""
    lens = list(range(40, 50))
    T, cu = sum(lens), np.concatenate([[0], np.cumsum(lens)]).tolist()
    q, k, v, g, beta, _ = make_inputs("default", seed=3, B=1, S=T, Hq=1, Hv=2)
    d = [t.cuda() for t in (q, k, v, g, beta)]
    want = gdn_chunk_varlen(*d, cu)
    odd = torch.empty(q.numel() + 1, dtype=q.dtype, device="cuda")[1:].view(q.shape).copy_(d[0])
    assert odd.is_contiguous() and odd.data_ptr() % 16
    got = gdn_chunk_varlen(odd, *d[1:], cu)
    for a, b in zip(got, want):
        assert ((a.float() - b.float()).norm() / b.float().norm()).item() <= 1e-2   # (padding changes where a chunk ends)


def test_a_long_sequence_among_short_ones_is_split():
    """Sequences are cut by what they hold of the batch's work: a long one costs about as much with short ones beside it as alone."""
    lens = [50] * 10 + [30000] + [100] * 10
    T, cu = sum(lens), np.concatenate([[0], np.cumsum(lens)]).tolist()
    q, k, v, g, beta, _ = make_inputs("default", seed=6, B=1, S=T, Hq=16, Hv=32)
    d = [t.cuda() for t in (q, k, v, g, beta)]
    own = [x[:, cu[10]:cu[11]].contiguous() for x in d]
    out, st = gdn_chunk_varlen(*d, cu)
    o1, s1 = gdn_chunk(*own)
    check_device_status()
    assert torch.equal(o1, out[:, cu[10]:cu[11]]) and torch.equal(s1, st[10:11])

    def best(call):
        times = []
        for _ in range(10):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            call()
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b))
        return min(times)

    alone, packed = best(lambda: gdn_chunk(*own)), best(lambda: gdn_chunk_varlen(*d, cu))
    assert packed < 2 * alone, f"{packed:.3f} ms, the long one alone {alone:.3f} ms"     # unsplit: more than three times


def test_short_sequences_of_different_lengths_share_a_launch():
    """A few new tokens per request, as many as each has: one launch besides the table's, not one per run of equal lengths."""
    lens = [1 + (i * 5) % 8 for i in range(300)]
    T, cu = sum(lens), np.concatenate([[0], np.cumsum(lens)]).tolist()
    q, k, v, g, beta, _ = make_inputs("default", seed=4, B=1, S=T, Hq=2, Hv=4)
    h0 = 0.1 * torch.randn(len(lens), 4, 128, 128, generator=torch.Generator().manual_seed(5)).cuda()
    d = [t.cuda() for t in (q, k, v, g, beta)]
    before = _lib.kernel_launches()
    out, st = gdn_chunk_varlen(*d, cu, initial_state=h0)
    assert _lib.kernel_launches() - before <= 2
    check_device_status()
    for i in list(range(20)) + [150, 298, 299]:
        a, b = cu[i], cu[i + 1]
        o1, s1 = gdn_chunk(*[x[:, a:b].contiguous() for x in d], initial_state=h0[i:i + 1])
        assert torch.equal(o1, out[:, a:b]) and torch.equal(s1, st[i:i + 1]), i


@pytest.mark.parametrize("lens", [[1] * 20 + [8] + [1] * 19, [8, 1], [3, 8, 2], [1, 70, 1], [5] * 7 + [4]])
@pytest.mark.parametrize("layer", [False, True])
def test_short_sequences_beside_a_longer_one(lens, layer):
    """Every sequence's own tokens are fetched and no more: among others of fewer tokens than the longest, and at the batch's end, where
    behind a sequence there is no further token."""
    T, cu = sum(lens), np.concatenate([[0], np.cumsum(lens)]).tolist()
    q, k, v, g, beta, _ = make_inputs("default", seed=T, B=1, S=T, Hq=2, Hv=4)
    h0 = 0.1 * torch.randn(len(lens), 4, 128, 128, generator=torch.Generator().manual_seed(T)).cuda()
    opts = {"use_qk_l2norm_in_kernel": True, "gate_activations": True} if layer else {}
    d = [t.cuda() for t in (q, k, v, g, beta)]
    out, st = gdn_chunk_varlen(*d, cu, initial_state=h0, **opts)
    check_device_status()
    for i, (a, b) in enumerate(zip(cu, cu[1:])):
        o1, s1 = gdn_chunk(*[x[:, a:b].contiguous() for x in d], initial_state=h0[i:i + 1], **opts)
        assert torch.equal(o1, out[:, a:b]) and torch.equal(s1, st[i:i + 1]), i

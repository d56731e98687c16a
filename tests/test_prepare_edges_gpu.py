"""P and T'' of the prepare kernel against float64 where its 16x16 fragments can go wrong: every remainder of a chunk, one and two value heads per CTA, several
items per CTA (tables, accumulators and exchange buffers in turn), with and without L2 normalisation, and keys that repeat (the inverse at its hardest)."""

import ctypes

import numpy as np
import pytest
import torch

from gdn_qsa_sm80 import gdn_chunk
from gdn_qsa_sm80_b200 import _lib
from gdn_qsa_sm80_b200 import gdn_chunk_interface as iface
from oracle import gdn_chunk_oracle as O

pytestmark = pytest.mark.gpu


def workspace(B, S, Hq, Hv):
    off = (ctypes.c_size_t * 5)()
    assert _lib.load().gdn_chunk_workspace_offsets(B, S, Hq, Hv, off) == 0
    raw = iface._scratch[(torch.cuda.current_device(), torch.cuda.current_stream().cuda_stream)]
    NT = (S + 63) // 64
    tiles = B * Hv * NT
    below = np.ones((64, 64), bool)
    below[:32, 32:] = False            # neither written nor read
    tile = lambda o: np.where(below, raw[o:o + tiles * 8192].view(torch.bfloat16).double().cpu().numpy().reshape(B, Hv, NT, 64, 64), 0)
    return tile(off[1]), tile(off[2]), raw[off[3]:off[3] + tiles * 1024].view(torch.float32).double().cpu().numpy().reshape(B, Hv, NT, 256)


def exact(q, k, g, beta, Hv, l2norm):
    B, S, _, D = k.shape
    q, k, g, beta = (t.double().cpu().numpy() for t in (q, k, g, beta))
    rk, rq = (1 / np.sqrt((t * t).sum(-1) + 1e-6) if l2norm else np.ones(t.shape[:3]) for t in (k, q))
    heads = lambda t: np.repeat(t, Hv // t.shape[2], 2)
    pad = lambda t: np.pad(np.moveaxis(t, 2, 1), ((0, 0), (0, 0), (0, -S % 64)) + ((0, 0),) * (t.ndim - 3)).reshape(B, Hv, -1, 64, *t.shape[3:])
    kn, qn = pad(heads(k * rk[..., None])), pad(heads(q * rq[..., None]))
    gam, beta = np.cumsum(pad(g), -1), pad(beta)
    low = np.tril(np.ones((64, 64), bool))
    dec = np.where(low, np.exp(np.where(low, gam[..., :, None] - gam[..., None, :], 0)), 0)
    P = qn @ kn.swapaxes(-1, -2) * dec * D ** -0.5
    T = np.linalg.inv(np.eye(64) + np.tril(kn @ kn.swapaxes(-1, -2) * dec * beta[..., None], -1)) * beta[..., None, :]
    pad1 = lambda t: np.pad(t, ((0, 0), (0, -S % 64), (0, 0)), constant_values=1e3 if l2norm else 1)   # rsqrt(1e-6) of a padding token
    rk = np.moveaxis(pad1(heads(rk)), 2, 1).reshape(B, Hv, -1, 64)
    return P, T, np.exp(gam) * rk


@pytest.mark.parametrize("l2norm", [False, True])
@pytest.mark.parametrize("Hq,Hv", [(1, 2), (3, 3)])
@pytest.mark.parametrize("B,S", [(1, s) for s in (1, 7, 8, 9, 15, 16, 17, 31, 32, 33, 47, 48, 49, 63, 64, 65)] + [(500, 130)])
def test_fragments(B, S, Hq, Hv, l2norm):
    gen = torch.Generator().manual_seed(S)
    r = lambda *s: torch.randn(*s, generator=gen)
    q, k = (t if l2norm else torch.nn.functional.normalize(t, dim=-1) for t in (r(B, S, Hq, 128), r(B, S, Hq, 128)))
    if S == 64 or B > 1:               # repeated keys, no decay: entries of A close to beta everywhere
        k = k[:, :1].expand(B, S, Hq, 128) + 1e-3 * k
    g, beta = -torch.nn.functional.softplus(r(B, S, Hv)) * (0.0 if S == 64 else 0.3), torch.sigmoid(r(B, S, Hv))
    d = [t.bfloat16().cuda() for t in (q, k, r(B, S, Hv, 128))] + [t.cuda() for t in (g, beta)]
    gdn_chunk(*d, path="prepare_only_r", use_qk_l2norm_in_kernel=l2norm)
    iface.check_device_status()
    P, T, vec = workspace(B, S, Hq, Hv)
    eP, eT, evec = exact(d[0], d[1], d[3], d[4], Hv, l2norm)
    # bf16 has 8 bits: rounding moves a value by 2^-8 of itself at most (a call of one token is one value); in T'' four TF32 roundings of 2^-11 at each of
    # two levels come on top
    assert O.rel_l2(P, eP) < 2.0 ** -8, O.rel_l2(P, eP)
    assert O.rel_l2(T, eT) < 2.0 ** -8 + 8 * 2.0 ** -11, O.rel_l2(T, eT)
    valid = S - 64 * (P.shape[2] - 1)
    assert np.abs(P[:, :, -1, valid:]).max(initial=0) == 0 and np.abs(T[:, :, -1, :, valid:]).max(initial=0) == 0
    assert O.rel_l2(vec[..., 192:], evec) < 1e-5


@pytest.mark.parametrize("l2norm", [False, True])
@pytest.mark.parametrize("Hq,Hv", [(1, 2), (3, 3)])
@pytest.mark.parametrize("down,up", [(5, 12), (5, 20), (20, 40), (40, 52)])     # across a line of 8, 16, 32 and 16 tokens
def test_gates_above_zero(down, up, Hq, Hv, l2norm):
    """gamma falls by 90 and rises by 85 again inside a chunk: exp(-90) alone is no fp32 number, the decay between the tokens before and behind is exp(-5).  The
    tokens between are not written (beta = 0)."""
    B, S = 2, 120
    gen = torch.Generator().manual_seed(down)
    r = lambda *s: torch.randn(*s, generator=gen)
    q, k = (t if l2norm else torch.nn.functional.normalize(t, dim=-1) for t in (r(B, S, Hq, 128), r(B, S, Hq, 128)))
    g, beta = -0.01 * torch.rand(B, S, Hv, generator=gen), torch.sigmoid(r(B, S, Hv))
    g[:, down], g[:, up], beta[:, down:up] = -90.0, 85.0, 0.0
    d = [t.bfloat16().cuda() for t in (q, k, r(B, S, Hv, 128))] + [t.cuda() for t in (g, beta)]
    gdn_chunk(*d, path="prepare_only_r", use_qk_l2norm_in_kernel=l2norm)
    iface.check_device_status()
    P, T, _ = workspace(B, S, Hq, Hv)
    eP, eT, _ = exact(d[0], d[1], d[3], d[4], Hv, l2norm)
    part = (slice(None), slice(None), 0, slice(up, None), slice(0, down))   # of the first chunk: rows behind the rise, columns before the fall
    for got, want, limit in ((P, eP, 2.0 ** -8), (T, eT, 2.0 ** -8 + 8 * 2.0 ** -11)):
        assert O.rel_l2(got[part], want[part]) < limit, O.rel_l2(got[part], want[part])


def tf32(x):
    """Rounded to the nearest number of 11 bits, halves to even."""
    b = x.astype(np.float32).view(np.uint32).astype(np.uint64)
    return ((b + 0xFFF + ((b >> 13) & 1)) & 0xFFFFE000).astype(np.uint32).view(np.float32).astype(np.float64)


def rounded_inverse(A):
    """(I + A)^-1 as the kernel rounds it: blocks of 16 exact, X21 = -X22 (A21 X11) of 32 and 64 with every factor a TF32 number."""
    T = np.zeros_like(A)
    for b in range(0, 64, 16):
        T[..., b:b + 16, b:b + 16] = np.linalg.inv(np.eye(16) + A[..., b:b + 16, b:b + 16])
    for s in (16, 32):
        for b in range(0, 64, 2 * s):
            lo, hi = slice(b, b + s), slice(b + s, b + 2 * s)
            T[..., hi, lo] = -tf32(T[..., hi, hi]) @ tf32(tf32(A[..., hi, lo]) @ tf32(T[..., lo, lo]))
    return T


@pytest.mark.parametrize("decay,alike", [(0.3, False), (0.01, False), (2.0, False), (0.1, True), (0.0, True)])
@pytest.mark.parametrize("Hq,Hv,l2norm", [(4, 8, False), (4, 8, True), (3, 3, True)])
def test_error_before_the_last_rounding(decay, alike, Hq, Hv, l2norm):
    """The rounding to bf16 hides what came before it but for the values it sends the other way, whose share grows with that error: of P (fp32 sums) next to none,
    of T'' as many as the roundings of the inverse's TF32 factors give by themselves."""
    B, S = 8, 640
    gen = torch.Generator().manual_seed(5)
    r = lambda *s: torch.randn(*s, generator=gen)
    q, k = (t if l2norm else torch.nn.functional.normalize(t, dim=-1) for t in (r(B, S, Hq, 128), r(B, S, Hq, 128)))
    if alike:
        k = k[:, :1] + 1e-3 * k
    g, beta = -torch.nn.functional.softplus(r(B, S, Hv)) * decay, torch.sigmoid(r(B, S, Hv))
    d = [t.bfloat16().cuda() for t in (q, k, r(B, S, Hv, 128))] + [t.cuda() for t in (g, beta)]
    gdn_chunk(*d, path="prepare_only_r", use_qk_l2norm_in_kernel=l2norm)
    iface.check_device_status()
    P, T, _ = workspace(B, S, Hq, Hv)
    eP, eT, _ = exact(d[0], d[1], d[3], d[4], Hv, l2norm)
    columns = np.moveaxis(beta.double().numpy(), 2, 1).reshape(B, Hv, -1, 1, 64)
    bf16 = lambda x: torch.from_numpy(np.ascontiguousarray(x)).float().bfloat16().double().numpy()

    def other_way(got, want):                # share of the values above a thousandth of the largest
        return (got != bf16(want))[np.abs(want) > 1e-3 * np.abs(want).max()].mean()

    expected = other_way(bf16(rounded_inverse(np.linalg.inv(eT / columns) - np.eye(64)) * columns), eT)
    # P: sums of 128 products and a decay in fp32, a few 2^-21 of a typical value (exponents of a hundred lose some bits more), against steps of 2^-8: a share of 2^-11
    # and less.  T'': some hundred (strong decay: 5e-4 of them are allowed for) to ten thousand values go the other way, so 15 % is outside their spread, and factors of
    # one bit less would double the share.
    assert other_way(P, eP) < 2.0 ** -10, other_way(P, eP)
    assert other_way(T, eT) < 1.15 * expected + 5e-4, (other_way(T, eT), expected)

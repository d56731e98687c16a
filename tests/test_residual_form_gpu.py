"""The lean prepare kernel and the residual-form chain (path "twopass_t") at the sizes where they can go wrong: one token,
chunk edges and remainders, one and several value heads per qk head, sequences split into segments or not.

Tolerance: the parity bar of the operator (rel-L2 <= 1e-2, max-abs <= 2e-2); bf16 operands (8 mantissa bits, half an ulp is
2^-9 = 2e-3 relative) enter four products in a row, so a correct result lies at 3-4e-3.
"""

import numpy as np
import pytest
import torch

from gdn_qsa_sm80 import gdn_chunk
from gdn_qsa_sm80_b200.gdn_chunk_interface import check_device_status
from gdn_qsa_sm80_b200.synthetic import make_inputs

from helpers import assert_close, oracle_f32

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,S,Hq,Hv,decay,h0", [
    (1, 1, 1, 2, 1.0, True), (2, 63, 1, 1, 1.0, False), (1, 64, 2, 4, 1.0, True), (1, 65, 3, 3, 1.0, True),
    (3, 127, 1, 4, 1.0, True), (1, 128, 2, 2, 1.0, False), (40, 300, 4, 8, 1.0, True),   # unsplit, two CTAs per SM
    (1, 511, 2, 4, 4.0, True),      # eight chunks: the shortest sequence that is split
    (2, 1500, 3, 3, 1.0, True), (1, 4096, 1, 2, 0.1, True),
    (1, 2048, 2, 4, 0.002, True),   # forgets nothing: the serial run inside a split launch
])
@pytest.mark.parametrize("layer", [False, True])
def test_matches_oracle(B, S, Hq, Hv, decay, h0, layer):
    q, k, v, g, beta, _ = make_inputs("default", seed=S + B, B=B, S=S, Hq=Hq, Hv=Hv)
    gen = torch.Generator().manual_seed(S)
    g = g * decay
    state = 0.1 * torch.randn(B, Hv, 128, 128, generator=gen) if h0 else None
    g_in, b_in = g, beta
    if layer:
        q, k = ((x.float() * torch.exp(torch.randn(B, S, Hq, 1, generator=gen))).bfloat16() for x in (q, k))
        g_in = torch.log(torch.expm1(-g).clamp_min(1e-30)).bfloat16()        # softplus(g_in) = -g up to bf16
        b_in = torch.logit(beta).bfloat16()
        g, beta = -torch.nn.functional.softplus(g_in.float()), torch.sigmoid(b_in.float())
    d = [t.cuda() for t in (q, k, v, g_in, b_in)]
    out, st = gdn_chunk(*d, initial_state=None if state is None else state.cuda(), path="twopass_t",
                        use_qk_l2norm_in_kernel=layer, gate_activations=layer)
    check_device_status()
    ro, rs = oracle_f32(q, k, v, g, beta, state, l2norm=layer)
    assert_close(out.float().cpu().numpy(), ro, "out")
    assert_close(st.cpu().numpy(), rs, "state")


@pytest.mark.parametrize("size", [-130.0, -1e4, -1e9, -3e38, float("-inf")])
@pytest.mark.parametrize("path", ["twopass_t", "twopass_nv64", "coop"])
@pytest.mark.parametrize("l2norm", [False, True])
def test_resets(size, path, l2norm):
    """Gates that end all memory, first, inside and last of a chunk: each token behind one keeps its own decay.  Held row by row;
    a row is a bf16 product of one to 64 terms, so its error is that of its largest operands: 2^-8 each, three in a row, and the row's
    own rounding."""
    B, S, Hq, Hv, at = 1, 300, 2, 4, [0, 64, 90, 100, 127, 191, 200]
    q, k, v, g, beta, h0 = make_inputs("default", seed=21, B=B, S=S, Hq=Hq, Hv=Hv)
    g[:, at] = size
    d = [t.cuda() for t in (q, k, v, g, beta)]
    h0 = h0[:, :Hv]
    out, st = gdn_chunk(*d, initial_state=h0.cuda(), path=path, use_qk_l2norm_in_kernel=l2norm)
    check_device_status()
    ro, rs = oracle_f32(q, k, v, g, beta, h0, form="recurrent", l2norm=l2norm)
    assert_close(out.float().cpu().numpy(), ro, "out")
    assert_close(st.cpu().numpy(), rs, "state")
    rows = np.linalg.norm(out.float().cpu().numpy() - ro, axis=-1) / np.linalg.norm(ro, axis=-1)
    assert rows[:, at].max() <= 2e-2 and np.median(rows) <= 1e-2

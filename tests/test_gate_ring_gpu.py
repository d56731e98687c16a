"""The normalisation kernel's rows on their way: where a thread's rows end in, at and behind its ring of five, and behind a forward pass, whose end it does not wait
for before it reads z."""

import pytest
import torch

from gdn_qsa_sm80 import gdn_chunk
from gdn_qsa_sm80_b200.gdn_chunk_interface import check_device_status, rmsnorm_gated

pytestmark = pytest.mark.gpu
WAVE = 2 * 32            # rows of an SM at a time


@pytest.mark.parametrize("rows", [lambda w: w - 1, lambda w: w + 1, lambda w: 5 * w - 33, lambda w: 5 * w, lambda w: 5 * w + 1, lambda w: 6 * w + 17, lambda w: 11 * w + 31])
def test_rows_against_float64(rows):
    n = rows(WAVE * torch.cuda.get_device_properties(0).multi_processor_count)
    gen = torch.Generator(device="cuda").manual_seed(n)
    y, z = (torch.randn(n, 128, generator=gen, device="cuda").bfloat16() for _ in range(2))
    w = (1 + 0.1 * torch.randn(128, generator=gen, device="cuda")).bfloat16()
    got = rmsnorm_gated(y, z, w).double()
    y, z = y.double(), z.double()
    want = y * (y.pow(2).mean(-1, keepdim=True) + 1e-6).rsqrt() * w.double() * z * torch.sigmoid(z)
    # one bf16 rounding, 2^-8 of a value at most, behind fp32 arithmetic
    assert ((got - want).abs() <= 2.0 ** -8 * want.abs() + 1e-30).all()


@pytest.mark.parametrize("B,S", [(1, 9), (1, 333), (4, 700)])
@pytest.mark.parametrize("path", ["auto", "simt"])
def test_behind_the_forward_pass_with_z_made_just_before(B, S, path):
    gen = torch.Generator(device="cuda").manual_seed(S)
    r = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    q, k = (torch.nn.functional.normalize(r(B, S, 4, 128), dim=-1).bfloat16() for _ in range(2))
    v, g, beta, x, w = r(B, S, 8, 128).bfloat16(), -torch.rand(B, S, 8, device="cuda"), torch.rand(B, S, 8, device="cuda"), r(B, S, 8, 128), torch.ones(128, device="cuda").bfloat16()
    plain, _ = gdn_chunk(q, k, v, g, beta, path=path)
    want = rmsnorm_gated(plain, x.bfloat16(), w)
    z = torch.zeros(B, S, 8, 128, dtype=torch.bfloat16, device="cuda")
    for _ in range(20):
        z.zero_()
        torch.cuda._sleep(20000)
        z.copy_(x)
        out, _ = gdn_chunk(q, k, v, g, beta, output_gate=(z, w), path=path)
        assert torch.equal(out, want)
    check_device_status()

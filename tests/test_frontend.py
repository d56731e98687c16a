"""Tensors that have no memory behind them reach the native front end as errors, not as a C++ exception through the
interpreter (which would end the process)."""
import threading

import pytest
import torch
from torch._subclasses.fake_tensor import FakeTensorMode

from gdn_qsa_sm80 import gdn_chunk


def _call(dev):
    q = torch.empty(1, 3, 2, 128, dtype=torch.bfloat16, device=dev)
    v = torch.empty(1, 3, 4, 128, dtype=torch.bfloat16, device=dev)
    g = torch.empty(1, 3, 4, device=dev)
    return gdn_chunk(q, q, v, g, g)


def test_fake_tensors_raise():
    with FakeTensorMode(), pytest.raises(Exception):
        _call("cuda")


@pytest.mark.gpu
def test_batched_tensors_raise():
    q = torch.zeros(2, 1, 3, 2, 128, dtype=torch.bfloat16, device="cuda")
    v = torch.zeros(2, 1, 3, 4, 128, dtype=torch.bfloat16, device="cuda")
    g = torch.zeros(2, 1, 3, 4, device="cuda")
    with pytest.raises(Exception):
        torch.vmap(lambda a, b, c: gdn_chunk(a, a, b, c, c)[0])(q, v, g)


def _inputs(B, S, Hq, Hv, seed):
    gen = torch.Generator().manual_seed(seed)
    q, k = (torch.nn.functional.normalize(torch.randn(B, S, Hq, 128, generator=gen), dim=-1).bfloat16().cuda() for _ in range(2))
    v = torch.randn(B, S, Hv, 128, generator=gen).bfloat16().cuda()
    return q, k, v, -torch.rand(B, S, Hv, generator=gen).cuda(), torch.rand(B, S, Hv, generator=gen).cuda()


@pytest.mark.gpu
@pytest.mark.parametrize("S", [4, 700])
def test_a_threads_first_cuda_call(S):
    """Nothing has given the thread a CUDA context before the call does."""
    x = _inputs(1, S, 2, 4, S)
    want, got = gdn_chunk(*x), []
    torch.cuda.synchronize()
    h0 = want[1].clone()

    def work():
        got.append(gdn_chunk(*x))
        got.append(gdn_chunk(*x, initial_state=h0))

    t = threading.Thread(target=work)
    t.start()
    t.join()
    assert len(got) == 2
    assert torch.equal(got[0][0], want[0]) and torch.equal(got[0][1], want[1])
    assert torch.equal(got[1][0], gdn_chunk(*x, initial_state=h0)[0])

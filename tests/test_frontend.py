"""Tensors that have no memory behind them reach the native front end as errors, not as a C++ exception through the
interpreter (which would end the process)."""
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

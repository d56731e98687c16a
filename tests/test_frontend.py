"""Tensors that have no memory behind them reach the native front end as errors, not as a C++ exception through the
interpreter (which would end the process)."""
import sys
import threading
import time

import pytest
import torch
from torch._subclasses.fake_tensor import FakeTensorMode

from gdn_qsa_sm80 import gdn_chunk, gdn_chunk_varlen
from gdn_qsa_sm80_b200 import _lib
from gdn_qsa_sm80_b200 import gdn_chunk_interface as interface

FRONTEND_PATH = _lib.FRONTEND_PATH


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


@pytest.mark.gpu
def test_other_threads_run_during_launches():
    """The forward call lets go of the interpreter while it launches.  With a switch interval of a minute another thread only
    runs when it does: enough calls of 50 us to fill the launch queue give it thousands of turns, or a few."""
    x = _inputs(64, 1, 16, 32, 0)
    gdn_chunk(*x)                          # scratch buffer and kernels in place
    torch.cuda.synchronize()
    turns, stop, started = [0], threading.Event(), threading.Event()

    def count():
        started.set()
        while not stop.is_set():
            turns[0] += 1
            time.sleep(0)

    t = threading.Thread(target=count)
    t.start()
    started.wait()
    old = sys.getswitchinterval()
    sys.setswitchinterval(60.0)
    try:
        before = turns[0]
        for _ in range(3000):
            gdn_chunk(*x)
        during = turns[0] - before
    finally:
        sys.setswitchinterval(old)
        stop.set()
        t.join()
    torch.cuda.synchronize()
    assert during > 100, during


@pytest.mark.gpu
def test_threads_on_one_stream():
    """Calls of several threads on one stream share its scratch buffer, which grows meanwhile: each gives the bits it gives alone."""
    def plain(seed, B, S):
        x = _inputs(B, S, 2, 4, seed)
        return lambda: gdn_chunk(*x)

    def converted(seed, S):                # through the Python wrapper
        q, k, v, g, beta = _inputs(1, S, 2, 4, seed)
        return lambda: gdn_chunk(q.float(), k, v, g, beta)

    def packed(seed, lens):
        x = _inputs(1, sum(lens), 2, 4, seed)
        cu = [sum(lens[:i]) for i in range(len(lens) + 1)]
        return lambda: gdn_chunk_varlen(*x, cu)

    jobs = [[plain(1, 1, 700), packed(2, [3, 100, 9, 64]), converted(3, 200)], [packed(4, [500, 20, 1, 1, 1500]), plain(5, 3, 130)],
            [converted(6, 2000), plain(7, 64, 1), packed(8, [5, 6, 7])], [plain(9, 8, 4), packed(10, [40] * 30), plain(11, 2, 3000)]]
    want = [[job() for job in mine] for mine in jobs]
    torch.cuda.synchronize()
    interface._scratch.clear()             # (the Python wrapper's buffers start small again)
    wrong = []

    def work(i):
        try:
            for _ in range(40):
                for job, (o, s) in zip(jobs[i], want[i]):
                    a, b = job()
                    if not (torch.equal(a, o) and torch.equal(b, s)):
                        wrong.append(i)
        except Exception as e:
            wrong.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    interface.check_device_status()
    assert not wrong


@pytest.fixture
def without_front_end(monkeypatch, tmp_path):
    """A front end that cannot be loaded here: built against another torch, or not at all."""
    monkeypatch.setattr(_lib, "FRONTEND_PATH", str(tmp_path / "_gdn_frontend.so"))
    monkeypatch.setattr(_lib, "_frontend", False)
    monkeypatch.setattr(interface, "_native_forward", None)


def test_the_wrapper_runs_without_the_front_end(without_front_end):
    with pytest.warns(RuntimeWarning, match="front end"), pytest.raises(RuntimeError, match="needs CUDA tensors"):
        _call("cpu")
    with pytest.raises(RuntimeError, match="needs CUDA tensors"):
        _call("cpu")


@pytest.mark.gpu
@pytest.mark.filterwarnings("ignore:gdn_chunk runs without")
def test_results_without_the_front_end(without_front_end):
    x = _inputs(2, 130, 2, 4, 1)
    wrapped, packed = gdn_chunk(*x), gdn_chunk_varlen(*[t.reshape(1, 260, *t.shape[2:]) for t in x], [0, 130, 260])
    assert _lib._frontend is None
    _lib._frontend = False
    _lib.FRONTEND_PATH, interface._native_forward = FRONTEND_PATH, None
    native = gdn_chunk(*x)
    assert _lib._frontend
    for a, b, c in zip(wrapped, native, packed):
        assert torch.equal(a, b) and torch.equal(c.reshape(a.shape), a)

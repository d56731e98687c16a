"""Waits of the chunked kernels under conditions that timing alone does not produce (test hooks, environment variable GDN_CHUNK_DBG)."""

import time

import pytest
import torch

from gdn_qsa_sm80 import gdn_chunk
from gdn_qsa_sm80_b200 import _lib
from gdn_qsa_sm80_b200.gdn_chunk_interface import check_device_status
from gdn_qsa_sm80_b200.synthetic import make_inputs

pytestmark = pytest.mark.gpu

LATE_PRODUCER, WARP_GIVES_UP, NO_TILE, NO_PRODUCT, LANE_GIVES_UP, LANE_WAITS = "8", "9", "10", "11", "12", "13"


def inputs(workload, **sizes):
    return [t.cuda() for t in make_inputs(workload, seed=3, **sizes)[:5]]


@pytest.mark.parametrize("workload,S", [("default", 2000), ("default", 1984), ("long_context", 8000)])   # warm-ups of about 5 and 23 chunks
def test_a_late_producer_is_not_overtaken_in_warm_up_chunks(workload, S, monkeypatch):
    """A wait names the parity of a barrier's phase: a role that comes to it after two of them waits for a third.  Chunks without
    outputs need nothing that the producer loads behind its wait for the chunk before."""
    d = inputs(workload, S=S, Hq=1, Hv=2)
    out, st = gdn_chunk(*d)
    check_device_status()
    monkeypatch.setenv("GDN_CHUNK_DBG", LATE_PRODUCER)
    late, st_late = gdn_chunk(*d)
    check_device_status()
    assert torch.equal(out, late) and torch.equal(st, st_late)


@pytest.mark.parametrize("B,S", [(1, 64 * 9), (2, 150), (1, 65), (200, 200)])
def test_a_late_producer_is_not_overtaken_by_the_outputs(B, S, monkeypatch):
    """All that a chunk's outputs need has been loaded when the producer waits for those of the chunk before to leave."""
    d = inputs("default", B=B, S=S, Hq=1, Hv=2)
    out, st = gdn_chunk(*d)
    check_device_status()
    monkeypatch.setenv("GDN_CHUNK_DBG", LATE_PRODUCER)
    late, st_late = gdn_chunk(*d)
    check_device_status()
    assert torch.equal(out, late) and torch.equal(st, st_late)


@pytest.mark.parametrize("hook,path,code", [(NO_TILE, "auto", "0x502"), (NO_PRODUCT, "prepare_only_t", "0x102")])
@pytest.mark.parametrize("Hq,Hv", [(1, 2), (3, 3)])
def test_a_wait_that_runs_out_is_reported_and_the_next_call_succeeds(hook, path, code, Hq, Hv, monkeypatch):
    """Two seconds, as everywhere: the first tile of V (or the first product) never comes and whoever needs it gives up."""
    d = inputs("default", S=40, Hq=Hq, Hv=Hv)
    out, st = gdn_chunk(*d)
    check_device_status()
    monkeypatch.setenv("GDN_CHUNK_DBG", hook)
    t0 = time.time()
    gdn_chunk(*d, path=path)
    with pytest.raises(_lib.GdnLibraryError, match=code):
        check_device_status()
    assert 1.5 < time.time() - t0 < 5.0      # all roles wait at the same time
    monkeypatch.delenv("GDN_CHUNK_DBG")
    again, st_again = gdn_chunk(*d)
    check_device_status()
    assert torch.equal(out, again) and torch.equal(st, st_again)


@pytest.mark.parametrize("S", [40, 64, 300])
def test_an_output_warp_that_gives_up_holds_up_the_others_for_a_limited_time(S, monkeypatch):
    """Each output warp counts its own tries, so one may leave while the others still see the barrier complete; they meet at a barrier
    without a limit when a chunk's outputs are staged.  What is reported is a wait that ran out first, not one behind it (0x50b: of the
    others, for the next chunk)."""
    d = inputs("default", S=S, Hq=1, Hv=2)
    out, st = gdn_chunk(*d)
    check_device_status()
    monkeypatch.setenv("GDN_CHUNK_DBG", WARP_GIVES_UP)
    t0 = time.time()
    gdn_chunk(*d)
    with pytest.raises(_lib.GdnLibraryError, match="0x5(?!0b)"):
        check_device_status()
    assert 1.5 < time.time() - t0 < 9.0      # its wait, then those of the others for the next chunk
    monkeypatch.delenv("GDN_CHUNK_DBG")
    again, st_again = gdn_chunk(*d)
    check_device_status()
    assert torch.equal(out, again) and torch.equal(st, st_again)


@pytest.mark.parametrize("Hq,Hv", [(1, 2), (3, 3)])
def test_a_single_lane_that_gave_up_is_reported(Hq, Hv, monkeypatch):
    """Each lane counts its own tries; the code of any of them is reported."""
    d = inputs("default", S=40, Hq=Hq, Hv=Hv)
    monkeypatch.setenv("GDN_CHUNK_DBG", LANE_GIVES_UP)
    gdn_chunk(*d, path="prepare_only_t")
    with pytest.raises(_lib.GdnLibraryError, match="0x101"):
        check_device_status()
    monkeypatch.delenv("GDN_CHUNK_DBG")
    gdn_chunk(*d)
    check_device_status()


@pytest.mark.parametrize("S", [40, 300])
@pytest.mark.parametrize("Hq,Hv", [(1, 2), (3, 3)])
def test_a_warp_leaves_when_one_of_its_lanes_has_given_up(Hq, Hv, S, monkeypatch):
    """The other lanes of its warp have seen their barriers complete: had they gone on, they would wait without a limit for the lane that left."""
    d = inputs("default", S=S, Hq=Hq, Hv=Hv)
    out, st = gdn_chunk(*d)
    check_device_status()
    monkeypatch.setenv("GDN_CHUNK_DBG", LANE_WAITS)
    t0 = time.time()
    gdn_chunk(*d, path="prepare_only_t")
    with pytest.raises(_lib.GdnLibraryError, match="0x102"):
        check_device_status()
    assert 1.5 < time.time() - t0 < 9.0      # its wait and those of the others for what its warp makes
    monkeypatch.delenv("GDN_CHUNK_DBG")
    again, st_again = gdn_chunk(*d)
    check_device_status()
    assert torch.equal(out, again) and torch.equal(st, st_again)

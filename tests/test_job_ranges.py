"""mvb_job_enqueue refuses, on the host, ranges that would compute slices from the
rotation, selection or beam of another time or chunk (a later frequency, or a later
chunk, continues the one time and chunk of the call before it)."""

import ctypes

import pytest

from matvis_b200 import _lib


def _job(ntime=3, nchunks=2, nfreq=4, freq_group=2):
    fake = 4096  # never dereferenced: the refused calls make no launch
    return _lib.Job(nsrc=10, chunk_size=5, cap=5, ntime=ntime, nchunks=nchunks, nfreq=nfreq, nant=2, nfeed=1,
                    freq_group=freq_group, rot=fake, sigmas=fake, nbeam=1, sflux=fake, freqs=fake, freqs_dev=fake,
                    vis=fake, mode=_lib.GEMM_F16_3, Mpad=128, Kcap=64)


@pytest.mark.parametrize("ranges", [
    (0, 3, 0, 1, 2, 4),  # later frequencies of several times: all would take the last time's sky
    (0, 1, 0, 2, 2, 4),  # of several chunks: the last chunk would be summed twice
    (0, 3, 0, 2, 2, 4),
    (0, 2, 1, 2, 0, 4),  # a later chunk of several times: one rotation for all of them
    (1, 3, 1, 2, 2, 4),
])
def test_ranges_without_their_own_prologue_are_refused(ranges):
    rc = _lib.lib.mvb_job_enqueue(ctypes.byref(_job()), *ranges, None)
    assert rc == _lib.MVB_ERR_ARG
    assert _lib.lib.mvb_last_error().decode().startswith("mvb_job_enqueue:")


@pytest.mark.parametrize("ranges", [(1, 1, 0, 2, 2, 4), (0, 3, 2, 2, 2, 4), (2, 1, 1, 2, 2, 4)])
def test_empty_ranges_are_accepted(ranges):
    assert _lib.lib.mvb_job_enqueue(ctypes.byref(_job()), *ranges, None) == _lib.MVB_OK

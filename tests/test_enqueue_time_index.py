"""VisEngine.enqueue_time takes a time index as an array does: counted from the end if
negative, any integer type, IndexError past the end (the native call is recorded, not made)."""

import numpy as np
import pytest
import torch

from matvis_b200 import _lib, workloads as wl
from matvis_b200.beam_models import GaussianBeam
from matvis_b200.engine import VisEngine, job_from_arrays


@pytest.fixture
def engine(monkeypatch):
    calls = []
    monkeypatch.setattr(_lib, "require_cuda", lambda device=None: torch.device("cpu"))
    monkeypatch.setattr(_lib, "stream_handle", lambda stream=None: None)
    # (job, t0, t1, c0, c1, f0, f1, stream), the integers as ctypes takes them
    monkeypatch.setattr(_lib.lib, "mvb_job_enqueue",
                        lambda job, *a: calls.append(tuple(_lib.c_int.from_param(x) and x for x in a[:6])) or 0)
    cfg = wl.subset(wl.config2(nfreq=4, ntimes=4), nsrc=50, nfreq=3, ntimes=3, nant=4, seed=4)
    eng = VisEngine(job_from_arrays(ants=cfg["antpos"], fluxes=cfg["fluxes"], ra=cfg["ra"], dec=cfg["dec"],
                                    freqs=cfg["freqs"], lsts=cfg["lsts"], latitude=cfg["latitude"],
                                    beams=[GaussianBeam(0.2)]))
    eng.allocate()
    return eng, calls


@pytest.mark.parametrize("t,want", [(0, 0), (-1, 2), (-3, 0), (np.int64(1), 1), (np.int32(-2), 1)])
def test_index_forms(engine, t, want):
    eng, calls = engine
    eng.enqueue_time(t)
    eng.enqueue_time(t, after=lambda f0, g: None)
    assert [c[:2] for c in calls] == [(want, want + 1)] * len(calls) and len(calls) == 2


@pytest.mark.parametrize("t", [3, -4])
def test_past_the_end(engine, t):
    with pytest.raises(IndexError):
        engine[0].enqueue_time(t)
    assert not engine[1]

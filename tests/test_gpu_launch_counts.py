"""The launch counts that the engine and the server report are the kernels that ran."""

import numpy as np
import pytest
import torch

from matvis_b200 import _lib, workloads as wl
from matvis_b200.beam_models import GaussianBeam
from matvis_b200.engine import VisEngine, job_from_arrays
from matvis_b200.serve import VisServer

pytestmark = pytest.mark.gpu


def _kernels(call):
    """The library's kernels that ran during ``call``, by the profiler."""
    torch.cuda.synchronize()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        call()
        torch.cuda.synchronize()
    return sum(e.count for e in prof.key_averages() if "mvb::" in e.key and "flux_sqrt_half" not in e.key)


def _spec(**kw):
    cfg = wl.subset(wl.config2(nfreq=16, ntimes=4), nsrc=2500, nfreq=5, ntimes=2, nant=24, seed=4)
    if kw.get("beams"):
        cfg["beams"], cfg["beam_idx"] = kw.pop("beams"), None
    return job_from_arrays(ants=cfg["antpos"], fluxes=cfg["fluxes"], ra=cfg["ra"], dec=cfg["dec"], freqs=cfg["freqs"],
                           lsts=cfg["lsts"], latitude=cfg["latitude"], beams=cfg["beams"], beam_idx=cfg["beam_idx"],
                           **kw)


CASES = [dict(polarized=True, freq_group=2), dict(polarized=True, nchunks=3), dict(beams=[GaussianBeam(0.2)]),
         dict(polarized=True, matprod="VectorDot", pair_product="vecdot", antpairs=np.array([[0, 1], [5, 3]]))]


@pytest.mark.parametrize("kw", CASES)
def test_engine_counts_its_launches(kw):
    eng = VisEngine(_spec(**kw))
    eng.upload()
    eng.enqueue()
    before = _lib.lib.mvb_launches()
    n = _kernels(eng.enqueue)
    assert n == _lib.lib.mvb_launches() - before > 0
    eng.capture()
    assert n == eng.launched == _kernels(eng.run) <= eng.launches_per_run()


@pytest.mark.parametrize("batch", [True, False])
def test_server_counts_its_launches(batch):
    srv = VisServer(max_active=3, batch_products=batch)
    jobs = [(0.0, _spec(**dict(kw))) for kw in CASES]
    n = _kernels(lambda: srv.serve_stream(jobs))
    assert n == srv.launches > 0

"""The native launch sequence of a job: the whole job in one call, a time at a time,
and a frequency group at a time (the results-copying run) give the same bits, for
every kind of beam, sky, rotation and product; ranges outside the job are refused."""

import ctypes

import numpy as np
import pytest
import torch

from matvis_b200 import _lib, workloads as wl
from matvis_b200.beam_models import GaussianBeam
from matvis_b200.beamfits import BeamFits
from matvis_b200.engine import VisEngine, job_from_arrays

pytestmark = pytest.mark.gpu


def _engine(kind, nchunks):
    cfg = wl.subset(wl.config2(nfreq=16, ntimes=4), nsrc=2500, nfreq=5, ntimes=2, nant=24, seed=4)
    kw = dict(polarized=True, beam_idx=cfg["beam_idx"], freq_group=2, nchunks=nchunks)
    if kind == "gauss":
        cfg["beams"], kw["polarized"], kw["beam_idx"] = [GaussianBeam(0.2)], False, None
    elif kind == "fits":
        g = cfg["beams"][0]
        data = np.stack([g.data, 0.9 * g.data], axis=2).astype(np.complex128)
        cfg["beams"] = [BeamFits("efield", data, g.az, g.za, np.array([90e6, 210e6]), ["x", "y"])]
        kw["beam_idx"] = None
    elif kind == "polsky":
        cfg["fluxes"] = wl.polarised_sky(cfg)
    elif kind == "erfa":
        kw["astrom"] = wl.synthetic_astrom(cfg["lsts"], cfg["latitude"])
    elif kind in ("vecdot", "herk"):
        kw.update(matprod="VectorDot", pair_product=kind, antpairs=np.array([[0, 1], [3, 3], [20, 7], [5, 23]]))
    return VisEngine(job_from_arrays(ants=cfg["antpos"], fluxes=cfg["fluxes"], ra=cfg["ra"], dec=cfg["dec"],
                                     freqs=cfg["freqs"], lsts=cfg["lsts"], latitude=cfg["latitude"],
                                     beams=cfg["beams"], **kw))


@pytest.mark.parametrize("kind", ["grid", "gauss", "fits", "polsky", "erfa", "vecdot", "herk"])
@pytest.mark.parametrize("nchunks", [1, 3])
def test_whole_time_and_group_calls_agree(kind, nchunks):
    eng = _engine(kind, nchunks)
    whole = eng.run().clone()
    assert whole.abs().max() > 0
    eng.vis.zero_()
    for t in range(len(eng.lsts)):
        eng.enqueue_time(t)
    assert torch.equal(eng.vis, whole)
    eng.vis.zero_()
    assert np.array_equal(eng.run_to_host(), whole.cpu().numpy())


def test_ranges_outside_the_job_are_refused():
    eng = _engine("grid", 1)
    eng.upload()
    job, _keep = eng._launches()
    for bad in ((-1, 1, 0, 1, 0, 5), (0, 3, 0, 1, 0, 5), (0, 2, 0, 2, 0, 5), (0, 2, 0, 1, 0, 6), (0, 2, 0, 1, 1, 5)):
        assert _lib.lib.mvb_job_enqueue(ctypes.byref(job), *bad, _lib.stream_handle()) == _lib.MVB_ERR_ARG

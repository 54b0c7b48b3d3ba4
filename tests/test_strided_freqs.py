"""Frequencies given as a view (every other channel, a column of a table) are the
frequencies of the job: the launch sequence reads them as a dense host array."""

import ctypes

import numpy as np
import pytest
import torch

from matvis_b200 import _lib, workloads as wl
from matvis_b200.beam_models import GaussianBeam
from matvis_b200.beamfits import BeamFits
from matvis_b200.engine import VisEngine, job_from_arrays


def _views(freqs):
    """The same values dense, strided in a longer array, and as a table's column."""
    wide = np.full((len(freqs), 2), 1.5e8)
    wide[:, 0] = freqs
    return dict(dense=freqs, every_other=wide.reshape(-1)[::2], column=wide[:, 0])


def _engine(kind, view, device=None):
    cfg = wl.subset(wl.config2(nfreq=16, ntimes=4), nsrc=2500, nfreq=5, ntimes=2, nant=24, seed=4)
    kw = dict(polarized=True, beam_idx=cfg["beam_idx"])
    if kind == "fits":
        g = cfg["beams"][0]
        data = np.stack([g.data, 0.9 * g.data], axis=2).astype(np.complex128)
        cfg["beams"] = [BeamFits("efield", data, g.az, g.za, np.array([90e6, 210e6]), ["x", "y"])]
        kw["beam_idx"] = None
    elif kind == "vecdot":
        kw.update(matprod="VectorDot", pair_product="vecdot", antpairs=np.array([[0, 1], [3, 3], [20, 7], [5, 23]]))
    elif kind == "gauss":
        cfg["beams"], kw = [GaussianBeam(0.2)], dict(freq_group=1)
    elif kind == "polsky":
        cfg["fluxes"] = wl.polarised_sky(cfg)
        kw["freq_group"] = 1
    else:
        kw["freq_group"] = 1 if kind == "group1" else 2
    freqs = _views(np.array(cfg["freqs"], dtype=np.float64))[view]
    return VisEngine(job_from_arrays(ants=cfg["antpos"], fluxes=cfg["fluxes"], ra=cfg["ra"], dec=cfg["dec"],
                                     freqs=freqs, lsts=cfg["lsts"], latitude=cfg["latitude"], beams=cfg["beams"],
                                     **kw), device=device)


@pytest.mark.parametrize("view", ["dense", "every_other", "column"])
def test_the_launch_sequence_points_at_dense_frequencies(view, monkeypatch):
    """What the native code reads through mvb_job.freqs, without a GPU."""
    monkeypatch.setattr(_lib, "require_cuda", lambda device=None: torch.device("cpu"))
    eng = _engine("gauss", view)
    eng.allocate()
    job, _keep = eng._launches()
    read = np.ctypeslib.as_array(ctypes.cast(job.freqs, ctypes.POINTER(ctypes.c_double)), (job.nfreq,))
    assert np.array_equal(read, np.asarray(eng.spec.freqs))


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["group1", "group2", "gauss", "fits", "vecdot", "polsky"])
def test_views_give_the_visibilities_of_a_dense_array(kind):
    want = _engine(kind, "dense").run().clone()
    assert want.abs().max() > 0
    for view in ("every_other", "column"):
        assert torch.equal(_engine(kind, view).run(), want), view
        assert np.array_equal(_engine(kind, view).run_to_host(), want.cpu().numpy()), view

"""Launches whose sources do not fill the GPU give each CTA a slice of the beams: every
slicing, an uneven one and one of whole lists among them, gives each beam's own result."""

import numpy as np
import pytest
import torch

import matvis_b200 as mv
from matvis_b200 import _lib, workloads

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


# 157 source blocks: 4 slices; 3 blocks: a beam each; 782: one slice
@pytest.mark.parametrize("nout", [300, 20000, 100000])
@pytest.mark.parametrize("polarized,nbeam", [(True, 7), (False, 9), (False, 30)])
def test_every_beam_is_its_own(polarized, nbeam, nout):
    rng = np.random.default_rng(nbeam)
    beams = workloads.dipole_beams(rng, nbeam, dgrid_deg=10.0)
    z, ph = rng.uniform(0, 1, nout), rng.uniform(0, 2 * np.pi, nout)
    crd = torch.as_tensor(np.stack([np.sqrt(1 - z * z) * np.cos(ph), np.sqrt(1 - z * z) * np.sin(ph)]), device=DEV)

    def interp(bl):
        bi = mv.B200BeamInterpolator(beam_list=bl, beam_idx=np.zeros(len(bl), int), polarized=polarized, nant=len(bl),
                                     freq=1e8, nsrc=nout)
        bi.setup()
        out = torch.full((len(bl), bi.nfeed, bi.nax, nout), 7.0, dtype=torch.complex64, device=DEV)
        _lib.check(_lib.lib.mvb_beam_interp(
            _lib.ptr(bi.grids), bi.grid_kind, bi.nbeam, bi.nax, bi.nfeed, bi.nza, bi.naz, _lib.ptr(bi.params),
            _lib.ptr(crd), nout, None, nout, _lib.ptr(out), 0, nout, None, None, 0, _lib.stream_handle()))
        return out

    every = interp(beams)
    for b, beam in enumerate(beams):
        assert torch.equal(every[b:b + 1], interp([beam])), b

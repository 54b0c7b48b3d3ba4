"""Beam gathers at the edges of their dispatch: packed and plane-by-plane grids,
power and complex grids, slots past the count, outputs off their alignment, and
positions on the grid's border and outside it, against the FP64 oracle."""

import numpy as np
import pytest
import torch

import matvis_b200 as mv
from matvis_b200 import _lib, workloads
from oracle import oracle as orc

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _launch(bi, crd, ld, n_dev, out, nout, ws, out_ptr=None):
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    _lib.check(_lib.lib.mvb_beam_interp(
        _lib.ptr(bi.grids), bi.grid_kind, bi.nbeam, bi.nax, bi.nfeed, bi.nza, bi.naz, _lib.ptr(bi.params),
        _lib.ptr(crd), ld, _lib.ptr(n_dev), nout, _lib.ptr(out) if out_ptr is None else out_ptr,
        1 if out.dtype in (torch.complex128, torch.float64) else 0, nout, _lib.ptr(status), _lib.ptr(ws),
        0 if ws is None else ws.numel() * 8, _lib.stream_handle()))
    return int(status.item())


# 10-degree grids (10 x 37 points) pack from 300,740 slot-beams on; 1-degree ones (91 x 361) from 365,702 slots
@pytest.mark.parametrize("polarized,dgrid,nbeam,nout", [
    (True, 10.0, 1, 1), (True, 10.0, 4, 75924), (True, 10.0, 4, 75927), (True, 10.0, 1, 300741), (True, 1.0, 1, 365703),
    (False, 10.0, 3, 129), (False, 1.0, 1, 400001)])
@pytest.mark.parametrize("c128", [False, True])
def test_gather_forms_match_oracle(polarized, dgrid, nbeam, nout, c128):
    rng = np.random.default_rng(nout)
    beams = workloads.dipole_beams(rng, nbeam, dgrid_deg=dgrid)
    bi = mv.B200BeamInterpolator(beam_list=beams, beam_idx=np.zeros(nbeam, int), polarized=polarized, nant=nbeam,
                                 freq=1e8, nsrc=nout, precision=2 if c128 else 1)
    bi.setup()
    n = max(nout - 5, 1)
    z, ph = rng.uniform(0, 1, nout), rng.uniform(0, 2 * np.pi, nout)
    e, nn = np.sqrt(1 - z * z) * np.cos(ph), np.sqrt(1 - z * z) * np.sin(ph)
    # zenith, the horizon, azimuth 0 and just below 360 degrees
    e[:1], nn[:1] = 0.0, 0.0
    if nout > 4:
        e[1:4], nn[1:4] = (1.0, 1.0 - 1e-12, 0.5), (0.0, -1e-9, 0.0)
    crd = torch.as_tensor(np.stack([e, nn]), device=DEV).contiguous()
    n_dev = torch.tensor([n], dtype=torch.int32, device=DEV)
    ws = torch.empty(2 * nbeam * nout, dtype=torch.float64, device=DEV)
    dt = torch.complex128 if c128 else torch.complex64
    F = bi.nfeed
    planes = torch.full((nbeam, F, F, nout), 7.0 + 7.0j, dtype=dt, device=DEV)
    with_ws = torch.full_like(planes, 7.0 + 7.0j)
    assert _launch(bi, crd, nout, n_dev, planes, nout, None) == 0
    assert _launch(bi, crd, nout, n_dev, with_ws, nout, ws) == 0
    assert torch.equal(planes, with_ws)
    assert (with_ws[..., n:] == 0).all()
    # an output that is aligned to its real type only
    real = torch.float64 if c128 else torch.float32
    flat = torch.full((planes.numel() * 2 + 1,), 7.0, dtype=real, device=DEV)
    assert _launch(bi, crd, nout, n_dev, flat, nout, ws, out_ptr=flat.data_ptr() + flat.element_size()) == 0
    assert torch.equal(flat[1:].view(-1, 2), torch.view_as_real(with_ws).reshape(-1, 2))
    ob = [orc.GridBeam(data=b.data.astype(np.complex128), az=b.az, za=b.za) for b in beams]
    ref = orc.beam_response(ob, polarized, e[:n], nn[:n])
    # grids are stored in 32 bits: two roundings of values of at most 1.1
    np.testing.assert_allclose(with_ws[..., :n].cpu().numpy(), ref, rtol=0, atol=1e-6)


@pytest.mark.parametrize("nout", [40, 80000])
def test_nonfinite_grid_is_reported(nout):
    rng = np.random.default_rng(3)
    beams = workloads.dipole_beams(rng, 4, dgrid_deg=10.0)
    beams[2].data[1, 0, 3, 5] = np.nan
    bi = mv.B200BeamInterpolator(beam_list=beams, beam_idx=np.zeros(4, int), polarized=True, nant=4, freq=1e8,
                                 nsrc=nout)
    bi.setup()
    za, az = np.deg2rad(30.0), np.deg2rad(50.0)  # the grid point itself, in uvbeam azimuth
    e = np.full(nout, np.sin(za) * np.cos(az))
    nn = np.full(nout, np.sin(za) * np.sin(az))
    crd = torch.as_tensor(np.stack([e, nn]), device=DEV).contiguous()
    out = torch.zeros((4, 2, 2, nout), dtype=torch.complex64, device=DEV)
    ws = torch.empty(8 * nout, dtype=torch.float64, device=DEV)
    n_dev = torch.tensor([nout], dtype=torch.int32, device=DEV)
    assert _launch(bi, crd, nout, n_dev, out, nout, ws) == _lib.MVB_DEV_NONFINITE

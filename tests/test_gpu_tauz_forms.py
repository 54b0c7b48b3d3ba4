"""The fused phase / Z writer at the edges of its launch shapes: each frequency of
a grouped launch equals the single-frequency launch bit for bit, columns past the
source count are zero, rows past the antennas are left alone, and the plain
complex64 panel agrees with FP64."""

import numpy as np
import pytest
import torch

from matvis_b200 import _lib

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _inputs(rng, A, F, X, n, cap, nf, nbeam):
    v = rng.normal(size=(3, cap))
    v /= np.linalg.norm(v, axis=0)
    return dict(ant=rng.uniform(-500, 500, (A, 3)), crd=v, freqs=rng.uniform(1e8, 2e8, nf),
                sflux=rng.uniform(0.1, 3, (nf, 2 * cap)).astype(np.float32),
                sidx=np.sort(rng.choice(2 * cap, cap, replace=False)).astype(np.int32),
                beam=(rng.normal(size=(nbeam, F, X, cap)) + 1j * rng.normal(size=(nbeam, F, X, cap))).astype(np.complex64),
                bidx=rng.integers(0, nbeam, A).astype(np.int32))


# counts around the 64-column CTAs, the 16-antenna lanes, 64-antenna blocks and the 8
# frequencies of a CTA; 9 and 20 beams do not fit the staged planes
@pytest.mark.parametrize("A,F,X,n,cap,nf,nbeam", [
    (1, 1, 1, 1, 1, 1, 1), (15, 1, 1, 63, 65, 9, 2), (17, 1, 1, 64, 200, 8, 1), (65, 2, 2, 33, 40, 3, 4),
    (64, 2, 2, 32, 32, 17, 1), (130, 1, 2, 97, 130, 2, 3), (129, 2, 1, 200, 333, 5, 20), (20, 2, 2, 0, 10, 4, 9),
    (70, 2, 2, 5000, 9000, 8, 4), (300, 1, 1, 20000, 20000, 8, 1)])
@pytest.mark.parametrize("mode", [_lib.Z_C64, _lib.GEMM_F16_3, _lib.GEMM_BF16_6, _lib.GEMM_TF32_3])
def test_grouped_launch_equals_single(A, F, X, n, cap, nf, nbeam, mode):
    rng = np.random.default_rng(A + n)
    h = _inputs(rng, A, F, X, n, cap, nf, nbeam)
    d = {k: torch.as_tensor(v, device=DEV).contiguous() for k, v in h.items()}
    n_dev = torch.tensor([n], dtype=torch.int32, device=DEV)
    mpad, kcap = _lib.zpanel_shape(mode, A * F, cap * X)
    nbytes = _lib.lib.mvb_zpanel_bytes(mode, mpad, kcap)
    scale = 16.0 if mode == _lib.GEMM_F16_3 else 1.0
    group = torch.full((nf, nbytes), 171, dtype=torch.uint8, device=DEV)
    one = torch.full((nf, nbytes), 171, dtype=torch.uint8, device=DEV)
    P = _lib.ptr
    _lib.check(_lib.lib.mvb_tau_z_grouped(
        P(d["ant"]), A, P(d["freqs"]), nf, P(d["crd"]), cap, P(n_dev), cap, P(d["sflux"]), 2 * cap, P(d["sidx"]),
        P(d["beam"]), cap, nbeam, P(d["bidx"]), F, X, mode, scale, P(group), nbytes, mpad, kcap, _lib.stream_handle()))
    for f in range(nf):
        _lib.check(_lib.lib.mvb_tau_z(
            P(d["ant"]), A, float(h["freqs"][f]), P(d["crd"]), cap, P(n_dev), cap, P(d["sflux"][f]), P(d["sidx"]),
            P(d["beam"]), cap, nbeam, P(d["bidx"]), F, X, mode, scale, P(one[f]), mpad, kcap, _lib.stream_handle()))
    assert torch.equal(group, one)
    if mode != _lib.Z_C64:
        return
    z = group.view(torch.complex64).reshape(nf, A * F, kcap).cpu().numpy()
    live = -(-n * X // 64) * 64
    assert (z[:, :, n * X:live] == 0).all()
    tau = (h["ant"] @ h["crd"][:, :n])[None] * (h["freqs"] / 299792458.0)[:, None, None]
    ext = np.exp(2j * np.pi * (tau - np.rint(tau)))
    fl = h["sflux"][:, h["sidx"][:n]].astype(np.float64)
    ref = np.einsum("gan,gn,afxn->gafnx", ext, fl, h["beam"][h["bidx"], :, :, :n].astype(np.complex128))
    # phase rounded to FP32 (pi 2^-24 of a turn), sincos, two products: under 8 units of 2^-24
    np.testing.assert_allclose(z[:, :, :n * X].reshape(nf, A, F, n, X), ref, rtol=0,
                               atol=8 * 2.0**-24 * max(np.abs(ref).max(initial=0.0), 1.0))

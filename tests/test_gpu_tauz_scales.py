"""The split panels of the fused phase / Z writer against FP64: the panel's scale is
divided between the beam and the sky inside the writer, so every sign and parity of its
exponent and a scale that is not a power of two are decoded and compared."""

import numpy as np
import pytest
import torch

from matvis_b200 import _lib
from matvis_b200.getz import ZPanel

pytestmark = pytest.mark.gpu
C = 299792458.0


def _ext(ant, crd, freqs):
    tau = (ant @ crd)[None] * (freqs / C)[:, None, None]
    return np.exp(2j * np.pi * (tau - np.rint(tau)))


def _factor(coh, ang):
    """(nf, n, 2, 2): lower L of R^T C R = L L^H, from (C00, C11, Re C01, Im C01)."""
    c01 = coh[..., 2] + 1j * coh[..., 3]
    m = np.stack([np.stack([coh[..., 0] + 0j, c01], -1), np.stack([c01.conj(), coh[..., 1] + 0j], -1)], -2)
    r = np.stack([np.stack([np.cos(ang), np.sin(ang)], -1), np.stack([-np.sin(ang), np.cos(ang)], -1)], -2)
    return np.linalg.cholesky(np.swapaxes(r, -1, -2) @ m @ r)


# counts off the CTA's 64 columns; more frequencies than a CTA takes; 20 beams are not staged
@pytest.mark.parametrize("A,F,X,n,cap,nf,nbeam,pol", [
    (17, 1, 1, 63, 70, 9, 2, False), (20, 2, 2, 33, 40, 3, 4, False), (5, 2, 1, 97, 120, 8, 20, False),
    (6, 1, 2, 31, 31, 1, 1, False), (20, 2, 2, 33, 40, 9, 4, True), (3, 2, 2, 95, 130, 1, 20, True)])
@pytest.mark.parametrize("mode,scale", [(_lib.GEMM_F16_3, s) for s in (2.0**-7, 2.0**5, 2.0**-49, 2.0**50, 12.0)] +
                         [(_lib.GEMM_F16_3, s) for s in (2.0**-100, 2.0**100)] +
                         [(_lib.GEMM_TF32_3, 1.0), (_lib.GEMM_BF16_6, 1.0)])
def test_split_panels_decode_to_fp64(A, F, X, n, cap, nf, nbeam, pol, mode, scale):
    if pol and not 2.0**-60 < scale < 2.0**60:
        pytest.skip("the coherency is the square: outside FP32")
    rng = np.random.default_rng(n + nf)
    dev, P, L = "cuda:0", _lib.ptr, _lib.lib
    up = lambda a: torch.as_tensor(a, device=dev).contiguous()
    crd = rng.normal(size=(3, cap))
    crd /= np.linalg.norm(crd, axis=0)
    ant, freqs = rng.uniform(-300, 300, (A, 3)), rng.uniform(1e8, 2e8, nf)
    beam = (rng.normal(size=(nbeam, F, X, cap)) + 1j * rng.normal(size=(nbeam, F, X, cap))).astype(np.complex64)
    bidx = rng.integers(0, nbeam, A).astype(np.int32)
    amp = 2.0**10 / scale  # |s Z| stays below 2^15: |beam| < 6, |L| < 2 amp
    panels = ZPanel.group(nf, mode, A, F, X, cap, dev)
    p0, n_dev = panels[0], torch.tensor([n], dtype=torch.int32, device=dev)
    d = [up(ant), up(freqs), up(crd), up(beam), up(bidx)]
    if pol:
        coh = (amp**2 * np.concatenate([rng.uniform(1, 2, (nf, cap, 2)), rng.uniform(-0.4, 0.4, (nf, cap, 2))], -1)
               ).astype(np.float32)
        ang = rng.uniform(0, 2 * np.pi, cap)
        dc, dr = up(coh), up(np.stack([np.cos(ang), np.sin(ang)], axis=1))
        _lib.check(L.mvb_tau_z_pol_grouped(P(d[0]), A, P(d[1]), nf, P(d[2]), cap, P(n_dev), cap, P(dc), cap, None, P(dr),
                                           P(d[3]), cap, nbeam, P(d[4]), mode, scale, P(p0.data), p0.nbytes, p0.Mpad,
                                           p0.Kcap, _lib.stream_handle()))
        lower = _factor(coh[:, :n].astype(np.float64), ang[:n])
    else:
        flux = (amp * rng.uniform(0.1, 2, (nf, cap))).astype(np.float32)
        df = up(flux)
        _lib.check(L.mvb_tau_z_grouped(P(d[0]), A, P(d[1]), nf, P(d[2]), cap, P(n_dev), cap, P(df), cap, None, P(d[3]),
                                       cap, nbeam, P(d[4]), F, X, mode, scale, P(p0.data), p0.nbytes, p0.Mpad, p0.Kcap,
                                       _lib.stream_handle()))
    b = beam[bidx][..., :n].astype(np.complex128)
    ext = _ext(ant, crd[:, :n], freqs)
    if pol:
        ref = np.einsum("gan,afxn,gnxy->gafny", ext, b, lower)
    else:
        ref = np.einsum("gan,gn,afxn->gafnx", ext, flux[:, :n].astype(np.float64), b)
    ref = ref.reshape(nf, A * F, n * X)
    assert np.abs(ref).max() * scale < 2.0**15
    # units of 2^-24 of the largest value: phase, sincos and products 8, the factor and its
    # second product 4, the split (22 bits or more) 4
    tol = 16 * 2.0**-24 * np.abs(ref).max()
    for g, panel in enumerate(panels):
        panel.n_host, panel.scale = n, scale if mode == _lib.GEMM_F16_3 else 1.0
        np.testing.assert_allclose(panel.to_complex().cpu().numpy(), ref[g], rtol=0, atol=tol)

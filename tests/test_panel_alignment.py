"""Panels that are not aligned to the writers' widest stores: a panel or a spacing of
panels aligned to the narrow stores holds the same bytes as an aligned one, and less
than that is refused on the host."""

import ctypes

import numpy as np
import pytest
import torch

from matvis_b200 import _lib

#: mode -> bytes of the narrowest store of the phase / Z writer
NARROW = {_lib.Z_C64: 16, _lib.GEMM_F16_3: 8, _lib.GEMM_BF16_3: 8, _lib.GEMM_BF16_6: 8, _lib.GEMM_TF32_3: 16}


def _shape(mode, rows, cols):
    mpad, kcap = _lib.zpanel_shape(mode, rows, cols)
    return mpad, kcap, _lib.lib.mvb_zpanel_bytes(mode, mpad, kcap)


@pytest.mark.parametrize("mode", sorted(NARROW))
@pytest.mark.parametrize("X", [1, 2])
def test_panels_below_the_narrow_stores_are_refused(mode, X):
    """On the host, before any CUDA call (every call here is refused)."""
    fake = ctypes.c_void_p(4096)
    A, n, L = 5, 100, _lib.lib
    mpad, kcap, nbytes = _shape(mode, A * X, n * X)
    bad = ctypes.c_void_p(4096 + NARROW[mode] // 2)
    calls = {
        "mvb_tau_z": (fake, A, 1e8, fake, n, None, n, fake, None, fake, n, 1, None, X, X, mode, 1.0, bad, mpad, kcap,
                      None),
        "mvb_tau_z_grouped": (fake, A, fake, 2, fake, n, None, n, fake, n, None, fake, n, 1, None, X, X, mode, 1.0,
                              bad, nbytes, mpad, kcap, None),
        "mvb_z_from_exptau": (fake, 0, n, A, n, fake, fake, n, 1, None, X, X, mode, 1.0, bad, mpad, kcap, None),
    }
    if X == 2:
        calls["mvb_tau_z_pol"] = (fake, A, 1e8, fake, n, None, n, fake, None, fake, fake, n, 1, None, mode, 1.0, bad,
                                  mpad, kcap, None)
    for name, args in calls.items():
        assert getattr(L, name)(*args) == _lib.MVB_ERR_ARG, name
        assert L.mvb_last_error().decode().startswith(name + ":")
    # the pair-wide stores of the packing and the sector stores of the exptau writer
    low = {_lib.Z_C64: 8, _lib.GEMM_TF32_3: 4, _lib.GEMM_F16_3: 1}.get(mode, 2)
    assert L.mvb_z_pack(fake, 0, A * X, n, n, mode, 1.0, ctypes.c_void_p(4096 + low), mpad, kcap, None) == _lib.MVB_ERR_ARG
    if mode == _lib.Z_C64 or (mode == _lib.GEMM_TF32_3 and X == 2):
        args = list(calls["mvb_z_from_exptau"])
        args[14] = ctypes.c_void_p(4096 + 16)
        assert L.mvb_z_from_exptau(*args) == _lib.MVB_ERR_ARG


@pytest.mark.gpu
@pytest.mark.parametrize("F,X,pol", [(1, 1, False), (2, 1, False), (2, 2, False), (2, 2, True)])
@pytest.mark.parametrize("mode", sorted(NARROW))
def test_narrow_panels_hold_the_aligned_bytes(mode, F, X, pol):
    rng = np.random.default_rng(5)
    dev, P, L = "cuda:0", _lib.ptr, _lib.lib
    A, cap, n, nf, nbeam = 21, 150, 133, 3, 2
    mpad, kcap, nbytes = _shape(mode, A * F, cap * X)
    up = lambda a: torch.as_tensor(a, device=dev).contiguous()
    crd = rng.normal(size=(3, cap))
    ant, crd = up(rng.uniform(-300, 300, (A, 3))), up(crd / np.linalg.norm(crd, axis=0))
    freqs = up(rng.uniform(1e8, 2e8, nf))
    beam = up((rng.normal(size=(nbeam, F, X, cap)) + 1j * rng.normal(size=(nbeam, F, X, cap))).astype(np.complex64))
    bidx = up(rng.integers(0, nbeam, A).astype(np.int32))
    n_dev = torch.tensor([n], dtype=torch.int32, device=dev)
    if pol:
        amp = rng.uniform(1, 2, (nf, cap, 4))
        amp[..., 2:] *= 0.3
        sky, ang = up(amp.astype(np.float32)), rng.uniform(0, 6, cap)
        rot = up(np.stack([np.cos(ang), np.sin(ang)], axis=1))
    else:
        sky = up(rng.uniform(0.1, 3, (nf, cap)).astype(np.float32))

    def write(base, stride):
        buf = torch.full((base + nf * stride,), 171, dtype=torch.uint8, device=dev)
        z = ctypes.c_void_p(buf.data_ptr() + base)
        if pol:
            rc = L.mvb_tau_z_pol_grouped(P(ant), A, P(freqs), nf, P(crd), cap, P(n_dev), cap, P(sky), cap, None, P(rot),
                                         P(beam), cap, nbeam, P(bidx), mode, 8.0, z, stride, mpad, kcap,
                                         _lib.stream_handle())
        else:
            rc = L.mvb_tau_z_grouped(P(ant), A, P(freqs), nf, P(crd), cap, P(n_dev), cap, P(sky), cap, None, P(beam),
                                     cap, nbeam, P(bidx), F, X, mode, 8.0, z, stride, mpad, kcap,
                                     _lib.stream_handle())
        _lib.check(rc)
        torch.cuda.synchronize()
        assert (buf[:base] == 171).all()
        rows = buf[base:].reshape(nf, stride)
        assert (rows[:, nbytes:] == 171).all()
        return rows[:, :nbytes].contiguous()

    want = write(0, nbytes)
    assert not (want == 171).all()
    for base, stride in ((NARROW[mode], nbytes), (0, nbytes + 16), (16, nbytes + 16)):
        assert torch.equal(write(base, stride), want), (base, stride)

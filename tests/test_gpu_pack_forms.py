"""Packing a caller's Z: the same panel whatever the alignment and pitch of the
source and the panel, zero columns up to the 64-column granule, values within the
split's precision, and the device-chosen fp16 scale equal to the host's rule."""

import numpy as np
import pytest
import torch

import matvis_b200 as mv
from matvis_b200 import _lib
from matvis_b200.getz import ZPanel

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
# relative error of the split: 2 fp16 terms 2^-22, 2 bf16 2^-16, 3 bf16 2^-24, 2 tf32 2^-22; FP32 source rounding 2^-24
REL = {_lib.GEMM_F16_3: 2.0**-21, _lib.GEMM_BF16_3: 2.0**-15, _lib.GEMM_BF16_6: 2.0**-22, _lib.GEMM_TF32_3: 2.0**-21,
       _lib.Z_C64: 2.0**-23}


@pytest.mark.parametrize("M,K", [(1, 1), (3, 65), (16, 128), (17, 127), (65, 640), (130, 1025), (2000, 40000)])
@pytest.mark.parametrize("c128", [False, True])
@pytest.mark.parametrize("mode", sorted(REL))
def test_pack_forms_agree(M, K, c128, mode):
    if M * K > 1e7 and mode not in (_lib.GEMM_F16_3, _lib.GEMM_TF32_3):
        pytest.skip("the large shape is for the four-row blocks, checked in two modes")
    gen = torch.Generator(device=DEV).manual_seed(M + K)
    dt = torch.complex128 if c128 else torch.complex64
    z = torch.randn((M, K), dtype=dt, device=DEV, generator=gen)
    odd = torch.randn((M * (K + 3) + 1,), dtype=dt, device=DEV, generator=gen)
    pitched = odd[1:].view(M, K + 3)
    pitched[:, :K] = z
    mpad, kcap = _lib.zpanel_shape(mode, M, K)
    nbytes = _lib.lib.mvb_zpanel_bytes(mode, mpad, kcap)
    scale = 4.0 if mode == _lib.GEMM_F16_3 else 1.0
    outs = []
    shifts = (0, 16) if mode == _lib.Z_C64 else (0, 16, 8)
    for src, ld in ((z, K), (pitched, K + 3)):
        for shift in shifts:
            buf = torch.zeros(nbytes + 64, dtype=torch.uint8, device=DEV)
            _lib.check(_lib.lib.mvb_z_pack(_lib.ptr(src), int(c128), M, K, ld, mode, scale, buf.data_ptr() + shift,
                                           mpad, kcap, _lib.stream_handle()))
            outs.append(buf[shift:shift + nbytes])
    assert all(torch.equal(outs[0], o) for o in outs[1:])
    data = outs[0].view(_lib.zpanel_dtype(mode)).view(ZPanel.data_shape(mode, M, mpad, kcap))
    panel = ZPanel(mode, M, 1, 1, kcap, DEV, data=data)
    panel.scale, panel.n_host = scale, -(-K // 64) * 64
    got = panel.to_complex()
    assert (got[:, K:] == 0).all()
    err = (got[:, :K] - z.to(torch.complex128)).abs().max().item()
    assert err <= 2 * REL[mode] * z.abs().max().item()  # both components


@pytest.mark.parametrize("value", [0.0, 1e-30, 3e-5, 1.0, 16368.0, 16384.0, 7e20, np.inf])
def test_device_scale_is_the_host_rule(value):
    z = torch.zeros((5, 70), dtype=torch.complex64, device=DEV)
    z[3, 69] = value
    mp = mv.B200MatMul(1, 1, 5, None, precision=2)
    mp.setup()
    panel = mp._as_panel(z, mp.mode)
    mx = float(torch.tensor(value, dtype=torch.float32))
    assert panel.scale == _lib.f16_scale(mx * (1 + 2**-10))
    if np.isfinite(value):
        out = mp(z, 0).cpu().numpy().reshape(5, 5)
        # two fp16 terms of one value: 2^-22 of it, squared
        assert abs(out[3, 3] - mx * mx) <= 2.0**-20 * mx * mx and np.count_nonzero(out) <= 1

"""The product with its live rows stated, around the line where the last block is
taken as 64 rows: small-integer Z, exact in every mode's steps, so the visibilities
are the integer result bit for bit (and those of the form without stated rows).  The
workspace starts as NaN: what the product does not write must not be read."""

import numpy as np
import pytest
import torch

import matvis_b200 as mv
from matvis_b200 import _lib
from matvis_b200._lib import check, ptr, stream_handle

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("m", [1, 32, 33, 64, 90, 97, 129, 160, 192, 193, 224, 225, 320])
@pytest.mark.parametrize("mode", ["bf16x3", "bf16x6", "tf32x3", "fp16x3"])
@pytest.mark.parametrize("ncol,k_chunk,drain", [(70, 64, 0), (1111, 128, 0), (640, 640, 1), (640, 256, 4)])
def test_stated_rows_are_exact(m, mode, ncol, k_chunk, drain):
    rng = np.random.default_rng(m + ncol)
    z = rng.integers(-8, 9, (2, m, ncol)) + 1j * rng.integers(-8, 9, (2, m, ncol))
    mp = mv.B200MatMul(1, 1, m, None, precision=1, gemm_mode=mode, k_chunk=k_chunk, drain_ksteps=drain)
    mp.setup()
    for zi in z:
        panel = mp._as_panel(torch.as_tensor(zi, device=DEV), mp.mode)
        mp.workspace(panel, k_chunk).fill_(255)  # a NaN in every word
        out = torch.empty(m * m, 1, 1, dtype=torch.complex64, device=DEV)
        mp.enqueue(panel, out)
        # |sums| <= 2 x 64 x 1,111 < 2^24: exact in FP32
        assert np.array_equal(out.cpu().numpy().reshape(m, m), zi.conj() @ zi.T)
        ws = mp.workspace(panel, k_chunk)
        check(_lib.lib.mvb_herk_grouped(ptr(panel.data), 0, 1, mp.mode, panel.Mpad, panel.Kcap, None, panel.n_host,
                                        panel.nax, k_chunk, drain, ptr(ws), ws.numel(), ptr(mp.status),
                                        stream_handle()))
        full = torch.empty_like(out)
        mp.reduce_grouped([panel], full[None], k_chunk=k_chunk)
        assert np.array_equal(full.cpu().numpy(), out.cpu().numpy())

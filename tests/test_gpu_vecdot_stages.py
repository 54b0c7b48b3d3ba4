"""The staged pair kernel at the edges of its stages (16, 8 or 4 columns, by the number
of rows), whole and partial, one and several units a CTA: small-integer Z, whose sums
are exact, so the visibilities equal the integer result bit for bit."""

import numpy as np
import pytest
import torch

import matvis_b200 as mv
from matvis_b200 import _lib

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("nant,nfeed,kb", [(9, 1, 16), (40, 2, 16), (350, 2, 16), (500, 2, 8), (1000, 2, 4)])
@pytest.mark.parametrize("ncol", [1, 2, 15, 16, 17, 33, 64, 2391, 2400])
def test_staged_pairs_are_exact(nant, nfeed, kb, ncol):
    assert _lib.lib.mvb_vecdot_stage_columns(nant, nfeed) == kb
    rng = np.random.default_rng(nant + ncol)
    m = nant * nfeed
    z = rng.integers(-8, 9, (m, ncol)) + 1j * rng.integers(-8, 9, (m, ncol))
    pairs = rng.integers(0, nant, (1500, 2))
    mp = mv.B200VectorDot(1, nfeed, nant, pairs, precision=1)
    mp.setup()
    out = mp(torch.as_tensor(z, device=DEV).to(torch.complex64), 0).cpu().numpy()
    zf = z.reshape(nant, nfeed, ncol)
    # |sums| <= 2 x 64 x 2,400 < 2^24: exact in FP32
    ref = np.einsum("nqk,npk->npq", zf[pairs[:, 0]].conj(), zf[pairs[:, 1]])
    assert np.array_equal(out, ref)

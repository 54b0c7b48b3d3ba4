"""The product's reduction at the edges of its 32 x 32 blocks and slice batches:
small-integer Z, whose products and sums are exact in every step, so the
visibilities equal the integer result bit for bit."""

import numpy as np
import pytest
import torch

import matvis_b200 as mv

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("nant,nfeed", [(1, 1), (31, 1), (33, 1), (64, 1), (97, 1), (129, 1), (16, 2), (17, 2), (65, 2),
                                        (80, 2), (143, 2)])
@pytest.mark.parametrize("ncol,k_chunk", [(64, 64), (640, 64), (1111, 128)])
@pytest.mark.parametrize("precision", [1, 2])
def test_reduction_blocks_are_exact(nant, nfeed, ncol, k_chunk, precision):
    rng = np.random.default_rng(nant * 7 + ncol)
    m = nant * nfeed
    z = rng.integers(-8, 9, (m, ncol)) + 1j * rng.integers(-8, 9, (m, ncol))
    g = (z.conj() @ z.T).reshape(nant, nfeed, nant, nfeed).transpose(0, 2, 3, 1).reshape(-1, nfeed, nfeed)
    mp = mv.B200MatMul(1, nfeed, nant, None, precision=precision, gemm_mode="fp16x3", k_chunk=k_chunk)
    mp.setup()
    out = mp(torch.as_tensor(z, device=DEV), 0)
    # |sums| <= 2 x 64 x 1,111 < 2^24: exact in FP32
    assert np.array_equal(out.cpu().numpy(), g)
    mp.enqueue(mp._as_panel(torch.as_tensor(z, device=DEV), mp.mode), out, accumulate=True)
    assert np.array_equal(out.cpu().numpy(), 2 * g)
    pairs = rng.integers(0, nant, (min(50, nant * nant), 2))
    mq = mv.B200MatMul(1, nfeed, nant, pairs, precision=precision, gemm_mode="fp16x3", k_chunk=k_chunk)
    mq.setup()
    some = mq(torch.as_tensor(z, device=DEV), 0)
    assert np.array_equal(some.cpu().numpy(), g.reshape(nant, nant, nfeed, nfeed)[pairs[:, 0], pairs[:, 1]])

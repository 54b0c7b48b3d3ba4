"""The horizon selection around the edges of its warps (128 sources) and blocks (1,024),
from an offset, with and without fluxes, and with fewer slots than sources above the
horizon: the kept sources in order, the count and the overflow bit."""

import numpy as np
import pytest
import torch

from matvis_b200 import _lib

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("count", [0, 1, 31, 32, 127, 128, 129, 1023, 1024, 1025, 5000])
@pytest.mark.parametrize("kind", ["mixed", "all", "none"])
@pytest.mark.parametrize("short", [False, True])
def test_selection(count, kind, short):
    rng = np.random.default_rng(count)
    c0, ld = 7, count + 20
    topo = rng.normal(size=(3, ld))
    topo[2] = {"mixed": topo[2], "all": np.abs(topo[2]) + 1e-3, "none": -np.abs(topo[2])}[kind]
    topo[2, c0:c0 + count:9] = 0.0  # on the horizon: not kept
    flux = rng.normal(size=ld)
    want = c0 + np.nonzero(topo[2, c0:c0 + count] > 0)[0]
    cap = max(len(want) - 3, 1) if short else len(want) + 5
    t, f = torch.as_tensor(topo, device=DEV), torch.as_tensor(flux, device=DEV)
    crd = torch.full((3, cap), 9.0, dtype=torch.float64, device=DEV)
    idx = torch.full((cap,), -1, dtype=torch.int32, device=DEV)
    fo = torch.full((cap,), 9.0, dtype=torch.float64, device=DEV)
    n, status = (torch.zeros(1, dtype=torch.int32, device=DEV) for _ in range(2))
    ws = torch.empty(max(_lib.lib.mvb_horizon_ws_bytes(count), 8), dtype=torch.uint8, device=DEV)
    P = _lib.ptr
    for with_flux in (True, False):
        _lib.check(_lib.lib.mvb_horizon_compact(P(t), ld, c0, c0 + count, P(f) if with_flux else None, P(crd), P(idx),
                                                P(fo) if with_flux else None, P(n), cap, P(status), P(ws), ws.numel(),
                                                _lib.stream_handle()))
        m = min(len(want), cap)
        assert int(n.item()) == len(want)
        assert int(status.item()) == (_lib.MVB_DEV_OVERFLOW if len(want) > cap else 0)
        assert np.array_equal(idx.cpu().numpy()[:m], want[:m]) and (idx[m:] == -1).all()
        assert np.array_equal(crd.cpu().numpy()[:, :m], topo[:, want[:m]]) and (crd[:, m:] == 9.0).all()
        if with_flux:
            assert np.array_equal(fo.cpu().numpy(), np.concatenate([flux[want[:m]], np.zeros(cap - m)]))

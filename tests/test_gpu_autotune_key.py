"""A tuned (k_chunk, drain interval) belongs to one form of the product: panels of one
padded size whose last blocks are of different widths are tuned apart."""

import pytest
import torch

from matvis_b200 import _lib, autotune
from matvis_b200.getz import ZPanel

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _own_cache(monkeypatch):
    monkeypatch.setattr(autotune, "_cache", {})


@pytest.mark.parametrize("with_run", [True, False])
def test_last_block_widths_are_tuned_apart(with_run):
    dev, mode, K = torch.device("cuda", 0), _lib.GEMM_F16_3, 2048
    status = torch.zeros(1, dtype=torch.int32, device=dev)
    timed = []
    run = (lambda kc, kd, st: timed.append((kc, kd))) if with_run else None
    for i, rows in enumerate((40, 90, 128)):  # last blocks of 64, 96 and 128 columns
        panel = ZPanel(mode, rows, 1, 1, K, dev)
        panel.n_host = K
        assert panel.Mpad == 128 and autotune.cached_choice(mode, 128, K, 0, rows=rows) is None
        n = len(timed)
        got = autotune.tune_product(panel, mode, status, run=run, kd_candidates=(2,))
        assert len(autotune._cache) == i + 1 and (not with_run or len(timed) > n)
        assert autotune.cached_choice(mode, 128, K, 0, rows=rows) == got
    assert autotune.cached_choice(mode, 128, K, 0) == got  # no rows given: a full last block
    assert autotune.cached_choice(mode, 128, K, 0, rows=50) is not None  # 64 columns as well
    assert int(status.item()) == 0

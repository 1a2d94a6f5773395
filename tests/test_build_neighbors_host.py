"""Any cut-off reaches the engine's neighbour build: the row capacity tried first stays finite.  No GPU: the
library is a stand-in that records the capacity."""
import types

import numpy as np
import pytest
import torch

from dmff_b200.engine import AdmpEngine


@pytest.mark.parametrize("rc", [0.0, 3.0, 1e200, float("inf"), float("nan")])
@pytest.mark.parametrize("edge", [10.0, 1e100, 0.0])
def test_capacity_is_finite(monkeypatch, rc, edge):
    seen = []

    def build(h, stream, pos, box, rc_, buf, cap, need):
        seen.append((rc_, cap))
        need._obj.value = 0
        return 0

    monkeypatch.setattr(torch.cuda, "current_stream", lambda d: types.SimpleNamespace(cuda_stream=0))
    eng = AdmpEngine.__new__(AdmpEngine)
    eng.lib, eng.h, eng.n, eng.device = types.SimpleNamespace(dmffb_build_neighbors=build), None, 50, "cpu"
    rows = eng.build_neighbors(torch.zeros((50, 3), dtype=torch.float64), np.eye(3) * edge, rc)
    assert rows.shape == (0, 3)
    (got, cap), = seen
    assert (got == rc or rc != rc) and 0 <= cap <= 50 * 49 // 2

"""Pair sets of coordinates that have drifted far apart, where FP32 differences no longer resolve the cut-off:
boxes below five half-width cells (every atom a candidate) and one of six, orthorhombic and triclinic, some
atoms a few boxes away and some 1e6 A, equal to the all-pairs FP64 test (whose own rounding is 1e-10 A there)."""
import numpy as np
import pytest
import torch

from dmff_b200.synthetic import water_box
from tests.helpers import make_engine
from tests.test_gpu_nb_build import TRI, _exact, _sorted

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nw,L,rc", [(50, 11.6, 5.6), (150, 16.6, 8.0), (150, 16.6, 5.0)])
@pytest.mark.parametrize("tri", [False, True])
@pytest.mark.parametrize("drift", [300.0, 2e4, 1e6])
def test_pair_sets(nw, L, rc, tri, drift):
    s = water_box(nw, L, seed=3 + nw, lmax=2, pol=True, rc=rc)
    box = np.asarray(s["box"]) @ TRI if tri else np.asarray(s["box"])
    rng = np.random.default_rng(nw)
    far = rng.integers(0, 2, size=(len(s["pos"]), 1)) * int(drift / L)
    pos = s["pos"] + (rng.integers(-3, 4, size=s["pos"].shape) + far * rng.choice([-1, 1], size=s["pos"].shape)) @ box
    eng = make_engine(s, precision="fp64", cg_tol=1e-10)
    p = torch.tensor(pos, dtype=torch.float64, device="cuda")
    want = _exact(pos, box, rc)
    for _ in range(2):
        eng.rebuild_internal_pairs(p, box)
        assert np.array_equal(_sorted(eng.internal_pairs())[:, :2], want)
        assert np.array_equal(_sorted(eng.build_neighbors(p, box, rc))[:, :2], want)

"""The scaled-row map of the two-pass build, whose count pass takes it from the covalent map: rows given twice, in
both orientations, with nbond 0, and partners beyond the cut-off.  Energies and forces of the engine's own list
against the same rows handed over by the caller, whose map is searched in the rows."""
import numpy as np
import pytest
import torch

from dmff_b200.engine import AdmpEngine
from dmff_b200.synthetic import water_box
from tests.helpers import rel_force_rms

pytestmark = pytest.mark.gpu

SCALES = [0.0, 0.3, 0.6, 1.0, 1.0, 1.0]


@pytest.mark.parametrize("nw,L,rc", [(700, 27.6, 11.0), (343, 21.8, 7.0), (150, 16.6, 8.0)])  # two-pass, staged, flat
def test_odd_covalent_rows(nw, L, rc):
    s = water_box(nw, L, seed=4, lmax=2, pol=True, rc=rc)
    n = 3 * nw
    rng = np.random.default_rng(nw)
    cov = np.asarray(s["cov_rows"]).reshape(-1, 3)
    far = np.stack([rng.integers(0, n // 2, 200), rng.integers(n // 2, n, 200), rng.integers(0, 4, 200)], 1)
    both = cov[:, [1, 0, 2]] + [0, 0, 2]  # the same pairs again, the other way round and with another nbond
    rows = np.concatenate([cov, both, far, far[:50]]).astype(np.int32)
    pos = torch.tensor(s["pos"], dtype=torch.float64, device="cuda")
    for precision, tol in (("fp64", 1e-11), ("fp32", 1e-6)):
        eng = AdmpEngine(n, 2, False, True, rc, s["kappa"], s["K"], s["axis_types"], s["axis_indices"], rows, SCALES,
                         precision=precision)
        eng.set_params(s["Q_local"])
        eng.rebuild_internal_pairs(pos, s["box"])
        r1, F1, _ = eng.compute(pos, s["box"])
        E1, F1 = r1.energy, F1.cpu().numpy().copy()
        own = eng.internal_pairs().clone()
        assert int((own[:, 2] != 0).sum()) > len(cov)
        r0, F0, _ = eng.compute(pos, s["box"], pairs=own)
        assert abs(E1 - r0.energy) <= tol * max(abs(r0.energy), abs(r0.e_self))
        assert rel_force_rms(F1, F0.cpu().numpy()) <= 10 * tol

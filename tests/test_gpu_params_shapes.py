"""CUDA parameters of other shapes than a row or value per atom: refused or broadcast as host arrays are,
never read past their end."""
import numpy as np
import pytest
import torch

from dmff_b200.engine import DispEngine
from dmff_b200.synthetic import water_box
from tests.helpers import make_engine

pytestmark = pytest.mark.gpu


def _cuda(x):
    return torch.tensor(np.asarray(x), dtype=torch.float64, device="cuda")


def test_admp_shapes():
    s = water_box(8, 9.3, seed=3, lmax=2, pol=True, rc=4.4)
    n = len(s["pos"])
    eng = make_engine(s, precision="fp64", cg_tol=1e-10)
    Q, pol, thole = _cuda(s["Q_local"]), _cuda(s["pol"]), _cuda(s["thole"])
    for args in ((Q[:-1], pol, thole), (Q[: n // 2], pol, thole), (torch.cat([Q, Q[:, :1]], 1), pol, thole),
                 (Q, pol[:-1], thole), (Q, pol, thole[:1])):
        with pytest.raises(ValueError):
            eng.set_params(*args)
    pos, box = _cuda(s["pos"]), s["box"]
    E = []
    for row in (Q[:1], Q[:1].cpu().numpy(), Q[:1].expand(n, 9)):  # one row for every site
        eng.set_params(row, pol, thole)
        E.append(eng.compute(pos, box)[0].energy)
    assert max(E) - min(E) <= 1e-9 * max(abs(E[0]), 1.0)


def test_dispersion_shapes():
    s = water_box(8, 9.3, seed=3, lmax=2, pol=True, rc=4.4)
    n = len(s["pos"])
    eng = DispEngine(n, 10, True, 4.4, 0.5, (12, 12, 12), None, (0, 0, 0, 1, 1, 1), tt=True)
    c, a = torch.ones((n, 3), dtype=torch.float64, device="cuda"), torch.ones(n, dtype=torch.float64, device="cuda")
    for args in ((c[:, :1], a, a, a), (c[:-1], a, a, a), (c, a[:-1], a, a), (c, a, a, a[:1])):
        with pytest.raises(ValueError):
            eng.set_params(*args)

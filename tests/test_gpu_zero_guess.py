"""The engine's zero-guess switch belongs to the caller: an energy of the drop-in layer that starts from zero
dipoles leaves it as it was, on or off."""
import numpy as np
import pytest
import torch

from dmff_b200.admp.pme import ADMPPmeForce
from dmff_b200.synthetic import water_box

pytestmark = pytest.mark.gpu

SCALES = [0.0, 0.0, 1.0, 1.0, 1.0, 1.0]


@pytest.mark.parametrize("on", [False, True])
def test_switch_survives_an_energy(on):
    s = water_box(8, 9.3, seed=3, lmax=2, pol=True, rc=4.4)
    cuda = lambda x: torch.tensor(np.asarray(x), dtype=torch.float64, device="cuda")  # noqa: E731
    pos, box = cuda(s["pos"]), np.asarray(s["box"])
    f = ADMPPmeForce(box, np.arange(len(s["pos"])), s["axis_types"], s["axis_indices"], s["rc"], 5e-4, 2, lpol=True,
                     cov_rows=s["cov_rows"])
    prm = [cuda(s[k]) for k in ("Q_local", "pol", "thole")]
    scales = [torch.tensor(SCALES, dtype=torch.float64)] * 3
    f.get_energy(pos, torch.tensor(box), None, *prm, *scales)
    eng = f.engine
    _, _, U = eng.compute(pos, box)
    exact = U.clone()
    eng.set_zero_guess(on)
    f.get_energy(pos, torch.tensor(box), None, *prm, *scales)
    # a solve that starts from its own solution has nothing left to do, one from zero has
    n_iter = eng.compute(pos, box, U=exact)[0].n_iter
    assert n_iter > 3 if on else n_iter <= 1

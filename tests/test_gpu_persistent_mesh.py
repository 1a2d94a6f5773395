"""The persistent dipole solve on meshes beyond 50 points per axis, up to the largest that its shared memory
takes, against the per-pass solve of the same engine (the FP32 dipoles' tolerance, 1e-5 of the largest); and
the rule that leaves large meshes of small systems to the per-pass solve."""
import numpy as np
import pytest
import torch

from dmff_b200.engine import AdmpEngine
from dmff_b200.synthetic import serving_system

pytestmark = pytest.mark.gpu

SCALES = [0.0, 0.0, 1.0, 1.0, 1.0, 1.0]


def _engine(s, K):
    eng = AdmpEngine(len(s["pos"]), 2, True, True, s["rc"], s["kappa"], K, s["axis_types"], s["axis_indices"],
                     s["cov_rows"], SCALES, SCALES, [1.0] * 6, precision="fp32", cg_tol=1e-7)
    eng.set_params(s["Q_local"], s["pol"], s["thole"])
    eng.set_zero_guess(True)
    return eng


@pytest.mark.parametrize("K", [(56, 56, 56), (57, 57, 57), (64, 64, 64), (73, 73, 73), (97, 97, 97), (112, 112, 112),
                               (16, 20, 128), (4, 96, 50)])
def test_against_the_per_pass_solve(K):
    s = serving_system(150, 21)
    pos = torch.tensor(s["pos"], dtype=torch.float64, device="cuda")
    eng = _engine(s, K)
    out = []
    for mode in (0, 1):
        eng.set_persistent_cg(mode)
        eng.rebuild_internal_pairs(pos, s["box"])
        r, _, U = eng.compute(pos, s["box"])
        out.append((r, U.cpu().numpy().copy(), eng.persistent_cg_blocks()))
    (r0, U0, b0), (r1, U1, b1) = out
    assert b0 == 0 and b1 > 0
    assert r0.converged == r1.converged == 1 and r1.n_iter <= r0.n_iter
    assert abs(r1.energy - r0.energy) <= 2e-6 * abs(r0.energy)
    assert np.abs(U1 - U0).max() <= 1e-5 * np.abs(U0).max()


@pytest.mark.parametrize("K,taken", [((72, 72, 72), True), ((80, 80, 80), False), ((32, 48, 96), True),
                                     ((112, 112, 112), False)])
def test_size_rule(K, taken):
    s = serving_system(150, 21)
    pos = torch.tensor(s["pos"], dtype=torch.float64, device="cuda")
    eng = _engine(s, K)
    eng.set_persistent_cg("auto")
    eng.compute(pos, s["box"])
    assert (eng.persistent_cg_blocks() > 0) == taken

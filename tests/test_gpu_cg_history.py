"""A dipole solve from zero leaves the same dipoles after the same steps whatever its engine solved before: after
a harder system (whose step count sets the head start), an easier one, one with nothing to solve, and whether it ran
in one persistent launch, through direct launches or replayed.  Against an engine that solves nothing else; the
sums' order differs (atomics), 1e-13 of the dipoles a step in FP64."""
import numpy as np
import pytest
import torch

from dmff_b200.synthetic import serving_system
from tests.helpers import make_engine

pytestmark = pytest.mark.gpu


def _solve(eng, pos, box):
    eng.rebuild_internal_pairs(pos, box)
    res, _, U = eng.compute(pos, box)
    assert res.converged == 1
    return res.n_iter, U.cpu().numpy().copy()


def _engine(s, **kw):
    eng = make_engine(s, **kw)
    eng.set_zero_guess(True)
    return eng


# 1400 waters are above the persistent solve's size rule: FP32 solves that stop at the reads
@pytest.mark.parametrize("precision,nw,tol", [("fp64", 200, 1e-6), ("fp64", 200, 1e-9), ("fp32", 200, 1e-6),
                                              ("fp32", 1400, 1e-6)])
def test_steps_do_not_depend_on_the_last_solve(precision, nw, tol):
    s = serving_system(nw, 3)
    pos = torch.tensor(s["pos"], dtype=torch.float64, device="cuda")
    scale = [1.0, 1.0, 0.02, 0.3, 0.0, 1.0, 0.02, 0.02, 1.0]
    want = {}
    for f in set(scale):
        eng = _engine(s, precision=precision, cg_tol=tol)
        if nw > 1366 or precision == "fp64":
            assert eng.lib.dmffb_set_graphs(eng.h, 0) == 0
        eng.set_params(np.asarray(s["Q_local"]) * (f != 0.0), np.asarray(s["pol"]) * (f or 1.0), s["thole"])
        want[f] = _solve(eng, pos, s["box"])
    assert want[1.0][0] > want[0.3][0] > want[0.02][0] > want[0.0][0] == 0
    eng = _engine(s, precision=precision, cg_tol=tol)
    for f in scale:
        eng.set_params(np.asarray(s["Q_local"]) * (f != 0.0), np.asarray(s["pol"]) * (f or 1.0), s["thole"])
        n, U = _solve(eng, pos, s["box"])
        assert n == want[f][0], (f, n, want[f][0])
        assert np.abs(U - want[f][1]).max() <= (1e-11 if precision == "fp64" else 1e-5) * np.abs(want[f][1]).max()


@pytest.mark.parametrize("tol", [1e-5, 1e-6, 1e-7, 1e-8])
def test_persistent_and_replayed_solves_take_the_same_steps(tol):
    s = serving_system(300, 8)
    pos = torch.tensor(s["pos"], dtype=torch.float64, device="cuda")
    eng = _engine(s, precision="fp32", cg_tol=tol)
    n = [_solve(eng, pos, s["box"])[0] for _ in range(4)]  # persistent, then captured and replayed
    assert len(set(n)) == 1, n


@pytest.mark.parametrize("max_iter", [1, 4, 6, 7, 8])
def test_step_limit_of_small_systems(max_iter):
    """Direct, replayed and persistent solves that run into max_iter stop there."""
    s = serving_system(200, 12)
    pos = torch.tensor(s["pos"], dtype=torch.float64, device="cuda")
    from dmff_b200.engine import AdmpEngine
    sc = [0.0, 0.0, 1.0, 1.0, 1.0, 1.0]
    eng = AdmpEngine(len(s["pos"]), 2, True, True, s["rc"], s["kappa"], s["K"], s["axis_types"], s["axis_indices"],
                     s["cov_rows"], sc, sc, [1.0] * 6, precision="fp32", cg_tol=1e-9, max_iter=max_iter)
    eng.set_params(s["Q_local"], s["pol"], s["thole"])
    eng.set_zero_guess(True)
    out = []
    for _ in range(4):
        eng.rebuild_internal_pairs(pos, s["box"])
        r, _, U = eng.compute(pos, s["box"])
        out.append((r.n_iter, r.converged, U.cpu().numpy().copy()))
    assert [(n, c) for n, c, _ in out] == [(max_iter, 0)] * 4
    for _, _, U in out[1:]:
        assert np.abs(U - out[0][2]).max() <= 1e-5 * np.abs(out[0][2]).max()

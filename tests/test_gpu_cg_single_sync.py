"""The dipole solve in its form with one synchronisation per iteration, and the reads' schedule after a
first solve from U = 0: atom counts either side of a CTA's atoms and of one round of the chip, replayed,
direct and persistent, against the float64 oracle on small boxes and against an FP64 solve to 1e-12 on
larger ones; a solve that stays on the schedule of the one before (same positions: the same step count),
one whose residual falls faster or slower than the last one's, and one with nothing to solve."""
import numpy as np
import pytest
import torch

from dmff_b200.synthetic import serving_system, water_box
from tests.helpers import make_engine, oracle_pairs, oracle_reference

pytestmark = pytest.mark.gpu


def _solve(eng, pos, box):
    eng.rebuild_internal_pairs(pos, box)
    res, _, U = eng.compute(pos, box)
    return res, U.cpu().numpy().copy()


@pytest.mark.parametrize("nw,L", [(3, 9.0), (8, 9.3), (27, 9.3)])
def test_against_the_oracle(nw, L):
    s = water_box(nw, L, seed=70 + nw, lmax=2, pol=True, rc=4.5)
    ref = oracle_reference(s, oracle_pairs(s), solver="cg", tol=1e-12)
    pos = torch.tensor(s["pos"], dtype=torch.float64, device="cuda")
    eng = make_engine(s, precision="fp64", cg_tol=1e-11)
    eng.set_zero_guess(True)
    counts = set()
    for _ in range(4):
        res, U = _solve(eng, pos, s["box"])
        assert res.converged == 1
        counts.add(res.n_iter)
        # the relative residual bounds the dipoles' error by the condition number, below ten here
        assert np.abs(U - ref["U"]).max() <= 1e-9 * np.abs(ref["U"]).max()
    assert len(counts) == 1, counts


# 148 x 4 x 8 = 4736 warps: 1578 waters stay within one round of the gather, 1579 take two
@pytest.mark.parametrize("nw", [85, 1578, 1579])
@pytest.mark.parametrize("mode", [0, 1])
def test_fp32_against_fp64(nw, mode):
    s = serving_system(nw, 5 + nw)
    pos = torch.tensor(s["pos"], dtype=torch.float64, device="cuda")
    ref = make_engine(s, precision="fp64", cg_tol=1e-12)
    ref.set_zero_guess(True)
    _, U0 = _solve(ref, pos, s["box"])
    eng = make_engine(s, precision="fp32", cg_tol=1e-7)
    eng.set_zero_guess(True)
    eng.set_persistent_cg(mode)
    for _ in range(3):
        res, U = _solve(eng, pos, s["box"])
        assert res.converged == 1
        assert np.abs(U - U0).max() <= 1e-4 * np.abs(U0).max()  # the FP32 dipoles' tolerance


def test_schedule_follows_the_system():
    s = serving_system(200, 3)
    pos = torch.tensor(s["pos"], dtype=torch.float64, device="cuda")
    eng = make_engine(s, precision="fp64", cg_tol=1e-8)
    eng.set_zero_guess(True)
    strong, weak = s["pol"], 0.05 * np.asarray(s["pol"])
    n = {}
    for pol in (strong, strong, weak, weak, weak, strong, strong):
        eng.set_params(s["Q_local"], pol, s["thole"])
        res, U = _solve(eng, pos, s["box"])
        fresh = make_engine(s, precision="fp64", cg_tol=1e-12)
        fresh.set_params(s["Q_local"], pol, s["thole"])
        fresh.set_zero_guess(True)
        _, U0 = _solve(fresh, pos, s["box"])
        assert res.converged == 1
        assert np.abs(U - U0).max() <= 1e-6 * max(np.abs(U0).max(), 1e-12)
        n.setdefault(float(np.sum(pol)), []).append(res.n_iter)
    assert n[float(np.sum(strong))][0] == n[float(np.sum(strong))][1]
    assert n[float(np.sum(weak))][-1] < n[float(np.sum(strong))][0]  # and it comes down again
    eng.set_params(np.zeros_like(np.asarray(s["Q_local"])), strong, s["thole"])
    res, U = _solve(eng, pos, s["box"])
    assert res.converged == 1 and res.n_iter == 0 and not U.any()

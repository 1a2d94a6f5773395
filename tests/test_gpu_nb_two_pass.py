"""The two-pass neighbour build (count and fill passes of a warp per atom), which takes neighbourhoods too large to
stage in shared memory: 2100 atoms in a box of five half-width cells of 5.5 A, orthorhombic and triclinic.  Rows
and nbond against the all-pairs FP64 test on the host, from the engine's own build and the caller-buffer entry, first
and later builds; and what a polarizable engine makes beside the rows (CSR, scaled-row map) against the same rows
handed over by the caller."""
import numpy as np
import pytest
import torch

from dmff_b200.synthetic import water_box
from tests.helpers import make_engine, rel_force_rms
from tests.test_gpu_nb_build import TRI, _exact, _sorted

pytestmark = pytest.mark.gpu

RC = 11.0


def _system(tri):
    s = water_box(700, 27.6, seed=9, lmax=2, pol=True, rc=RC)
    box = np.asarray(s["box"]) @ TRI if tri else np.asarray(s["box"])
    pos = np.asarray(s["pos"]) + np.random.default_rng(1).integers(-3, 4, size=s["pos"].shape) @ box
    return s, box, pos


def _widths(box):
    V = abs(np.linalg.det(box))
    return [V / np.linalg.norm(np.cross(box[(k + 1) % 3], box[(k + 2) % 3])) for k in range(3)]


@pytest.mark.parametrize("tri", [False, True])
def test_rows(tri):
    s, box, pos = _system(tri)
    rc = RC if not tri else min(_widths(box)) / 2.5 - 0.01  # five half-width cells on the narrowest axis
    n = len(pos)
    nc = [int(w / (0.5 * rc)) for w in _widths(box)]
    assert min(nc) >= 5 and 16 * (1.5 * 125 * n / np.prod(nc) + 64) > 44 << 10  # neither flat nor staged
    p = torch.tensor(pos, dtype=torch.float64, device="cuda")
    want = _exact(pos, box, rc)
    cov = {(min(i, j), max(i, j)): nb for i, j, nb in np.asarray(s["cov_rows"]).reshape(-1, 3)}
    nbond = np.array([cov.get((int(i), int(j)), 0) for i, j in want])
    eng = make_engine(dict(s, rc=rc), precision="fp64", cg_tol=1e-10)
    for _ in range(3):
        eng.rebuild_internal_pairs(p, box)
        rows = _sorted(eng.internal_pairs())
        assert np.array_equal(rows[:, :2], want) and np.array_equal(rows[:, 2], nbond)
        assert np.array_equal(_sorted(eng.build_neighbors(p, box, rc)), rows)
        assert np.array_equal(_sorted(eng.build_neighbors(p, box, rc, capacity=1)), rows)  # too small: grown


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_csr_and_scaled_rows(precision):
    s, box, pos = _system(False)
    p = torch.tensor(pos, dtype=torch.float64, device="cuda")
    eng = make_engine(s, precision=precision, cg_tol=1e-9 if precision == "fp64" else 1e-7)
    eng.set_zero_guess(True)
    eng.rebuild_internal_pairs(p, box)
    rows = eng.internal_pairs().clone()
    out = []
    for kw in ({"pairs": rows}, {}, {}):
        if not kw:
            eng.rebuild_internal_pairs(p, box)
        r, F, U = eng.compute(p, box, **kw)
        out.append((r.energy, r.n_iter, F.cpu().numpy().copy(), U.cpu().numpy().copy()))
    tol = 1e-11 if precision == "fp64" else 1e-6
    E0, n0, F0, U0 = out[0]
    for E, n, F, U in out[1:]:
        assert n == n0 and abs(E - E0) <= tol * abs(E0)
        assert rel_force_rms(F, F0) <= 10 * tol and np.abs(U - U0).max() <= 10 * tol * np.abs(U0).max()

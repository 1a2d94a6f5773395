"""The dipole solve's full CSR of a caller's rows (k_csr_count, k_csr_fill add runs of rows with one first
atom): rows grouped by that atom, in any order, and with ignored rows between them, against the float64
oracle.  Numbers of rows that leave a partly filled last warp come with the sizes."""
import numpy as np
import pytest
import torch

from dmff_b200.synthetic import water_box
from tests.helpers import make_engine, oracle_pairs, oracle_reference

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nw,L", [(1, 9.0), (3, 9.0), (8, 9.3), (27, 9.3)])
def test_caller_rows_in_any_order(nw, L):
    s = water_box(nw, L, seed=90 + nw, lmax=2, pol=True, rc=4.5)
    rows = oracle_pairs(s)
    ref = oracle_reference(s, rows, solver="cg", tol=1e-12)
    rows = np.asarray(rows, np.int32)
    n = s["n_atoms"]
    rng = np.random.default_rng(nw)
    grouped = rows[np.argsort(rows[:, 0], kind="stable")]
    padded = np.full((2 * len(rows) + 37, 3), n, np.int32)
    padded[np.sort(rng.permutation(len(padded))[:len(rows)])] = grouped
    pos = torch.tensor(s["pos"], dtype=torch.float64, device="cuda")
    eng = make_engine(s, precision="fp64", cg_tol=1e-11)
    for r in (grouped, rng.permutation(rows), padded):
        eng.set_zero_guess(True)
        res, _, U = eng.compute(pos, s["box"], pairs=torch.tensor(r, device="cuda"))
        assert res.converged == 1
        # the relative residual bounds the dipoles' error by the condition number, below ten here
        assert np.abs(U.cpu().numpy() - ref["U"]).max() <= 1e-9 * np.abs(ref["U"]).max()

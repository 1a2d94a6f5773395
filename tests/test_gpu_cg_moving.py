"""The dipole solve's graph while atoms move: positions, rows and the number of pairs change at every step, the
graph's step reads none of them.  Dipoles against an engine without graphs at each step; from the third step on
the launches of a step are those of a replayed per-pass solve (six a CG step), not of the persistent one."""
import numpy as np
import pytest
import torch

from dmff_b200.synthetic import serving_system
from tests.helpers import make_engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,nw", [("fp32", 150), ("fp32", 1400), ("fp64", 150)])
def test_moving_atoms_replay(precision, nw):
    s = serving_system(nw, 6)
    box = s["box"]
    x0 = torch.tensor(s["pos"], dtype=torch.float64, device="cuda")
    step = torch.tensor(np.random.default_rng(2).normal(0.0, 0.01, size=s["pos"].shape), device="cuda")
    eng, ref = (make_engine(s, precision=precision, cg_tol=1e-6) for _ in range(2))
    assert ref.lib.dmffb_set_graphs(ref.h, 0) == 0
    for e in (eng, ref):
        e.set_zero_guess(True)
    pos = x0.clone()
    pairs, launches = [], []
    for k in range(6):
        pos += step
        out = []
        for e in (eng, ref):
            n0 = e.counters()["launches"]
            e.rebuild_internal_pairs(pos, box)
            r, _, U = e.compute(pos, box)
            out.append((r, U.cpu().numpy().copy(), e.counters()["launches"] - n0))
        (r, U, n), (r0, U0, _) = out
        assert r.converged == 1 and r.n_iter == r0.n_iter
        assert np.abs(U - U0).max() <= (1e-11 if precision == "fp64" else 1e-5) * np.abs(U0).max()
        pairs.append(r.n_pairs)
        launches.append(n - 6 * r.n_iter)
    assert len(set(pairs)) > 3, pairs
    assert min(launches[2:]) > 0, launches

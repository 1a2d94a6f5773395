"""Neighbour builds in boxes of many cells with few atoms (a cluster in a vacuum, a dilute gas), where the scan
over the cells is a kernel of its own beyond two tiles of 4096: cell counts either side of that and the largest,
64^3; cut-offs that change between builds of one engine, so that each finds the counters the last one left.
Pair sets against the all-pairs FP64 test on the host; and the classical cell pass on the same cells against the list."""
import numpy as np
import pytest
import torch

from dmff_b200.engine import AdmpEngine, ClassicalEngine
from tests.helpers import rel_force_rms
from tests.test_gpu_nb_build import TRI, _exact, _sorted

pytestmark = pytest.mark.gpu


def _atoms(n, box, seed, cluster):
    rng = np.random.default_rng(seed)
    x = rng.uniform(0.0, 1.0, (n, 3)) @ box
    if cluster:  # a ball around a corner, wrapped over all faces
        x = rng.normal(0.0, 6.0, (n, 3))
    return x


@pytest.mark.parametrize("n", [1, 40, 300])
@pytest.mark.parametrize("cluster", [False, True])
@pytest.mark.parametrize("tri", [False, True])
def test_pair_sets(n, cluster, tri):
    box = np.eye(3) * 100.0
    box = box @ TRI if tri else box
    pos = _atoms(n, box, n + tri, cluster)
    p = torch.tensor(pos, dtype=torch.float64, device="cuda")
    eng = AdmpEngine(n, 0, False, False, 5.0, 0.0, (0, 0, 0), None, None, None, [1.0] * 6, precision="fp64")
    want = {rc: _exact(pos, box, rc) for rc in (2.5, 5.0, 9.5, 9.9, 12.0, 20.0)}  # 64^3 cells .. 10^3
    for rc in (5.0, 2.5, 20.0, 9.5, 2.5, 9.9, 5.0, 12.0, 9.5):
        assert np.array_equal(_sorted(eng.build_neighbors(p, box, rc))[:, :2], want[rc]), rc
        eng.rebuild_internal_pairs(p, box)
        assert np.array_equal(_sorted(eng.internal_pairs())[:, :2], want[5.0])


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_cell_pass(precision):
    n, box = 2000, np.eye(3) * 100.0
    rng = np.random.default_rng(3)
    g = np.stack(np.meshgrid(*[np.arange(13)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
    p = torch.tensor(g * 3.0 + rng.uniform(-0.2, 0.2, (n, 3)) - 18.0, dtype=torch.float64, device="cuda")
    q = rng.choice([-0.4, 0.4], n)
    out = []
    for cell in (False, True):
        e = ClassicalEngine(n, n_types=1, coulomb="rf", rc=6.0, precision=precision)
        e.set_params(q, np.zeros(n, np.int32), np.array([[3.0]]), np.array([[0.5]]))
        e.set_cell_pass(cell)
        for _ in range(2):
            if not cell:
                e.rebuild_internal_pairs(p, box)
            r, F = e.compute(p, box)
        out.append((r, F.cpu().numpy().copy()))
    (r0, F0), (r1, F1) = out
    tol = 1e-11 if precision == "fp64" else 1e-5
    assert r1.n_pairs == r0.n_pairs > n
    assert abs(r1.energy - r0.energy) <= tol * abs(r0.e_lj) and rel_force_rms(F1, F0) <= 10 * tol

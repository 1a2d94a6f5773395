"""The neighbour builds (cells sorted by k_bin_count / k_bin_fill, k_pairs_cell or k_pairs_flat,
k_nb_place) against the all-pairs FP64 test on the host, with the pair set required equal: boxes at the
edges between the builds (every-atom scan below five half-width cells on an axis, five exactly, several
CTAs and runs), triclinic boxes, atoms far outside the box, first and later builds, both entry
points; and the scaled-row map and CSR made with the list against those searched from the same rows
handed over by the caller."""
import numpy as np
import pytest
import torch

from dmff_b200.synthetic import water_box
from tests.helpers import make_engine, rel_force_rms

pytestmark = pytest.mark.gpu


def _exact(pos, box, rc):
    hinv = np.linalg.inv(box)
    out = []
    for i in range(len(pos) - 1):
        d = pos[i + 1:] - pos[i]
        s = d @ hinv
        s -= np.floor(s + 0.5)
        r = np.sqrt(((s @ box) ** 2).sum(1))
        out += [(i, i + 1 + j) for j in np.nonzero(r < rc)[0]]
    return np.array(out, dtype=np.int64).reshape(-1, 2)


def _sorted(rows):
    rows = rows.cpu().numpy()
    assert np.all(np.diff(rows[:, 0]) >= 0)
    return rows[np.lexsort((rows[:, 1], rows[:, 0]))]


TRI = np.array([[1.0, 0.0, 0.0], [0.21, 1.0, 0.0], [-0.17, 0.12, 1.0]])


# waters, box edge, rc: 2.4, 2.5 + and 3.1 rc wide; 1023 / 1026 atoms either side of one run of sums
@pytest.mark.parametrize("nw,L,rc,tri", [(1, 9.0, 4.0, False), (50, 11.6, 5.6, False), (150, 16.6, 8.0, True),
                                         (150, 16.6, 6.63, False), (341, 21.8, 7.0, False),
                                         (342, 21.8, 8.7, True), (700, 27.6, 5.0, True)])
def test_pair_sets(nw, L, rc, tri):
    s = water_box(nw, L, seed=3 + nw, lmax=2, pol=True, rc=rc)
    box = np.asarray(s["box"]) @ TRI if tri else np.asarray(s["box"])
    rng = np.random.default_rng(nw)
    pos = s["pos"] + rng.integers(-40, 41, size=s["pos"].shape) @ box  # images far outside the box
    eng = make_engine(s, precision="fp64", cg_tol=1e-10)
    p = torch.tensor(pos, dtype=torch.float64, device="cuda")
    want = _exact(pos, box, rc)
    cov = {(min(i, j), max(i, j)): nb for i, j, nb in np.asarray(s["cov_rows"]).reshape(-1, 3)}
    nbond = np.array([cov.get((int(i), int(j)), 0) for i, j in want])
    for _ in range(3):  # first build (slots from the mean density) and later ones
        eng.rebuild_internal_pairs(p, box)
        rows = _sorted(eng.internal_pairs())
        assert np.array_equal(rows[:, :2], want)
        assert np.array_equal(rows[:, 2], nbond)
        assert np.array_equal(_sorted(eng.build_neighbors(p, box, rc)), rows)
        # another cut-off between two builds of the engine's own list
        near = _sorted(eng.build_neighbors(p, box, 0.6 * rc, capacity=1))
        assert np.array_equal(near[:, :2], _exact(pos, box, 0.6 * rc))


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-10), ("fp32", 2e-6)])
@pytest.mark.parametrize("nw,L", [(60, 12.3), (500, 24.7)])
def test_own_list_against_the_same_rows_from_the_caller(nw, L, precision, tol):
    # own list: scaled rows and CSR from the build; the caller's rows: both searched from the rows
    s = water_box(nw, L, seed=21, lmax=2, pol=True, rc=6.0)
    pos = torch.tensor(s["pos"], dtype=torch.float64, device="cuda")
    eng = make_engine(s, precision=precision, cg_tol=1e-10 if precision == "fp64" else 1e-7)
    eng.set_zero_guess(True)
    for _ in range(2):
        eng.rebuild_internal_pairs(pos, s["box"])
        ra, Fa, _ = eng.compute(pos, s["box"])
        Fa = Fa.cpu().numpy().copy()
        rb, Fb, _ = eng.compute(pos, s["box"], pairs=eng.internal_pairs())
        assert ra.n_pairs == rb.n_pairs
        assert abs(ra.energy - rb.energy) <= tol * abs(rb.energy)
        assert rel_force_rms(Fa, Fb.cpu().numpy()) <= 10 * tol


def test_clustered_atoms_outgrow_the_slots():
    # everything in one corner of a large box: counts far above the mean density's, and cells whose
    # neighbourhood does not fit the stage
    s = water_box(300, 20.8, seed=9, lmax=2, pol=True, rc=6.0)
    box = np.eye(3) * 64.0
    eng = make_engine(s, precision="fp64", cg_tol=1e-10)
    p = torch.tensor(s["pos"], dtype=torch.float64, device="cuda")
    want = _exact(s["pos"], box, 6.0)
    for _ in range(2):
        eng.rebuild_internal_pairs(p, box)
        assert np.array_equal(_sorted(eng.internal_pairs())[:, :2], want)
    assert np.array_equal(_sorted(eng.build_neighbors(p, box, 6.0))[:, :2], want)

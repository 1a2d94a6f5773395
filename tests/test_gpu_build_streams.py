"""Builds and evaluations of one engine on different streams share arrays (the scaled-row map, the cells and
their counters, which stay zero between calls).  A build queued behind 20 ms of other work on a side stream returns
at once; an evaluation that does not use its list then runs on the current stream, and one build and
evaluation after both.  All equal an engine that does the same on one stream, to the sums' order (atomics)."""
import numpy as np
import pytest
import torch

from dmff_b200.synthetic import polymer_water_box, water_box
from tests.helpers import make_engine, rel_force_rms
from tests.test_gpu_classical import _engine

pytestmark = pytest.mark.gpu


def _late_build(eng, pos, box):
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        torch.cuda._sleep(40_000_000)
        eng.rebuild_internal_pairs(pos, box)


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_rows_of_the_caller_beside_a_build(precision):
    s = water_box(343, 21.8, seed=5, lmax=2, pol=True, rc=7.0)
    box = s["box"]
    pos = torch.tensor(s["pos"], dtype=torch.float64, device="cuda")
    near = pos * 0.97  # other rows, denser
    ref, eng = (make_engine(s, precision=precision, cg_tol=1e-9) for _ in range(2))
    rows = ref.build_neighbors(near, box * 0.97, s["rc"]).clone()
    tol = 1e-11 if precision == "fp64" else 1e-5
    for e in (ref, eng):
        e.set_zero_guess(True)
        e.rebuild_internal_pairs(pos, box)

    def both(e):
        out = []
        for p, b, kw in ((near, box * 0.97, {"pairs": rows}), (pos, box, {})):
            r, F, _ = e.compute(p, b, **kw)
            out.append((r.energy, r.n_iter, F.cpu().numpy().copy()))
        return out

    want = both(ref)
    for _ in range(3):
        _late_build(eng, pos, box)
        for (E, n, F), (E0, n0, F0) in zip(both(eng), want):
            assert n == n0 and abs(E - E0) <= tol * abs(E0) and rel_force_rms(F, F0) <= 10 * tol


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_cell_pass_beside_a_build(precision):
    s = polymer_water_box(4, 20, 500, 24.6, seed=4, rc=8.0)
    pos = torch.tensor(s["pos"], dtype=torch.float64, device="cuda")
    far = pos[torch.randperm(len(pos), generator=torch.Generator().manual_seed(1)).cuda()].contiguous()  # other cells
    ref, eng = _engine(s, precision, "pme"), _engine(s, precision, "pme")
    for e in (ref, eng):
        e.rebuild_internal_pairs(pos, s["box"])
    ref.set_cell_pass(True)
    r0, F0 = ref.compute(pos, s["box"])
    F0 = F0.cpu().numpy().copy()
    tol = 1e-11 if precision == "fp64" else 1e-5
    for _ in range(3):
        _late_build(eng, far, s["box"])
        for cell in (True, False, True):
            eng.set_cell_pass(cell)
            if not cell:
                eng.rebuild_internal_pairs(pos, s["box"])
            r, F = eng.compute(pos, s["box"])
            assert r.n_pairs == r0.n_pairs
            assert abs(r.energy - r0.energy) <= tol * max(abs(r0.energy), abs(r0.e_coul_real))
            assert rel_force_rms(F.cpu().numpy(), F0) <= 10 * tol

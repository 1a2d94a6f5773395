"""Device memory of an engine's first evaluation: neighbour rows (12 bytes), the CSR of both directions and its pair
tensors (4 and 16 bytes an entry) with one headroom of 1.3, the slots, and per-atom arrays (below 400 bytes).  The
bound takes 1.45 for the headroom and 8 MB for the driver's 2 MB pages."""
import pytest
import torch

from dmff_b200.synthetic import serving_system
from tests.helpers import make_engine

pytestmark = pytest.mark.gpu


def test_first_lists_carry_one_headroom():
    s = serving_system(4096, 2)
    n = len(s["pos"])
    pos = torch.tensor(s["pos"], dtype=torch.float64, device="cuda")
    for _ in range(2):  # kernels and libraries of the first engine are loaded, the second is measured
        eng = make_engine(s, precision="fp32", cg_tol=1e-6)
        eng.set_zero_guess(True)
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        eng.rebuild_internal_pairs(pos, s["box"])
        res, _, _ = eng.compute(pos, s["box"])
        torch.cuda.synchronize()
        used = before - torch.cuda.mem_get_info()[0]
        last = eng, res
    pairs = last[1].n_pairs
    mean = 2 * pairs / n
    assert used <= 1.45 * 52 * pairs + 4 * n * (1.45 * mean + 24) + 400 * n + (8 << 20), (used, pairs)

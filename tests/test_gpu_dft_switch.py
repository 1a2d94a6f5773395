"""The convolution's switch returns to the engine's own choice by size."""
import pytest
import torch

from dmff_b200.synthetic import water_box
from tests.helpers import make_engine

pytestmark = pytest.mark.gpu


def test_switch_returns_to_the_size_rule():
    s = water_box(27, 9.3, seed=2, lmax=2, pol=True, rc=4.4)
    pos = torch.tensor(s["pos"], dtype=torch.float64, device="cuda")
    eng = make_engine(s, precision="fp32", cg_tol=1e-6)
    eng.set_zero_guess(True)
    seen, E = [], []
    for mode in (None, False, "auto", True, False, "auto"):
        if mode is not None:
            eng.set_fused_fft(mode)
        E.append(eng.compute(pos, s["box"])[0].energy)
        seen.append(eng.fused_fft_active())
    assert seen == [True, False, True, True, False, True]  # the rule takes the DFT kernels at this size
    assert max(E) - min(E) <= 1e-5 * abs(E[0])

"""The common factor of FP32 spline values, divided out of the direct-DFT convolution.  Unit charges, positive in
one half of the box and negative in the other: the reciprocal energy is that of one wave, whose amplitude adds
up over 2000 charges, so that their splines' roundings (6e-8 each) leave 1e-9 of it.  The transforms leave 3e-8
from the DFT matrices and at most 3e-8 from the wave's own last rounding, twice that in the energy: below 1e-7 in a
mean over four boxes, against 2.7e-7 of the factor."""
import numpy as np
import pytest
import torch

from dmff_b200.engine import AdmpEngine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [36, 45, 50])
def test_reciprocal_energy_has_no_common_factor(K):
    n, L = 2000, 30.0
    err = []
    for seed in range(4):
        pos = np.random.default_rng(seed).uniform(0.0, L, (n, 3))
        q = np.where(pos[:, :1] < 0.5 * L, 1.0, -1.0)
        x = torch.tensor(pos, dtype=torch.float64, device="cuda")
        E = {}
        for precision in ("fp64", "fp32"):
            eng = AdmpEngine(n, 0, False, True, 2.0, 0.35, (K,) * 3, None, None, None, [1.0] * 6, precision=precision)
            eng.set_params(q)
            eng.set_fused_fft(True)
            E[precision] = np.mean([eng.compute(x, np.eye(3) * L)[0].e_recip for _ in range(4)])
        err.append((E["fp32"] - E["fp64"]) / E["fp64"])
    assert abs(np.mean(err)) <= 1e-7, err

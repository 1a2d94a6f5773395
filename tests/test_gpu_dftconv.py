"""The direct-DFT mesh convolution (admp_dftconv.cuh) against cuFFT on the same engine kind: extents
around the size rule's lines and the tile switch, odd, even and prime ones, different per axis, and
a triclinic box; the Coulomb and the three dispersion influence functions, energies, forces and the box
gradient.

FP64 tolerance: both transforms are sums of at most 3 * 128 rounded terms per mesh point (1e-16 each,
accumulating as a random walk, about 2e-15) and the box gradient adds cancelling terms a few hundred
times larger than their sum: 1e-12.  FP32: the spread, the transforms and the gather round at 6e-8 in
as many terms (1e-6) against FP64: 1e-5."""
import numpy as np
import pytest
import torch

from dmff_b200.engine import ClassicalEngine, DispEngine

pytestmark = pytest.mark.gpu

BOX = np.diag([21.0, 24.0, 19.0])
TRICLINIC = np.array([[21.0, 0.0, 0.0], [2.5, 24.0, 0.0], [-1.5, 3.0, 19.0]])


def _coulomb(K, box, precision, mode, n=301):
    rng = np.random.default_rng(3)
    q = rng.normal(size=n)
    eng = ClassicalEngine(n, coulomb="pme", rc=8.0, kappa=0.35, K=K, precision=precision)
    eng.set_params(q - q.mean(), np.zeros(n, np.int32))
    if mode is not None:
        assert eng.lib.dmffb_set_fused_fft(eng.h, mode) == 0
    pos = torch.tensor(rng.uniform(0, 1, (n, 3)) @ box, device="cuda")
    res, F = eng.compute(pos, box, pairs=torch.zeros((0, 3), dtype=torch.int32, device="cuda"))
    return res.e_coul_recip, F.cpu().numpy().copy(), np.array(res.box_grad[:]), eng.lib.dmffb_fused_fft_active(eng.h)


def _largest_prime(k):
    return max([p for p in range(2, k + 1) if k % p == 0 and all(p % f for f in range(2, p))] or [1])


def _close(a, b, tol):
    assert abs(a[0] - b[0]) <= tol * abs(b[0])
    assert np.linalg.norm(a[1] - b[1]) <= tol * np.linalg.norm(b[1])
    assert np.abs(a[2] - b[2]).max() <= tol * np.abs(b[2]).max()


@pytest.mark.parametrize("K", [(4, 5, 6), (8, 8, 8), (17, 20, 15), (31, 30, 29), (48, 49, 47), (49, 49, 49), (50, 41, 23),
                               (56, 56, 56), (57, 8, 56), (63, 61, 62), (68, 40, 33), (85, 85, 85), (97, 64, 16)])
def test_dft_convolution_matches_cufft(K):
    for box in (BOX, TRICLINIC):
        ref = _coulomb(K, box, "fp64", 0)
        assert ref[3] == 0
        own = _coulomb(K, box, "fp64", None)
        assert own[3] == (max(K) <= 49 or (max(K) <= 73 and max(map(_largest_prime, K)) > 16))
        _close(own, ref, 1e-12)
        f32 = _coulomb(K, box, "fp32", None)
        assert f32[3] == 1
        _close(f32, ref, 1e-5)


@pytest.mark.parametrize("K", [(64, 64, 64), (96, 80, 72), (100, 33, 47)])
def test_size_rule_keeps_cufft(K):
    assert _coulomb(K, BOX, "fp32", None)[3] == 0


@pytest.mark.parametrize("K", [(16, 18, 17), (40, 40, 40), (61, 33, 20)])
def test_dispersion_influence_functions(K):
    rng = np.random.default_rng(5)
    n = 211
    c = np.abs(rng.normal(1.0, 0.3, (n, 3))) * np.array([30.0, 90.0, 300.0])
    pos = torch.tensor(rng.uniform(0, 1, (n, 3)) @ TRICLINIC, device="cuda")
    none = torch.zeros((0, 3), dtype=torch.int32, device="cuda")
    out = []
    for precision, mode in (("fp64", 0), ("fp64", None), ("fp32", None)):
        eng = DispEngine(n, 10, True, 8.0, 0.35, K, None, (0, 0, 0, 1, 1, 1), precision=precision)
        eng.set_params(c)
        if mode is not None:
            eng.lib.dmffb_set_fused_fft(eng.h, mode)
        eng.set_param_grads(True)
        res, (F, _) = eng.compute(pos, TRICLINIC, pairs=none)
        out.append((res.e_recip, F.cpu().numpy().copy(), np.array(res.box_grad[:]),
                    eng.param_grads()["c"].cpu().numpy()))
    for k, tol in ((1, 1e-12), (2, 1e-5)):
        _close(out[k], out[0], tol)
        assert np.abs(out[k][3] - out[0][3]).max() <= tol * np.abs(out[0][3]).max()

"""Parameters handed over as CUDA tensors (no copy through the host) against the same values from host
arrays: energies, forces, parameter adjoints and the second-order pass of ADMP engines, the self energy and
short range of dispersion engines; values changed in place between calls, padded and strided
tensors, and a stream other than the default one.  Same kernels on the same values: the FP64 energies agree
to rounding of the atomics' order (1e-12), the second-order pass to its own step's error (1e-6)."""
import numpy as np
import pytest
import torch

from dmff_b200.engine import DispEngine
from dmff_b200.synthetic import water_box
from tests.helpers import make_engine, rel_force_rms

pytestmark = pytest.mark.gpu


def _cuda(x):
    return torch.tensor(np.asarray(x), dtype=torch.float64, device="cuda")


@pytest.mark.parametrize("nw,L,lmax", [(1, 9.0, 2), (43, 11.0, 2), (43, 11.0, 1)])
def test_admp(nw, L, lmax):
    s = water_box(nw, L, seed=12 + nw, lmax=lmax, pol=True, rc=4.4)
    pos, box = _cuda(s["pos"]), s["box"]
    ref = make_engine(s, precision="fp64", cg_tol=1e-11)
    eng = make_engine(s, precision="fp64", cg_tol=1e-11)
    Q = _cuda(s["Q_local"])
    rng = np.random.default_rng(4)
    side = torch.cuda.Stream()
    for k in range(3):
        Q *= 1.0 + 0.01 * k
        pol, thole = _cuda(s["pol"]) * (1.0 + 0.02 * k), _cuda(s["thole"]) + 0.01 * k
        wide = torch.stack([thole, thole], 1)[:, 0]  # strided
        ref.set_params(Q.cpu().numpy(), pol.cpu().numpy(), thole.cpu().numpy())
        if k == 2:
            side.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(side):
                eng.set_params(Q[:, : (lmax + 1) ** 2], pol, wide)
            torch.cuda.current_stream().wait_stream(side)
        else:
            eng.set_params(Q[:, : (lmax + 1) ** 2], pol, wide)
        for e in (ref, eng):
            e.set_param_grads(True)
        r0, F0, _ = ref.compute(pos, box)
        r1, F1, _ = eng.compute(pos, box)
        assert abs(r1.energy - r0.energy) <= 1e-12 * max(abs(r0.energy), abs(r0.e_self))
        assert rel_force_rms(F1.cpu().numpy(), F0.cpu().numpy()) <= 1e-9
        g0, g1 = ref.param_grads(), eng.param_grads(with_global=False)
        assert g1["Q_global"] is None
        for name in ("Q_local", "pol", "thole"):
            assert (g1[name] - g0[name]).abs().max() <= 1e-9 * max(float(g0[name].abs().max()), 1e-12)
    c = _cuda(rng.normal(size=s["pos"].shape))
    b0, b1 = ref.backward(c_pos=c), eng.backward(c_pos=c)  # fetches the device parameters
    for name in ("pos", "Q_local", "pol", "thole"):
        assert (b1[name] - b0[name]).abs().max() <= 1e-6 * max(float(b0[name].abs().max()), 1e-12)


@pytest.mark.parametrize("n", [1, 255, 257])
@pytest.mark.parametrize("tt,precision,tol", [(False, "fp64", 1e-12), (True, "fp64", 1e-12), (True, "fp32", 1e-6)])
def test_disp(n, tt, precision, tol):
    rng = np.random.default_rng(n)
    L = 16.0
    box = np.eye(3) * L
    side = int(np.ceil(n ** (1 / 3)))
    grid = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n] * (L / side)
    pos = _cuda(grid + rng.uniform(0, 0.2, (n, 3)))
    mk = lambda: DispEngine(n, 10, True, 5.0, 0.4, (16, 16, 16), np.zeros((0, 3), np.int32), [1.0] * 6, tt=tt,
                            precision=precision)
    ref, eng = mk(), mk()
    for k in range(2):
        c = np.abs(rng.normal(3.0, 1.0, (n, 3))) * (k + 1)
        abq = [rng.uniform(1.0, 2.0, n) for _ in range(3)] if tt else [None] * 3
        ref.set_params(c, *abq)
        eng.set_params(_cuda(c.T.copy()).T, *[None if x is None else _cuda(x) for x in abq])
        r0, F0 = ref.compute(pos, box)
        r1, F1 = eng.compute(pos, box)
        assert abs(r1.e_self - r0.e_self) <= 1e-13 * abs(r0.e_self)
        size = abs(r0.e_self) + abs(r0.e_recip)
        assert abs(r1.energy - r0.energy) <= tol * size
        assert abs(r1.e_sr - r0.e_sr) <= tol * max(abs(r0.e_sr), size)
        for a, b in zip(F1, F0):
            assert (a - b).abs().max() <= 100 * tol * max(float(b.abs().max()), size / (n * L))

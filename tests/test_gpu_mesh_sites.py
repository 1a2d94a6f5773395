"""The general mesh spread and gather (a CTA per group of sites, charges alone and full multipoles) and
the influence kernel, through engines whose sums are checked against a plain float64 evaluation: an
atom count either side of every group size, meshes narrower than, as wide as and not a multiple of
the six-point stencil, extents that take cuFFT (the influence kernel) and the direct DFTs, and triclinic boxes."""
import numpy as np
import pytest
import torch

from dmff_b200.engine import ClassicalEngine
from dmff_b200.synthetic import water_box
from tests.helpers import make_engine, oracle_pairs, oracle_reference, rel_force_rms

pytestmark = pytest.mark.gpu


def _structure(pos, q, box, K, kappa):
    """Reciprocal energy of point charges by a float64 B-spline sum (order 6) and torch's FFT, over the
    half spectrum with its conjugates by weight (at the middle frequency of an even extent of a
    triclinic box the two halves' k^2 differ; the engine evaluates this one)."""
    pos = torch.tensor(pos, dtype=torch.float64, requires_grad=True)
    K = list(K)
    x = pos @ torch.linalg.inv(box) * torch.tensor(K, dtype=torch.float64)
    up = torch.ceil(x.detach())
    w = up - x

    def spline(w):
        m = torch.stack([w, 1 - w], -1)
        for k in range(3, 7):
            z = torch.zeros_like(m[..., :1])
            u = w[..., None] + torch.arange(k, dtype=w.dtype)
            m = (u * torch.cat([m, z], -1) + (k - u) * torch.cat([z, m], -1)) / (k - 1)
        return m

    M = spline(w)  # [n, 3, 6]
    g = (up.long()[:, :, None] - 3 + torch.arange(6))
    g = torch.stack([g[:, d] % K[d] for d in range(3)], 1)
    idx = (g[:, 0, :, None, None] * K[1] + g[:, 1, None, :, None]) * K[2] + g[:, 2, None, None, :]
    val = torch.tensor(q)[:, None, None, None] * M[:, 0, :, None, None] * M[:, 1, None, :, None] * M[:, 2, None, None, :]
    mesh = torch.zeros(K[0] * K[1] * K[2], dtype=torch.float64).index_add(0, idx.reshape(-1), val.reshape(-1)).reshape(K)
    S = torch.fft.rfftn(mesh)
    m6 = spline(torch.zeros(()).double())  # the spline at the integers
    ms = []
    th = 1.0
    for d in range(3):
        k = torch.fft.fftfreq(K[d], 1.0 / K[d]).double()[: S.shape[d]]
        ms.append(k)
        b = sum(m6[j] * torch.cos(2 * np.pi * k * (j - 3) / K[d]) for j in range(6))
        shape = [1, 1, 1]
        shape[d] = len(k)
        th = th * b.reshape(shape)
    kv = 2 * np.pi * torch.einsum("cd,dijk->cijk", torch.linalg.inv(box), torch.stack(torch.meshgrid(*ms, indexing="ij")))
    k2 = (kv ** 2).sum(0)
    k2[0, 0, 0] = 1.0
    G = 2 * np.pi / torch.linalg.det(box) * torch.exp(-k2 / (4 * kappa ** 2)) / k2 / th ** 2
    G[0, 0, 0] = 0.0
    wt = torch.full((S.shape[2],), 2.0, dtype=torch.float64)
    wt[0] = 1.0
    if K[2] % 2 == 0:
        wt[-1] = 1.0
    E = 1389.35455846 * (wt * G * (S.real ** 2 + S.imag ** 2)).sum()
    return float(E.detach()), torch.autograd.grad(E, pos)[0].numpy()


TRI = torch.tensor([[1.0, 0.0, 0.0], [0.15, 1.0, 0.0], [-0.1, 0.2, 1.0]], dtype=torch.float64)


# FP64 sums of some 10^4 terms: 1e-11; FP32 meshes: 216 products of six-digit splines, transforms: 2e-5
@pytest.mark.parametrize("precision,tol", [("fp64", 1e-11), ("fp32", 2e-5)])
@pytest.mark.parametrize("n,K,tri", [(1, (6, 6, 6), False), (7, (7, 6, 9), True), (9, (65, 10, 12), False),
                                     (33, (12, 66, 7), True), (500, (30, 27, 67), True),
                                     (9480, (24, 22, 20), False), (18961, (20, 68, 16), False)])
def test_charges_against_float64(n, K, tri, precision, tol):
    rng = np.random.default_rng(n)
    L = 14.0
    box = torch.eye(3, dtype=torch.float64) * L
    box = box @ TRI if tri else box
    pos = rng.uniform(-L, 2 * L, (n, 3))
    q = rng.normal(0.0, 1.0, n)
    kappa = 0.35
    eng = ClassicalEngine(n, n_types=0, coulomb="pme", rc=2.0, kappa=kappa, K=K, cov_rows=np.zeros((0, 3), np.int32),
                          mscales_coul=[1.0] * 6, mscales_lj=[1.0] * 6, precision=precision)
    eng.set_params(q)
    p = torch.tensor(pos, device="cuda")
    res, F = eng.compute(p, box.numpy(), pairs=torch.tensor([[n, n, 0]], dtype=torch.int32, device="cuda"))
    E, G = _structure(pos, q, box, K, kappa)
    assert abs(res.e_coul_recip - E) <= tol * abs(E)
    # a lone charge's force is what the mesh leaves of zero: compare with the energy per length there
    scale = np.sqrt((G ** 2).mean()) + abs(E) / (n * L)
    assert np.sqrt(((F.cpu().numpy() + G) ** 2).mean()) <= 10 * tol * scale


@pytest.mark.parametrize("nw,L,lmax", [(3, 9.0, 2), (11, 9.5, 2), (27, 10.2, 1)])
def test_multipoles_against_the_oracle(nw, L, lmax):
    # FP64: the tolerances of the other comparisons with the oracle (1e-10 energy, 1e-8 forces)
    s = water_box(nw, L, seed=40 + nw, lmax=lmax, pol=True, rc=4.2)
    pr = oracle_pairs(s)
    ref = oracle_reference(s, pr, solver="cg", tol=1e-12)
    eng = make_engine(s, precision="fp64", cg_tol=1e-11)
    pos = torch.tensor(s["pos"], dtype=torch.float64, device="cuda")
    res, F, _ = eng.compute(pos, s["box"], pairs=torch.tensor(pr, dtype=torch.int32, device="cuda"))
    assert abs(res.energy - ref["E"]) <= 1e-10 * abs(ref["E"])
    assert rel_force_rms(F.cpu().numpy(), ref["F"]) <= 1e-8

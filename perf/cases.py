"""Performance cases of the energy / force framework, as a simulation program calls it.

Every case is one evaluation of a molecular system by one public entry point: an engine step of an
MD or serving program (neighbour rebuild, induced dipoles where the model has them, energy, forces
and box gradient) or a differentiable energy of the drop-in layer with its gradients (training).
The systems are liquid water (0.0334 molecules / A^3, the density of the serving stream) built from
the seed, with the cut-offs, Ewald tolerances, multipoles, polarizabilities and dispersion
parameters of the benchmark workloads; the classical systems add short polymer chains.

``exact`` restates the same energies in 64-bit torch (pair sums over all pairs within the cut-off,
B-spline meshes with torch.fft, conjugate gradients for the dipoles) and differentiates them by
autograd.  Engines of precision "fp32" compute in 32 bits, and a program that chose them keeps
their vectors in 32 bits, so these cases return them so.
"""
import math

import numpy as np
import torch

DENSITY = 0.0334  # molecules / A^3
DIEL = 1389.35455846  # kJ/mol A / e^2
RT3 = math.sqrt(3.0)
CG_TOL = 1e-6  # the benchmark's relative tolerance of the dipole solve


def listed():
    return [
        # a small fixed-charge (multipole) box: every step is launches and latency
        {"name": "fixed_216", "kind": "admp", "waters": 216, "pol": False, "precision": "fp32", "rc": 6.0},
        # the small end of the serving stream: dipole solve of a few hundred atoms
        {"name": "pol_150", "kind": "admp", "waters": 150, "pol": True, "precision": "fp32", "rc": 8.0},
        # an ordinary request of the stream, odd in atoms (3999) and mesh
        {"name": "pol_1333", "kind": "admp", "waters": 1333, "pol": True, "precision": "fp32", "rc": 8.0},
        # the headline benchmark's size: an MD step of 12288 polarizable atoms
        {"name": "pol_4096", "kind": "admp", "waters": 4096, "pol": True, "precision": "fp32", "rc": 8.0},
        # the largest request of the stream
        {"name": "pol_10000", "kind": "admp", "waters": 10000, "pol": True, "precision": "fp32", "rc": 8.0},
        # double precision, as used to validate a run or for energy conservation
        {"name": "pol64_2048", "kind": "admp", "waters": 2048, "pol": True, "precision": "fp64", "rc": 8.0},
        # one sample of a parameter fit: neighbour list, energy, gradients of positions, box,
        # multipoles, polarizabilities and Thole widths
        {"name": "train_2048", "kind": "train", "waters": 2048, "precision": "fp32", "rc": 8.0},
        # the same for dispersion PME with Tang-Toennies short range
        {"name": "disp_2048", "kind": "disp", "waters": 2048, "precision": "fp32", "rc": 8.0},
        # classical MD step of a polymer solution on its neighbour list
        {"name": "classical_1000", "kind": "classical", "waters": 1000, "chains": 2, "cell_pass": False,
         "precision": "fp32", "rc": 8.0},
        # the 100 000-atom classical step, pairs straight from the cell grid
        {"name": "classical_33000", "kind": "classical", "waters": 33000, "chains": 20, "cell_pass": True,
         "precision": "fp32", "rc": 10.0},
    ]


def draw(rng):
    def waters(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    k = rng.randrange(10)
    if k < 1:
        return {"kind": "admp", "waters": waters(100, 4000), "pol": False, "precision": "fp32",
                "rc": rng.choice([6.0, 7.0, 8.0])}
    if k < 4:
        return {"kind": "admp", "waters": waters(100, 10000), "pol": True, "precision": "fp32",
                "rc": rng.choice([6.0, 7.0, 8.0])}
    if k < 5:
        return {"kind": "admp", "waters": waters(100, 2500), "pol": True, "precision": "fp64",
                "rc": rng.choice([6.0, 8.0])}
    if k < 6:
        return {"kind": "train", "waters": waters(100, 2500), "precision": "fp32", "rc": rng.choice([6.0, 8.0])}
    if k < 7:
        return {"kind": "disp", "waters": waters(100, 4000), "precision": "fp32", "rc": rng.choice([6.0, 8.0])}
    if k < 8:
        return {"kind": "classical", "waters": waters(300, 4000), "chains": rng.randrange(0, 4), "cell_pass": False,
                "precision": "fp32", "rc": rng.choice([8.0, 9.0])}
    return {"kind": "classical", "waters": waters(1500, 33000), "chains": rng.randrange(0, 12), "cell_pass": True,
            "precision": "fp32", "rc": rng.choice([8.0, 9.0, 10.0])}


# ------------------------------------------------------------------------------- systems
def _rotations(gen, n):
    q = torch.randn((n, 4), generator=gen, dtype=torch.float64)
    w, x, y, z = (q / q.norm(dim=1, keepdim=True)).T
    return torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w),
                        2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w),
                        2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)], 1).reshape(n, 3, 3)


def _body():
    r, th = 0.9572, math.radians(104.52)
    return torch.tensor([[0.0, 0.0, 0.0], [r * math.sin(th / 2), 0.0, r * math.cos(th / 2)],
                         [-r * math.sin(th / 2), 0.0, r * math.cos(th / 2)]], dtype=torch.float64)


def _place(gen, m, a, keep, contact=1.7, rounds=400):
    """Rigid waters near the sites ``keep`` of an m^3 lattice of spacing ``a``: jitter of 0.3 A and
    random orientations, redrawn while an atom is within ``contact`` of another molecule's, each
    redraw kept only where it widens the molecule's closest contact (as equilibrated water has none
    so close).  Returns [n, 3, 3] positions (O, H, H)."""
    sites = torch.tensor(keep, dtype=torch.long)
    n = len(keep)
    ijk = torch.stack([sites // (m * m), (sites // m) % m, sites % m], 1)
    body = _body()

    def draw_mol(k, jitter):
        c = (ijk[k].double() + 0.5) * a + (torch.rand((len(k), 3), generator=gen, dtype=torch.float64) * 2 - 1) * jitter
        return c[:, None, :] + torch.einsum("nij,aj->nai", _rotations(gen, len(k)), body)

    slot = torch.full((m ** 3,), -1, dtype=torch.long)
    slot[sites] = torch.arange(n)
    r = (-1, 0, 1) if m >= 3 else ((0, 1) if m == 2 else (0,))
    offs = torch.tensor([(i, j, k) for i in r for j in r for k in r if (i, j, k) != (0, 0, 0)])
    nb = (ijk[:, None, :] + offs[None]) % m
    nb = slot[(nb[..., 0] * m + nb[..., 1]) * m + nb[..., 2]]  # [n, 26], -1 where empty
    L = a * m

    def closest(mol, idx):
        o = nb[idx]
        d = mol[:, None, :, None, :] - pos[o.clamp(min=0)][:, :, None, :, :]
        d = d - L * torch.round(d / L)
        d = (d * d).sum(-1).reshape(len(idx), o.shape[1], 9)
        d[o < 0] = 1e9
        return d.reshape(len(idx), -1).amin(1).sqrt()

    everyone = torch.arange(n)
    pos = draw_mol(everyone, 0.3)
    near = closest(pos, everyone)
    for rnd in range(rounds):
        bad = (near < contact).nonzero()[:, 0]
        if not len(bad):
            break
        # molecules that move at the same time are not neighbours
        pri = torch.full((n + 1,), -1.0, dtype=torch.float64)
        pri[bad] = torch.rand(len(bad), generator=gen, dtype=torch.float64)
        bad = bad[pri[bad] >= pri[nb[bad]].amax(1)] if nb.shape[1] else bad
        cand = draw_mol(bad, 0.3 if rnd < 200 else 0.15)
        d = closest(cand, bad)
        ok = d > near[bad]
        pos[bad[ok]] = cand[ok]
        touched = torch.zeros(n + 1, dtype=torch.bool)
        touched[bad[ok]] = True
        touched[nb[bad[ok]].reshape(-1)] = True
        touched = touched[:n].nonzero()[:, 0]
        if len(touched):
            near[touched] = closest(pos[touched], touched)
    return pos


def _ewald(rc, ethresh, L):
    kappa = math.sqrt(-math.log(2 * ethresh)) / rc
    return kappa, int(math.ceil(2 * kappa * L / 3 / ethresh ** 0.2))


def _harmonics(rng, n_types):
    """Per-type multipoles in the framework's harmonic order: charges of water, dipoles and traceless
    quadrupoles N(0, 0.1)."""
    rows = []
    for q in (-0.8, 0.4)[:n_types]:
        dx, dy, dz = rng.normal(0.0, 0.1, 3)
        xx, yy, xy, xz, yz = rng.normal(0.0, 0.1, 5)
        rows.append([q, dz, dx, dy, -xx - yy, 2 / RT3 * xz, 2 / RT3 * yz, (xx - yy) / RT3, 2 / RT3 * xy])
    return np.array(rows)


def _water(case, seed):
    """Positions (A), topology and parameters of a water box, all from the seed."""
    nw = case["waters"]
    rng = np.random.default_rng([17, int(seed)])
    gen = torch.Generator().manual_seed(int(seed) + 7919)
    L = (nw / DENSITY) ** (1.0 / 3.0)
    m = int(math.ceil(nw ** (1.0 / 3.0) - 1e-9))
    keep = np.sort(rng.choice(m ** 3, nw, replace=False)) if nw < m ** 3 else np.arange(m ** 3)
    pos = _place(gen, m, L / m, keep.tolist()).reshape(-1, 3)
    o = 3 * np.arange(nw)
    n = 3 * nw
    ax_t = np.tile([1, 0, 0], nw).astype(np.int32)  # O bisector, H z-then-x
    ax_i = np.full((n, 3), -1, np.int32)
    ax_i[o, 0], ax_i[o, 1] = o + 1, o + 2
    ax_i[o + 1, 0], ax_i[o + 1, 1] = o, o + 2
    ax_i[o + 2, 0], ax_i[o + 2, 1] = o, o + 1
    one = np.ones_like(o)
    cov = np.stack([np.stack([o, o + 1, one], 1), np.stack([o, o + 2, one], 1), np.stack([o + 1, o + 2, 2 * one], 1)],
                   1).reshape(-1, 3).astype(np.int32)
    types = np.tile([0, 1, 1], nw)
    rc = min(case["rc"], 0.5 * L * (1 - 1e-6))
    kappa, K = _ewald(rc, 5e-4, L)
    C = np.stack([np.exp(rng.normal(math.log(c), 0.5, 2)) for c in (1e-3, 1e-4, 1e-5)], 1)[types]
    return dict(n=n, pos=pos, L=L, box=np.eye(3) * L, axis_types=ax_t, axis_indices=ax_i, cov=cov, types=types, rc=rc,
                ethresh=5e-4, kappa=kappa, K=K, Q=_harmonics(rng, 2)[types],
                alpha=np.where(types == 0, 1.0, 0.5), thole=np.full(n, 0.33),
                c=np.sqrt(C * np.array([1e6, 1e8, 1e10])), tt_a=np.array([1203470.743, 83.2283563])[types] / 2625.5,
                tt_b=np.full(n, 35.0 * 0.0529177249), tt_q=np.array([-0.741706, 0.370853])[types])


def _mixture(case, seed):
    """Water with straight zig-zag chains (bond 1.53 A) along z, each in a 2 x 2 column of lattice
    sites left free of water; harmonic bonds and angles everywhere, torsions along the chains."""
    rng = np.random.default_rng([23, int(seed)])
    gen = torch.Generator().manual_seed(int(seed) + 104729)
    nch = case["chains"]
    m = 3
    while m ** 3 - 4 * m * min(nch, (m // 3) ** 2) < case["waters"]:
        m += 1
    nch = min(nch, (m // 3) ** 2)
    L = ((case["waters"] + 4 * m * nch) / DENSITY) ** (1.0 / 3.0)
    a = L / m
    taken = np.zeros((m, m, m), bool)
    spots = [(3 * i, 3 * j) for i in range(m // 3) for j in range(m // 3)]
    spots = [spots[k] for k in rng.permutation(len(spots))[:nch]]
    nb = max(2, int((L - 4.0) / 1.27))
    chains = []
    for i, j in spots:
        taken[i:i + 2, j:j + 2, :] = True
        k = np.arange(nb)
        x = np.stack([(i + 1) * a + 0.427 * (-1.0) ** k, np.full(nb, (j + 1) * a), 2.0 + 1.27 * k], 1)
        chains.append(x + rng.normal(0.0, 0.08, x.shape))
    free = np.nonzero(~taken.reshape(-1))[0]
    keep = np.sort(rng.choice(free, case["waters"], replace=False))
    wat = _place(gen, m, a, keep.tolist()).reshape(-1, 3)
    nw, n0 = case["waters"], nch * nb
    n = n0 + 3 * nw
    pos = torch.cat([torch.tensor(np.concatenate(chains) if chains else np.zeros((0, 3))), wat])
    o = n0 + 3 * np.arange(nw)
    q = [c - c.mean() for c in rng.normal(0.0, 0.3, (nch, nb))]
    q = np.concatenate(q + [np.tile([-0.834, 0.417, 0.417], nw)])
    types = np.concatenate([np.tile(np.arange(nb) % 8, nch), np.tile([8, 9, 9], nw)]).astype(np.int32)
    sig = np.concatenate([rng.uniform(3.0, 3.8, 8), [3.15061, 0.0]])
    eps = np.concatenate([rng.uniform(0.2, 0.8, 8), [0.6364, 0.0]])
    base = (np.arange(nch) * nb)[:, None]
    step = lambda w: (base + np.arange(nb - w)[None]).reshape(-1)  # noqa: E731
    b0, a0, t0 = step(1), step(2), step(3)
    bonds = np.concatenate([np.stack([b0, b0 + 1], 1), np.stack([o, o + 1], 1), np.stack([o, o + 2], 1)])
    bond_p = np.concatenate([np.stack([np.full(len(b0), 2000.0), rng.uniform(1.48, 1.58, len(b0))], 1),
                             np.tile([4500.0, 0.96], (2 * nw, 1))])
    angles = np.concatenate([np.stack([a0, a0 + 1, a0 + 2], 1), np.stack([o + 1, o, o + 2], 1)])
    angle_p = np.concatenate([np.tile([400.0, math.radians(110.0)], (len(a0), 1)),
                              np.tile([380.0, math.radians(104.52)], (nw, 1))])
    tors = np.repeat(np.stack([t0, t0 + 1, t0 + 2, t0 + 3], 1), 3, axis=0)
    tors_p = np.stack([rng.uniform(0.5, 2.0, len(tors)), rng.choice([0.0, math.pi], len(tors)),
                       np.tile([1.0, 2.0, 3.0], len(t0))], 1)
    one = np.ones_like
    cov = [np.stack([step(w), step(w) + w, w * one(step(w))], 1) for w in range(1, min(6, nb - 1) + 1)]
    cov = np.concatenate(cov + [np.stack([o, o + 1, one(o)], 1), np.stack([o, o + 2, one(o)], 1),
                                np.stack([o + 1, o + 2, 2 * one(o)], 1)])
    cov = cov[np.lexsort((cov[:, 1], cov[:, 0]))].astype(np.int32)
    rc = min(case["rc"], 0.5 * L * (1 - 1e-6))
    kappa, K = _ewald(rc, 1e-5, L)
    return dict(n=n, pos=pos, L=L, box=np.eye(3) * L, cov=cov, rc=rc, kappa=kappa, K=K, q=q, types=types,
                sig=(sig[:, None] + sig[None]) * 0.5, eps=np.sqrt(eps[:, None] * eps[None] + 1e-32),
                bonds=bonds, bond_p=bond_p, angles=angles, angle_p=angle_p, tors=tors, tors_p=tors_p)


M_SCALES = [0.0, 0.0, 1.0, 1.0, 1.0, 1.0]
D_SCALES = [1.0] * 6
DISP_SCALES = [0.0, 0.0, 0.0, 1.0, 1.0, 1.0]
COUL_SCALES = [0.0, 0.0, 0.8333333333333334, 1.0, 1.0, 1.0]
LJ_SCALES = [0.0, 0.0, 0.5, 1.0, 1.0, 1.0]


# ------------------------------------------------------------------------------- cases
def prepare(case, seed):
    kind = case["kind"]
    s = _mixture(case, seed) if kind == "classical" else _water(case, seed)
    K = (s["K"],) * 3
    pos = s["pos"].cuda().contiguous()
    state = {"kind": kind, "half": case["precision"] == "fp32", "pos": pos, "box": s["box"]}
    if kind == "admp":
        from dmff_b200.engine import AdmpEngine
        pol = case["pol"]
        eng = AdmpEngine(s["n"], 2, pol, True, s["rc"], s["kappa"], K, s["axis_types"], s["axis_indices"], s["cov"],
                         M_SCALES, M_SCALES if pol else None, D_SCALES if pol else None, precision=case["precision"],
                         cg_tol=CG_TOL)
        eng.set_params(s["Q"], s["alpha"] if pol else None, s["thole"] if pol else None)
        if pol:
            eng.set_zero_guess(True)
        return dict(state, eng=eng, pol=pol)
    if kind == "classical":
        from dmff_b200.engine import ClassicalEngine
        eng = ClassicalEngine(s["n"], n_types=10, coulomb="pme", rc=s["rc"], kappa=s["kappa"], K=K, cov_rows=s["cov"],
                              mscales_coul=COUL_SCALES, mscales_lj=LJ_SCALES, precision=case["precision"])
        eng.set_params(s["q"], s["types"], s["sig"], s["eps"])
        eng.set_terms("bond", s["bonds"], s["bond_p"])
        eng.set_terms("angle", s["angles"], s["angle_p"])
        if len(s["tors"]):
            eng.set_terms("torsion", s["tors"], s["tors_p"])
        eng.set_cell_pass(case["cell_pass"])
        return dict(state, eng=eng, list=not case["cell_pass"])
    from dmff_b200.api.topology import CovalentMap
    from dmff_b200.common.nblist import NeighborList
    cov = CovalentMap(s["n"], s["cov"])
    nl = NeighborList(s["box"], s["rc"], cov)
    box = torch.tensor(s["box"], requires_grad=True)
    leaf = lambda x: torch.tensor(x, dtype=torch.float64, device="cuda", requires_grad=True)  # noqa: E731
    pos.requires_grad_(True)
    state = dict(state, nl=nl, box=box)
    if kind == "train":
        from dmff_b200.admp.pme import ADMPPmeForce
        f = ADMPPmeForce(s["box"], np.arange(s["n"]), s["axis_types"], s["axis_indices"], s["rc"], s["ethresh"], 2,
                         lpol=True, cov_rows=s["cov"], precision=case["precision"], cg_tol=CG_TOL)
        return dict(state, force=f, prm=[leaf(s["Q"]), leaf(s["alpha"]), leaf(s["thole"])],
                    scales=[torch.tensor(x, dtype=torch.float64) for x in (M_SCALES, M_SCALES, D_SCALES)])
    from dmff_b200.admp.disp_pme import ADMPDispPmeForce
    f = ADMPDispPmeForce(s["box"], s["rc"], s["ethresh"], 10, cov_rows=s["cov"], tt_damping=True,
                         precision=case["precision"])
    return dict(state, force=f, prm=[leaf(s["c"]), leaf(s["tt_a"]), leaf(s["tt_b"]), leaf(s["tt_q"])],
                scales=torch.tensor(DISP_SCALES, dtype=torch.float64))


def run(state):
    kind, pos = state["kind"], state["pos"]
    keep = (lambda t: t.float()) if state["half"] else (lambda t: t)
    if kind == "admp":
        eng = state["eng"]
        eng.rebuild_internal_pairs(pos, state["box"])
        res, F, U = eng.compute(pos, state["box"])
        out = {"energy": res.energy, "forces": keep(F), "box_grad": keep(torch.tensor(res.box_grad[:], dtype=torch.float64))}
        if state["pol"]:
            out["dipoles"] = keep(U)
        return out
    if kind == "classical":
        eng = state["eng"]
        if state["list"]:
            eng.rebuild_internal_pairs(pos, state["box"])
        res, F = eng.compute(pos, state["box"])
        # the terms of the energy, as a program logs them (their sum cancels to any small value)
        return {"e_coul": [res.e_coul_real, res.e_coul_recip], "e_lj": res.e_lj,
                "e_bonded": res.e_bond + res.e_angle + res.e_torsion, "forces": keep(F), "box_grad": keep(torch.tensor(res.box_grad[:], dtype=torch.float64))}
    pairs = state["nl"].allocate(pos)
    prm, box = state["prm"], state["box"]
    if kind == "train":
        E = state["force"].get_energy(pos, box, pairs, *prm, *state["scales"])
    else:
        E = state["force"].get_energy(pos, box, pairs, prm[0], state["scales"], tt=tuple(prm[1:]))
    g = torch.autograd.grad(E, [pos, box, *prm])
    return {"energy": float(E.detach()), "g_pos": keep(g[0]), "g_box": keep(g[1]), "g_prm": [keep(x) for x in g[2:]]}


def work(case):
    n = 3 * case["waters"] + (case.get("chains", 0) * 50)
    L = (case["waters"] / DENSITY) ** (1.0 / 3.0)
    rc = min(case["rc"], 0.5 * L)
    pairs = n * 0.5 * 4.0 / 3.0 * math.pi * rc ** 3 * 3 * DENSITY
    wide = 8 if case["precision"] == "fp64" else 4
    kind = case["kind"]
    K = _ewald(rc, 1e-5 if kind == "classical" else 5e-4, L)[1]
    K3 = float(K) ** 3
    fft = 5.0 * K3 * math.log2(K3)  # a forward and an inverse real transform
    # positions in, forces out, parameters in; the mesh once out and back for each transform pair
    if kind == "admp":
        it = 12 if case["pol"] else 0
        return {"bytes": n * (24 + 24 + 72 + (40 if case["pol"] else 0)) + (1 + it) * 2 * wide * K3,
                "flops": pairs * ((1900 + 600 + 200 + it * 2 * 24) if case["pol"] else 1450) + (1 + it) * fft
                + (2 + it) * n * 216 * 8}
    if kind == "train":
        return {"bytes": n * (24 + 24 + 2 * 88) + 14 * 2 * wide * K3,
                "flops": pairs * (1900 + 600 + 200 + 2000 + 12 * 48) + 14 * fft + 14 * n * 216 * 8}
    if kind == "disp":
        return {"bytes": n * (24 + 24 + 2 * 48) + 3 * 2 * wide * K3, "flops": pairs * 500 + 3 * fft + 6 * n * 216 * 4}
    return {"bytes": n * (24 + 24 + 12) + 2 * wide * K3, "flops": pairs * 120 + fft + 2 * n * 216 * 4}


# ------------------------------------------------------------------------------- 64-bit values
def _all_pairs(pos, L, rc):
    """Every i < j with minimum-image distance < rc."""
    n, out = pos.shape[0], []
    step = max(1, 40_000_000 // n)
    for a in range(0, n, step):
        d = pos[a:a + step, None, :] - pos[None, :, :]
        d -= L * torch.floor(d / L + 0.5)
        i, j = ((d * d).sum(-1) < rc * rc).nonzero(as_tuple=True)
        i = i + a
        ok = i < j
        out.append(torch.stack([i[ok], j[ok]]))
    return torch.cat(out, 1)


def _nbond(ij, cov, n):
    """Topological distance of each pair (0: none)."""
    key, order = np.unique(cov[:, 0].astype(np.int64) * n + cov[:, 1], return_index=True)
    key = torch.tensor(key, device=ij.device)
    val = torch.tensor(cov[order, 2].astype(np.int64), device=ij.device)
    q = ij[0] * n + ij[1]
    at = torch.searchsorted(key, q).clamp(max=len(key) - 1)
    return torch.where(key[at] == q, val[at], 0)


def _scale(table, nb):
    t = torch.tensor(table, dtype=torch.float64, device=nb.device)
    return t[torch.where(nb > 0, nb - 1, 5)]


def _image(d, box):
    """Minimum-image vectors; the image numbers are constants of the differentiation."""
    with torch.no_grad():
        k = torch.floor(d @ torch.linalg.inv(box) + 0.5)
    return d - k @ box


def _splines(w):
    """Order-6 B-spline at w + 0 .. w + 5 (last axis) with its first and second derivatives."""
    def up(m, k):  # order k - 1 -> k
        z = torch.zeros_like(m[..., :1])
        lo, hi = torch.cat([m, z], -1), torch.cat([z, m], -1)
        u = w[..., None] + torch.arange(k, dtype=w.dtype, device=w.device)
        return (u * lo + (k - u) * hi) / (k - 1)

    def diff(m):
        z = torch.zeros_like(m[..., :1])
        return torch.cat([m, z], -1) - torch.cat([z, m], -1)

    m4 = up(up(torch.stack([w, 1 - w], -1), 3), 4)
    m5 = up(m4, 5)
    return up(m5, 6), diff(m5), diff(diff(m4))


def _mesh_energy(pos, box, K, q, mu, Th, green):
    """sum_k green(k^2, V) |S(k) / b(k)|^2 of charges, dipoles and quadrupoles (q + mu.d + Th:dd / 3).
    Mesh derivatives are taken with the transpose of the scaled inverse box, as the model defines
    them (it differs from the inverse box itself only where a box gradient is taken)."""
    hinv = torch.linalg.inv(box)
    x = K * (pos @ hinv)
    with torch.no_grad():
        c = torch.ceil(x)
    M, D, DD = _splines(c - x)  # [n, 3, 6]; a point's distance u = c - x + j falls with x
    at = [(c[:, d].long()[:, None] - 3 + torch.arange(6, device=pos.device)) % K for d in range(3)]
    flat = ((at[0][:, :, None, None] * K + at[1][:, None, :, None]) * K + at[2][:, None, None, :])
    ein = lambda a, b, e: a[:, :, None, None] * b[:, None, :, None] * e[:, None, None, :]  # noqa: E731
    v = q[:, None, None, None] * ein(M[:, 0], M[:, 1], M[:, 2])
    if mu is not None:
        m = -K * (mu @ hinv.T)
        v = v + ein(m[:, 0, None] * D[:, 0], M[:, 1], M[:, 2]) + ein(m[:, 1, None] * M[:, 0], D[:, 1], M[:, 2]) \
            + ein(m[:, 2, None] * M[:, 0], M[:, 1], D[:, 2])
    if Th is not None:
        t = K * K / 3.0 * torch.einsum("cj,njk,dk->ncd", hinv, Th, hinv)
        v = v + ein(t[:, 0, 0, None] * DD[:, 0], M[:, 1], M[:, 2]) + ein(t[:, 1, 1, None] * M[:, 0], DD[:, 1], M[:, 2]) \
            + ein(t[:, 2, 2, None] * M[:, 0], M[:, 1], DD[:, 2]) \
            + 2 * ein(t[:, 0, 1, None] * D[:, 0], D[:, 1], M[:, 2]) \
            + 2 * ein(t[:, 0, 2, None] * D[:, 0], M[:, 1], D[:, 2]) \
            + 2 * ein(t[:, 1, 2, None] * M[:, 0], D[:, 1], D[:, 2])
    S = torch.zeros(K ** 3, dtype=torch.float64, device=pos.device).index_add(0, flat.reshape(-1), v.reshape(-1))
    S = torch.fft.rfftn(S.reshape(K, K, K))
    k = torch.arange(K, device=pos.device)
    k = torch.where(k < (K + 1) // 2, k, k - K).double()
    b5 = torch.tensor([1.0, 26.0, 66.0, 26.0, 1.0], dtype=torch.float64, device=pos.device) / 120.0
    off = torch.arange(-2, 3, device=pos.device).double()
    bm = (b5 * torch.cos(2 * math.pi * k[:, None] * off / K)).sum(1)
    h = K // 2 + 1
    kk = torch.stack(torch.meshgrid(k, k, k[:h], indexing="ij"), -1)
    ksq = ((2 * math.pi * kk @ hinv.T) ** 2).sum(-1)
    w = torch.full((h,), 2.0, dtype=torch.float64, device=pos.device)
    w[0] = 1.0
    if K % 2 == 0:
        w[-1] = 1.0
    b = bm[:, None, None] * bm[None, :, None] * bm[None, None, :h]
    return (green(ksq, torch.linalg.det(box)) * w * (S.real ** 2 + S.imag ** 2) / (b * b)).sum()


def _green_coulomb(kappa):
    def green(ksq, V):
        zero = ksq == 0
        k = torch.where(zero, torch.ones_like(ksq), ksq)
        return torch.where(zero, torch.zeros_like(k), 2 * math.pi / V / k * torch.exp(-k / 4 / kappa ** 2))
    return green


def _green_disp(kappa, p):
    def green(ksq, V):
        x2 = ksq.clamp(min=1e-16) / 4 / kappa ** 2
        x = x2.sqrt()
        e, f = torch.exp(-x2), math.sqrt(math.pi) * torch.special.erfc(x)
        if p == 6:
            g, d = (1 - 2 * x2) * e + 2 * x ** 3 * f, 3
        elif p == 8:
            g, d = (3 - 2 * x2 + 4 * x2 ** 2) * e - 4 * x ** 5 * f, 45
        else:
            g, d = (15 - 6 * x2 + 4 * x2 ** 2 - 8 * x2 ** 3) * e + 8 * x ** 7 * f, 1260
        return math.pi ** 1.5 / 2 / V * kappa ** (p - 3) * g / d
    return green


def _global_multipoles(pos, box, s, Q):
    """Charges, dipoles and traceless quadrupole tensors of the waters in the laboratory frame."""
    dev = pos.device
    ia = torch.tensor(s["axis_indices"].astype(np.int64), device=dev)
    unit = lambda v: v / v.norm(dim=1, keepdim=True)  # noqa: E731
    z = unit(_image(pos[ia[:, 0]] - pos, box))
    x = unit(_image(pos[ia[:, 1]] - pos, box))
    bis = torch.tensor(s["axis_types"] == 1, device=dev)[:, None]
    z = torch.where(bis, unit(z + x), z)
    x = unit(x - z * (x * z).sum(1, keepdim=True))
    R = torch.stack([x, torch.linalg.cross(z, x), z], 1)  # rows: local axes
    mu = torch.einsum("na,nab->nb", Q[:, [2, 3, 1]], R)
    zz, xz, yz, dd, xy = (Q[:, 4], Q[:, 5] * RT3 / 2, Q[:, 6] * RT3 / 2, Q[:, 7] * RT3 / 2, Q[:, 8] * RT3 / 2)
    xx, yy = -zz / 2 + dd, -zz / 2 - dd
    Th = torch.stack([xx, xy, xz, xy, yy, yz, xz, yz, zz], 1).reshape(-1, 3, 3)
    return Q[:, 0], mu, torch.einsum("nai,nab,nbj->nij", R, Th, R)


def _pair_multipole(d, mp, ij, U, s, alpha, thole, nb):
    """Real-space energy of the pairs (vectors d = r_i - r_j): permanent multipoles with the
    screened 1/r operators, induced dipoles with Thole-damped ones."""
    kap = s["kappa"]
    q, mu, Th = mp
    i, j = ij
    r = d.norm(dim=1)
    z = d / r[:, None]
    a = kap * r
    X = 2 / math.sqrt(math.pi) * torch.exp(-a * a)
    m = _scale(M_SCALES, nb)
    e1 = torch.special.erfc(a) - 1
    e2 = e1 + a * X
    e3 = e2 + 2 / 3 * a ** 3 * X
    e4 = e3 + 4 / 15 * a ** 5 * X
    dot = lambda u, v: (u * v).sum(-1)  # noqa: E731
    di, dj = dot(mu[i], z), dot(mu[j], z)
    dperp = dot(mu[i], mu[j]) - di * dj
    Ai, Aj = torch.einsum("nab,nb->na", Th[i], z), torch.einsum("nab,nb->na", Th[j], z)
    ti, tj = dot(Ai, z), dot(Aj, z)
    c = 2 / RT3
    pij = c * (dot(mu[j], Ai) - dj * ti)  # transverse dipole of j with quadrupole of i
    pji = c * (dot(mu[i], Aj) - di * tj)
    aa = c * c * (dot(Ai, Aj) - ti * tj)
    # transverse blocks: tr(P_i P_j) with P = (1 - zz) Th (1 - zz)
    tt = torch.einsum("nab,nab->n", Th[i], Th[j]) - 2 * dot(Ai, Aj) + ti * tj
    bb = 2 / 3 * (tt - ti * tj / 2)
    a3, a5 = a ** 3 * X, a ** 5 * X
    cc = (m + e1) / r
    cd = (m + e2) / r ** 2
    dd0 = -2 / 3 * (3 * (m + e3) + a3) / r ** 3
    dd1 = (m + e3 - 2 / 3 * a3) / r ** 3
    cq = (m + e3) / r ** 3
    dq0 = (3 * (m + e3) + 4 / 3 * a5) / r ** 4
    dq1 = -RT3 * (m + e3) / r ** 4
    qq0 = (6 * (m + e4) + 4 / 45 * (10 * a * a - 3) * a5) / r ** 5
    qq1 = -4 / 15 * (15 * (m + e4) + a5) / r ** 5
    qq2 = (m + e4 - 4 / 15 * a5) / r ** 5
    qi, qj = q[i], q[j]
    E = cc * qi * qj + cd * (qi * dj - qj * di) + dd0 * di * dj + dd1 * dperp + cq * (qi * tj + qj * ti) \
        + dq0 * (dj * ti - di * tj) + dq1 * (pij - pji) + qq0 * ti * tj + qq1 * aa + qq2 * bb
    if U is not None:
        p, ds = m, _scale(D_SCALES, nb)
        wid = torch.where(p > 0, torch.full_like(p, 5.0), thole[i] + thole[j])
        au = wid * r / (alpha[i] * alpha[j]) ** (1 / 6)
        ee = torch.where(au < 50, torch.exp(-au.clamp(max=50.0)), torch.zeros_like(au))
        P = 1 + au + au * au / 2
        tc, td0 = 1 - ee * P, 1 - ee * (P + au ** 3 / 4)
        tq0, tq1 = 1 - ee * (P + au ** 3 / 6 + au ** 4 / 18), 1 - ee * (P + au ** 3 / 6)
        ui, uj = dot(U[i], z), dot(U[j], z)
        cud = (p * tc + e2) / r ** 2
        dud0 = -2 / 3 * (3 * (p * td0 + e3) + a3) / r ** 3
        dud1 = (p * tc + e3 - 2 / 3 * a3) / r ** 3
        udq0 = (3 * (p * tq0 + e3) + 4 / 3 * a5) / r ** 4
        udq1 = -RT3 * (p * tq1 + e3) / r ** 4
        uu0 = -2 / 3 * (3 * (ds * td0 + e3) + a3) / r ** 3
        uu1 = (ds * tc + e3 - 2 / 3 * a3) / r ** 3
        E = E + cud * (qi * uj - qj * ui) + dud0 * (dj * ui + di * uj) \
            + dud1 * (dot(mu[j], U[i]) - dj * ui + dot(mu[i], U[j]) - di * uj) + udq0 * (uj * ti - ui * tj) \
            + udq1 * c * (dot(U[j], Ai) - uj * ti - dot(U[i], Aj) + ui * tj) \
            + uu0 * ui * uj + uu1 * (dot(U[i], U[j]) - ui * uj)
    return DIEL * E.sum()


def _admp_exact(s, pol, dev, want_prm):
    pos = s["pos"].clone().to(dev).requires_grad_(True)
    box = torch.tensor(s["box"], device=dev, requires_grad=True)
    Q, al, th = (torch.tensor(s[k], device=dev, requires_grad=True) for k in ("Q", "alpha", "thole"))
    ij = _all_pairs(pos.detach(), s["L"], s["rc"])
    nb = _nbond(ij, s["cov"], s["n"])
    kap, K = s["kappa"], s["K"]

    def energy(U, mp, d):
        e = _pair_multipole(d, mp, ij, U, s, al, th, nb)
        q, mu, Th = mp
        mt = mu if U is None else mu + U
        e = e + DIEL * _mesh_energy(pos, box, K, q, mt, Th, _green_coulomb(kap))
        f0 = kap / math.sqrt(math.pi)
        # quadrupole self term over the five harmonics: (2/3) Th:Th
        e = e - DIEL * f0 * ((q * q).sum() + 2 / 3 * kap ** 2 * (mt * mt).sum()
                             + 4 / 15 * kap ** 4 * 2 / 3 * (Th * Th).sum())
        return e if U is None else e + DIEL * 0.5 * ((U * U).sum(1) / al).sum()

    def geometry():
        return _global_multipoles(pos, box, s, Q), _image(pos[ij[0]] - pos[ij[1]], box)

    U = None
    if pol:
        with torch.no_grad():
            mp0, d0 = geometry()

        def grad_U(u):
            u = u.detach().requires_grad_(True)
            return torch.autograd.grad(energy(u, mp0, d0), u)[0]

        x = torch.zeros_like(pos).detach()
        g0 = grad_U(x)
        r = -g0
        pre = al.detach()[:, None] / DIEL
        p = z = r * pre
        rz, stop = (r * z).sum(), 1e-11 * g0.norm()
        for _ in range(100):
            Ap = grad_U(p) - g0
            a = rz / (p * Ap).sum()
            x, r = x + a * p, r - a * Ap
            if r.norm() < stop:
                break
            z = r * pre
            rz, old = (r * z).sum(), rz
            p = z + rz / old * p
        U = x
    E = energy(U, *geometry())
    wrt = [pos, box] + ([Q, al, th] if want_prm else [])
    return E.detach(), torch.autograd.grad(E, wrt), U


def _disp_exact(s, dev):
    pos = s["pos"].clone().to(dev).requires_grad_(True)
    box = torch.tensor(s["box"], device=dev, requires_grad=True)
    c, A, B, q = (torch.tensor(s[k], device=dev, requires_grad=True) for k in ("c", "tt_a", "tt_b", "tt_q"))
    ij = _all_pairs(pos.detach(), s["L"], s["rc"])
    i, j = ij
    m = _scale(DISP_SCALES, _nbond(ij, s["cov"], s["n"]))
    kap = s["kappa"]
    r = _image(pos[i] - pos[j], box).norm(dim=1)
    x2 = (kap * r) ** 2
    e = torch.exp(-x2)
    g6 = 1 + x2 + x2 ** 2 / 2
    g8 = g6 + x2 ** 3 / 6
    g10 = g8 + x2 ** 4 / 24
    cc = c[i] * c[j]
    lr = ((m + g6 * e - 1) * cc[:, 0] / r ** 6 + (m + g8 * e - 1) * cc[:, 1] / r ** 8
          + (m + g10 * e - 1) * cc[:, 2] / r ** 10).sum()
    for k, p in enumerate((6, 8, 10)):
        lr = lr + _mesh_energy(pos, box, s["K"], c[:, k], None, None, _green_disp(kap, p))
    sq = (c * c).sum(0)
    lr = lr - kap ** 6 / 12 * sq[0] - kap ** 8 / 48 * sq[1] - kap ** 10 / 240 * sq[2]
    rb = r * 1.889726878
    x = torch.sqrt(B[i] * B[j]) * rb
    poly = 1 + x + x ** 2 / 2 + x ** 3 / 6 + x ** 4 / 24 + x ** 5 / 120 + x ** 6 / 720
    sr = (m * torch.exp(-x) * (2625.5 * torch.sqrt(A[i] * A[j]) - 2625.5 * (1 + x) * q[i] * q[j] / rb
                               + poly * cc[:, 0] / r ** 6)).sum()
    E = sr - lr
    return E.detach(), torch.autograd.grad(E, [pos, box, c, A, B, q])


def _classical_exact(s, dev):
    pos = s["pos"].clone().to(dev).requires_grad_(True)
    box = torch.tensor(s["box"], device=dev, requires_grad=True)
    q, types = torch.tensor(s["q"], device=dev), torch.tensor(s["types"].astype(np.int64), device=dev)
    sig, eps = torch.tensor(s["sig"], device=dev), torch.tensor(s["eps"], device=dev)
    kap, e_real, e_lj = s["kappa"], 0.0, 0.0
    gp, gb = torch.zeros_like(pos).detach(), torch.zeros_like(box).detach()

    def add(e):
        a, b = torch.autograd.grad(e, [pos, box], allow_unused=True)
        gp.add_(a)
        if b is not None:
            gb.add_(b)
        return float(e.detach())

    every = _all_pairs(pos.detach(), s["L"], s["rc"])
    for ij in every.split(4_000_000, dim=1):
        i, j = ij
        nb = _nbond(ij, s["cov"], s["n"])
        r = _image(pos[i] - pos[j], box).norm(dim=1)
        coul = (DIEL * q[i] * q[j] * (_scale(COUL_SCALES, nb) - 1 + torch.special.erfc(kap * r)) / r).sum()
        s6 = (sig[types[i], types[j]] / r) ** 6
        lj = (4 * eps[types[i], types[j]] * _scale(LJ_SCALES, nb) * (s6 * s6 - s6)).sum()
        e_lj += float(lj.detach())
        e_real += float(coul.detach())
        add(coul + lj)
    e_recip = add(DIEL * _mesh_energy(pos, box, s["K"], q, None, None, _green_coulomb(kap)))
    b, bp = torch.tensor(s["bonds"], device=dev), torch.tensor(s["bond_p"], device=dev)
    a, ap = torch.tensor(s["angles"], device=dev), torch.tensor(s["angle_p"], device=dev)
    bonded = add((bp[:, 0] / 2 * ((pos[b[:, 1]] - pos[b[:, 0]]).norm(dim=1) - bp[:, 1]) ** 2).sum())
    unit = lambda v: v / v.norm(dim=1, keepdim=True)  # noqa: E731
    cs = (unit(pos[a[:, 1]] - pos[a[:, 0]]) * unit(pos[a[:, 1]] - pos[a[:, 2]])).sum(1)
    bonded += add((ap[:, 0] / 2 * (torch.arccos(cs) - ap[:, 1]) ** 2).sum())
    if len(s["tors"]):
        t, tp = torch.tensor(s["tors"], device=dev), torch.tensor(s["tors_p"], device=dev)
        b1, b2, b3 = (pos[t[:, k + 1]] - pos[t[:, k]] for k in range(3))
        n1, n2 = torch.linalg.cross(b1, b2), torch.linalg.cross(b2, b3)
        phi = torch.atan2(b2.norm(dim=1) * (b1 * n2).sum(1), (n1 * n2).sum(1))
        bonded += add((tp[:, 0] * (1 + torch.cos(tp[:, 2] * phi - tp[:, 1]))).sum())
    return [e_real, e_recip], e_lj, bonded, gp, gb


def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    kind = case["kind"]
    if kind == "classical":
        e_coul, e_lj, bonded, gp, gb = _classical_exact(_mixture(case, seed), dev)
        return {"e_coul": e_coul, "e_lj": e_lj, "e_bonded": bonded, "forces": -gp, "box_grad": gb.reshape(9)}
    s = _water(case, seed)
    if kind == "disp":
        E, g = _disp_exact(s, dev)
        return {"energy": float(E), "g_pos": g[0], "g_box": g[1], "g_prm": list(g[2:])}
    E, g, U = _admp_exact(s, kind == "train" or case["pol"], dev, kind == "train")
    if kind == "train":
        return {"energy": float(E), "g_pos": g[0], "g_box": g[1], "g_prm": list(g[2:])}
    out = {"energy": float(E), "forces": -g[0], "box_grad": g[1].reshape(9)}
    if case["pol"]:
        out["dipoles"] = U
    return out

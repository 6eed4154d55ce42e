"""The work that a user of this framework has it do, as cases that can be
timed and compared: the Hamiltonian product, the block products of the
eigensolver, one GCG call, densities, the Coulomb solve and one self-consistent
update, each through the public entry points. An HF iteration is one such
update and one GCG call per species.

Sizes are those of the repository's own configurations (16O on 30^3, 24Mg on
32^3, 40Ca on 36^3, the 40^3 x 64 block, 120Sn on 48^3 with HFB pairing) and
generic ones around them. Inputs are made on the GPU from the seed alone,
without the library: localised orbitals, Woods-Saxon-like wells, Fermi-shaped
densities.

Eigenvectors are only defined up to a rotation inside a degenerate level, and
every level here is a Kramers pair, so the eigensolver cases return what a
self-consistent loop reads from the block: the eigenvalues, and the densities
rho and tau of all its columns. The unconverged corrections of one GCG
iteration amplify rounding to about 1e-7 of the orbitals (second order in the
eigenvalues), so those densities are returned in single precision, as the
repository's fixtures keep theirs.
"""
import ctypes as C
import math
import random

import numpy as np
import torch

import nuclearcgm_gb300 as ng
from nuclearcgm_gb300 import abi, config

DEV = "cuda"
PREC = {"fp64": abi.FP64, "fp32": abi.FP32, "fp32_tc": abi.FP32_TC}
H2M = 20.7355  # hbar^2 / 2m [MeV fm^2]
E2 = 1.43996446  # e^2 of the Poisson halo and source [MeV fm]


def listed():
    return [
        # one small H.X in the form the correction solver uses: a launch and
        # little else (a 16O block)
        {"name": "hx_small", "kind": "hx", "n": 30, "cols": 12,
         "precision": "fp32"},
        # the headline H.X: the 40^3 x 64 block in FP32
        {"name": "hx_block64", "kind": "hx", "n": 40, "cols": 64,
         "precision": "fp32"},
        # H.X in FP64 on a 40Ca Rayleigh-Ritz search space (60 columns)
        {"name": "hx_rr60", "kind": "hx", "n": 36, "cols": 60,
         "precision": "fp64"},
        # the reference-facing call: complex128 host arrays in the Eigen
        # layout, default precision, copies included
        {"name": "hx_host", "kind": "hx_host", "n": 30, "cols": 16,
         "precision": "fp64"},
        # the orthonormalisation's products at the 40Ca size: V^H V, V C
        {"name": "dense_ca40", "kind": "dense", "n": 36, "m": 60, "k": 60,
         "precision": "fp64"},
        # densities of the occupied 40Ca orbitals
        {"name": "densities_ca40", "kind": "densities", "n": 36, "cols": 20},
        # Coulomb solve on the 120Sn lattice from a cold start
        {"name": "poisson_sn120", "kind": "poisson", "n": 48, "Z": 50,
         "warm": False},
        # one GCG call of an HF iteration: 16O, default precision
        {"name": "gcg_o16", "kind": "gcg", "n": 30, "nev": 8, "pcols": 8,
         "precision": "fp64"},
        # 40Ca in the tensor-core form
        {"name": "gcg_ca40_tc", "kind": "gcg", "n": 36, "nev": 20,
         "pcols": 20, "precision": "fp32_tc"},
        # the 64-column block with conjugate directions, default precision
        {"name": "gcg_block64", "kind": "gcg", "n": 40, "nev": 64,
         "pcols": 64, "precision": "fp64"},
        # one self-consistent update with HFB pairing (a reduced 120Sn)
        {"name": "state_hfb", "kind": "state", "n": 40, "A": 120, "Z": 50,
         "basis": 80, "pairing": "HFB"},
        # the same call for 40Ca in the default precision
        {"name": "gcg_ca40", "kind": "gcg", "n": 36, "nev": 20,
         "pcols": 20, "precision": "fp64"},
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["hx", "hx", "hx_host", "dense", "densities",
                       "poisson", "gcg", "gcg", "state"])
    if kind == "hx":
        prec = rng.choice(["fp32", "fp64"])
        n = rng.randint(30 if prec == "fp32" else 16, 48)
        lo = 10 if prec == "fp32" else 4
        cols = _logint(rng, lo, min(64, 40 ** 3 * 64 // n ** 3))
        return {"kind": kind, "n": n, "cols": cols, "precision": prec}
    if kind == "hx_host":
        return {"kind": kind, "n": rng.randint(12, 32),
                "cols": _logint(rng, 1, 24),
                "precision": rng.choice(["fp32", "fp64"])}
    if kind == "dense":
        m = _logint(rng, 4, 120)
        return {"kind": kind, "n": rng.randint(12, 40), "m": m,
                "k": rng.randint(max(1, m // 3), m),
                "precision": rng.choice(["fp64", "fp32_tc"])}
    if kind == "densities":
        return {"kind": kind, "n": rng.randint(12, 48),
                "cols": _logint(rng, 2, 64)}
    if kind == "poisson":
        return {"kind": kind, "n": rng.randint(12, 48),
                "Z": 2 * rng.randint(2, 40), "warm": rng.random() < 0.7}
    if kind == "gcg":
        n = rng.randint(18, 40)
        nev = 2 * _logint(rng, 1, 32)
        return {"kind": kind, "n": n, "nev": nev,
                "pcols": rng.choice([0, nev, nev]),
                "precision": rng.choice(["fp64", "fp32", "fp32_tc"])}
    if kind == "state":
        Z = 2 * rng.randint(6, 20)
        A = 2 * Z + 2 * rng.randint(0, 5)
        return {"kind": kind, "n": 2 * rng.randint(10, 18), "A": A, "Z": Z,
                "basis": A - Z + 2 * rng.randint(6, 14),
                "pairing": rng.choice(["BCS", "HFB"])}
    raise ValueError(kind)


# ---- inputs ---------------------------------------------------------------

def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _axis(n, h):
    return (torch.arange(n, dtype=torch.float64, device=DEV) -
            0.5 * (n - 1)) * h


def _mesh(n, h):
    x = _axis(n, h)
    # [k][j][i]: i (x) fastest
    return (x.view(1, 1, n), x.view(1, n, 1), x.view(n, 1, 1))


def _gauss_sum(rng, x, y, z, a, count, dlo, dhi):
    G = torch.zeros_like(x + y + z)
    grad = [torch.zeros_like(G) for _ in range(3)]
    for _ in range(count):
        c = [rng.uniform(-a / 2, a / 2) for _ in range(3)]
        w, d = rng.uniform(1.5, 3.0), rng.uniform(dlo, dhi)
        u = [x - c[0], y - c[1], z - c[2]]
        e = d * torch.exp(-(u[0] ** 2 + u[1] ** 2 + u[2] ** 2) / w ** 2)
        G += e
        for q in range(3):
            grad[q] += -2.0 * u[q] / w ** 2 * e
    return G, torch.stack([g.reshape(-1) for g in grad])


def _fields(n, h, seed):
    """f (m*), grad f, U, W and UC of a lumpy nucleus, as in the
    repository's standalone workload."""
    rng = random.Random(int(seed) * 31 + 5)
    x, y, z = _mesh(n, h)
    a = 0.5 * (n - 1) * h
    G, _ = _gauss_sum(rng, x, y, z, a, 8, 5.0, 60.0)
    U = (-G).clamp(-60.0, 0.0).reshape(-1)
    g, dg = _gauss_sum(rng, x, y, z, a, 8, 0.1, 1.0)
    gmax = g.max()
    f = (H2M * (1.0 - 0.3 * g / gmax)).reshape(-1)
    gradf = -H2M * 0.3 * dg / gmax
    _, dG = _gauss_sum(rng, x, y, z, a, 8, 0.1, 1.0)
    W = 10.0 * dG / dG.square().sum(0).max().sqrt()
    r = (x * x + y * y + z * z).sqrt().reshape(-1)
    UC = E2 * 20.0 / r.clamp_min(3.0)
    return [t.contiguous() for t in (f, gradf, U, W, UC)]


def _random_block(N, cols, seed):
    v = torch.randn(cols, N, 2, dtype=torch.float64, device=DEV,
                    generator=_gen(seed))
    return torch.view_as_complex(v) / math.sqrt(2.0 * N)


def _ho1d(n, h, b, count):
    """Oscillator functions H_k(x/b) exp(-x^2/2b^2), k < count, normalised
    on the mesh."""
    x = _axis(n, h) / b
    out = [torch.exp(-0.5 * x * x)]
    out.append(math.sqrt(2.0) * x * out[0])
    for k in range(2, count):
        out.append(math.sqrt(2.0 / k) * x * out[-1] -
                   math.sqrt((k - 1.0) / k) * out[-2])
    P = torch.stack(out[:count])
    return P / P.norm(dim=1, keepdim=True)


def _orbitals(n, h, cols, seed, orthonormal=False):
    """Localised spinors: anisotropic oscillator states with mixed spin and
    complex phases, in time-reversed pairs (columns 2p, 2p + 1)."""
    rng = random.Random(int(seed) * 101 + 3)
    pairs = (cols + 1) // 2
    top = 1
    while (top + 1) * (top + 2) * (top + 3) // 6 < pairs + 4:
        top += 1
    lists = sorted(((i + j + k), i, j, k) for i in range(top + 1)
                   for j in range(top + 1 - i) for k in range(top + 1 - i - j))
    b = [rng.uniform(1.7, 2.1) for _ in range(3)]
    P = [_ho1d(n, h, bb, top + 2) for bb in b]

    def g(q):
        _, i, j, k = lists[q % len(lists)]
        return (P[2][k].view(n, 1, 1) * P[1][j].view(1, n, 1) *
                P[0][i].view(1, 1, n)).reshape(-1)

    X = torch.zeros(2 * pairs, n ** 3, 2, dtype=torch.complex128, device=DEV)
    for p in range(pairs):
        c = [rng.gauss(0, 0.35) for _ in range(6)]
        u, v, w = g(p), g(p + 1), g(p + 3)
        X[2 * p, :, 0] = u * complex(1.0, c[0]) + v * complex(c[1], c[2])
        X[2 * p, :, 1] = v * complex(c[3], 0.2) + w * complex(c[4], c[5])
        X[2 * p + 1, :, 0] = -X[2 * p, :, 1].conj()
        X[2 * p + 1, :, 1] = X[2 * p, :, 0].conj()
    X = X.reshape(2 * pairs, 2 * n ** 3)
    X /= X.norm(dim=1, keepdim=True)
    if orthonormal:
        for _ in range(2):
            G = X.conj() @ X.T  # G_ab = <a|b>
            L = torch.linalg.cholesky(G)
            X = torch.linalg.solve_triangular(L.conj(), X, upper=False)
    return X[:cols].contiguous()


def _fermi(n, h, Z, seed):
    rng = random.Random(int(seed) * 13 + 1)
    x, y, z = _mesh(n, h)
    R = 1.2 * (2.2 * Z) ** (1.0 / 3.0)
    s = [rng.uniform(0.9, 1.1) for _ in range(3)]
    o = [rng.uniform(-0.2, 0.2) for _ in range(3)]
    r = (((x - o[0]) / s[0]) ** 2 + ((y - o[1]) / s[1]) ** 2 +
         ((z - o[2]) / s[2]) ** 2).sqrt()
    rho = 1.0 / (1.0 + torch.exp((r - R) / 0.55))
    rho = rho * (Z / (rho.sum() * h ** 3))
    return rho.reshape(-1).contiguous()


def _second_difference(n):
    """30/12, -16/12, 1/12: minus the 5-point second derivative at h = 1."""
    T = torch.zeros(n, n, dtype=torch.float64, device=DEV)
    for d, v in ((0, 2.5), (1, -4.0 / 3.0), (2, 1.0 / 12.0)):
        o = torch.full((n - d,), v, dtype=torch.float64, device=DEV)
        T += torch.diag(o, d) + (torch.diag(o, -d) if d else 0)
    return T


def _well(n, h, pairs, seed):
    """A separable well whose levels are known: eigenpairs of the lattice
    Hamiltonian are products of 1-D ones. Widths are drawn until the levels
    of the block are separated from the next one."""
    rng = random.Random(int(seed) * 53 + 11)
    T = _second_difference(n).cpu() * H2M / h ** 2
    x = _axis(n, h).cpu()
    best = None
    for _ in range(60):
        e1, v1, us = [], [], []
        for q in range(3):
            w, D = rng.uniform(2.8, 4.6), rng.uniform(18.0, 24.0)
            u = -D * torch.exp(-(x / w) ** 2)
            e, v = torch.linalg.eigh(T + torch.diag(u))
            e1.append(e.tolist())
            v1.append(v)
            us.append(u)
        top = min(n, 14)
        lv = sorted((e1[0][i] + e1[1][j] + e1[2][k], i, j, k)
                    for i in range(top) for j in range(top)
                    for k in range(top))
        gap = lv[pairs][0] - lv[pairs - 1][0]
        if best is None or gap > best[0]:
            best = (gap, lv, v1, us)
        if gap > 0.6:
            break
    return best[1:]


def _spinor_products(n, lv, v1, first, pairs):
    V = [v.to(DEV) for v in v1]
    X = torch.zeros(2 * pairs, n ** 3, 2, dtype=torch.complex128, device=DEV)
    for p in range(pairs):
        _, i, j, k = lv[first + p]
        g = (V[2][:, k].view(n, 1, 1) * V[1][:, j].view(1, n, 1) *
             V[0][:, i].view(1, 1, n)).reshape(-1)
        X[2 * p, :, 0] = g
        X[2 * p + 1, :, 1] = g
    return X.reshape(2 * pairs, 2 * n ** 3)


def _directions(n, lv, v1, pairs, seed):
    """Conjugate directions: changes of the orbitals, unit columns."""
    a = torch.randn(pairs, pairs, dtype=torch.float64, device=DEV,
                    generator=_gen(seed))
    q, _ = torch.linalg.qr(a)
    nxt = _spinor_products(n, lv, v1, pairs, pairs).view(pairs, 2, -1)
    P = torch.einsum("ab,bsr->asr", q.to(torch.complex128), nxt)
    return P.reshape(2 * pairs, -1).contiguous()


def _step(n):
    return 0.55 if n >= 24 else 13.0 / (n - 1)


def _context(n, h, cols):
    # tensors made on torch's stream are handed to the context's own one
    torch.cuda.synchronize()
    return ng.Context(ng.Grid(n, 0.5 * (n - 1) * h), cols)


def prepare(case, seed):
    kind, n = case["kind"], case["n"]
    h = _step(n)
    s = {"kind": kind, "n": n, "ns": n ** 3, "N": 2 * n ** 3}
    if kind in ("hx", "hx_host"):
        cols = case["cols"]
        f = _fields(n, h, seed)
        ctx = _context(n, h, cols)
        s["H"] = ng.Hamiltonian(ctx, abi.PROTON).set_fields(*f)
        s["ctx"], s["cols"] = ctx, cols
        s["prec"] = PREC[case["precision"]]
        X = _random_block(s["N"], cols, seed)
        if kind == "hx":
            s["X"] = X.to(torch.complex64) if s["prec"] == abi.FP32 else X
            s["Y"] = torch.empty_like(s["X"])
        else:
            s["X"] = np.asfortranarray(X.cpu().numpy().T)
    elif kind == "dense":
        m, k = case["m"], case["k"]
        s["ctx"] = _context(n, h, 4)
        s["m"], s["k"], s["prec"] = m, k, PREC[case["precision"]]
        # orbitals and the corrections to them, which are far smaller
        V = _orbitals(n, h, m, seed)
        x, y, z = _mesh(n, h)
        env = torch.exp(-(x * x + y * y + z * z) / 30.0).reshape(-1, 1)
        d = torch.randn(m, n ** 3, 4, dtype=torch.float64, device=DEV,
                        generator=_gen(seed))
        d = torch.view_as_complex(d.view(m, n ** 3, 2, 2)) * env
        d = d.reshape(m, -1) / d.reshape(m, -1).norm(dim=1, keepdim=True)
        third = max(1, m // 3)
        V += 0.3 * d
        V[2 * third:] = 3e-3 * d[2 * third:]
        s["V"] = V.contiguous()
        c = torch.randn(k, m, 2, dtype=torch.float64, device=DEV,
                        generator=_gen(seed + 1))
        s["C"] = torch.view_as_complex(c).contiguous()  # [k][m]: column-major
        s["G"] = torch.empty(m, m, dtype=torch.complex128, device=DEV)
        s["Y"] = torch.empty(k, s["N"], dtype=torch.complex128, device=DEV)
    elif kind == "densities":
        s["ctx"] = _context(n, h, case["cols"])
        s["cols"] = case["cols"]
        s["X"] = _orbitals(n, h, case["cols"], seed)
        s["out"] = torch.empty(12, n ** 3, dtype=torch.float64, device=DEV)
    elif kind == "poisson":
        s["ctx"] = _context(n, h, 4)
        s["Z"] = case["Z"]
        s["rho"] = _fermi(n, h, case["Z"], seed)
        s["guess"] = None
        if case["warm"]:
            # the previous iteration's potential
            x, y, z = _mesh(n, h)
            r = (x * x + y * y + z * z).sqrt().reshape(-1)
            s["guess"] = (E2 * case["Z"] / r.clamp_min(4.0)).contiguous()
        s["out"] = torch.empty(2, n ** 3, dtype=torch.float64, device=DEV)
    elif kind == "gcg":
        nev, pc = case["nev"], case["pcols"]
        pairs = nev // 2
        lv, v1, us = _well(n, h, pairs, seed)
        x, y, z = _mesh(n, h)
        # the mean field has moved a little since the orbitals were solved
        # for: an effective mass and a bump, as between two HF iterations.
        # No spin-orbit field: H is not Hermitian on the lattice, and the
        # Rayleigh-Ritz step reads one triangle, so with it the result would
        # depend on the arbitrary rotation inside each Kramers pair.
        rng = random.Random(int(seed) * 71 + 2)
        g, dg = _gauss_sum(rng, x, y, z, 6.0, 4, 0.2, 1.0)
        eps = 4e-4
        f = (H2M * (1.0 - eps * g)).reshape(-1)
        U = (us[0].to(DEV).view(1, 1, n) + us[1].to(DEV).view(1, n, 1) +
             us[2].to(DEV).view(n, 1, 1)).reshape(-1)
        b, _ = _gauss_sum(rng, x, y, z, 6.0, 4, -30.0, 30.0)
        U = U + eps * b.reshape(-1)
        ctx = _context(n, h, 3 * nev + pc)
        s["H"] = ng.Hamiltonian(ctx, abi.NEUTRON).set_fields(
            f, (-H2M * eps * dg).contiguous(), U.contiguous(), None, None)
        s["ctx"], s["nev"], s["pcols"] = ctx, nev, pc
        s["X"] = _spinor_products(n, lv, v1, 0, pairs).contiguous()
        s["P"] = None
        if pc:
            s["P"] = _directions(n, lv, v1, pairs, seed)
        s["prm"] = config._gcg(config.HF_GCG, PREC[case["precision"]])
        s["Xo"] = torch.empty_like(s["X"])
        s["lam"] = np.zeros(nev)
        s["out"] = torch.empty(12, n ** 3, dtype=torch.float64, device=DEV)
    elif kind == "state":
        cfg = _state_config(case, h)
        s["cfg"], s["st"] = cfg, ng.IterationData(cfg)
        cols = case["basis"]
        s["cols"] = cols
        s["X"] = [_orbitals(n, h, cols, 2 * seed + q, True) for q in range(2)]
        rng = random.Random(int(seed) * 17)
        e = []
        for q in range(2):
            # a well-paired open shell: close levels at the Fermi energy
            steps = [rng.uniform(0.3, 1.1) for _ in range(cols // 2)]
            lv = np.cumsum(steps)
            lv -= lv[(case["A"] - case["Z"] if q == 0 else case["Z"]) // 2]
            lv -= 8.0
            e.append(np.repeat(lv, 2).astype(np.float64))
        s["e"] = e
        s["out"] = torch.empty(2, 11, n ** 3, dtype=torch.float64, device=DEV)
        torch.cuda.synchronize()
        # the iterations before this one: BCS, then the first HFB step
        first = 1 if case["pairing"] == "BCS" else cfg.start_hfb_iter
        for it in range(first + 1):
            _update(s, it)
        s["it"] = first + 1
    else:
        raise ValueError(kind)
    torch.cuda.synchronize()
    return s


def _state_config(case, h):
    n = case["n"]
    return config.from_input({
        "functional": "SLy4", "nucleus": {"A": case["A"], "Z": case["Z"]},
        "box": {"boxSize": (n - 1) * h, "axisMeshPoints": n},
        "startHFBIter": 1,
        "pairing": {"type": case["pairing"], "HFbasisSize": case["basis"],
                    "V0": 300.0, "window": 60.0},
        "maxIterations": 10, "energyTol": 1e-3})


# ---- one pass -------------------------------------------------------------

def _p(t):
    return None if t is None else t.data_ptr()


def _densities(s, X, cols):
    o = s["out"]
    ng._check(ng.load().ncgm_densities(s["ctx"].h, _p(X), cols, _p(o[0]),
                                       _p(o[1]), _p(o[2]), _p(o[11])))
    return o


def _update(s, it):
    (Xn, Xp), (en, ep) = s["X"], s["e"]
    ng._check(ng.load().ncgm_state_update(
        s["st"].h, _p(Xn), en.ctypes.data, s["cols"], _p(Xp), ep.ctypes.data,
        s["cols"], it, abi.UPDATE_NORMALIZE | abi.UPDATE_TRORDER))


def run(s):
    kind, L = s["kind"], ng.load()
    if kind == "hx":
        ng._check(L.ncgm_apply_h_device(s["ctx"].h, abi.PROTON, _p(s["X"]),
                                        _p(s["Y"]), s["cols"], s["prec"], 0.0))
        return s["Y"]
    if kind == "hx_host":
        return s["H"].apply(s["X"], s["prec"])
    if kind == "dense":
        h, V, m = s["ctx"].h, _p(s["V"]), s["m"]
        ng._check(L.ncgm_gram(h, V, m, V, m, _p(s["G"]), s["prec"]))
        ng._check(L.ncgm_vc(h, V, m, _p(s["C"]), s["k"], _p(s["Y"]),
                            s["prec"]))
        return {"gram": s["G"], "rotated": s["Y"]}
    if kind == "densities":
        o = _densities(s, s["X"], s["cols"])
        return {"rho": o[0], "tau": o[1], "J": o[2:11], "divJ": o[11]}
    if kind == "poisson":
        o, its = s["out"], C.c_int()
        ng._check(L.ncgm_poisson(s["ctx"].h, _p(s["rho"]), s["Z"],
                                 _p(s["guess"]), _p(o[0]), _p(o[1]),
                                 C.byref(its)))
        return {"direct": o[0], "UC": o[1]}
    if kind == "gcg":
        st = abi.GcgStats()
        ng._check(L.ncgm_gcg(s["ctx"].h, abi.NEUTRON, _p(s["X"]), s["nev"],
                             _p(s["P"]), s["pcols"], s["nev"],
                             C.byref(s["prm"]), _p(s["Xo"]),
                             s["lam"].ctypes.data, C.byref(st)))
        o = _densities(s, s["Xo"], s["nev"])
        # without spin-orbit J and div J vanish: only their rounding is left
        return {"lambda": s["lam"], "rho": o[0].float(), "tau": o[1].float()}
    if kind == "state":
        _update(s, s["it"])
        out = {}
        for q in range(2):
            o = s["out"][q]
            ng._check(L.ncgm_state_fields(s["st"].h, q, _p(o[0]), _p(o[1]),
                                          _p(o[4]), _p(o[5]), _p(o[8])))
            ng._check(L.ncgm_state_densities(s["st"].h, q, _p(o[9]),
                                             _p(o[10])))
            out["fields%d" % q], out["densities%d" % q] = o[:9], o[9:]
        out["E"] = list(s["st"].energies(*s["e"]))
        return out
    raise ValueError(kind)


def work(case):
    n = case["n"]
    ns, N = n ** 3, 2 * n ** 3
    kind = case["kind"]
    hxf = 185.0  # flops of H per point and column
    if kind in ("hx", "hx_host"):
        b = 4 if case["precision"] == "fp32" and kind == "hx" else 8
        return {"bytes": N * case["cols"] * 2 * b * 2 + 8 * ns * b,
                "flops": hxf * ns * case["cols"]}
    if kind == "dense":
        m, k = case["m"], case["k"]
        return {"bytes": 16 * (N * (m + k) + m * (m + k)),
                "flops": 8.0 * N * m * k + 4.0 * N * m * m}
    if kind == "densities":
        return {"bytes": 16 * N * case["cols"] + 8 * 12 * ns,
                "flops": 300.0 * ns * case["cols"]}
    if kind == "poisson":
        return {"bytes": 8 * ns * (3 + bool(case["warm"])),
                "flops": 12.0 * n * ns}
    if kind == "gcg":
        nev, pc = case["nev"], case["pcols"]
        m = 2 * nev + pc
        return {"bytes": 16 * N * (2 * nev + pc) + 8 * (8 + 2) * ns,
                "flops": 8.0 * N * (1.5 * m * m + m * m + 2 * m * nev) +
                hxf * ns * (m + 12 * nev) + 300.0 * ns * nev}
    if kind == "state":
        B = case["basis"]
        return {"bytes": 2 * (16 * N * B + 8 * ns * 11),
                "flops": 2 * (300.0 * ns * B + 8.0 * N * B * B * 2)}
    raise ValueError(kind)


# ---- what the results are in 64 bits --------------------------------------

def _shift(v, axis, d):
    """v[.. a + d ..] with zeros outside the box; v: [cols][k][j][i][spin]."""
    out = torch.zeros_like(v)
    n = v.shape[axis]
    if abs(d) < n:
        src = [slice(None)] * v.dim()
        dst = [slice(None)] * v.dim()
        src[axis] = slice(max(d, 0), n + min(d, 0))
        dst[axis] = slice(max(-d, 0), n + min(-d, 0))
        out[tuple(dst)] = v[tuple(src)]
    return out


def _exact_hx(n, h, fields, X):
    """H X for X [cols][N] complex128."""
    f, gf, U, W, UC = fields
    sh = (1, n, n, n, 1)
    f, U, UC = f.view(sh), U.view(sh), UC.view(sh)
    out = []
    for x in X.split(8):
        v = x.view(-1, n, n, n, 2)
        y = (U + UC + 7.5 * f / h ** 2) * v
        for a in range(3):
            ax = 3 - a  # x: axis 3
            p1, m1 = _shift(v, ax, 1), _shift(v, ax, -1)
            p2, m2 = _shift(v, ax, 2), _shift(v, ax, -2)
            y = y - f / h ** 2 * (4.0 / 3.0 * (p1 + m1) - (p2 + m2) / 12.0)
            D = (8.0 * (p1 - m1) - (p2 - m2)) / (12.0 * h)
            y = y - gf[a].view(sh) * D
            w = [W[q].view(sh[:-1]) for q in range(3)]
            # -i (sigma x W)_a = -i (sigma_b W_c - sigma_c W_b)
            b, c = (a + 1) % 3, (a + 2) % 3
            y = y - 1j * (_sigma(b, D) * w[c].unsqueeze(-1) -
                          _sigma(c, D) * w[b].unsqueeze(-1))
        out.append(y.reshape(y.shape[0], -1))
    return torch.cat(out)


def _sigma(q, v):
    u, d = v[..., 0], v[..., 1]
    if q == 0:
        return torch.stack([d, u], -1)
    if q == 1:
        return torch.stack([-1j * d, 1j * u], -1)
    return torch.stack([u, -d], -1)


def _d1(n, h):
    """First derivative along an axis: 9-point inside, order dropping to a
    one-sided difference at the faces."""
    D = torch.zeros(n, n, dtype=torch.float64)
    rules = {1: ([1], [0.5]), 2: ([1, 2], [8 / 12, -1 / 12]),
             3: ([1, 2, 3], [45 / 60, -9 / 60, 1 / 60]),
             4: ([1, 2, 3, 4], [672 / 840, -168 / 840, 32 / 840, -3 / 840])}
    for i in range(n):
        # the rule is chosen face by face, the nearer layers first
        if i == 0:
            D[0, 1], D[0, 0] = 1.0, -1.0
            continue
        if i in (1, n - 2):
            r = 1
        elif i == n - 1:
            D[i, i], D[i, i - 1] = 1.0, -1.0
            continue
        elif i in (2, n - 3):
            r = 2
        elif i in (3, n - 4):
            r = 3
        else:
            r = 4
        for d, c in zip(*rules[r]):
            D[i, i + d] += c
            D[i, i - d] -= c
    return (D / h).to(DEV)


def _exact_densities(n, h, X):
    D = _d1(n, h).to(torch.complex128)
    rho = torch.zeros(n, n, n, dtype=torch.float64, device=DEV)
    tau, dj = torch.zeros_like(rho), torch.zeros_like(rho)
    J = torch.zeros(9, n, n, n, dtype=torch.float64, device=DEV)
    for x in X:
        v = x.view(n, n, n, 2)
        g = [torch.einsum("ai,kjis->kjas", D, v),
             torch.einsum("aj,kjis->kais", D, v),
             torch.einsum("ak,kjis->ajis", D, v)]
        rho += (v.real ** 2 + v.imag ** 2).sum(-1)
        for mu in range(3):
            tau += (g[mu].real ** 2 + g[mu].imag ** 2).sum(-1)
            for nu in range(3):
                J[mu * 3 + nu] += (v.conj() * _sigma(nu, g[mu])).sum(-1).imag
        for mu, nu, la, e in ((0, 1, 2, 1), (1, 2, 0, 1), (2, 0, 1, 1),
                              (2, 1, 0, -1), (0, 2, 1, -1), (1, 0, 2, -1)):
            dj -= e * (g[nu].conj() * _sigma(la, g[mu])).sum(-1).imag
    return {"rho": rho.reshape(-1), "tau": tau.reshape(-1),
            "J": J.reshape(9, -1), "divJ": dj.reshape(-1)}


def _exact_poisson(n, h, Z, rho):
    a = 0.5 * (n - 1) * h
    x, y, z = _mesh(n, h)
    r3 = rho.view(n, n, n)
    t = torch.ones(n, dtype=torch.float64, device=DEV)
    t[0] = t[-1] = 0.5
    w = t.view(n, 1, 1) * t.view(1, n, 1) * t.view(1, 1, n) * h ** 3
    q20 = float((r3 * (2 * z * z - x * x - y * y) * w).sum()) * math.sqrt(
        5 / (16 * math.pi))
    q22 = float((r3 * (x * x - y * y) * w).sum()) * math.sqrt(
        15 / (32 * math.pi))
    # potential on the box with two halo layers, index [i][j][k] of the halo
    u = -a - 2 * h + torch.arange(n + 4, dtype=torch.float64, device=DEV) * h
    X, Y, Zc = u.view(-1, 1, 1), u.view(1, -1, 1), u.view(1, 1, -1)
    r = (X * X + Y * Y + Zc * Zc).sqrt().clamp_min(1e-9)
    ct = Zc / r
    phi = torch.atan2(Y.expand_as(r), X.expand_as(r))
    y20 = math.sqrt(5 / (16 * math.pi)) * (3 * ct * ct - 1)
    y22 = math.sqrt(15 / (32 * math.pi)) * torch.cos(2 * phi) * (1 - ct * ct)
    V = E2 * Z / r + E2 * (y20 * q20 + 2 * y22 * q22) / r
    inner = torch.zeros(n + 4, dtype=torch.bool, device=DEV)
    inner[2:-2] = True
    ins = inner.view(-1, 1, 1) & inner.view(1, -1, 1) & inner.view(1, 1, -1)
    V = torch.where(ins, torch.zeros_like(V), V)
    # what the halo adds to L U: the first halo index goes with the slowest
    # lattice index (the x and z roles of the halo are exchanged)
    b = torch.zeros(n, n, n, dtype=torch.float64, device=DEV)
    for ax in range(3):
        for d, c in ((1, 16 / 12), (2, -1 / 12)):
            for sgn in (1, -1):
                lo = 2 + sgn * d
                sl = [slice(2, n + 2)] * 3
                sl[ax] = slice(lo, lo + n)
                b += c * V[tuple(sl)] / h ** 2
    rhs = 4 * math.pi * E2 * r3 + b  # -L U = 4 pi e^2 rho + halo
    e, Q = torch.linalg.eigh(_second_difference(n) / h ** 2)
    s = torch.einsum("ka,jb,ic,kji->abc", Q, Q, Q, rhs)
    s = s / (e.view(-1, 1, 1) + e.view(1, -1, 1) + e.view(1, 1, -1))
    U = torch.einsum("ka,jb,ic,abc->kji", Q, Q, Q, s).reshape(-1)
    ex = -E2 * (3 / math.pi) ** (1 / 3) * rho ** (1 / 3)
    return {"direct": U, "UC": U + ex}


def exact(case, seed):
    kind, n = case["kind"], case["n"]
    h = _step(n)
    if kind in ("hx", "hx_host"):
        X = _random_block(2 * n ** 3, case["cols"], seed)
        if kind == "hx" and case["precision"] == "fp32":
            X = X.to(torch.complex64).to(torch.complex128)
        Y = _exact_hx(n, h, _fields(n, h, seed), X)
        return Y if kind == "hx" else np.asfortranarray(Y.cpu().numpy().T)
    if kind == "dense":
        s = prepare(case, seed)
        V, c = s["V"], s["C"]
        G = torch.zeros_like(s["G"])
        for r in V.split(8192, dim=1):  # rows in parts: shorter sums
            G += r @ r.conj().T  # [j][i] = conj(v_i) . v_j
        return {"gram": G, "rotated": c @ V}
    if kind == "densities":
        return _exact_densities(n, h, _orbitals(n, h, case["cols"], seed))
    if kind == "poisson":
        return _exact_poisson(n, h, case["Z"], _fermi(n, h, case["Z"], seed))
    # an eigensolver stopped after one iteration and pairing to a stopping
    # rule have no closed value
    return None

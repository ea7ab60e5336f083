"""Timed workloads of the package, from the smallest calls to the largest.

Every case goes through an entry point that programs call: the Python functions
of the reference (host arrays in and out) for the Coulomb tensor of small
systems, the sTDDFT tensors and the grid densities, and the device-buffer and
batched calls for Coulomb tensors of larger systems. Molecules, bases and
states follow common/synthetic.py's definitions (sizes of its benchmark
configurations and of the 5-60 atom batch between and around them); elements
come from the case, geometry, exponents, orbitals and CI vectors from the seed.

A case is a dict of plain values:
  kind      what is called (see run)
  natoms    atoms of the molecule (batch: of the smallest molecule)
  lmax, lauxmax, nstates, nmos, npoints   sizes, where the kind has them
  boys      "reference" (the library's default) or "exact"
  shift     metric shift; 0 is the default, and large synthetic auxiliary bases
            are linearly dependent without one
  precision "fp64" or "mixed"
"""

import ctypes
import math
import sys
from pathlib import Path

import numpy as np
import torch

ROOT = Path(__file__).resolve().parents[1]
if str(ROOT / "pysisyphus-addons_b200") not in sys.path:
    sys.path.insert(0, str(ROOT / "pysisyphus-addons_b200"))

from pysisyphus_addons import _native as nat  # noqa: E402
from pysisyphus_addons.common import synthetic  # noqa: E402
from pysisyphus_addons.diabatization import intor as diab  # noqa: E402
from pysisyphus_addons.gdma import prim_dens  # noqa: E402
from pysisyphus_addons.grid import grid  # noqa: E402
from pysisyphus_addons.std import intor as std  # noqa: E402

NOCC, NVIRT = 6, 6


def _case(kind, natoms, lmax, lauxmax=0, nstates=0, boys="exact", shift=0.0, precision="fp64", **more):
    return dict(kind=kind, natoms=natoms, lmax=lmax, lauxmax=lauxmax, nstates=nstates, boys=boys, shift=shift,
                precision=precision, **more)


def listed():
    return [
        # A diatomic or triatomic, two states: the smallest drop-in call, all latency.
        dict(_case("coulomb_host", 3, 2, 2, 2, boys="reference"), name="coulomb_3atoms"),
        # The 8-atom configuration through the drop-in call, library defaults.
        dict(_case("coulomb_host", 8, 2, 2, 4, boys="reference"), name="coulomb_8atoms"),
        # Fitted densities of a small molecule (2d call), f shells, odd sizes.
        dict(_case("df_host", 11, 3, 3, 3, shift=1e-6), name="df_11atoms"),
        # The 40-atom configuration, densities resident on the device.
        dict(_case("coulomb_device", 40, 3, 4, 8, shift=1e-7), name="coulomb_40atoms"),
        # A larger molecule with many states (91 densities), FP32 recurrences for weak triplets.
        dict(_case("coulomb_device", 75, 3, 4, 13, shift=1e-7, precision="mixed"), name="coulomb_75atoms_mixed"),
        # The 200-atom configuration: g orbital and h auxiliary shells.
        dict(_case("coulomb_device", 200, 4, 5, 8, shift=1e-7), name="coulomb_200atoms"),
        # Sixteen molecules of 5 to 35 atoms in one call, e.g. the frames or fragments of a data set.
        dict(_case("coulomb_batch", 5, 3, 4, 6, shift=1e-7, nmol=16, step=2), name="coulomb_batch16"),
        # sTDDFT: one-center tensors of a mid-sized molecule.
        dict(_case("eri2c", 60, 3, 4, boys="reference", shift=1e-5), name="eri2c_60atoms"),
        # sTDDFT: MO-pair tensor of a small molecule, library defaults.
        dict(_case("df2c_mo", 8, 2, 2, boys="reference", nmos=21), name="df2c_mo_8atoms"),
        # sTDDFT: MO-pair tensor, 20 occupied and 40 virtual orbitals, 40 atoms.
        dict(_case("df2c_mo", 40, 3, 4, shift=1e-5, nmos=60), name="df2c_mo_40atoms"),
        # A density on a cube file's 64^3 points around the 40-atom molecule.
        dict(_case("grid", 40, 3, npoints=64**3), name="grid_40atoms"),
        # GDMA: density of the diffuse primitive pairs on a molecular grid.
        dict(_case("prim", 20, 3, npoints=60007), name="prim_20atoms"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["coulomb_host", "coulomb_host", "df_host", "coulomb_device", "coulomb_device", "coulomb_device",
                       "coulomb_batch", "eri2c", "df2c_mo", "df2c_mo", "grid", "prim"])
    boys = rng.choice(["reference", "exact"])
    if kind == "coulomb_host":
        return _case(kind, _log(rng, 2, 14), 2, 2, rng.randint(2, 6), boys=boys, shift=1e-6)
    if kind == "df_host":
        return _case(kind, _log(rng, 3, 14), rng.randint(2, 3), rng.randint(2, 4), rng.randint(1, 5), boys=boys, shift=1e-6)
    if kind == "coulomb_device":
        high = rng.random() < 0.4
        return _case(kind, _log(rng, 12, 110), 4 if high else 3, 5 if high else 4, rng.randint(3, 14), shift=1e-7,
                     precision=rng.choice(["fp64", "mixed"]))
    if kind == "coulomb_batch":
        return _case(kind, rng.randint(4, 8), 3, 4, rng.randint(3, 9), shift=1e-7, nmol=rng.randint(3, 16), step=rng.randint(1, 2))
    if kind == "eri2c":
        return _case(kind, _log(rng, 5, 80), rng.randint(2, 3), rng.randint(2, 4), boys=boys, shift=1e-5)
    if kind == "df2c_mo":
        return _case(kind, _log(rng, 5, 40), rng.randint(2, 3), rng.randint(2, 4), boys=boys, shift=1e-5, nmos=rng.randint(5, 60))
    if kind == "grid":
        return _case(kind, _log(rng, 4, 45), rng.randint(2, 4), npoints=_log(rng, 3000, 250000))
    return _case(kind, _log(rng, 4, 24), rng.randint(2, 3), npoints=_log(rng, 2000, 60000))


# ---------------------------------------------------------------- inputs

def _ncart(L):
    return (L + 1) * (L + 2) // 2


def _cart_size(shells):
    return sum(_ncart(s.L) for s in shells)


def _molecule(case, seed):
    """Bases of a molecule whose elements belong to the case, its geometry and exponents to the seed."""
    mol = synthetic.random_molecule(case["natoms"], seed=seed)
    mol.atomic_nums = np.random.default_rng(case["natoms"]).choice(synthetic.ELEMENTS, size=case["natoms"])
    return synthetic.orbital_basis(mol, lmax=case["lmax"], seed=seed), synthetic.aux_basis(mol, lauxmax=case["lauxmax"])


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) + 77)


def _orbitals(nbf, n, gen):
    return torch.linalg.qr(torch.randn(nbf, n, dtype=torch.float64, device="cuda", generator=gen))[0]


def _densities(nbf, nstates, seed):
    """State and transition densities (ndens, nbf, nbf) on the GPU, lower triangular order,
    of CIS-like states in random orthonormal orbitals (as synthetic.random_states)."""
    gen = _gen(seed)
    no = min(NOCC, nbf // 2)
    nv = min(NVIRT, nbf - no)
    C = _orbitals(nbf, no + nv, gen)
    Co, Cv = C[:, :no], C[:, no:]
    X = torch.randn(nstates, no, nv, dtype=torch.float64, device="cuda", generator=gen)
    X /= X.flatten(1).norm(dim=1)[:, None, None]
    D = torch.empty(nstates * (nstates + 1) // 2, nbf, nbf, dtype=torch.float64, device="cuda")
    D00 = 2.0 * Co @ Co.T
    k = 0
    for i in range(nstates):
        for j in range(i + 1):
            if i == j == 0:
                D[k] = D00
            elif j == 0:
                D[k] = math.sqrt(2.0) * Co @ X[i] @ Cv.T
            else:
                D[k] = Cv @ (X[i].T @ X[j]) @ Cv.T - Co @ (X[j] @ X[i].T) @ Co.T
                if i == j:
                    D[k] += D00
            k += 1
    return D


def _points(shells, npoints, seed):
    """A regular grid for whole cubes, else scattered points, around the molecule."""
    C = np.array([s.center for s in shells])
    lo, hi = C.min(0) - 3.0, C.max(0) + 3.0
    n = round(npoints ** (1.0 / 3.0))
    if n**3 == npoints:
        X = np.meshgrid(*[np.linspace(lo[d], hi[d], n) for d in range(3)], indexing="ij")
        return np.stack([x.ravel() for x in X], axis=1)
    # points around atoms, as a molecular grid has them
    rng = np.random.default_rng(seed)
    at = C[np.sort(rng.integers(0, len(C), size=npoints))]
    return at + rng.normal(size=(npoints, 3)) * rng.uniform(0.2, 2.5, size=(npoints, 1))


def _cart_density(n, seed):
    Cc = torch.randn(n, 20, dtype=torch.float64, device="cuda", generator=_gen(seed)) / math.sqrt(n)
    return (Cc @ Cc.T).cpu().numpy()


def _norm_coeffs(sh):
    c, e, lp = sh.coeffs, sh.exps, sh.L + 1.5
    pair = np.outer(c, c) / np.add.outer(e, e) ** lp * np.sqrt(np.outer(e, e)) ** lp
    return c * np.sqrt(e**lp / (np.pi**1.5 / 2**sh.L * pair.sum()))


def _prim_data(shells):
    inds, data, off = [], [], 0
    for s in shells:
        for c, e in zip(_norm_coeffs(s), s.exps):
            inds.append((s.L, off))
            data.append((c, e, *s.center))
        off += _ncart(s.L)
    return np.array(inds, dtype=np.int32), np.array(data)


def prepare(case, seed):
    kind = case["kind"]
    st = dict(case=case)
    if kind == "coulomb_batch":
        st["shells"], st["D"], st["orb"], st["aux"], st["out"] = [], [], [], [], []
        for m in range(case["nmol"]):
            one = dict(case, natoms=case["natoms"] + case["step"] * m)
            o, a = _molecule(one, seed + 1000 * m)
            st["orb"].append(nat.Basis(o, "orbital"))
            st["aux"].append(nat.Basis(a, "aux"))
            st["D"].append(_densities(st["orb"][-1].nsph, case["nstates"], seed + 1000 * m))
            st["out"].append(torch.empty((case["nstates"],) * 4, dtype=torch.float64, device="cuda"))
        return st
    shells, aux = _molecule(case, seed)
    st["shells"], st["shells_aux"] = shells, aux
    if kind == "coulomb_device":
        st["orb"], st["aux"] = nat.Basis(shells, "orbital"), nat.Basis(aux, "aux")
        st["D"] = _densities(st["orb"].nsph, case["nstates"], seed)
        st["out"] = torch.empty((case["nstates"],) * 4, dtype=torch.float64, device="cuda")
    elif kind in ("coulomb_host", "df_host"):
        st["D"] = _densities(shells.sph_size, case["nstates"], seed).cpu().numpy()
    elif kind == "df2c_mo":
        nbf = shells.sph_size
        st["C"] = np.asfortranarray(_orbitals(nbf, min(case["nmos"], nbf), _gen(seed)).cpu().numpy())
    elif kind == "grid":
        st["points"] = _points(shells, case["npoints"], seed)
        st["D"] = _cart_density(_cart_size(shells), seed)
    elif kind == "prim":
        st["points"] = _points(shells, case["npoints"], seed)
        st["P"] = _cart_density(_cart_size(shells), seed)
        st["inds"], st["data"] = _prim_data(shells)
        st["rho"] = np.zeros(case["npoints"])
    return st


SWITCH = 4.0  # GDMA: pairs with an exponent sum below it go to the grid


def run(st):
    case = st["case"]
    kind = case["kind"]
    nat.set_boys_mode(case["boys"])
    nat.set_metric_shift(case["shift"])
    nat.set_precision(case["precision"])
    if kind == "coulomb_host":
        return diab.contract_coulomb_densities_4d(st["shells"], st["shells_aux"], st["D"])
    if kind == "df_host":
        return diab.contract_coulomb_densities_2d(st["shells"], st["shells_aux"], st["D"])
    if kind == "coulomb_device":
        D = st["D"]
        nat.check(nat.load().pa_df_4d(st["orb"].handle, st["aux"].handle, D.shape[0], D.shape[1], D.data_ptr(),
                                      nat.PA_LAYOUT_C, case["nstates"], st["out"].data_ptr(),
                                      ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
        return st["out"]
    if kind == "coulomb_batch":
        # a data set's batches differ from call to call, so no graph is recorded for replay
        nat.df_4d_batch(st["orb"], st["aux"], st["D"], [case["nstates"]] * case["nmol"], st["out"], use_graph=False,
                        stream=ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        return st["out"]
    if kind == "eri2c":
        return std.int_df1c(st["shells"], st["shells_aux"]), std.int_eri2c(st["shells"], st["shells_aux"])
    if kind == "df2c_mo":
        return std.int_df2c_mo(st["shells"], st["shells_aux"], st["C"])
    if kind == "grid":
        return grid.eval_density(st["shells"], st["points"], st["D"])
    return prim_dens.eval_prim_density(st["inds"], st["data"], st["points"], st["P"], SWITCH, st["rho"])


# ---------------------------------------------------------------- necessary work

def _pairs(shells):
    """(la, lb, primitive pairs) sums of the shell pairs whose overlap is not negligible:
    number of pairs' spherical functions, and of pairs weighted by primitives."""
    x = np.array([s.center for s in shells])
    e = np.array([s.exps.min() for s in shells])
    n = np.array([2 * s.L + 1 for s in shells], dtype=float)
    r2 = ((x[:, None] - x[None]) ** 2).sum(-1)
    near = e[:, None] * e[None] / (e[:, None] + e[None]) * r2 < 23.0
    full = np.outer(n, n)
    return float((full * near).sum() + (n * n).sum()) / 2, float((n * np.diag(full / n)).sum())


def work(case):
    kind = case["kind"]
    if kind == "coulomb_batch":
        w = [work(dict(case, kind="coulomb_device", natoms=case["natoms"] + case["step"] * m)) for m in range(case["nmol"])]
        return {k: sum(x[k] for x in w) for k in ("bytes", "flops")}
    shells, aux = _molecule(case, 0)
    nbf, naux = shells.sph_size, aux.sph_size
    if kind in ("grid", "prim"):
        nc, npt = _cart_size(shells), case["npoints"]
        near = min(1.0, 60.0 / nc)  # functions that reach a point
        return {"bytes": 8.0 * (4 * npt + nc * nc), "flops": npt * (60.0 * nc * near + (nc * near) ** 2)}
    pairs, diag = _pairs(shells)
    chol = naux**3 / 3.0
    if kind == "eri2c":
        return {"bytes": 8.0 * (2 * nbf * naux + nbf * nbf),
                "flops": 2 * (20.0 * diag * naux + chol + nbf * naux**2) + 2.0 * nbf * nbf * naux}
    if kind == "df2c_mo":
        nm = min(case["nmos"], nbf)
        rows = nm * (nm + 1) / 2
        return {"bytes": 8.0 * (nbf * nm + rows * naux),
                "flops": pairs * naux * (20.0 + 4.0 * nm) + 2.0 * nbf * nm * nm * naux + chol + rows * naux**2}
    nd = case["nstates"] * (case["nstates"] + 1) / 2
    out = nd * naux if kind == "df_host" else case["nstates"] ** 4
    return {"bytes": 8.0 * (nd * nbf * nbf + out), "flops": pairs * naux * (20.0 + 2.0 * nd) + chol + nd * naux**2}


# ---------------------------------------------------------------- values in 64 bits
# Plain torch: real solid harmonics by their recursion, Hermite (McMurchie-Davidson)
# expansions of primitive pairs, every triplet without screening.

EXACT_ATOMS = 12  # integrals of larger molecules take too long here


def _carts(l):
    return [(i, j, l - i - j) for i in range(l, -1, -1) for j in range(l - i, -1, -1)]


def _dfact(n):
    return 1.0 if n <= 1 else n * _dfact(n - 2)


def _solid(l):
    """Rows m = -l..l over _carts(l), each normalized for primitives with unit x^l norm."""
    def mul(p, e, f):
        return {tuple(a + b for a, b in zip(k, e)): v * f for k, v in p.items()}

    def add(*ps):
        out = {}
        for p in ps:
            for k, v in p.items():
                out[k] = out.get(k, 0.0) + v
        return out
    X, Y, Z = (1, 0, 0), (0, 1, 0), (0, 0, 1)
    prev, cur = {}, {0: {(0, 0, 0): 1.0}}
    for n in range(l):
        nxt = {}
        f = math.sqrt((2.0 if n == 0 else 1.0) * (2 * n + 1) / (2 * n + 2))
        low = cur[-n] if n else {}
        nxt[n + 1] = add(mul(cur[n], X, f), mul(low, Y, -f))
        nxt[-n - 1] = add(mul(cur[n], Y, f), mul(low, X, f))
        for m in range(-n, n + 1):
            d = math.sqrt((n + m + 1) * (n - m + 1))
            r = [mul(prev[m], tuple(2 * c for c in e), -math.sqrt((n + m) * (n - m)) / d) for e in (X, Y, Z)] if m in prev else []
            nxt[m] = add(mul(cur[m], Z, (2 * n + 1) / d), *r)
        prev, cur = cur, nxt
    T = np.array([[cur[m].get(c, 0.0) for c in _carts(l)] for m in range(-l, l + 1)])
    ov = np.array([[np.prod([0.0 if (p + q) % 2 else _dfact(p + q - 1) for p, q in zip(a, b)]) for b in _carts(l)]
                   for a in _carts(l)])
    return T / np.sqrt(np.einsum("mi,ij,mj->m", T, ov, T))[:, None]


def _herm_list(L):
    return [c for l in range(L + 1) for c in _carts(l)]


def _hermite(la, lb, a, b, AB):
    """E[i][j][t] of one dimension, tensors over primitive pairs."""
    p = a + b
    E = {(0, 0, 0): torch.exp(-a * b / p * AB**2)}
    get = lambda i, j, t: E.get((i, j, t), 0.0) if 0 <= t <= i + j else 0.0  # noqa: E731
    for i in range(la + 1):
        for j in range(lb + 1):
            for t in range(i + j + 1):
                if i == j == 0:
                    continue
                if i > 0:
                    E[i, j, t] = get(i - 1, j, t - 1) / (2 * p) - b / p * AB * get(i - 1, j, t) + (t + 1) * get(i - 1, j, t + 1)
                else:
                    E[i, j, t] = get(i, j - 1, t - 1) / (2 * p) + a / p * AB * get(i, j - 1, t) + (t + 1) * get(i, j - 1, t + 1)
    return E


def _charges(la, lb, a, b, A, B, w):
    """Hermite expansion [pair, ma * mb, tuv] of contracted spherical products."""
    Es = [_hermite(la, lb, a, b, A[:, d] - B[:, d]) for d in range(3)]
    herm = {c: k for k, c in enumerate(_herm_list(la + lb))}
    Sa, Sb = _solid(la), _solid(lb)
    H = torch.zeros(len(a), len(Sa), len(Sb), len(herm), dtype=torch.float64, device="cuda")
    for ka, ca in enumerate(_carts(la)):
        for kb, cb in enumerate(_carts(lb)):
            co = torch.tensor(np.outer(Sa[:, ka], Sb[:, kb]), device="cuda")
            if not co.any():
                continue
            for t in range(ca[0] + cb[0] + 1):
                for u in range(ca[1] + cb[1] + 1):
                    for v in range(ca[2] + cb[2] + 1):
                        e = Es[0][ca[0], cb[0], t] * Es[1][ca[1], cb[1], u] * Es[2][ca[2], cb[2], v] * w
                        H[:, :, :, herm[t, u, v]] += e[:, None, None] * co
    return H.flatten(1, 2)


def _boys(N, T):
    """F_0..F_N: power series of the highest order and downward recursion, or for large T
    the complete integral and upward recursion."""
    small = T < 36.0
    Ts, Tl = torch.where(small, T, 0.0), torch.where(small, 40.0, T)
    ex, exl = torch.exp(-Ts), torch.exp(-Tl)
    term = torch.full_like(T, 1.0 / (2 * N + 1))
    s = term.clone()
    for k in range(1, 170):
        term = term * (2.0 * Ts / (2 * N + 2 * k + 1))
        s += term
    F = [None] * (N + 1)
    F[N] = ex * s
    for n in range(N - 1, -1, -1):
        F[n] = (2.0 * Ts * F[n + 1] + ex) / (2 * n + 1)
    up = torch.sqrt(math.pi / Tl) / 2.0 * torch.erf(torch.sqrt(Tl))
    for n in range(N + 1):
        F[n] = torch.where(small, F[n], up)
        up = ((2 * n + 1) * up - exl) / (2.0 * Tl)
    return F


def _coulomb(L1, p, P, H1, L2, q, Q, H2):
    """sum over Hermite components of both sides: [n1, s1, n2, s2]."""
    L = L1 + L2
    al = p[:, None] * q[None] / (p[:, None] + q[None])
    X = P[:, None] - Q[None]
    F = _boys(L, al * (X**2).sum(-1))
    lev = [{(0, 0, 0): (-2.0 * al) ** n * F[n]} for n in range(L + 1)]
    for deg in range(1, L + 1):
        for n in range(L - deg + 1):
            for c in _carts(deg):
                d = next(k for k in range(3) if c[k])
                m1 = tuple(x - (k == d) for k, x in enumerate(c))
                m2 = tuple(x - 2 * (k == d) for k, x in enumerate(c))
                v = X[..., d] * lev[n + 1][m1]
                if c[d] > 1:
                    v = v + (c[d] - 1) * lev[n + 1][m2]
                lev[n][c] = v
    R = lev[0]
    pref = 2.0 * math.pi**2.5 / (p[:, None] * q[None] * torch.sqrt(p[:, None] + q[None]))
    h1, h2 = _herm_list(L1), _herm_list(L2)
    out = torch.zeros(len(p), H1.shape[1], len(q), H2.shape[1], dtype=torch.float64, device="cuda")
    for k, tau in enumerate(h2):
        Y = torch.stack([R[tuple(a + b for a, b in zip(t, tau))] for t in h1])
        out += torch.einsum("nst,tnm,mr->nsmr", H1, Y, (-1.0) ** sum(tau) * H2[:, :, k])
    return out * pref[:, None, :, None]


def _by_l(shells):
    """Per L: exponents, centers, coefficients and shell of every primitive; first function of every shell."""
    off = np.concatenate(([0], np.cumsum([2 * s.L + 1 for s in shells])))
    out = {}
    for L in sorted({s.L for s in shells}):
        rows = [(e, c, *s.center, off[i]) for i, s in enumerate(shells) if s.L == L for c, e in zip(_norm_coeffs(s), s.exps)]
        r = torch.tensor(np.array(rows), dtype=torch.float64, device="cuda")
        out[L] = r[:, 0], r[:, 2:5], r[:, 1], r[:, 5].long()
    return out


def _single(L, e, x, c):
    """One-center expansion of auxiliary shells (a partner s function of exponent 0)."""
    z = torch.zeros_like(e)
    return _charges(L, 0, e, z, x, x, c)


def _integrals(shells, aux):
    """(mu nu|P) as [nbf, nbf, naux] and (P|Q)."""
    O, A = _by_l(shells), _by_l(aux)
    nbf, naux = shells.sph_size, aux.sph_size
    V = torch.zeros(naux, naux, dtype=torch.float64, device="cuda")
    T = torch.zeros(nbf, nbf, naux, dtype=torch.float64, device="cuda")
    sph = lambda L: torch.arange(2 * L + 1, device="cuda")  # noqa: E731
    for lc, (ec, xc, cc, oc) in A.items():
        Hc = _single(lc, ec, xc, cc)
        ic = (oc[:, None] + sph(lc)).flatten()
        for ld, (ed, xd, cd, od) in A.items():
            G = _coulomb(lc, ec, xc, Hc, ld, ed, xd, _single(ld, ed, xd, cd))
            V[ic[:, None], (od[:, None] + sph(ld)).flatten()[None]] = G.flatten(2, 3).flatten(0, 1)
        for la, (ea, xa, ca, oa) in O.items():
            for lb, (eb, xb, cb, ob) in O.items():
                if lb > la:
                    continue
                i, j = torch.meshgrid(torch.arange(len(ea), device="cuda"), torch.arange(len(eb), device="cuda"), indexing="ij")
                i, j = i.flatten(), j.flatten()
                step = max(1, 40_000_000 // (len(ec) * len(_herm_list(la + lb + lc))))
                for k in range(0, len(i), step):
                    a, b = i[k : k + step], j[k : k + step]
                    p = ea[a] + eb[b]
                    P = (ea[a][:, None] * xa[a] + eb[b][:, None] * xb[b]) / p[:, None]
                    H = _charges(la, lb, ea[a], eb[b], xa[a], xb[b], ca[a] * cb[b])
                    G = _coulomb(la + lb, p, P, H, lc, ec, xc, Hc).flatten(2, 3)
                    G = G.view(len(a), 2 * la + 1, 2 * lb + 1, -1)
                    mu = (oa[a][:, None, None] + sph(la)[None, :, None]).expand(G.shape[:3])
                    nu = (ob[b][:, None, None] + sph(lb)[None, None, :]).expand(G.shape[:3])
                    blk = torch.zeros(nbf, nbf, G.shape[3], dtype=torch.float64, device="cuda")
                    blk.index_put_((mu.flatten(), nu.flatten()), G.flatten(0, 2), accumulate=True)
                    T[:, :, ic] += blk if la == lb else blk + blk.transpose(0, 1)
    return T, V


def exact(case, seed):
    kind = case["kind"]
    if kind in ("grid", "prim"):
        return _exact_grid(case, seed)
    if kind == "coulomb_batch" or case["natoms"] > EXACT_ATOMS:
        return None
    shells, aux = _molecule(case, seed)
    nbf, naux = shells.sph_size, aux.sph_size
    T, V = _integrals(shells, aux)
    L = torch.linalg.cholesky(V + case["shift"] * torch.eye(naux, dtype=torch.float64, device="cuda"))
    fit = lambda raw: torch.linalg.solve_triangular(L, raw, upper=False)  # noqa: E731
    if kind == "eri2c":
        df = fit(torch.diagonal(T).contiguous()).T
        return df, df @ df.T
    if kind == "df2c_mo":
        C = _orbitals(nbf, min(case["nmos"], nbf), _gen(seed))
        M = torch.einsum("mp,mnP,nq->pqP", C, T, C)
        p, q = torch.tril_indices(C.shape[1], C.shape[1], device="cuda")
        return fit(M[p, q].T).T
    D = _densities(nbf, case["nstates"], seed)
    df = fit(T.flatten(0, 1).T @ D.flatten(1).T)
    if kind == "df_host":
        return df
    G = df.T @ df
    ns = case["nstates"]
    at = torch.tensor([[max(i, j) * (max(i, j) + 1) // 2 + min(i, j) for j in range(ns)] for i in range(ns)], device="cuda")
    return G[at.flatten()[:, None], at.flatten()[None]].reshape((ns,) * 4)


def _exact_grid(case, seed):
    shells, _ = _molecule(case, seed)
    pts = torch.tensor(_points(shells, case["npoints"], seed), device="cuda")
    D = torch.tensor(_cart_density(_cart_size(shells), seed), device="cuda")
    prim = case["kind"] == "prim"
    # one row per function (grid), or per function of each primitive (prim)
    rows, e, x, w, pw, of = [], [], [], [], [], 0
    for s in shells:
        cs = list(zip(_norm_coeffs(s), s.exps))
        for group in ([[t] for t in cs] if prim else [cs]):
            for k, c in enumerate(_carts(s.L)):
                rows.append(of + k)
                nrm = 1.0 / math.sqrt(np.prod([_dfact(2 * i - 1) for i in c]))
                e.append([t[1] for t in group] + [1.0] * (3 - len(group)))
                w.append([t[0] * nrm for t in group] + [0.0] * (3 - len(group)))
                x.append(s.center)
                pw.append(c)
        of += _ncart(s.L)
    put = lambda v: torch.tensor(np.array(v), dtype=torch.float64, device="cuda")  # noqa: E731
    e, w, x, pw, rows = put(e), put(w), put(x), put(pw).long(), torch.tensor(rows, device="cuda")
    M = D[rows][:, rows]
    if prim:
        M = M * (e[:, None, 0] + e[None, :, 0] < SWITCH)
    rho = []
    for k in range(0, len(pts), 4000):
        d = pts[k : k + 4000, None] - x[None]
        r2 = (d**2).sum(-1)
        chi = torch.stack([torch.exp(-e[:, t] * r2) * w[:, t] for t in range(3)]).sum(0)
        for t in range(3):
            chi = chi * d[..., t] ** pw[:, t]
        rho.append(((chi @ M) * chi).sum(1))
    return torch.cat(rho)

"""The work that programs have this library do, as measurable cases.

listed() gives the standard cases, draw() more of the same ranges; prepare() makes what a program has in
hand before the call (device grids with a basis, matrices, kept tensors), run() is one pass through the
public API, exact() the same result in plain 64-bit torch.  Kinds:

  fock         one direct-form Fock build (RCS or UOS) at a mid-SCF density: the call of every SCF iteration
  scf          a whole RCS SCF from the zero density to 1e-8 Eh
  batch        one fock_build_batch call over many small atoms and ions
  one_electron grid upload, basis values and gradients, S and H by quadrature, grid release
  precomputed  the per-iteration Fock build from a kept Fji tensor
  tc_build     the per-iteration transcorrelated build from kept Fji / Vji tensors
  tc_cycle     the transcorrelated precompute (two computeF, two computeV) and the build on it
"""
import math
import random

import numpy as np
import torch

from tcscf_b200 import api, ffi, grids

PRECISION = {"fp64": ffi.PREC_FP64, "bf16x3": ffi.PREC_BF16X3}
# closed subshells of atoms: electrons -> occupied radial functions per l
CLOSED = {2: "1", 4: "2", 10: "2,1", 12: "3,1", 18: "3,2", 20: "4,2", 30: "4,2,1", 36: "4,3,1"}
LEBEDEV = {11: 50, 17: 110, 19: 146, 21: 170, 23: 194, 25: 230, 27: 266, 29: 302, 31: 350, 35: 434, 41: 590, 47: 770, 53: 974, 59: 1202,
           77: 2030}
A12 = 1.0   # u = r12 / (2 (1 + r12)): the Jastrow factor of the Be transcorrelated configuration


def listed():
    he = {"Z": 2, "shells": "8,4", "z0": 0.5, "ratio": 1.8, "up": "1"}
    ne = {"Z": 10, "shells": "14,3,2,1", "z0": 0.3, "ratio": 1.7, "up": "2,1"}
    kr = {"Z": 36, "shells": "32,10,6,4", "z0": 0.2, "ratio": 1.45, "up": "4,3,1"}
    be = {"Z": 4, "shells": "12,4", "z0": 0.4, "ratio": 1.8, "up": "2", "down": "2"}
    return [
        # He, 20 functions on 50 x 50 points: the smallest configuration, where launches and latency count
        {"name": "he_fock_fp64", "kind": "fock", "prec": "fp64", "nrad": 50, "order": 11, **he},
        # a whole He SCF through RCSHartreeFock.compute, eigen-solves and convergence tests included
        {"name": "he_scf_fp64", "kind": "scf", "prec": "fp64", "nrad": 50, "order": 11, **he},
        # Ne, 40 functions on 100 x 590 points: an ordinary atom, reference precision and mixed precision
        {"name": "ne_fock_fp64", "kind": "fock", "prec": "fp64", "nrad": 100, "order": 41, **ne},
        {"name": "ne_fock_bf16x3", "kind": "fock", "prec": "bf16x3", "nrad": 100, "order": 41, **ne},
        # unrestricted open shell on two different scrambled-Sobol grids of ragged sizes (r1 and r2 drawn separately)
        {"name": "uos_qmc_fp64", "kind": "fock", "prec": "fp64", "n1": 16381, "n2": 8191, "Z": 7, "shells": "9,4,1", "z0": 0.4, "ratio": 1.7,
         "up": "2,1", "down": "2"},
        # Kr, 120 functions: reference precision on a coarse grid, mixed precision on the full 200 x 2030 grid (the largest build)
        {"name": "kr_fock_fp64", "kind": "fock", "prec": "fp64", "nrad": 40, "order": 77, **kr},
        {"name": "kr_fock_bf16x3", "kind": "fock", "prec": "bf16x3", "nrad": 200, "order": 77, **kr},
        # many small atoms and ions in one call, mixed precision
        {"name": "batch16_bf16x3", "kind": "batch", "prec": "bf16x3", "set": 20261203, "count": 16},
        # setting an atom up: grid, basis values and gradients, overlap and core Hamiltonian by quadrature
        {"name": "ne_one_electron", "kind": "one_electron", "nrad": 100, "order": 41, **ne},
        # the reference's iteration from a stored Fji (complex, from a 3-D r2 grid)
        {"name": "precomputed_fp64", "kind": "precomputed", "n1": 16384, "n2": 2048, "dim2": 3, **ne},
        # Be transcorrelated HF: one SCF iteration on kept tensors, and a cycle with its mixed-precision precompute
        {"name": "be_tc_build", "kind": "tc_build", "prec": "fp64", "n1": 65536, "n2": 1024, **be},
        {"name": "be_tc_cycle_bf16x3", "kind": "tc_cycle", "prec": "bf16x3", "n1": 65536, "n2": 65536, **be},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _atom(rng):
    ne = rng.choice(list(CLOSED))
    occ = [int(x) for x in CLOSED[ne].split(",")] + [0] * 4
    shells = [rng.randint(occ[0] + 3, 14), rng.randint(occ[1] + 1, 7) if occ[1] else rng.randint(0, 3),
              rng.randint(occ[2] + 1, 5) if occ[2] else rng.randint(0, 2), rng.randint(0, 2)]
    return {"Z": ne + rng.randint(0, 2), "shells": ",".join(map(str, shells)), "z0": round(rng.uniform(0.25, 0.5), 3),
            "ratio": round(rng.uniform(1.6, 1.8), 3), "up": CLOSED[ne]}


def _nb(case):
    return sum((2 * l + 1) * int(k) for l, k in enumerate(case["shells"].split(",")))


def draw(rng):
    kind = rng.choice(["fock", "fock", "fock", "fock", "scf", "batch", "one_electron", "precomputed", "tc_build", "tc_cycle"])
    if kind == "batch":
        return {"kind": "batch", "prec": "bf16x3", "set": rng.randint(1, 1 << 30), "count": rng.randint(3, 24)}
    if kind in ("tc_build", "tc_cycle"):
        up, down = rng.choice([("1", "1"), ("2", "2"), ("2", "1"), ("2,1", "2,1")])
        c = {"kind": kind, "prec": "fp64" if kind == "tc_build" else "bf16x3", "n1": _log_int(rng, 2000, 60000),
             "n2": _log_int(rng, 500, 1500) if kind == "tc_build" else _log_int(rng, 2000, 60000), "Z": 10 if "," in up else 4,
             "shells": "%d,%d" % (rng.randint(5, 12), rng.randint(2, 5)), "z0": round(rng.uniform(0.3, 0.6), 3), "ratio": 1.8, "up": up, "down": down}
        return c
    c = {"kind": kind, **_atom(rng)}
    if kind == "precomputed":
        while _nb(c) > 64:
            c.update(_atom(rng))
        return {**c, "n1": _log_int(rng, 2000, 20000), "n2": _log_int(rng, 500, 3000), "dim2": rng.choice([2, 3])}
    if kind == "scf":
        # atoms whose every level is full from the core-Hamiltonian step on (2 or 10 electrons)
        while _nb(c) > 40 or c["up"] not in ("1", "2,1"):
            c.update(_atom(rng))
        return {**c, "prec": "fp64", "nrad": rng.randint(30, 50), "order": rng.choice([11, 17, 19, 21])}
    if kind == "one_electron":
        return {**c, "nrad": rng.randint(30, 150), "order": rng.choice([11, 17, 23, 29, 35, 41])}
    c["prec"] = rng.choice(["fp64", "bf16x3"])
    if rng.random() < 0.3:   # two different grids, now and then open shell
        c.update(n1=_log_int(rng, 1000, 30000), n2=_log_int(rng, 1000, 30000))
        if rng.random() < 0.5 and "," in c["up"]:
            c["down"] = ",".join(c["up"].split(",")[:-1])
        return c
    n, orders = _log_int(rng, 2000, 60000 if c["prec"] == "fp64" else 250000), list(LEBEDEV)
    order = min(orders, key=lambda o: abs(math.log(LEBEDEV[o] / (2.0 * math.sqrt(n)) / math.exp(rng.uniform(-0.7, 0.7)))))
    return {**c, "nrad": max(20, min(200, round(n / LEBEDEV[order]))), "order": order}


# ---- inputs (the same for prepare and exact; numpy only, but for the quadrature points) -----------------------
def _basis(case, rs=None):
    """[(zeta, n, l, m)], even-tempered per l; rs: exponents of this seed (jittered by up to 2 %)."""
    f = 1.0 if rs is None else 1.0 + 0.02 * rs.uniform(-1, 1)
    return [(float(case["z0"] * f * case["ratio"] ** k), l + 1, l, m) for l, cnt in enumerate(case["shells"].split(",")) for k in range(int(cnt))
            for m in range(-l, l + 1)]


def _unitary(basis):
    """Complex to real harmonics, phiR = U phi (m > 0: cos type, m < 0: sin type)."""
    at = {b: i for i, b in enumerate(basis)}
    U, h = np.zeros((len(basis),) * 2, dtype=complex), math.sqrt(0.5)
    for k, (z, n, l, m) in enumerate(basis):
        p = at[(z, n, l, -m)]
        if m == 0:
            U[k, k] = 1
        elif m > 0:
            U[k, k] = U[k, p] = h
        else:
            U[k, p], U[k, k] = -1j * h, 1j * h
    return U


def _radial(z, l, Z):
    """Overlap and core Hamiltonian of the radial STOs r^l exp(-z r) of one l, in closed form."""
    n, z = l + 1, np.asarray(z)
    N = (2 * z) ** (n + 0.5) / math.sqrt(math.factorial(2 * n))
    a, NN = z[:, None] + z[None, :], N[:, None] * N[None, :]
    g = lambda k: math.factorial(k) / a ** (k + 1)  # noqa: E731
    S = NN * g(2 * n)
    H = NN * ((z[None, :] * n - Z) * g(2 * n - 1) - 0.5 * z[None, :] ** 2 * g(2 * n))
    return S, 0.5 * (H + H.T)


def _one_electron(basis, Z):
    S, H = np.zeros((len(basis),) * 2), np.zeros((len(basis),) * 2)
    for l in sorted({b[2] for b in basis}):
        at = [[i for i, b in enumerate(basis) if b[2:] == (l, m)] for m in range(-l, l + 1)]
        s, h = _radial([basis[i][0] for i in at[0]], l, Z)
        for ix in at:
            S[np.ix_(ix, ix)], H[np.ix_(ix, ix)] = s, h
    return S, H


def _orbitals(basis, Z, occ, rs):
    """Occupied orbitals [nb][n] in the real-harmonic basis, as in the middle of an SCF: the lowest eigenvectors per l of the
    core Hamiltonian with a random screening of a few per cent, filled over all m."""
    cols = []
    for l, cnt in enumerate(int(x) for x in occ.split(",") if x):
        at = [[i for i, b in enumerate(basis) if b[2:] == (l, m)] for m in range(-l, l + 1)]
        s, h = _radial([basis[i][0] for i in at[0]], l, Z)
        e, V = np.linalg.eigh(s)
        X = V[:, e > 1e-9 * e[-1]] / np.sqrt(e[e > 1e-9 * e[-1]])
        hx = X.T @ h @ X
        e, V = np.linalg.eigh(hx)
        noise = rs.normal(size=(cnt + 1,) * 2) * 0.05
        k = min(cnt + 1, len(e))
        V[:, :k] = V[:, :k] @ np.linalg.qr(np.eye(k) + noise[:k, :k])[0]
        for ix in at:
            for c in range(cnt):
                col = np.zeros(len(basis))
                col[ix] = X @ V[:, c]
                cols.append(col)
    return np.stack(cols, axis=1) if cols else np.zeros((len(basis), 0))


def _density(basis, C):
    U = _unitary(basis)
    return np.ascontiguousarray(U.T @ (C @ C.T) @ U.conj())


def _points(case, seed, which=0):
    """Quadrature points and weights: radial x Lebedev, or the scrambled-Sobol grid of electron `which`."""
    if "nrad" in case:
        return grids.product_grid(case["nrad"], case["order"])
    ndim = case.get("dim2", 3) if which else 3
    return grids.qmc_grid(ndim, case["n2"] if which else case["n1"], 3 * int(seed) + which)


def _inputs(case, seed):
    """basis, S, h, densities [nspin][nb][nb] (reference basis) and orbitals per spin (real harmonics)."""
    rs = np.random.RandomState(int(seed) % (1 << 31))
    basis = _basis(case, rs if case["kind"] in ("scf", "one_electron") else None)
    S, h = _one_electron(basis, case["Z"])
    C = [_orbitals(basis, case["Z"], case[s], rs) for s in ("up", "down") if s in case]
    return basis, S, h, np.stack([_density(basis, c) for c in C]), C


def _tc_orbitals(basis, C, seed):
    """Occupied orbitals [n][nb] in the reference basis with the arbitrary phases an eigen-solver returns."""
    rs = np.random.RandomState((int(seed) + 77) % (1 << 31))
    return [np.ascontiguousarray((_unitary(basis).T @ c * np.exp(2j * np.pi * rs.rand(c.shape[1]))).T) for c in C]


def _instances(case):
    rng = random.Random(case["set"])
    return [{"kind": "fock", "nrad": rng.randint(40, 120), "order": rng.choice([17, 19, 21, 23, 25, 27, 29, 31, 35]), **_atom(rng)}
            for _ in range(case["count"])]


# ---- the program's side ---------------------------------------------------------------------------------------
_CTX = []


def _context():
    if not _CTX:
        _CTX.append(api.Context(0))
    return _CTX[0]


class Held(dict):
    """What a program holds; its device grids and tensors go when it goes."""

    def __del__(self):
        for x in self.get("own", []):
            x.close()


def _grid(state, points, basis, gradients=False):
    G = api.QMCGrid(_context(), points)
    state["own"].append(G)
    G.setBasisFunctions(basis, storeGradients=gradients)
    return G


def _jastrow():
    return ffi.ochi_struct(A12, A12, [((1, 0, 0), -A12 / 2, -A12 / 4)])


def _tc_tensors(case, G1, G2, G3, u):
    p = PRECISION[case["prec"]]
    return [api.computeF(G1, G2, k, u, keep=True, copy=False, precision=p)[1] for k in (ffi.K_TC_SCALAR_SAME, ffi.K_TC_SCALAR_OPPO)] + \
           [api.computeV(G1, G3, k, u, keep=True, copy=False, precision=p)[1] for k in (ffi.K_GRAD_U_SAME, ffi.K_GRAD_U_OPPO)]


def prepare(case, seed):
    s = Held(case=case, own=[])
    if case["kind"] == "batch":
        s["grids"], s["D"], s["h"] = [], [], []
        for k, inst in enumerate(_instances(case)):
            basis, _, h, D, _ = _inputs(inst, seed + k)
            s["grids"].append(_grid(s, _points(inst, seed), basis))
            s["D"].append(D[0])
            s["h"].append(h)
        return s
    s["basis"], s["S"], s["h"], s["D"], C = _inputs(case, seed)
    s["n_occ"] = C[0].shape[1]
    if case["kind"] == "one_electron":
        s["points"] = _points(case, seed)
        return s
    tc = case["kind"].startswith("tc_")
    s["G1"] = _grid(s, _points(case, seed), s["basis"], gradients=tc)
    s["G2"] = s["G1"] if "nrad" in case else _grid(s, _points(case, seed, 1), s["basis"])
    if tc:
        s["occ"], s["u"] = _tc_orbitals(s["basis"], C, seed), _jastrow()
        s["G3"] = _grid(s, _points(case, seed, 2), s["basis"])
        if case["kind"] == "tc_build":
            s["tensors"] = _tc_tensors(case, s["G1"], s["G2"], s["G3"], s["u"])
            s["own"] += s["tensors"]
    if case["kind"] == "precomputed":
        s["F"] = api.computeF(s["G1"], s["G2"], ffi.K_INV_R12, keep=True, copy=False)[1]
        s["own"].append(s["F"])
    return s


def run(s):
    case, kind = s["case"], s["case"]["kind"]
    if kind == "fock":
        return api.fock_build(s["G1"], s["G2"], s["D"], s["h"], precision=PRECISION[case["prec"]])
    if kind == "scf":
        hf = api.RCSHartreeFock(s["n_occ"], s["n_occ"], len(s["basis"]))
        e = hf.compute(s["S"], s["h"], s["G1"], s["G2"], precision=PRECISION[case["prec"]], tol=1e-8)
        return e, hf.density, hf.eigenvalues
    if kind == "batch":
        return api.fock_build_batch(s["grids"], s["grids"], s["D"], s["h"], precision=PRECISION[case["prec"]], want_fock=True)
    if kind == "one_electron":
        G = api.QMCGrid(_context(), s["points"])
        G.setBasisFunctions(s["basis"], storeGradients=True)
        SH = api.overlap_core_quadrature(G, case["Z"])
        G.close()
        return SH
    if kind == "precomputed":
        return api.fock_build_precomputed(s["G1"], s["F"], s["D"], s["h"])
    t = s["tensors"] if kind == "tc_build" else _tc_tensors(case, s["G1"], s["G2"], s["G3"], s["u"])
    out = api.tc_fock_build(s["G1"], *t, len(s["occ"][0]), len(s["occ"][1]), s["D"], s["occ"][0], s["occ"][1], s["h"])
    if kind == "tc_cycle":
        for x in t:
            x.close()
    return out


def _sizes(case):
    n1 = case["nrad"] * LEBEDEV[case["order"]] if "nrad" in case else case["n1"]
    return n1, n1 if "nrad" in case else case["n2"], _nb(case)


def work(case):
    if case["kind"] == "batch":
        each = [work({**c, "prec": case["prec"]}) for c in _instances(case)]
        return {k: sum(w[k] for w in each) for k in ("bytes", "flops")}
    n1, n2, nb = _sizes(case)
    occ = [sum((2 * l + 1) * int(x) for l, x in enumerate(case[s].split(",")) if x) for s in ("up", "down") if s in case]
    np_, mats = nb * (nb + 1) // 2, 16 * 4 * nb * nb * len(occ)
    if case["kind"] in ("fock", "scf"):
        # each pair of points once (unordered where r1 and r2 are one grid): distance and 1/r12 (10), rho, the exchange row and
        # the Coulomb sum; an SCF takes about ten builds
        pairs = n1 * (n1 + 1) // 2 if "nrad" in case else n1 * n2
        k = 10 if case["kind"] == "scf" else 1
        pts = n1 if "nrad" in case else n1 + n2
        return {"bytes": k * (pts * (nb + 4) * 8 + mats), "flops": k * pairs * (10 + sum(2 * (r + nb) + 2 for r in occ))}
    if case["kind"] == "one_electron":
        # points in; S and H are sums over n1 of one value and three gradient components per pair of functions, complex
        return {"bytes": n1 * 32 + n1 * nb * 8 * 9 + mats, "flops": n1 * (np_ * 4 * 8 + nb * 100)}
    if case["kind"] == "precomputed":
        # the kernel integrals are real and symmetric in the real-harmonic basis: n1 np doubles
        return {"bytes": n1 * (np_ + 2 * nb + 1) * 8 + mats, "flops": n1 * len(occ) * nb * nb * 8}
    build = {"bytes": n1 * (8 * np_ + 8 * nb + 1) * 8 + mats,
             "flops": n1 * 2 * (8 * nb * nb * 4 * 3 + nb * nb * 8 * (4 + 3 * sum(occ)))}
    if case["kind"] == "tc_build":
        return build
    return {"bytes": build["bytes"] + (n1 + 2 * n2) * (nb + 4) * 8, "flops": build["flops"] + n1 * n2 * 8 * (2 * np_ + 10)}


# ---- the same results in plain 64-bit torch -------------------------------------------------------------------
def _dev(a):
    return torch.as_tensor(np.ascontiguousarray(a), device="cuda" if torch.cuda.is_available() else "cpu")


def _legendre(l, m, x, s):
    """Y_l^m(theta, 0) with the Condon-Shortley phase, m >= 0; 0 for m > l."""
    if m > l:
        return torch.zeros_like(x)
    p = torch.full_like(x, math.sqrt((2 * m + 1) / (4 * math.pi)))
    for k in range(1, m + 1):
        p = p * -s * math.sqrt((2 * k - 1) / (2 * k))
    below = torch.zeros_like(x)
    for j in range(m + 1, l + 1):
        a = math.sqrt((4 * j * j - 1) / (j * j - m * m))
        b = math.sqrt(((j - 1) ** 2 - m * m) / (4 * (j - 1) ** 2 - 1)) if j > 1 else 0.0
        p, below = a * (x * p - b * below), p
    return p


def _cartesian(g):
    p = _dev(g.points)
    return p if p.shape[0] == 3 else torch.stack([p[0], torch.zeros_like(p[0]), p[1]])


def _values(points, basis, gradients=False):
    """Complex values [n][nb] (and gradients [n][nb][3], with the reference's formula) of the STOs."""
    x, y, z = points
    r = torch.sqrt(x * x + y * y + z * z)
    ct, st, ph = z / r, torch.sqrt(x * x + y * y) / r, torch.atan2(y, x)
    th = torch.acos(ct)
    sth, cth, sp, cp = torch.sin(th), torch.cos(th), torch.sin(ph), torch.cos(ph)
    vals, grads = [], []
    for a, n, l, m in basis:
        R = (2 * a) ** (n + 0.5) / math.sqrt(math.factorial(2 * n)) * r ** (n - 1) * torch.exp(-a * r)
        Y = _legendre(l, abs(m), ct, st) * torch.exp(1j * m * ph)
        vals.append(R * Y)
        if gradients:
            c1 = math.sqrt((l - m) * (l + m + 1)) if l != m else 0.0
            up = c1 * torch.exp(-1j * ph) * _legendre(l, abs(m + 1), ct, st) * torch.exp(1j * (m + 1) * ph)
            gr, gt, gp = ((n - 1) / r - a) * R * Y, (m * Y / torch.tan(th) + up) * R / r, 1j * m * Y * R / (r * sth)
            grads.append(torch.stack([gr * cp * sth + gt * cp * cth - gp * sp, gr * sp * sth + gt * sp * cth + gp * cp, gr * cth - gt * sth], -1))
    vals = torch.stack(vals, 1)
    return (vals, torch.stack(grads, 1)) if gradients else vals


def _real(vals, U):
    return (vals @ U.T).real.contiguous()


def _distance(a, b):
    """r12 of points a [3][n] and b [3][m]."""
    d2 = torch.zeros((a.shape[1], b.shape[1]), dtype=a.dtype, device=a.device)
    for k in range(3):
        d2.add_((a[k][:, None] - b[k][None, :]).square_())
    return d2.sqrt_()


def _inverse(r):
    return torch.where(r == 0, torch.zeros((), dtype=r.dtype, device=r.device), 1 / r)


def _finish(G, G3, D, h, factor):
    """Masked G, F and the energy of the reference's constructSCFOperator."""
    mask = (h != 0).to(G.dtype)
    G, G3 = G * mask, G3 * mask
    e = factor * torch.einsum("sij,sji->", D, h + G / 2 - G3 / 3).real
    return G, G3, h + G - G3, float(e)


def _exact_fock(g1, g2, basis, D, C, h):
    U = _dev(_unitary(basis))
    p1, p2, w1, w2 = _cartesian(g1), _cartesian(g2), _dev(g1.weights), _dev(g2.weights)
    f1, f2 = _real(_values(p1, basis), U), _real(_values(p2, basis), U)
    C, D, h = [_dev(c) for c in C], _dev(D), _dev(h)
    psi1, psi2 = [f1 @ c for c in C], [f2 @ c for c in C]
    wf2, src = w2[:, None] * f2, [w2 * (q * q).sum(1) for q in psi2]
    GR = [torch.zeros(len(basis), len(basis), dtype=f1.dtype, device=f1.device) for _ in C]
    step = max(1, (1 << 27) // p2.shape[1])
    for a in range(0, p1.shape[1], step):
        b = slice(a, a + step)
        g = _inverse(_distance(p1[:, b], p2))
        VH = sum(g @ s for s in src)
        wf = w1[b, None] * f1[b]
        for k in range(len(C)):
            T = ((psi1[k][b] @ psi2[k].T).mul_(g)) @ wf2
            GR[k] += wf.T @ ((2.0 if len(C) == 1 else 1.0) * VH[:, None] * f1[b] - T)
    G = torch.stack([U.T @ x.to(U.dtype) @ U.conj() for x in GR])
    G, _, F, e = _finish(G, torch.zeros_like(G), D, h, 2.0 if len(C) == 1 else 1.0)
    return G, F, e


def _exact_scf(g, basis, S, h, nocc):
    U = _dev(_unitary(basis))
    p, w = _cartesian(g), _dev(g.weights)
    f = _real(_values(p, basis), U)
    kern, hd = _inverse(_distance(p, p)), _dev(h)
    L = torch.linalg.cholesky(_dev(S))
    DR, e, W = torch.zeros_like(hd), float("inf"), None
    for _ in range(50):
        q = f @ DR
        VH, T = kern @ (w * (q * f).sum(1)), ((q @ f.T) * kern) @ (w[:, None] * f)
        G = (w[:, None] * f).T @ (2 * VH[:, None] * f - T) * (hd != 0)
        ne = float(2 * (DR * (hd + G / 2)).sum())
        if abs(ne - e) < 1e-8:
            break
        e = ne
        A = torch.linalg.solve_triangular(L, torch.linalg.solve_triangular(L, hd + G, upper=False).T, upper=False)
        W, V = torch.linalg.eigh(0.5 * (A + A.T))
        c = torch.linalg.solve_triangular(L.T, V[:, :nocc], upper=True)
        DR = c @ c.T
    return ne, (U.T @ DR.to(U.dtype) @ U.conj())[None], W[None]


def _exact_pairs(p1, kern, p2, f2, w2, U):
    """kern(r1, r2) integrated against conj(phi_j) phi_i over r2: the components kern gives, complex [n1][nb][nb] each."""
    nb = f2.shape[1]
    k, l = torch.triu_indices(nb, nb, device=f2.device)
    W = w2[:, None] * f2[:, k] * f2[:, l]
    full = torch.zeros(nb, nb, dtype=torch.long, device=f2.device)
    full[k, l] = full[l, k] = torch.arange(len(k), device=f2.device)
    return [U.T @ (K @ W)[:, full].to(U.dtype) @ U.conj() for K in kern(p1, p2)]


def _tc_scalar(c):
    def kern(p1, p2):
        r = _distance(p1, p2)
        f = c * A12 / (r + A12) ** 2   # |grad u| of u = c r / (r + a)
        return [torch.where(r == 0, torch.zeros((), dtype=r.dtype, device=r.device), 2 / r - 2 * f * f)]
    return kern


def _grad_u(c):
    def kern(p1, p2):
        r = _distance(p1, p2)
        f = torch.where(r == 0, torch.zeros((), dtype=r.dtype, device=r.device), c * A12 / (r * (r + A12) ** 2))
        return [f * (p1[k][:, None] - p2[k][None, :]) for k in range(3)]
    return kern


def _exact_tc(case, seed, basis, D, C, h):
    U = _dev(_unitary(basis))
    g = [_points(case, seed, k) for k in range(3)]
    p, w = [_cartesian(x) for x in g], [_dev(x.weights) for x in g]
    v1, gr1 = _values(p[0], basis, True)
    f2, f3 = _real(_values(p[1], basis), U), _real(_values(p[2], basis), U)
    occ, D, h = [_dev(c) for c in _tc_orbitals(basis, C, seed)], _dev(D), _dev(h)
    sums = torch.zeros((3, 2) + h.shape, dtype=U.dtype, device=U.device)
    step = max(16, (1 << 25) // max(case["n2"], 2 * len(basis) ** 2))
    es = torch.einsum
    for a in range(0, case["n1"], step):
        b = slice(a, a + step)
        q, v, gr, wt = p[0][:, b], v1[b], gr1[b], w[0][b].to(U.dtype)
        F = [_exact_pairs(q, _tc_scalar(c), p[1], f2, w[1], U)[0] for c in (-A12 / 4, -A12 / 2)]
        V = [torch.stack(_exact_pairs(q, _grad_u(c), p[2], f3, w[2], U), -1) for c in (-A12 / 4, -A12 / 2)]
        VT, SG, occd, sumN, VTs, SCV = [], [], [], [], [], []
        Vjb = [[es("bi,rjic->rjbc", occ[s], V[t]) for t in (0, 1)] for s in (0, 1)]
        for s in (0, 1):
            o, cv = 1 - s, v.conj()
            VT.append(es("rjic,ij->rc", V[0], D[s]) + es("rjic,ij->rc", V[1], D[o]))
            SG.append(es("ij,rj,ric->rc", D[s], cv, gr))
            kv = v @ D[s]
            occd.append((cv * kv).sum(1).real.to(U.dtype))
            sumN.append([es("aj,rjbc->rabc", occ[s].conj(), Vjb[s][t]).abs().square().sum((1, 2, 3)) for t in (0, 1)])
            VTs.append(es("rj,rjic->ric", kv, V[0]))
            SCV.append(es("rkc,rk->rc", VTs[s].conj(), kv))
        for s in (0, 1):
            o, cv, kv = 1 - s, v.conj(), v @ D[s]
            faa = es("rji,ij->r", F[0], D[s]) + es("rji,ij->r", F[1], D[o])
            fai = es("rj,rji->ri", kv, F[0])
            vai = es("rjic,rjc->ri", V[0], es("kj,rkc->rjc", D[s], gr))
            vja = es("rj,rijc->ric", cv @ D[s].T, V[0])
            svd = es("rkic,rkc->ri", V[0], es("lk,rlc->rkc", D[s], VTs[s]))
            wv = wt[:, None] * cv
            sums[0, s] += wv.T @ (faa[:, None] * v - fai)
            sums[1, s] += wv.T @ (es("rc,ric->ri", VT[s], gr) - vai) + es("r,rjic,rc->ji", wt, V[0], SG[s]) + es("r,rjic,rc->ji", wt, V[1], SG[o]) \
                - es("r,rjc,ric->ji", wt, vja, gr)
            x = (VT[s].abs().square().sum(1) - sumN[s][0] - sumN[o][1])[:, None] * v + 2 * (svd - es("rc,ric->ri", VT[s], VTs[s]))
            sums[2, s] += wv.T @ x + 2 * (wt[:, None] * (svd.conj() - es("rjc,rc->rj", VTs[s].conj(), VT[s]))).T @ v
            sums[2, s] += 2 * es("r,ric,rjc->ji", wt, VTs[s], VTs[s].conj())
            for t, k in ((0, s), (1, o)):
                sums[2, s] += 2 * es("r,rjic,rc->ji", wt, V[t], occd[k][:, None] * VT[k] - SCV[k])
                sums[2, s] -= 2 * es("r,rjbc,ribc->ji", wt * occd[k], Vjb[s][t], Vjb[s][t].conj())
    G2 = 0.5 * (sums[0] + sums[1] - sums[1].mH)
    G2, G3, F, e = _finish(G2, 0.5 * sums[2], D, h, 1.0)
    return G2, G3, F, e


def exact(case, seed):
    if case["kind"] == "batch":
        es, Fs = [], []
        for k, inst in enumerate(_instances(case)):
            basis, _, h, D, C = _inputs(inst, seed + k)
            g = _points(inst, seed)
            _, F, e = _exact_fock(g, g, basis, D, C, h)
            es.append(e)
            Fs.append(F[0])
        return np.array(es), Fs
    basis, S, h, D, C = _inputs(case, seed)
    if case["kind"].startswith("tc_"):
        return _exact_tc(case, seed, basis, D, C, h)
    g1 = _points(case, seed)
    g2 = g1 if "nrad" in case else _points(case, seed, 1)
    if case["kind"] == "scf":
        return _exact_scf(g1, basis, S, h, C[0].shape[1])
    if case["kind"] == "one_electron":
        v, gr = _values(_cartesian(g1), basis, True)
        w, r = _dev(g1.weights), _cartesian(g1).square().sum(0).sqrt()
        over = lambda x: (v * x[:, None]).mH @ v  # noqa: E731
        return over(w), 0.5 * sum((gr[:, :, k] * w[:, None]).mH @ gr[:, :, k] for k in range(3)) - case["Z"] * over(w / r)
    if case["kind"] == "precomputed" and case["dim2"] == 2:
        g2 = grids.QuadratureGrid(g2.points, 2 * math.pi * g2.weights)
    return _exact_fock(g1, g2, basis, D, C, h)

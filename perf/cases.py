"""The calls whose time counts: the work a program gives this engine, through
its public entry points (william_ci_b200.engine, william_ci_b200.df).

A case is a dict of plain values.  `kind` picks the call:

  jk       J and K of one SCF iteration from a resident engine handle
           (Engine.direct_JK on host arrays, or Engine.direct_JK_device on
           device buffers with the pass captured as a CUDA graph), with the
           system's fixed t-rule or with the learned grid;
  stored   the stored two-electron integrals and J, K from them
           (Engine.ERI_integral_toroidal, Engine.stored_JK);
  nuclear  the nuclear attraction matrix (Engine.nuclear_attraction);
  kmo      k-space MO integrals from the stored ones (Engine.ao_to_kmo);
  dfjk     density-fitted J and K (df.DFJK);
  dfmp2    density-fitted k-MP2 energy (df.DeviceDF.dfmp2).

Systems are the named workloads of william_ci_b200.system on `cells` cells:
`ring` (STO-3G hydrogens), `chain` (3 contracted s + 1 p per H, one periodic
direction), `sheet` (s, p, d; two periodic directions), `cube` (s, p; three).
`basis` is the seed of the workload's exponents, `spacing` a factor on its cell length.  The seed given to prepare
makes the density, the orbitals and the fitted coefficients.
"""
import dataclasses
import math

import numpy as np
import torch

from william_ci_b200 import df as DF
from william_ci_b200.engine import TCE_METHOD_LEARNED, Engine
from william_ci_b200.system import AOSystem, build_system, scaled_down, workload


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # the smallest call: a two-cell STO-3G ring, host arrays in and out
        # (tests and first steps of a user's program); launches and copies count
        _case("ring2-host", "jk", "ring", (2, 1, 1), route="host"),
        # the headline configuration with the default method: the 64-cell chain,
        # one J/K pass of an SCF iteration, the 32-node rule, device buffers
        _case("chain64-fixed", "jk", "chain", (64, 1, 1)),
        # the same pass with the learned grid, the engine's accurate method
        _case("chain64-learned", "jk", "chain", (64, 1, 1), learned=True),
        # a ragged chain with the 40-node rule (the reference's nquad_128 setting),
        # J and K through host arrays as scf.py calls them
        _case("chain27-40nodes-host", "jk", "chain", (27, 1, 1), nquad=40, route="host"),
        # a learned-grid chain of ordinary size
        _case("chain16-learned", "jk", "chain", (16, 1, 1), learned=True),
        # two periodic directions, s, p and d shells
        _case("sheet3x2-fixed", "jk", "sheet", (3, 2, 1)),
        _case("sheet3x3-learned", "jk", "sheet", (3, 3, 1), learned=True),
        # three periodic directions, s and p shells
        _case("cube2-learned", "jk", "cube", (2, 2, 2), learned=True),
        # the stored path of a small system: all integrals, then J and K from them
        _case("chain13-stored", "stored", "chain", (13, 1, 1)),
        # the nuclear attraction of the headline chain (once per geometry)
        _case("chain64-nuclear", "nuclear", "chain", (64, 1, 1)),
        # (ov|ov) over k for a correlated method after the SCF
        _case("chain20-kmo", "kmo", "chain", (20, 1, 1)),
        # density-fitted k-MP2 of a chain at the size of the named 128-cell one
        _case("chain96-dfmp2", "dfmp2", "chain", (96, 1, 1)),
    ]


def draw(rng):
    """One more case of the ranges above: sizes spread over each path's range,
    odd ones among them."""
    kind = rng.choice(["ring", "chain", "chain", "chain-l", "chain-l", "sheet", "sheet", "cube", "stored",
                       "nuclear", "kmo", "dfjk", "dfmp2"])
    basis = rng.choice([2026, 2026, 7, 11, 19])
    spacing = round(rng.uniform(1.0, 1.3), 3)

    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    if kind == "ring":
        return _case(None, "jk", "ring", (size(2, 6), 1, 1), route=rng.choice(["host", "device"]), spacing=spacing)
    if kind == "chain":
        return _case(None, "jk", "chain", (size(4, 48), 1, 1), nquad=rng.choice([32, 32, 40]), basis=basis,
                     spacing=spacing, route=rng.choice(["host", "device"]))
    if kind == "chain-l":
        return _case(None, "jk", "chain", (size(8, 48), 1, 1), learned=True, basis=basis, spacing=spacing)
    if kind == "sheet":
        n = rng.choice([(2, 2, 1), (3, 2, 1), (2, 3, 1), (3, 3, 1)])
        return _case(None, "jk", "sheet", n, learned=rng.random() < 0.5, spacing=spacing)
    if kind == "cube":
        n = rng.choice([(2, 2, 2), (2, 2, 2), (3, 2, 2)])
        return _case(None, "jk", "cube", n, learned=rng.random() < 0.5, spacing=spacing)
    if kind == "stored":
        return _case(None, "stored", "chain", (size(3, 16), 1, 1), nquad=rng.choice([32, 40]), basis=basis, spacing=spacing)
    if kind == "nuclear":
        return _case(None, "nuclear", "chain", (size(6, 64), 1, 1), nquad=rng.choice([32, 40]), basis=basis, spacing=spacing)
    if kind == "kmo":
        return _case(None, "kmo", "chain", (size(5, 22), 1, 1), spacing=spacing)
    if kind == "dfjk":
        return _case(None, "dfjk", "chain", (size(8, 100), 1, 1), spacing=spacing)
    return _case(None, "dfmp2", "chain", (size(10, 96), 1, 1), spacing=spacing)


def _case(name, kind, system, cells, nquad=32, learned=False, route="device", basis=2026,
          spacing=1.0):
    c = {"kind": kind, "system": system, "nx": cells[0], "ny": cells[1], "nz": cells[2], "nquad": nquad,
         "learned": learned, "route": route, "basis": basis, "spacing": spacing}
    if name is not None:
        c["name"] = name
    return c


# ---------------------------------------------------------------------------
# systems and inputs
# ---------------------------------------------------------------------------
AUX_BANDS = 16    # auxiliary functions per cell of the density fitting below: 4 s + 2 p + 1 d shells


def _cells(case):
    return case["nx"], case["ny"], case["nz"]


def _system(case) -> AOSystem:
    """The workload's supercell with coefficients normalised as real Gaussians."""
    name = {"ring": "h2_ring", "chain": "h_chain64", "sheet": "h2_sheet", "cube": "li_cube"}[case["system"]]
    cell, basis = workload(name, seed=case["basis"])
    cell = dataclasses.replace(cell, spacing=cell.spacing * case["spacing"])
    return _normalised(build_system(scaled_down(cell, _cells(case)), basis))


def _normalised(s: AOSystem) -> AOSystem:
    dfact = (1.0, 1.0, 3.0)     # (2l - 1)!!
    for f in range(s.nbas):
        p0, p1 = s.prim_off[f], s.prim_off[f + 1]
        a = s.exps[p0:p1]
        l3 = [int(x) for x in s.lxyz[f]]
        l = sum(l3)
        nrm = (2.0 * a / math.pi) ** 0.75 * (4.0 * a) ** (0.5 * l) / math.sqrt(math.prod(dfact[x] for x in l3))
        c = s.coefs[p0:p1] * nrm
        m = a[:, None] + a[None, :]
        ov = (math.pi / m) ** 1.5 * math.prod(dfact[x] for x in l3) / (2.0 * m) ** l
        s.coefs[p0:p1] = c / math.sqrt(float(c @ ov @ c))
    return s


def _density(s: AOSystem, seed: int) -> np.ndarray:
    """A symmetric density of the supercell's translations, decaying with the
    distance on the torus, as an SCF iteration hands it over."""
    rng = np.random.default_rng(seed)
    n, nf = s.ncell, s.nfuc
    crd = np.array([[x, y, z] for z in range(n[2]) for y in range(n[1]) for x in range(n[0])])
    nc = len(crd)
    far = np.minimum(crd, np.array(n) - crd)
    blk = rng.standard_normal((nc, nf, nf)) * np.exp(-0.9 * np.sqrt((far ** 2).sum(1)))[:, None, None]
    blk[0] += np.eye(nf)
    idx = (crd[None, :, :] - crd[:, None, :]) % np.array(n)      # cell of (column - row)
    idx = idx[..., 0] + n[0] * (idx[..., 1] + n[1] * idx[..., 2])
    P = blk[idx].transpose(0, 2, 1, 3).reshape(nc * nf, nc * nf)
    return np.asfortranarray(0.5 * (P + P.T))


def _orbitals(case, nf, seed):
    """Unitary k blocks, energies with a gap, two electrons per cell."""
    rng = np.random.default_rng(seed)
    n = case["nx"]
    z = rng.standard_normal((n, nf, nf)) + 1j * rng.standard_normal((n, nf, nf))
    C = np.linalg.qr(z)[0]
    eps = np.sort(rng.uniform(0.1, 2.0, (n, nf)), axis=1)
    eps[:, 0] = -rng.uniform(0.2, 0.8, n)
    occ = np.zeros((n, nf), dtype=np.int32)
    occ[:, 0] = 2
    return C, eps, occ


def prepare(case, seed):
    kind = case["kind"]
    if kind == "dfjk":          # the fitted coefficients of a fit done before (host arrays, as df.DFJK takes them)
        B, Bh, P, ncl, nf, nau = _fitted(case, seed)
        return {"case": case, "h": DF.DFJK(B, Bh, ncl, nf, nau), "P": P}
    s = _system(case)
    st = {"case": case, "sys": s}
    if kind == "dfmp2":
        cell, _ = workload("h_chain64", seed=case["basis"])
        cell = dataclasses.replace(cell, spacing=cell.spacing * case["spacing"])
        aux = _normalised(build_system(scaled_down(cell, _cells(case)), DF.even_tempered_aux([1])))
        st["h"] = DF.DeviceDF(s, aux)
        st["C"], st["eps"], st["occ"] = _orbitals(case, s.nfuc, seed)
        return st
    e = Engine(s, nquad=case["nquad"])
    st["h"] = e
    if kind == "nuclear":       # the charges move: each step of a geometry search asks again
        rng = np.random.default_rng(seed)
        st["geo"] = np.asfortranarray(s.geometry + rng.uniform(-0.05, 0.05, s.geometry.shape) * [1.0, 0.0, 0.0])
        return st
    st["P"] = _density(s, seed)
    if kind == "kmo":
        e.ERI_integral_toroidal()
        st["C"] = _orbitals(case, s.nfuc, seed)[0]
        return st
    if case["learned"]:
        e.lg_setup(n_train=3000, seed=2026, epochs=40)
        e.set_method(TCE_METHOD_LEARNED)
    if kind == "jk" and case["route"] == "device":
        e.set_graph(True)
        n, nf = s.nbas, s.nfuc
        st["dP"] = torch.from_numpy(np.ascontiguousarray(st["P"].T)).cuda()     # column-major n x n
        st["dJ"] = torch.zeros((n, nf), dtype=torch.float64, device="cuda")     # column-major nf x n
        st["dK"] = torch.zeros((n, nf), dtype=torch.float64, device="cuda")
    return st


def run(state):
    case, h = state["case"], state["h"]
    kind = case["kind"]
    if kind == "jk":
        if case["route"] == "host":
            return h.direct_JK(state["P"])
        h.direct_JK_device(state["dP"].data_ptr(), state["dJ"].data_ptr(), state["dK"].data_ptr(),
                           torch.cuda.current_stream().cuda_stream)
        return state["dJ"], state["dK"]
    if kind == "stored":
        eri = h.ERI_integral_toroidal()
        J, K = h.stored_JK(state["P"])
        return eri, J, K
    if kind == "nuclear":
        return h.nuclear_attraction(geometry=state["geo"])
    if kind == "kmo":
        nf = state["sys"].nfuc
        return h.ao_to_kmo(state["C"], (0, 1), (1, nf))
    if kind == "dfjk":
        return h(state["P"])
    r = h.dfmp2(state["C"], state["eps"], state["occ"], mode=0)
    return r["emp2"], r["e2d"], r["e2x"]


# ---------------------------------------------------------------------------
# the fit handed to the density-fitted J/K: decaying three-index coefficients
# ---------------------------------------------------------------------------
def _fitted(case, seed):
    rng = np.random.default_rng(seed)
    s = _system(case)
    n, nf, nau = case["nx"], s.nfuc, AUX_BANDS
    far = np.minimum(np.arange(n), n - np.arange(n))
    B = rng.standard_normal((nf, n, nf, n, nau))
    B *= np.exp(-0.7 * far)[None, :, None, None, None] * np.exp(-0.4 * far)[None, None, None, :, None]
    B = np.asfortranarray(B.reshape(nf, n * nf, n, nau).reshape(nf, n * nf, n * nau))
    nkh = int((DF.khalf((n, 1, 1)) >= 0).sum())
    Bh = rng.standard_normal((nf, nau, nf, n, nkh)) + 1j * rng.standard_normal((nf, nau, nf, n, nkh))
    return B, np.asfortranarray(Bh), _density(s, seed + 1), (n, 1, 1), nf, nau


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _pair_counts(s: AOSystem):
    """Significant function pairs (first function in the unit cell) and primitive
    pairs, by the product's Gaussian prefactor with the nearest image."""
    nc = int(np.prod(s.ncell))
    npair = nprim = 0.0
    L = np.array([x if x > 0 else 1e30 for x in s.L])
    shells = {}
    for f in range(s.nbas):
        shells.setdefault((int(s.atom_of[f]), float(s.exps[s.prim_off[f]]), int(s.lxyz[f].sum()),
                           float(s.coefs[s.prim_off[f]]) if s.lxyz[f].sum() == 0 else 0.0), []).append(f)
    reps = [(v[0], len(v)) for v in shells.values()]
    uc = [(f, m) for f, m in reps if f < s.nfuc]
    for f, m in uc:
        a = s.exps[s.prim_off[f]:s.prim_off[f + 1]]
        for g, mg in reps:
            b = s.exps[s.prim_off[g]:s.prim_off[g + 1]]
            d = np.abs(s.ctr[f] - s.ctr[g])
            r2 = float((np.minimum(d, np.abs(L - d)) ** 2).sum())
            k = np.exp(-(a[:, None] * b[None, :]) / (a[:, None] + b[None, :]) * r2) > 1e-13
            nprim += float(k.sum())
            npair += m * mg * float(k.any())
    return npair, nprim, nc


def work(case):
    """Inputs read once, outputs written once; operations of the quartet paths:
    one multiply-add per node and periodic or real direction of every primitive
    quartet that the pair prefactors leave (8-fold and translation unique)."""
    s = _system(case)
    n, nf, nc = s.nbas, s.nfuc, s.nbas // s.nfuc
    kind = case["kind"]
    if kind in ("jk", "stored"):
        npair, nprim, nc = _pair_counts(s)
        flops = nprim * nprim * nc / 8.0 * case["nquad"] * 6.0 + npair * npair * nc / 8.0 * 32.0
        out = 2.0 * 8.0 * n * (n if case["route"] == "host" else nf)
        if kind == "stored":
            return {"bytes": 8.0 * (n * n + nf * float(n) ** 3 + 2.0 * n * n),
                    "flops": flops + 4.0 * nf * float(n) ** 3}
        return {"bytes": 8.0 * n * n + out, "flops": flops}
    if kind == "nuclear":
        npair, nprim, nc = _pair_counts(s)
        return {"bytes": 8.0 * n * n + 32.0 * len(s.charges), "flops": nprim * len(s.charges) * case["nquad"] * 6.0}
    if kind == "kmo":
        nv = nf - 1
        return {"bytes": 8.0 * nf * float(n) ** 3 + 16.0 * nv * nv * float(nc) ** 3 + 16.0 * n * nf,
                "flops": 8.0 * nf * nv * nv * float(nc) ** 3}
    nau = AUX_BANDS
    if kind == "dfjk":
        nkh = nc // 2 + 1
        return {"bytes": 8.0 * nf * n * nau * nc + 16.0 * nf * nf * nau * nc * nkh + 3 * 8.0 * n * n,
                "flops": 4.0 * nf * n * nau * nc + 16.0 * nf * nf * nf * nau * nc * nc}
    nv = nf - 1
    return {"bytes": 8.0 * nf * n * nau * nc + 16.0 * n * nf,
            "flops": 8.0 * nau * nv * nv * float(nc) ** 3}


# ---------------------------------------------------------------------------
# the same numbers in 64 bits without the engine
# ---------------------------------------------------------------------------
def exact(case, seed):
    if case["kind"] == "dfjk":
        return _exact_dfjk(*_fitted(case, seed))
    if case["kind"] == "jk" and case["system"] == "ring" and case["nx"] <= 6:
        s = _system(case)
        J, K = _exact_jk_s(s, _density(s, seed), case["nquad"])
        if case["route"] == "host":
            return J, K
        nf = s.nfuc
        return torch.from_numpy(np.ascontiguousarray(J[:nf].T)), torch.from_numpy(np.ascontiguousarray(K[:nf].T))
    return None


def _bessel(x, nmax):
    """e^{-x} I_n(x), n = 0..nmax, by downward recurrence, normalised with
    e^{-x} (I_0 + 2 sum I_n) = 1."""
    x = np.asarray(x, dtype=np.float64)
    out = np.zeros((nmax + 1,) + x.shape)
    top = nmax + 60 + int(4.0 * math.sqrt(float(x.max()) + 1.0) * 5.0)
    hi, cur = np.zeros_like(x), np.full_like(x, 1e-290)
    tot = 2.0 * cur
    xs = np.where(x > 0, x, 1.0)
    for n in range(top, 0, -1):
        hi, cur = cur, hi + 2.0 * n / xs * cur
        big = np.abs(cur) > 1e200
        if big.any():
            f = np.where(big, 1e-200, 1.0)
            hi, cur, tot = hi * f, cur * f, tot * f
            out *= f
        tot = tot + (cur if n == 1 else 2.0 * cur)
        if n - 1 <= nmax:
            out[n - 1] = cur
    out /= tot
    zero = x <= 0
    if zero.any():
        out[:, zero] = 0.0
        out[0, zero] = 1.0
    return out


def _rule(n):
    """Gauss-Legendre on [0, 1] mapped by t = 0.6 u / (1 - u)."""
    x, w = np.polynomial.legendre.leggauss(n)
    u = 0.5 * (1.0 + x)
    return 0.6 * u / (1.0 - u), 0.5 * w * 0.6 / (1.0 - u) ** 2


def _exact_jk_s(s, P, nquad):
    n, a, L = s.nbas, 2.0 * math.pi / s.L[0], s.L[0]
    t, w = _rule(nquad)
    rows = []
    for f in range(n):
        for g in range(n):
            for i in range(s.prim_off[f], s.prim_off[f + 1]):
                for j in range(s.prim_off[g], s.prim_off[g + 1]):
                    e1, e2 = s.exps[i], s.exps[j]
                    z = e1 * np.exp(1j * a * s.ctr[f, 0]) + e2 * np.exp(1j * a * s.ctr[g, 0])
                    p = abs(z) if abs(z) > 1e-12 * (e1 + e2) else 0.0
                    rows.append((f * n + g, e1 + e2, p, math.atan2(z.imag, z.real),
                                 s.coefs[i] * s.coefs[j] * math.exp(-2.0 * (e1 + e2 - p) / a ** 2)))
    pair = np.array([r[0] for r in rows])
    es, pe, th, cf = (np.array([r[k] for r in rows]) for k in (1, 2, 3, 4))
    A, C = 2.0 * pe / a ** 2, 2.0 * t * t / a ** 2
    nmax = 40 + int(math.ceil(10.0 * math.sqrt(A.max())))
    G, T = _bessel(A, nmax), _bessel(C, nmax)
    T[1:] *= 2.0
    E = np.zeros((n * n, n * n))
    order = np.arange(nmax + 1)
    for x in range(len(pair)):
        if pair[x] // n >= s.nfuc:
            continue
        F = G[:, x:x + 1] * G * np.cos(order[:, None] * (th[x] - th)[None, :])
        I = np.einsum("nq,nk->qk", F, T)
        D = 1.0 / (es[x] * es[:, None] + (es[x] + es[:, None]) * (t * t)[None, :])
        v = 2.0 / math.sqrt(math.pi) * L * L * cf[x] * cf * math.pi ** 2 * ((I * D) @ w)
        np.add.at(E[pair[x]], pair, v)
    E = E.reshape(n, n, n, n)
    J = np.einsum("abcd,cd->ab", E, P)
    K = -0.5 * np.einsum("abcd,bc->ad", E, P)
    J[s.nfuc:] = 0.0
    K[s.nfuc:] = 0.0
    return J, K


def _exact_dfjk(B, Bh, P, ncl, nf, nau):
    """J = B gamma with gamma = sum over cells of B^T P; K(k) = -1/(2N) sum_k1,Q
    B_Q(k1, k - k1) P(k1) B_Q^H, on the host's matrices."""
    N = ncl[0]
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    Bt = torch.from_numpy(np.ascontiguousarray(B.reshape(nf, N, nf, N, nau))).to(dev)     # a, R, b, C, q
    Pt = torch.from_numpy(np.ascontiguousarray(P)).to(dev).reshape(N, nf, N, nf)           # r, a, c, b
    c = torch.arange(N, device=dev)
    # Ps(a, R, b, r) = P(r a, (R + r) b); G(C, q, r); gamma(C', q) = sum_r G(C' - r, q, r)
    Ps = Pt[c[None, :], :, (c[:, None] + c[None, :]) % N, :]                               # R, r, a, b
    G = torch.einsum("aRbCq,Rrab->Cqr", Bt, Ps)
    gam = torch.zeros((N, nau), dtype=torch.float64, device=dev)
    for r in range(N):
        gam += torch.roll(G[:, :, r], shifts=r, dims=0)
    J0 = torch.einsum("aRbCq,Cq->aRb", Bt, gam).reshape(nf, N * nf)
    ph = torch.exp(2j * math.pi * (c[:, None] * c[None, :] % N).to(torch.float64) / N)
    P0 = Pt[0].to(torch.complex128)                                                        # a, R, b
    Pk = torch.einsum("kR,aRb->kab", ph, P0)
    Pk = 0.5 * (Pk + Pk.conj().transpose(1, 2))
    khi = torch.from_numpy(DF.khalf(ncl)).to(dev)
    Bt2 = torch.from_numpy(np.ascontiguousarray(Bh)).to(dev)                               # a, Q, b, k1, kh
    Kk = torch.zeros((N, nf, nf), dtype=torch.complex128, device=dev)
    for kk in range(N):
        k2 = (kk - c) % N
        direct = khi[k2] >= 0
        k1s = torch.where(direct, c, (-c) % N)
        khs = torch.where(direct, khi[k2], khi[(-k2) % N])
        X = Bt2[:, :, :, k1s, khs].permute(3, 0, 1, 2)                                     # k1, a, Q, b
        X = torch.where(direct[:, None, None, None], X, X.conj())
        M = torch.einsum("kaQb,kbc->kaQc", X, Pk)
        Kk[kk] = -0.5 / N * torch.einsum("kaQc,keQc->ae", M, X.conj())
    K0 = torch.einsum("kab,kR->aRb", Kk, ph.conj()).real / N
    n = N * nf
    J, K = np.zeros((n, n)), np.zeros((n, n))
    J[:nf] = J0.cpu().numpy()
    K[:nf] = K0.reshape(nf, n).cpu().numpy()
    return J, K

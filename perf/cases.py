"""Performance cases of the Green-function library: the work a user's program has it do.

A case is one call sequence through ``titan_b200.native.GreenGPU`` (the binding of
``include/titan_gpu.h``) on a seeded Slater-Koster model of one of the shapes of
``titan_b200.host.synthetic``, on a mesh of the sizes that the tests, the decks and the
benchmark use.  ``prepare`` sets a context up the way a program does before its loop (system,
local Hamiltonian, meshes), ``run`` makes one pass of the loop's body, ``exact`` restates the
result with plain torch in 64 bits from the same tables.

    path       pass
    ---------  ------------------------------------------------------------------------
    rpa        chi0 for a few frequencies, then the RPA Dyson solve of each one
    chi0       chi0 for the frequencies of one wave vector (tg_chi0_batch)
    qbatch     chi0 for a few wave vectors of an adaptive mesh (tg_chi0_qbatch)
    dyson      the RPA Dyson solve alone
    scf        new local Hamiltonian, occupations and moments, Jacobian (one Newton step)
    she        the disturbance-response integral
    ldos       the local density of states on an energy grid
    jij        the exchange-coupling tensor at one wave vector
"""
from __future__ import annotations

import math

import numpy as np
import torch

from titan_b200.host import mesh as M
from titan_b200.host import synthetic
from titan_b200.host.deck import Deck
from titan_b200.host.system import initial_state
from titan_b200.native import GreenGPU, jacobian_layout

N_ORB = 9     # spd sites
N_D = 5

# sites and dimension of the lattice of each shape ("slabL": L layers, two-dimensional)
SITES = {"bcc1": 1, "sq2": 2, "bcc4": 4}
THREE_D = ("bcc1", "bcc4")


def sites(shape):
    return SITES[shape] if shape in SITES else int(shape[4:])


def case(path, shape, nk, n_e, n_real=0, n_omega=1, n_q=1, q=0.0, precision="fp64", d_only=False, adaptive=0,
         name=None):
    c = {"path": path, "shape": shape, "nk": nk, "n_e": n_e, "n_real": n_real, "n_omega": n_omega, "n_q": n_q,
         "q": q, "precision": precision, "d_only": d_only, "adaptive": adaptive}
    if name:
        c = {"name": name, **c}
    return c


def listed():
    return [
        # one static and one dynamic point of a bulk ferromagnet's spin susceptibility with its
        # RPA enhancement: the smallest deck (one atom, dimH 18), a converged-enough test mesh
        case("rpa", "bcc1", 8, 32, n_real=16, n_omega=2, name="bulk_rpa"),
        # the spin-wave spectrum of a two-atom monolayer at q = 0: several frequencies share
        # G(k, E); the benchmark's workload on a reduced mesh, split precision
        case("chi0", "sq2", 99, 64, n_real=32, n_omega=4, precision="split", name="mono_spectrum"),
        # one point of its dispersion at a finite q in FP64 (the default precision)
        case("chi0", "sq2", 100, 64, n_real=32, q=0.21, name="mono_q_fp64"),
        # two wave vectors of a five-layer film (dimH 90) on an adaptive mesh, dense k near the
        # real axis and few k far from it
        case("qbatch", "slab5", 40, 64, n_real=24, n_q=2, q=0.17, precision="split", adaptive=8, name="film_q"),
        # the d-only susceptibility of a 16-layer film (dimH 288)
        case("chi0", "slab16", 14, 32, n_real=24, precision="split", d_only=True, name="thick_film_d"),
        # the RPA solve of that film's d block, once per frequency (dimension 1600)
        case("dyson", "slab16", 0, 0, d_only=True, name="thick_film_rpa"),
        # one Newton step of a four-atom magnetic bulk cell (dimH 72)
        case("scf", "bcc4", 9, 40, name="newton_cell"),
        # one Newton step of the one-atom bulk on its production mesh
        case("scf", "bcc1", 24, 64, name="newton_bulk"),
        # spin-orbit torque of the monolayer: its response to an electric field at one frequency
        case("she", "sq2", 61, 64, n_real=32, name="mono_torque"),
        # densities of states of the four-atom cell over the band width
        case("ldos", "bcc4", 11, 501, name="cell_ldos"),
        # the exchange coupling of the monolayer at one q
        case("jij", "sq2", 81, 48, q=0.13, name="mono_exchange"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["rpa", "chi0", "chi0", "chi0", "qbatch", "dyson", "scf", "scf", "she", "ldos", "jij"])
    n_e = rng.randint(17, 64)
    q = rng.choice([0.0, rng.uniform(0.02, 0.4)])
    if path == "rpa":
        return case(path, "bcc1", rng.randint(5, 14), n_e, n_real=rng.randint(8, 32), n_omega=rng.randint(1, 3), q=q)
    if path == "chi0":
        shape = rng.choice(["bcc1", "sq2", "slab3", "bcc4", "slab%d" % rng.randint(6, 15)])
        prec = rng.choice(["split", "fp64"])
        n_real = rng.randint(8, 32)
        if shape in ("bcc1", "sq2"):
            nk = rng.randint(9, 20) if shape == "bcc1" else _log_int(rng, 13, 99)
            return case(path, shape, nk, n_e, n_real=n_real, n_omega=rng.randint(1, 3), q=q, precision=prec)
        if shape in ("slab3", "bcc4"):
            nk = rng.randint(4, 9) if shape == "bcc4" else _log_int(rng, 9, 40)
            return case(path, shape, nk, n_e, n_real=n_real, q=q, precision=prec, d_only=rng.random() < 0.5)
        return case(path, shape, rng.randint(5, 14), rng.randint(17, 32), n_real=rng.randint(8, 24), q=q,
                    precision=prec, d_only=True)
    if path == "qbatch":
        return case(path, rng.choice(["sq2", "slab4", "slab5"]), _log_int(rng, 15, 40), n_e, n_real=rng.randint(8, 24),
                    n_q=rng.randint(1, 3), q=rng.uniform(0.05, 0.3), precision=rng.choice(["split", "fp64"]),
                    adaptive=rng.randint(4, 9))
    if path == "dyson":
        layers = _log_int(rng, 1, 16)
        return case(path, "slab%d" % layers, 0, 0, d_only=layers > 4 or rng.random() < 0.5)
    if path == "scf":
        shape = rng.choice(["bcc1", "sq2", "slab3", "bcc4"])
        nk = {"bcc1": rng.randint(6, 24), "sq2": _log_int(rng, 13, 80), "slab3": _log_int(rng, 9, 30),
              "bcc4": rng.randint(4, 9)}[shape]
        return case(path, shape, nk, min(n_e, 40) if shape == "bcc4" else n_e)
    if path == "she":
        shape = rng.choice(["bcc1", "sq2", "slab3"])
        nk = {"bcc1": rng.randint(5, 14), "sq2": _log_int(rng, 13, 61), "slab3": _log_int(rng, 9, 30)}[shape]
        return case(path, shape, nk, n_e, n_real=rng.randint(8, 32), q=q)
    if path == "ldos":
        shape = rng.choice(["bcc1", "sq2", "bcc4"])
        nk = {"bcc1": rng.randint(8, 24), "sq2": _log_int(rng, 21, 99), "bcc4": rng.randint(4, 11)}[shape]
        return case(path, shape, nk, rng.randint(101, 501))
    shape = rng.choice(["bcc1", "sq2", "bcc4"])
    nk = {"bcc1": rng.randint(6, 18), "sq2": _log_int(rng, 21, 81), "bcc4": rng.randint(4, 9)}[shape]
    return case(path, shape, nk, min(n_e, 48), q=rng.uniform(0.02, 0.4))


# --------------------------------------------------------------------------- inputs
def _d_orbitals(system):
    return [list(d) for d in system.dorbs]


def _u_matrix(n_sites, d_only, U=1.0):
    """Local Coulomb matrix of spd sites with Un = Um = U on the d orbitals, in the row order of
    chi (site, mu, nu, spin pair): U on (mu mu) <-> (nu nu) pairs of equal spin pair, minus U on
    the longitudinal pairs of equal (mu, nu)."""
    n = N_D if d_only else N_ORB
    d = range(n) if d_only else range(N_ORB - N_D, N_ORB)
    blk = np.zeros((n, n, 4, n, n, 4), complex)
    for mu in d:
        for ga in d:
            for s in range(4):
                blk[mu, mu, s, ga, ga, s] += U
    for mu in d:
        for nu in d:
            for a in (1, 2):
                for b in (1, 2):
                    blk[mu, nu, a, nu, mu, b] -= U
    m = 4 * n * n
    out = np.zeros((n_sites * m, n_sites * m), complex)
    for i in range(n_sites):
        out[i * m:(i + 1) * m, i * m:(i + 1) * m] = blk.reshape(m, m)
    return out


def _chi_dim(c):
    n = N_D if c["d_only"] else N_ORB
    return 4 * n * n * sites(c["shape"])


def _deck(c, seed):
    sysm = synthetic.make_system(c["shape"], seed=20000 + int(seed))
    nk = c["nk"]
    kp = (nk, nk, nk) if c["shape"] in THREE_D else (nk, nk, 1)
    total = int(np.prod(kp))
    p = dict(kp_in=kp, kptotal=total, minimumBZmesh=total, parts=1, n1gl=c["n_e"], parts3=1,
             n3gl=max(c["n_real"], 1), emin=0.0, emax=0.3, nEner=3)
    if c["adaptive"]:
        t = np.linspace(0.0, 1.0, c["n_e"])
        p["nk_per_energy"] = np.rint(np.exp(math.log(total) * (1 - t) + math.log(c["adaptive"] ** 2) * t)).astype(int)
    return Deck.from_system(sysm, p, mesh=c["path"] != "ldos")


def _frequencies(c):
    """n_omega frequencies up to 0.15 eV; several include the static one."""
    if c["n_omega"] == 1:
        return [0.07] if c["n_real"] else [0.0]
    return [0.15 * i / (c["n_omega"] - 1) for i in range(c["n_omega"])]


def prepare(case, seed):
    c = case
    rng = np.random.default_rng(9000 + int(seed))
    st = {"case": c}
    if c["path"] == "dyson":
        D = _chi_dim(c)
        st["gpu"] = GreenGPU(0)
        st["U"] = _u_matrix(sites(c["shape"]), c["d_only"])
        x = rng.standard_normal((D, D)) + 1j * rng.standard_normal((D, D))
        # a response matrix: negative definite on average, weaker off the diagonal
        st["chi"] = 0.05 * x / math.sqrt(D) - 0.1 * np.diag(rng.uniform(0.2, 1.0, D))
        return st
    if c["path"] == "ldos":
        deck = _deck(c, seed)
        s = deck.system
        kp = (c["nk"],) * 3 if c["shape"] in THREE_D else (c["nk"], c["nk"], 1)
        deck.real_kp, deck.real_w = M.bz_fraction(s.a1, s.a2, s.a3, s.sysdim, kp)
    else:
        deck = _deck(c, seed)
    s = deck.system
    m = rng.uniform(-1.0, 1.0, 3) + np.array([0.0, 0.0, 2.0])
    h0 = s.h0(initial_state(s, tuple(m)))
    gpu = GreenGPU(0)
    gpu.set_system(s)
    gpu.set_h0(h0)
    if deck.ek is not None:
        gpu.set_imag_mesh(deck.ek)
    gpu.set_real_mesh(deck.real_kp, deck.real_w)
    st.update(gpu=gpu, deck=deck, system=s, h0=h0)
    b1 = np.asarray(s.reciprocal()[0], float)
    st["qs"] = [c["q"] * (i + 1) / c["n_q"] * b1 for i in range(c["n_q"])]
    st["es"] = _frequencies(c)
    reals = [deck.real_points(e, s.Ef) for e in st["es"]] if c["n_real"] else None
    st["x2"] = [r[0] for r in reals] if reals else None
    st["p2"] = [r[1] for r in reals] if reals else None
    if c["d_only"]:
        gpu.set_chi_orbitals(_d_orbitals(s))
    if c["path"] == "rpa":
        st["U"] = _u_matrix(s.n_atoms, False)
    elif c["path"] == "ldos":
        st["grid"] = s.Ef + np.linspace(-6.0, 6.0, c["n_e"])
    elif c["path"] == "jij":
        v = rng.standard_normal((s.n_atoms, 3))
        st["evec"] = v / np.linalg.norm(v, axis=1)[:, None]
        st["Um"] = s.Um()
    elif c["path"] == "she":
        st["efield"] = (1.0, 0.0, 0.0)
    return st


# --------------------------------------------------------------------------- one pass
def run(state):
    st, c = state, state["case"]
    gpu, path = st["gpu"], c["path"]
    if path == "dyson":
        return {"chi": gpu.dyson(st["chi"], st["U"])}
    s = st["system"]
    if path == "chi0":
        return {"chi0": gpu.chi0_batch(st["qs"][0], st["es"], s.Ef, s.eta, s.etap, st["x2"], st["p2"],
                                       c["precision"])}
    if path == "rpa":
        chi0 = gpu.chi0_batch(st["qs"][0], st["es"], s.Ef, s.eta, s.etap, st["x2"], st["p2"], c["precision"])
        return {"chi0": chi0, "chi": [gpu.dyson(x, st["U"]) for x in chi0]}
    if path == "qbatch":
        return {"chi0": gpu.chi0_qbatch(st["qs"], st["es"], s.Ef, s.eta, s.etap, st["x2"], st["p2"],
                                        c["precision"])}
    if path == "scf":
        gpu.set_h0(st["h0"])
        rho, mx, my, mz, mp = gpu.expectation(s.Ef, s.eta)
        return {"rho": rho, "mx": mx, "my": my, "mz": mz, "mp": mp, "jacobian": gpu.jacobian(s.Ef, s.eta)}
    if path == "she":
        return {"tchi": gpu.she(st["qs"][0], st["es"][0], s.Ef, s.eta, s.etap, st["x2"][0], st["p2"][0],
                                st["efield"])}
    if path == "ldos":
        up, dn = gpu.ldos(st["grid"], s.eta)
        return {"up": up, "dn": dn}
    return {"J": gpu.jij(st["qs"][0], s.Ef, s.eta, st["evec"], st["Um"])}


# --------------------------------------------------------------------------- what a pass needs
def _nk_folded(c):
    return c["nk"] ** (3 if c["shape"] in THREE_D else 2)


def work(case):
    """Each point's resolvent (4 n^3 flops where one factorisation of H(k) serves every energy:
    G = X + i Y with X, Y Hermitian; 8 n^3 for an inversion of its own), the reductions over it,
    and the mesh, tables and results once."""
    c = case
    D = _chi_dim(c)
    if c["path"] == "dyson":
        return {"bytes": 16.0 * 3 * D * D, "flops": 8.0 * (2.0 + 1.0 / 3.0) * D ** 3}
    n_at = sites(c["shape"])
    n = 2 * N_ORB * n_at
    ns = 2 * N_D * n_at if c["d_only"] else n
    nk = _nk_folded(c)
    if c["adaptive"]:
        lo, hi = c["adaptive"] ** 2, nk
        n_imag = c["n_e"] * (hi - lo) / math.log(hi / lo)
    else:
        n_imag = nk * c["n_e"]
    pts_real = nk * c["n_real"]
    mesh = 40.0 * n_imag + 32.0 * nk
    g = 4.0 * ns * ns * n
    if c["path"] in ("chi0", "rpa", "qbatch"):
        n_dyn = c["n_omega"] - (1 if c["n_omega"] > 1 else 0) if c["n_real"] else 0
        units = c["n_q"] * (c["n_omega"] * n_imag + n_dyn * pts_real)
        g_imag = 2.0 * g if c["adaptive"] else g
        flops = 8.0 * D * D * units + g_imag * n_imag * (1 + c["n_q"] * c["n_omega"]) + \
            g * pts_real * n_dyn * (1 + c["n_q"])
        out = 16.0 * D * D * c["n_omega"] * c["n_q"]
        if c["path"] == "rpa":
            flops += c["n_omega"] * 8.0 * (2.0 + 1.0 / 3.0) * D ** 3
            out *= 3.0
        return {"bytes": mesh + out, "flops": flops}
    if c["path"] == "scf":
        return {"bytes": mesh + 16.0 * n * n, "flops": (g + 32.0 * n * n) * n_imag}
    if c["path"] == "she":
        vertex = 8.0 * (2 * n * (n // 2) ** 2 + 4 * D * (n // 2))
        return {"bytes": mesh + 64.0 * D, "flops": 2.0 * g * (n_imag + pts_real) + vertex * (2 * n_imag + pts_real)}
    if c["path"] == "ldos":
        return {"bytes": 32.0 * nk + 16.0 * n * c["n_e"], "flops": nk * (2.0 * n * n * c["n_e"] + 40.0 * n ** 3)}
    return {"bytes": mesh, "flops": (2.0 * g + 2.0 * 128.0 * (N_D * n_at) ** 2) * n_imag}


# --------------------------------------------------------------------------- plain 64-bit result
class _Plain:
    """H(k) and its resolvents from the tables of a system, with torch in 64 bits."""

    def __init__(self, system, h0):
        dev = torch.device("cuda")
        self.dev = dev
        cv, bi, ish, t = system.neighbor_table()
        self.nat, self.norb = system.n_atoms, N_ORB
        self.n = 2 * N_ORB * self.nat
        self.R = torch.tensor(cv, dtype=torch.float64, device=dev)
        self.h0 = torch.tensor(np.ascontiguousarray(h0), dtype=torch.complex128, device=dev)
        n, m = self.n, N_ORB
        T = np.zeros((cv.shape[0], n, n), complex)
        S = np.zeros((cv.shape[0], self.nat * m, self.nat * m), complex)   # without spin
        for k in range(cv.shape[0]):
            j = int(bi[k])
            for i in range(self.nat):
                if ish[k, i]:
                    blk = t[k, i]
                    S[k, j * m:(j + 1) * m, i * m:(i + 1) * m] += blk
                    for sp in range(2):
                        r, cc = 2 * m * j + sp * m, 2 * m * i + sp * m
                        T[k, r:r + m, cc:cc + m] += blk
        self.T = torch.tensor(T, device=dev).reshape(cv.shape[0], n * n)
        self.S = torch.tensor(S, device=dev).reshape(cv.shape[0], -1)

    def t(self, x, dtype=torch.float64):
        return torch.as_tensor(np.ascontiguousarray(x), dtype=dtype, device=self.dev)

    def phase(self, kp):
        a = kp @ self.R.T
        return torch.complex(torch.cos(a), torch.sin(a))

    def hk(self, kp):
        return self.h0 + (self.phase(kp) @ self.T).reshape(-1, self.n, self.n)

    def dtdk(self, kp, ue):
        f = 1j * (self.R @ self.t(ue))
        m = self.nat * self.norb
        return ((self.phase(kp) * f) @ self.S).reshape(-1, m, m)

    def green(self, z, kp):
        eye = torch.eye(self.n, dtype=torch.complex128, device=self.dev)
        return torch.linalg.inv(z[:, None, None] * eye - self.hk(kp))

    def site(self, G, i, j):
        """[p, spin, orb, spin, orb] block of sites (i, j)."""
        w = 2 * self.norb
        return G[:, i * w:(i + 1) * w, j * w:(j + 1) * w].reshape(-1, 2, self.norb, 2, self.norb)


def _blocks(n, total):
    step = max(256, int(4.0e7 / (n * n)))
    return [(a, min(total, a + step)) for a in range(0, total, step)]


def _exact_chi(st, q, w):
    """chi0 of wave vector q and frequency number w."""
    c, s, deck = st["case"], st["system"], st["deck"]
    P = _Plain(s, st["h0"])
    e = st["es"][w]
    orb = list(range(N_ORB - N_D, N_ORB)) if c["d_only"] else list(range(N_ORB))
    no, nat = len(orb), s.n_atoms
    rows = torch.tensor([i * 2 * N_ORB + sp * N_ORB + o for i in range(nat) for sp in range(2) for o in orb],
                        device=P.dev)
    m = 4 * no * no
    C = torch.zeros(nat, nat, m, m, dtype=torch.complex128, device=P.dev)
    D = torch.zeros_like(C)
    qv = P.t(q)
    sgn = P.n

    def add(acc, A, B):
        a = A.reshape(-1, nat, 2 * no, nat, 2 * no)
        b = B.reshape(-1, nat, 2 * no, nat, 2 * no)
        for i in range(nat):
            for j in range(nat):
                acc[i, j] += a[:, i, :, j].reshape(-1, m).T @ b[:, i, :, j].reshape(-1, m)

    y, kp, wt = P.t(deck.ek.point_energy()), P.t(deck.ek.kp), P.t(deck.ek.weight)
    for a, b in _blocks(sgn, kp.shape[0]):
        G2 = P.green(torch.complex(torch.full_like(y[a:b], s.Ef), y[a:b] + s.etap), kp[a:b])
        G1 = P.green(torch.complex(torch.full_like(y[a:b], s.Ef + e), y[a:b] + s.eta), kp[a:b] + qv)
        G1, G2 = G1[:, rows][:, :, rows], G2[:, rows][:, :, rows]
        add(C, wt[a:b, None, None] * G1, G2.transpose(1, 2))
    if abs(e) >= 1e-15:
        rk, rw = P.t(deck.real_kp), P.t(deck.real_w)
        nk = rk.shape[0]
        x2, p2 = P.t(st["x2"][w]), P.t(st["p2"][w])
        for a, b in _blocks(sgn, nk * x2.shape[0]):
            ix = torch.arange(a, b, device=P.dev)
            x, wr, k = x2[ix // nk], p2[ix // nk] * rw[ix % nk], rk[ix % nk]
            G2 = P.green(torch.complex(x, torch.full_like(x, s.etap)), k)[:, rows][:, :, rows]
            G1 = P.green(torch.complex(x + e, torch.full_like(x, s.eta)), k + qv)[:, rows][:, :, rows]
            add(D, wr[:, None, None] * (G1 - G1.conj().transpose(1, 2)), G2.conj())
    # spins (a, b) of the four spin pairs
    sa, sb = [1, 0, 1, 0], [0, 0, 1, 1]
    out = torch.zeros(nat, no, no, 4, nat, no, no, 4, dtype=torch.complex128, device=P.dev)
    for i in range(nat):
        for j in range(nat):
            Cij = C[i, j].reshape(2, no, 2, no, 2, no, 2, no)     # a1 nu a2 ga b1 mu b2 xi
            Cji = C[j, i].reshape(2, no, 2, no, 2, no, 2, no)     # a2 ga a1 nu b2 xi b1 mu
            Dij = D[i, j].reshape(2, no, 2, no, 2, no, 2, no)
            for s1 in range(4):
                for s2 in range(4):
                    a1, b1, a2, b2 = sa[s1], sb[s1], sa[s2], sb[s2]
                    f = Cij[a1, :, a2, :, b1, :, b2, :] - 1j * Dij[a1, :, a2, :, b1, :, b2, :]   # nu ga mu xi
                    g = Cji[a2, :, a1, :, b2, :, b1, :].conj()                                   # ga nu xi mu
                    out[i, :, :, s1, j, :, :, s2] = f.permute(2, 0, 1, 3) + g.permute(3, 1, 0, 2)
    dim = nat * no * no * 4
    return (out.reshape(dim, dim) / (2.0 * math.pi)).cpu().numpy()


def _exact_dyson(chi, U):
    x = torch.as_tensor(np.ascontiguousarray(chi), device="cuda")
    u = torch.as_tensor(np.ascontiguousarray(U), device="cuda")
    eye = torch.eye(x.shape[0], dtype=torch.complex128, device="cuda")
    return torch.linalg.solve(eye + x @ u, x).cpu().numpy()


_PAULI = np.array([[[1, 0], [0, 1]], [[0, 1], [1, 0]], [[0, -1j], [1j, 0]], [[1, 0], [0, -1]]], complex)


def _exact_scf(st):
    s, deck = st["system"], st["deck"]
    P = _Plain(s, st["h0"])
    nat, w2 = s.n_atoms, 2 * N_ORB
    y, kp, wt = P.t(deck.ek.point_energy()), P.t(deck.ek.kp), P.t(deck.ek.weight)
    d = list(range(N_ORB - N_D, N_ORB))
    # vertices of the unknowns of a site: d occupations, then the three moments (U = 1)
    verts = []
    pd = np.zeros((N_ORB, N_ORB))
    pd[d, d] = 1.0
    for mu in d:
        one = np.zeros((N_ORB, N_ORB))
        one[mu, mu] = 1.0
        verts.append(-0.5 * np.kron(_PAULI[0], pd - 2.0 * one))
    for a in (1, 2, 3):
        verts.append(-0.5 * np.kron(_PAULI[a], pd))
    nv = len(verts)
    V = P.t(np.array(verts), torch.complex128)
    # observables of a site as matrices under the trace: d occupations, d moments, total charge
    obs = []
    for mu in d:
        one = np.zeros((N_ORB, N_ORB))
        one[mu, mu] = 1.0
        obs.append(np.kron(_PAULI[0], one))
    for a in (1, 2, 3):
        obs.append(np.kron(_PAULI[a], pd))
    obs.append(np.eye(w2))
    O = P.t(np.array(obs), torch.complex128)
    acc = torch.zeros(P.n, P.n, dtype=torch.complex128, device=P.dev)
    K = torch.zeros(nat, nv, nat, w2, w2, dtype=torch.complex128, device=P.dev)   # (G V_b G)_ii
    for a, b in _blocks(2 * P.n, kp.shape[0]):
        G = P.green(torch.complex(torch.full_like(y[a:b], s.Ef), y[a:b] + s.eta), kp[a:b])
        w = wt[a:b, None, None].to(torch.complex128)
        acc += (w * G).sum(0)
        for j in range(nat):
            left = w * G[:, :, j * w2:(j + 1) * w2]
            right = G[:, j * w2:(j + 1) * w2, :]
            for v in range(nv):
                LV = left @ V[v]
                for i in range(nat):
                    r = slice(i * w2, (i + 1) * w2)
                    K[j, v, i] += torch.einsum("prk,pkc->rc", LV[:, r], right[:, :, r])
    neq = nat * nv + 1
    if jacobian_layout(s)[0] != neq:
        return None
    J = np.zeros((neq, neq))
    tr = torch.einsum("oab,jviba->iojv", O, K).real.cpu().numpy()
    for i in range(nat):
        J[i * nv:(i + 1) * nv, :neq - 1] = tr[i, :nv].reshape(nv, -1)
    J[neq - 1, :neq - 1] = tr[:, nv].sum(0).reshape(-1)
    F = torch.zeros(P.n, P.n, dtype=torch.complex128, device=P.dev)
    rk, rw = P.t(deck.real_kp), P.t(deck.real_w)
    for a, b in _blocks(P.n, rk.shape[0]):
        z = torch.full((b - a,), complex(s.Ef, s.eta), dtype=torch.complex128, device=P.dev)
        F += (rw[a:b, None, None] * P.green(z, rk[a:b])).sum(0)
    fi = torch.stack([F[i * w2:(i + 1) * w2, i * w2:(i + 1) * w2] for i in range(nat)])
    fe = torch.einsum("oab,iba->io", O, fi).imag.cpu().numpy()
    for i in range(nat):
        J[i * nv:(i + 1) * nv, neq - 1] = -fe[i, :nv]
    J[neq - 1, neq - 1] = -fe[:, nv].sum()
    J /= math.pi
    J[np.arange(neq - 1), np.arange(neq - 1)] -= 1.0
    A = acc.cpu().numpy()
    rho, mz = np.zeros((nat, N_ORB)), np.zeros((nat, N_ORB))
    mp = np.zeros((nat, N_ORB), complex)
    for i in range(nat):
        u = np.arange(i * w2, i * w2 + N_ORB)
        dn = u + N_ORB
        nu, nd = 0.5 + A[u, u].real / math.pi, 0.5 + A[dn, dn].real / math.pi
        rho[i], mz[i] = nu + nd, nu - nd
        ud, du = A[u, dn], A[dn, u]
        mp[i] = (du.real + ud.real) / math.pi + 1j * (du.imag - ud.imag) / math.pi
    return {"rho": rho, "mx": mp.real.copy(), "my": mp.imag.copy(), "mz": mz, "mp": mp, "jacobian": J}


# spin blocks (row, column; 0 = up, 1 = down) of the response's two factors: entry (s, s') takes
# G1 rows of spin a(s) and columns of spin a'(s'), G2 rows of spin b'(s') and columns of spin b(s)
def _exact_she(st):
    s, deck = st["system"], st["deck"]
    P = _Plain(s, st["h0"])
    nat, m = s.n_atoms, N_ORB
    up = torch.tensor([i * 2 * m + o for i in range(nat) for o in range(m)], device=P.dev)
    spin = (up, up + m)
    e, qv = st["es"][0], P.t(st["qs"][0])
    sa, sb = [1, 0, 1, 0], [0, 0, 1, 1]
    df = torch.zeros(nat, m, m, 4, 4, dtype=torch.complex128, device=P.dev)   # site mu nu s s'

    def blk(G, a, b):
        return G[:, spin[a]][:, :, spin[b]]

    def put(t, w, s1, s2, rows_nu):
        t = (w[:, None, None] * t).sum(0).reshape(nat, m, nat, m)
        for i in range(nat):
            x = t[i, :, i]
            df[i, :, :, s1, s2] += x.T if rows_nu else x

    y, kp, wt = P.t(deck.ek.point_energy()), P.t(deck.ek.kp), P.t(deck.ek.weight)
    for a, b in _blocks(P.n, kp.shape[0]):
        G1 = P.green(torch.complex(torch.full_like(y[a:b], s.Ef + e), y[a:b] + s.eta), kp[a:b] + qv)
        G2 = P.green(torch.complex(torch.full_like(y[a:b], s.Ef), y[a:b] + s.etap), kp[a:b])
        Dk = P.dtdk(kp[a:b], st["efield"])
        DT = Dk.transpose(1, 2)
        for s1 in range(4):
            for s2 in range(4):
                put(blk(G1, sa[s1], sa[s2]) @ Dk @ blk(G2, sb[s2], sb[s1]), wt[a:b], s1, s2, True)
                put(blk(G2, sb[s1], sb[s2]).conj() @ DT @ blk(G1, sa[s2], sa[s1]).conj(), wt[a:b], s1, s2, False)
    rk, rw = P.t(deck.real_kp), P.t(deck.real_w)
    nk = rk.shape[0]
    x2, p2 = P.t(st["x2"][0]), P.t(st["p2"][0])
    for a, b in _blocks(P.n, nk * x2.shape[0]):
        ix = torch.arange(a, b, device=P.dev)
        x, wr, k = x2[ix // nk], p2[ix // nk] * rw[ix % nk], rk[ix % nk]
        G1 = P.green(torch.complex(x + e, torch.full_like(x, s.eta)), k + qv)
        G2 = P.green(torch.complex(x, torch.full_like(x, s.etap)), k)
        A = G1 - G1.conj().transpose(1, 2)
        Dk = P.dtdk(k, st["efield"])
        for s1 in range(4):
            for s2 in range(4):
                t = blk(A, sa[s1], sa[s2]) @ Dk @ blk(G2, sb[s1], sb[s2]).conj().transpose(1, 2)
                put(-1j * t, wr, s1, s2, True)
    return {"tchi": (df.reshape(-1, 4) / (2.0 * math.pi)).cpu().numpy()}


def _exact_ldos(st):
    s, deck = st["system"], st["deck"]
    P = _Plain(s, st["h0"])
    rk, rw = P.t(deck.real_kp), P.t(deck.real_w)
    grid = P.t(st["grid"])
    out = torch.zeros(grid.shape[0], P.n, dtype=torch.float64, device=P.dev)
    for a, b in _blocks(P.n, rk.shape[0]):
        lam, U = torch.linalg.eigh(P.hk(rk[a:b]))
        W = (U.real ** 2 + U.imag ** 2) * rw[a:b, None, None]                  # k r a
        for k in range(b - a):
            L = (s.eta / math.pi) / ((grid[:, None] - lam[k][None, :]) ** 2 + s.eta ** 2)
            out += L @ W[k].T
    r = out.reshape(-1, s.n_atoms, 2, N_ORB).cpu().numpy()
    return {"up": np.ascontiguousarray(r[:, :, 0]), "dn": np.ascontiguousarray(r[:, :, 1])}


def _exact_jij(st):
    s, deck = st["system"], st["deck"]
    P = _Plain(s, st["h0"])
    nat, w2 = s.n_atoms, 2 * N_ORB
    d = list(range(N_ORB - N_D, N_ORB))
    pd = np.zeros((N_ORB, N_ORB))
    pd[d, d] = 1.0
    A = np.zeros((nat, 3, w2, w2), complex)
    for i in range(nat):
        ev = st["evec"][i]
        for mu in range(3):
            for x in range(3):
                A[i, mu] += -0.5 * st["Um"][i] * ((mu == x) - ev[mu] * ev[x]) * np.kron(_PAULI[x + 1], pd)
    A = P.t(A, torch.complex128)
    J = torch.zeros(nat, nat, 3, 3, dtype=torch.complex128, device=P.dev)
    y, kp, wt = P.t(deck.ek.point_energy()), P.t(deck.ek.kp), P.t(deck.ek.weight)
    qv = P.t(st["qs"][0])
    for a, b in _blocks(2 * P.n, kp.shape[0]):
        z = torch.complex(torch.full_like(y[a:b], s.Ef), y[a:b] + s.eta)
        G, Gq = P.green(z, kp[a:b]), P.green(z, kp[a:b] - qv)
        w = wt[a:b, None, None]
        for i in range(nat):
            for j in range(nat):
                ri, rj = slice(i * w2, (i + 1) * w2), slice(j * w2, (j + 1) * w2)
                for mu in range(3):
                    for nu in range(3):
                        t1 = torch.einsum("pab,pba->", w * (A[i, mu] @ G[:, ri, rj]), A[j, nu] @ Gq[:, rj, ri])
                        t2 = torch.einsum("pab,pba->", w * (A[i, mu] @ Gq[:, ri, rj]), A[j, nu] @ G[:, rj, ri])
                        J[i, j, mu, nu] += t1 + t2.conj()
    return {"J": (-J / (2.0 * math.pi)).cpu().numpy()}


def exact(case, seed):
    """What ``run`` returns for these inputs, with torch in 64 bits."""
    st = prepare(case, seed)
    path = case["path"]
    if path == "dyson":
        return {"chi": _exact_dyson(st["chi"], st["U"])}
    st.pop("gpu").close()
    if path in ("chi0", "rpa"):
        chi = np.array([_exact_chi(st, st["qs"][0], w) for w in range(case["n_omega"])])
        if path == "chi0":
            return {"chi0": chi}
        return {"chi0": chi, "chi": [_exact_dyson(x, st["U"]) for x in chi]}
    if path == "qbatch":
        return {"chi0": np.array([[_exact_chi(st, q, w) for w in range(case["n_omega"])] for q in st["qs"]])}
    return {"scf": _exact_scf, "she": _exact_she, "ldos": _exact_ldos, "jij": _exact_jij}[path](st)

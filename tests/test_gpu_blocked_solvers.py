"""Blocked FP64 tensor-core solvers at the sizes where their tiling can go wrong (needs a B200):
the Gauss-Jordan inversion (panels of 4 columns, blocks of 8), the pair sums over its Green
functions, the Dyson LU (panels of 8, blocks of 64), the disturbance vertex, the tridiagonal
resolvents and the eigensolver."""
import numpy as np
import pytest

from oracle import titan_oracle as O
from titan_b200.host import synthetic
from titan_b200.host.system import initial_state

from gg_numpy import fermi_column_numpy, gg_tensor_numpy

pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps


@pytest.fixture(scope="module")
def gpu():
    from titan_b200.native import GreenGPU
    g = GreenGPU(0)
    yield g
    g.close()


@pytest.mark.parametrize("shape,scale", [("bcc1", 0.0), ("sq2", 0.0), ("slab3", 1.0), ("slab3", 0.0), ("bcc4", 0.0),
                                         ("slab5", 0.0)])
def test_inversion_needs_its_pivots(gpu, shape, scale):
    """z - H with H = scale * model + a permutation-like Hermitian matrix: every diagonal entry
    is tiny, so elimination without row exchanges loses all digits.  Each entry within 1e-12 n
    of the largest one of LAPACK's inverse (the bound of the plain inversion test)."""
    deck = synthetic.make_deck(shape, mesh=False)
    s = deck.system
    n = s.dimH
    rng = np.random.default_rng(7)
    gpu.set_system(s)
    p = rng.permutation(n)
    h0 = np.zeros((n, n), complex)
    for a, b in zip(p[0::2], p[1::2]):
        t = np.exp(2j * np.pi * rng.uniform()) * rng.uniform(0.5, 2.0)
        h0[a, b], h0[b, a] = t, np.conj(t)
    gpu.set_h0(h0)
    kp = rng.uniform(-2, 2, size=(5, 3))
    Hk = gpu.hamiltk_batch(kp)
    if scale == 0.0:   # remove the hoppings: h0 - H_nl(k) at each k in turn
        zs, out, ref = [], [], []
        for k in range(5):
            gpu.set_h0(2.0 * h0 - Hk[k])
            z = np.array([1e-9j + 1e-7 * k])
            out.append(gpu.green_batch(z, kp[k:k + 1])[0])
            ref.append(np.linalg.inv(z[0] * np.eye(n) - h0))
    else:
        z = 1e-3j + 0.01 * np.arange(5)
        out = gpu.green_batch(z, kp)
        ref = [np.linalg.inv(z[k] * np.eye(n) - Hk[k]) for k in range(5)]
    for a, b in zip(out, ref):
        assert np.max(np.abs(a - b)) <= 1e-12 * n * np.max(np.abs(b))


@pytest.mark.parametrize("shape,nk", [("slab3", (2, 2, 1)), ("bcc4", (2, 2, 2)), ("slab5", (2, 3, 1))])
def test_pair_sums_of_larger_cells(gpu, shape, nk):
    """GG tensor (orbital-resolved and summed), Fermi column and J_ij against numpy: products of
    two Green functions, each within 1e-12 n of its largest entry."""
    deck = synthetic.make_deck(shape, nk=nk, n1gl=5, parts=1, n3gl=4)
    s = deck.system
    h0 = s.h0(initial_state(s))
    gpu.setup(deck, h0)
    m = O.Model(s, h0)
    ek = deck.ek
    tol = 2e-12 * s.dimH
    G = m.green(s.Ef + 1j * (ek.point_energy() + s.eta), ek.kp)
    for resolved in (True, False):
        T = gpu.gg_tensor(s.Ef, s.eta, resolved)
        Tr = gg_tensor_numpy(s, G, ek.weight, resolved)
        assert np.max(np.abs(T - Tr)) <= tol * np.max(np.abs(Tr))
    Gr = m.green(np.full(deck.real_kp.shape[0], s.Ef + 1j * s.eta), deck.real_kp)
    D, Dr = gpu.fermi_column(s.Ef, s.eta), fermi_column_numpy(s, Gr, deck.real_w)
    assert np.max(np.abs(D - Dr)) <= tol * np.max(np.abs(Dr))
    ev = np.random.default_rng(2).standard_normal((s.n_atoms, 3))
    ev /= np.linalg.norm(ev, axis=1)[:, None]
    q = np.array([0.1, -0.05, 0.0])
    J, Jr = gpu.jij(q, s.Ef, s.eta, ev, s.Um()), O.jij(m, ek, q, s.Ef, s.eta, ev, s.Um(), s.dorbs)
    assert np.max(np.abs(J - Jr)) <= tol * np.max(np.abs(Jr))


@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 63, 64, 65, 72, 129])
@pytest.mark.parametrize("order", ["C", "F"])
def test_dyson_at_the_edges_of_its_panels(gpu, n, order):
    """Random chi and U: 1 + chi U has no dominant diagonal, so rows are exchanged in every
    panel.  Two backward-stable solves differ by at most ~ n eps cond."""
    rng = np.random.default_rng(n)
    x, u = (np.asarray(rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)), order=order) for _ in range(2))
    got = gpu.dyson(x, u)
    M = np.eye(n) + x @ u
    ref = np.linalg.solve(M, x)
    assert np.linalg.norm(got - ref) <= 10.0 * n * EPS * np.linalg.cond(M) * np.linalg.norm(ref)


@pytest.mark.parametrize("n", [1024, 1025, 1300, 1620])
def test_dyson_exchanges_rows_in_every_panel_kernel(gpu, n):
    """Random chi and U where panels have up to 1024 rows (a row per thread in registers), up to 1607
    (shared memory) and more (global memory), with the switches between them inside one solve: the
    backward error of the solution and its distance from LAPACK's, each within 10 n eps (times the
    condition)."""
    rng = np.random.default_rng(n)
    x, u = (rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)) for _ in range(2))
    got = gpu.dyson(x, u)
    M = np.eye(n) + x @ u
    assert np.linalg.norm(M @ got - x) <= 10.0 * n * EPS * np.linalg.norm(M) * np.linalg.norm(got)
    ref = np.linalg.solve(M, x)
    assert np.linalg.norm(got - ref) <= 10.0 * n * EPS * np.linalg.cond(M, 1) * np.linalg.norm(ref)


@pytest.mark.parametrize("n", [70, 1300, 1700])   # column 67 in a panel of each of the three kernels
def test_dyson_reports_a_singular_system(gpu, n):
    from titan_b200.native import TitanGPUError
    x = np.eye(n, dtype=complex)
    u = -np.eye(n, dtype=complex)
    with pytest.raises(TitanGPUError) as err:
        gpu.dyson(x, 0.5 * u - 0.5 * np.diag(np.arange(n) == 66))
    assert err.value.code == 67


@pytest.mark.parametrize("shape,nk", [("bcc1", (2, 3, 2)), ("sq2", (3, 2, 1)), ("slab3", (2, 2, 1))])
def test_disturbance_fragments(gpu, shape, nk):
    """The vertex products in 8 x 8 fragments: one site (25 fragments for eight warps, a last column
    block of two orbitals), two sites (50), and three (75, more than the warps hold: the staged
    kernel).  Both axes, one after the other into the same sums, q and frequency nonzero; within
    1e-10 of the oracle, the bound of the plain test."""
    deck = synthetic.make_deck(shape, nk=nk, n1gl=5, parts=1, n3gl=3)
    s = deck.system
    h0 = s.h0(initial_state(s))
    gpu.setup(deck, h0)
    e, q, ue = 0.04, np.array([0.1, 0.05, 0.0]), np.array([0.6, 0.0, 0.8])
    x2, p2 = deck.real_points(e, s.Ef)
    ref = O.eintshe(O.Model(s, h0), deck.ek, (deck.real_kp, deck.real_w), q, e, s.Ef, s.eta, s.etap, x2, p2, ue)
    got = gpu.she(q, e, s.Ef, s.eta, s.etap, x2, p2, ue)
    assert np.max(np.abs(got - ref)) <= 1e-10 * np.max(np.abs(ref)), shape


# 60 of 108 rows (tiles of 64 x 64), all 126 rows (128 x 64; no multiple of the reduction's panels
# of 8), 50 of 90 rows (64 x 64, reduction in shared memory), all 90 rows (96 x 96)
@pytest.mark.parametrize("shape,d_only", [("slab6", True), ("slab7", False), ("slab5", True), ("slab5", False)])
def test_tridiagonal_tiles_equal_gauss_jordan(gpu, shape, d_only):
    """chi0 from tridiagonalised Green functions at the tile shapes of their products equals the
    Gauss-Jordan path to 1e-12, the bound of the plain test (which has the 160 x 80 tiles)."""
    deck = synthetic.make_deck(shape, nk=(2, 2, 1), n1gl=3, parts=1, n3gl=3)
    s = deck.system
    gpu.setup(deck, s.h0(initial_state(s)))
    gpu.set_chi_orbitals([list(d) for d in s.dorbs] if d_only else None)
    e, q = 0.05, np.array([0.1, 0.0, 0.0])
    x2, p2 = deck.real_points(e, s.Ef)
    try:
        auto = gpu.chi0(q, e, s.Ef, s.eta, s.etap, x2, p2, precision="fp64")
        gpu.set_green_method("gauss-jordan")
        gj = gpu.chi0(q, e, s.Ef, s.eta, s.etap, x2, p2, precision="fp64")
    finally:
        gpu.set_green_method("auto")
        gpu.set_chi_orbitals(None)
    assert np.linalg.norm(auto - gj) < 1e-12 * np.linalg.norm(gj)


@pytest.mark.parametrize("shape", ["bcc1", "sq2", "slab3", "bcc4", "slab5"])
@pytest.mark.parametrize("kind", ["model", "two_levels", "diagonal"])
def test_eigensolver_edges(gpu, shape, kind):
    """Eigenpairs at the dimensions of the solver's variants, also of matrices that are diagonal
    already or have two eigenvalues only: residual, orthogonality and eigenvalues within
    10 n eps (times |H|), the backward error of a reduction of n reflectors."""
    deck = synthetic.make_deck(shape, mesh=False)
    s = deck.system
    n = s.dimH
    h0 = s.h0(initial_state(s))
    kp = np.random.default_rng(3).uniform(-2, 2, (1 if kind != "model" else 37, 3))
    gpu.set_system(s)
    gpu.set_h0(h0)
    if kind != "model":   # h0 such that H(k) is the wanted matrix up to roundoff
        want = np.diag(np.arange(n) - 0.5 * n) if kind == "diagonal" else np.kron(np.diag([1.0, -1.0]), np.eye(n // 2))
        gpu.set_h0(want.astype(complex) - (gpu.hamiltk_batch(kp)[0] - h0))
    H = gpu.hamiltk_batch(kp)
    lam, U = gpu.eig_batch(kp)
    tol = 10 * n * EPS
    for k in range(len(kp)):
        h = np.linalg.norm(H[k], 2)
        assert np.max(np.abs(U[k].conj().T @ U[k] - np.eye(n))) <= tol
        assert np.max(np.abs((U[k] * lam[k]) @ U[k].conj().T - H[k])) <= tol * h
        assert np.max(np.abs(np.sort(lam[k]) - np.linalg.eigvalsh(H[k]))) <= tol * h


@pytest.mark.parametrize("shape,d_only,counts", [("bcc1", False, (9, 19, 29)), ("slab6", True, (9, 21, 31))])
def test_launches_are_counted(gpu, shape, d_only, counts):
    """tg_last_timing's number of kernels of chi0 (static; at finite q and frequency, FP64 and split):
    two per H(k) table; four per eigendecomposition, then one launch per Green function (or pair of
    operands), or one per tridiagonalisation, then two launches and a gather per operand; the
    contraction one per axis, in split precision two more per operand and one per axis; the epilogue."""
    deck = synthetic.make_deck(shape, nk=(3, 3, 3) if shape == "bcc1" else (3, 3, 1), n1gl=4, parts=1, n3gl=3)
    s = deck.system
    gpu.setup(deck, s.h0(initial_state(s)))
    gpu.set_chi_orbitals([list(d) for d in s.dorbs] if d_only else None)
    x2, p2 = deck.real_points(0.05, s.Ef)
    q = np.array([0.1, 0.0, 0.0])
    got = []
    try:
        gpu.chi0(0.0 * q, 0.0, s.Ef, s.eta, s.etap)
        got.append(int(gpu.last_timing()[10]))
        for precision in ("fp64", "split"):
            gpu.chi0(q, 0.05, s.Ef, s.eta, s.etap, x2, p2, precision)
            got.append(int(gpu.last_timing()[10]))
    finally:
        gpu.set_chi_orbitals(None)
    assert tuple(got) == counts


class MixedSites:
    """A chain of sites of `norbs` orbitals with random Hermitian hoppings to two cells: what the
    binding and the oracle read of a system."""

    def __init__(self, norbs, rng):
        self.norbs, self.n_atoms = list(norbs), len(norbs)
        self.dimH, self.dimens = 2 * sum(norbs), 4 * sum(n * n for n in norbs)
        nat, nm = self.n_atoms, max(norbs)
        cells, basis, t = [], [], []
        for R in (np.array([1.0, 0.2, 0.0]), np.array([0.1, 1.1, 0.0])):
            b = {(j, i): 0.3 * (rng.standard_normal((norbs[j], norbs[i])) + 1j * rng.standard_normal((norbs[j], norbs[i])))
                 for j in range(nat) for i in range(nat)}
            for sign in (1, -1):
                for j in range(nat):
                    blk = np.zeros((nat, nm, nm), complex)
                    for i in range(nat):
                        blk[i, :norbs[j], :norbs[i]] = b[j, i] if sign > 0 else b[i, j].conj().T
                    cells.append(sign * R)
                    basis.append(j)
                    t.append(blk)
        self.table = (np.array(cells), np.array(basis, np.int32), np.ones((len(t), nat), np.int32), np.array(t))

    def neighbor_table(self):
        return self.table

    def ia(self):
        from titan_b200.host import onsite
        return onsite.site_offsets(self.norbs)

    def sigmaimunu2i(self):
        from titan_b200.host.system import TBSystem
        return TBSystem.sigmaimunu2i(self)


@pytest.mark.parametrize("norbs", [(4, 5), (2, 3, 4), (9, 4, 5), (1, 8, 9), (9, 9, 2), (9, 5, 9, 4), (5, 9, 9, 9, 4),
                                   (10, 9, 8, 9, 9), (13, 9, 9, 9, 8)])
def test_sites_of_different_orbital_counts(gpu, norbs):
    """chi0 (spectral, tridiagonalised from 90 on, and Gauss-Jordan) and, up to 90, the disturbance
    integral on both axes where no site starts or ends at a fragment's or a tile's edge: dimensions
    18 to 96 with a kernel of their own, within 1e-10 of the oracle, the bound of the plain tests."""
    from titan_b200.host.mesh import EKMesh
    rng = np.random.default_rng(sum(norbs) * 31 + len(norbs))
    s = MixedSites(norbs, rng)
    h = rng.standard_normal((s.dimH, s.dimH)) + 1j * rng.standard_normal((s.dimH, s.dimH))
    h = 0.5 * (h + h.conj().T)
    nk, y, wy = 5, np.array([0.01, 0.2, 3.0]), rng.uniform(0.2, 1.0, 3)
    k = rng.uniform(-2, 2, (nk, 3))
    ek = EKMesh(y, wy, np.repeat(np.arange(3), nk), np.tile(k, (3, 1)), np.repeat(wy, nk) / nk)
    Ef, eta, etap, e, q, ue = 0.1, 2e-3, 1e-3, 0.07, np.array([0.2, 0.1, 0.0]), np.array([0.6, 0.3, 0.0])
    x2, p2 = np.linspace(Ef - e, Ef, 3), np.full(3, 0.02)
    gpu.set_system(s)
    gpu.set_h0(h)
    gpu.set_imag_mesh(ek)
    gpu.set_real_mesh(k, np.full(nk, 1.0 / nk))
    m, bz = O.Model(s, h), (k, np.full(nk, 1.0 / nk))
    ref = O.eintshechi(m, ek, bz, q, e, Ef, eta, etap, x2, p2)
    single = s.dimH in (18, 36, 40, 54, 72, 90)   # (the cluster kernel has no disturbance integral)
    try:
        for method in ("auto", "gauss-jordan"):
            gpu.set_green_method(method)
            got = gpu.chi0(q, e, Ef, eta, etap, x2, p2)
            assert np.linalg.norm(got - ref) <= 1e-10 * np.linalg.norm(ref), method
            if single:
                she = gpu.she(q, e, Ef, eta, etap, x2, p2, ue)
                sref = O.eintshe(m, ek, bz, q, e, Ef, eta, etap, x2, p2, ue)
                assert np.max(np.abs(she - sref)) <= 1e-10 * np.max(np.abs(sref)), method
    finally:
        gpu.set_green_method("auto")

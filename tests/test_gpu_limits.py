"""Calls where device memory is short, from several threads, and on Hamiltonians with entries whose
squares underflow (needs a B200)."""
import threading
import time

import numpy as np
import pytest

from titan_b200.host import synthetic
from titan_b200.host.system import initial_state

pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps
MIB = 1 << 20


def context(deck, h0):
    from titan_b200.native import GreenGPU
    g = GreenGPU(0)
    g.setup(deck, h0)
    return g


class filled_device:
    """Leaves `free` bytes of the device's memory to the calls inside."""

    def __init__(self, free):
        self.free = free

    def __enter__(self):
        import torch
        torch.cuda.empty_cache()
        left = torch.cuda.mem_get_info(0)[0]
        assert left > self.free
        self.block = torch.empty(left - self.free, dtype=torch.uint8, device="cuda:0")

    def __exit__(self, *exc):
        import torch
        del self.block
        torch.cuda.empty_cache()


def test_a_call_after_one_that_ran_out_of_memory():
    """The failed call reports TG_ERR_NOMEM; what is called next is not touched by it."""
    from titan_b200.native import GreenGPU, TitanGPUError
    g = GreenGPU(0)
    rng = np.random.default_rng(2)
    x = rng.standard_normal((8, 8)) + 1j * rng.standard_normal((8, 8))
    want = np.linalg.solve(np.eye(8) + x @ x, x)
    g.dyson(x, x)   # (loads the kernels)
    with filled_device(64 * MIB):
        with pytest.raises(TitanGPUError) as err:
            g.dyson(np.eye(1600, dtype=complex), np.eye(1600, dtype=complex))
        assert err.value.code == -5
        assert np.allclose(g.dyson(x, x), want, rtol=0, atol=1e-12 * np.abs(want).max())
    g.close()


def calls_of(deck):
    s = deck.system
    ev = np.tile([[0.6, 0.0, 0.8]], (s.n_atoms, 1))
    return {"smunu": lambda g: g.smunu(s.Ef, s.eta), "gs_orbital": lambda g: g.gs_orbital(s.Ef, s.eta),
            "gg_tensor": lambda g: g.gg_tensor(s.Ef, s.eta), "fermi_column": lambda g: g.fermi_column(s.Ef, s.eta),
            "jacobian": lambda g: g.jacobian(s.Ef, s.eta), "adjoint_vb": lambda g: g.adjoint_vb(s.Ef, s.eta),
            "jij": lambda g: g.jij(np.array([0.1, 0.05, 0.0]), s.Ef, s.eta, ev, s.Um())}


@pytest.mark.parametrize("free,names", [(640, ("smunu", "gs_orbital", "gg_tensor", "fermi_column", "jacobian",
                                                "adjoint_vb")), (2600, ("jij",))])
def test_sums_without_room_for_their_tables(free, names):
    """31329 k of two spd sites: an H(k) table is 650 MB and the Green functions of a pass are up to
    1 GiB.  With `free` MiB left the sums form H(k) in the inversion and take shorter passes; they
    differ from the others by the order of the sum only (1e-12)."""
    deck = synthetic.make_deck("sq2", nk=(177, 177, 1), n1gl=2, parts=1, n3gl=2)
    h0 = deck.system.h0(initial_state(deck.system))
    calls = calls_of(deck)
    for name in names:
        g = context(deck, h0)
        want = calls[name](g)   # (also loads the kernels)
        g.close()
        g = context(deck, h0)
        with filled_device(free * MIB):
            got = calls[name](g)
            g.close()
        assert np.max(np.abs(got - want)) <= 1e-12 * np.max(np.abs(want)), name


def test_ldos_without_room_for_every_rotation():
    """The LDOS of 16900 k of two spd sites keeps 700 MB of matrices and eigenvectors; the list of
    their rotations, 1 GiB where there is room, is worked off in shorter parts with 1 GiB left."""
    deck = synthetic.make_deck("sq2", nk=(130, 130, 1), n1gl=2, parts=1, n3gl=2)
    s = deck.system
    h0 = s.h0(initial_state(s))
    es = s.Ef + np.linspace(-1.0, 1.0, 5)
    g = context(deck, h0)
    want = g.ldos(es, s.eta)
    g.close()
    g = context(deck, h0)
    with filled_device(1024 * MIB):
        got = g.ldos(es, s.eta)
        g.close()
    for a, b in zip(got, want):
        assert np.max(np.abs(a - b)) <= 1e-12 * np.max(np.abs(b))


def without_hoppings(shape):
    s = synthetic.make_system(shape)
    cv, bi, ish, t = s.neighbor_table()
    s.neighbor_table = lambda: (cv, bi, ish, 0.0 * t)
    return s


def weakly_coupled(n, tiny, rng):
    """Random Hermitian matrix whose first three rows couple to each other and to the rest by
    imaginary entries of size `tiny` alone."""
    h = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    h = 0.5 * (h + h.conj().T)
    for r in range(3):
        d = h[r, r]
        h[r, :], h[:, r] = 1j * tiny, -1j * tiny
        h[r, r] = d
    for r in range(3):
        h[r, :r], h[:r, r] = -1j * tiny, 1j * tiny
    return h


@pytest.mark.parametrize("tiny", [1e-145, 1e-158, 1e-170])
@pytest.mark.parametrize("shape", ["bcc1", "sq2", "bcc4", "slab5"])
def test_eigenvectors_of_couplings_that_underflow(shape, tiny):
    """A reflector of a column whose squares are denormal or zero is unitary all the same:
    orthogonality and residual within 10 n eps (times |H|)."""
    from titan_b200.native import GreenGPU
    s = without_hoppings(shape)
    h = weakly_coupled(s.dimH, tiny, np.random.default_rng(4))
    g = GreenGPU(0)
    g.set_system(s)
    g.set_h0(h)
    lam, U = g.eig_batch(np.zeros((3, 3)))
    g.close()
    tol = 10 * s.dimH * EPS
    for l, u in zip(lam, U):
        assert np.max(np.abs(u.conj().T @ u - np.eye(s.dimH))) <= tol
        assert np.max(np.abs((u * l) @ u.conj().T - h)) <= tol * np.linalg.norm(h, 2)


@pytest.mark.parametrize("shape", ["slab5", "slab7"])
def test_resolvents_of_couplings_that_underflow(shape):
    """The same for the resolvents from tridiagonalised H(k) (in shared memory, and in panels
    beyond dimension 96): chi0 equals the Gauss-Jordan path to 1e-12."""
    from titan_b200.native import GreenGPU
    deck = synthetic.make_deck(shape, nk=(2, 2, 1), n1gl=3, parts=1, n3gl=3)
    s = without_hoppings(shape)
    g = GreenGPU(0)
    g.set_system(s)
    g.set_h0(weakly_coupled(s.dimH, 1e-158, np.random.default_rng(4)))
    g.set_imag_mesh(deck.ek)
    g.set_chi_orbitals([list(d) for d in s.dorbs])
    q = np.array([0.1, 0.0, 0.0])
    auto = g.chi0(q, 0.0, s.Ef, s.eta, s.etap)
    g.set_green_method("gauss-jordan")
    gj = g.chi0(q, 0.0, s.Ef, s.eta, s.etap)
    g.close()
    assert np.linalg.norm(auto - gj) < 1e-12 * np.linalg.norm(gj)


def test_threads_with_different_shared_memory():
    """Six contexts of one process whose kernels need different amounts of shared memory (dimensions
    36, 54 and 72, one or two shells of neighbours): every call of every thread is carried out."""
    from titan_b200.native import GreenGPU
    errors = []

    def work(shape, n_stages, seconds=3.0):
        try:
            s = synthetic.make_system(shape, n_stages=n_stages)
            g = GreenGPU(0)
            g.set_system(s)
            g.set_h0(s.h0(initial_state(s)))
            kp, z = np.random.default_rng(1).uniform(-2, 2, (4, 3)), s.Ef + 0.1j * np.arange(1, 5)
            end = time.monotonic() + seconds
            while time.monotonic() < end:
                g.eig_batch(kp)
                g.green_batch(z, kp)
            g.close()
        except Exception as ex:
            errors.append(ex)

    threads = [threading.Thread(target=work, args=a) for a in (("sq2", 1), ("bcc4", 2), ("slab3", 1)) * 2]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors

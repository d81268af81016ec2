"""The orbital side of a step by one cluster of blocks (csrc/orbstep.cu) and
the one-warp rho1 synchronisation against the oracle, at the sizes where they
change shape: grids around the 64-point pieces of g_ksql, the 256-point pieces
of the other sums and the points a Gram-Schmidt thread owns (1, 2, 4, 8, 16),
2 to 8 orbitals, every tableau, both boundary conditions, the split step on
both, the robust projector; and densities that need regularisation.

Tolerance: 1e-10 of the largest element, the parity target of whole steps."""
import numpy as np
import pytest

from helpers import rand_coef, rel_err

pytestmark = pytest.mark.gpu

XI, XF = -4.0, 4.0

# N, M, G, periodic, imag, rk, der, split, robust
CASES = [
    (4, 2, 5, True, True, 5, 302, False, False),
    (3, 3, 63, True, True, 2, 302, False, False),
    (3, 3, 64, True, False, 4, 302, False, True),
    (3, 4, 65, False, True, 5, 302, False, False),
    (3, 5, 255, True, False, 5, 302, False, False),
    (2, 6, 257, True, True, 4, 301, False, False),
    (2, 7, 513, False, True, 5, 302, False, False),
    (2, 8, 130, True, False, 5, 302, False, True),
    (3, 4, 1025, True, True, 5, 302, False, False),
    (3, 3, 2049, True, True, 4, 302, False, False),
    (3, 4, 129, True, True, 4, 300, True, False),
    (3, 3, 96, False, False, 5, 302, True, False),
]


def orbitals(rng, M, G, periodic):
    """smooth random orbitals, orthonormal in the Simpson metric's plain sum"""
    x = np.linspace(XI, XF, G)
    f = np.zeros((M, G), np.complex128)
    for k in range(M):
        for j in range(M + 1):
            ph = 2 * np.pi * j * (x - XI) / (XF - XI)
            a = rng.normal(size=4)
            f[k] += (a[0] + 1j * a[1]) * np.cos(ph) + (a[2] + 1j * a[3]) * np.sin(ph)
    if not periodic:
        f *= np.exp(-x ** 2)
    return f


def simpson(G, dx, oracle):
    """the oracle's weights, one grid function at a time"""
    return np.array([oracle.simpson(dx, np.eye(G)[i].astype(np.complex128)).real
                     for i in range(G)])


@pytest.mark.parametrize("N,M,G,per,imag,rk,der,split,rob", CASES)
def test_step_vs_oracle(gpu, oracle, N, M, G, per, imag, rk, der, split, rob):
    rng = np.random.default_rng(1000 * M + G)
    dx = (XF - XI) / (G - 1)
    w = simpson(G, dx, oracle)
    f = orbitals(rng, M, G, per)
    for i in range(M):
        for j in range(i):
            f[i] -= np.sum(w * f[j].conj() * f[i]) * f[j]
        f[i] /= np.sqrt(np.sum(w * np.abs(f[i]) ** 2))
    pot = 0.5 * np.linspace(XI, XF, G) ** 2
    dt, g, lz = min(1e-3, 0.2 * dx * dx), 0.3, 4
    c = rand_coef(rng, oracle.dim(N, M))
    s = gpu.Solver(N, M, G, XI, XF, dt, imag, rk_order=rk, lanczos_iter=lz, periodic=per)
    s.set_derivative(der)
    s.set_orb_method(31 if split else 30)
    s.set_orthogonality(rob)
    s.set_potential(pot)
    s.set_interaction(g)
    s.set_state(f, c)
    st = {"orb": f.copy(), "coef": c.copy(), "hob": np.zeros((M, M), complex),
          "hint": np.zeros(M ** 4, complex)}
    st["rho1"] = np.ascontiguousarray(oracle.onebody_dm(N, M, c))
    st["rho2"] = np.ascontiguousarray(oracle.twobody_dm(N, M, c)).reshape(-1)
    st["rinv"] = np.ascontiguousarray(np.linalg.inv(st["rho1"]))
    for _ in range(2):
        s.step(1)
        oracle.propagate_step(st, N, dx, dt, -0.5, 0.0, g, per, imag, rk, lz, pot, robust=rob,
                              der=der, orb_method=31 if split else 30)
    got = s.get()
    for k in ("orb", "coef", "hob", "hint", "rho1", "rho2", "rinv"):
        assert rel_err(got[k], st[k]) < 1e-10, k


@pytest.mark.parametrize("M", [1, 2, 3, 5, 8])
def test_regularised_inverse(gpu, oracle, M):
    """every boson in the first orbital: rho1 has M - 1 zero eigenvalues, so
    rho1 + x exp(-rho1 / x), x = N 1e-9, is inverted (synchronize.c:42-57)"""
    N, G = 3, 33
    rng = np.random.default_rng(M)
    c = np.zeros(oracle.dim(N, M), np.complex128)
    c[0] = 1.0
    dx = (XF - XI) / (G - 1)
    w = simpson(G, dx, oracle)
    f = orbitals(rng, M, G, True)
    s = gpu.Solver(N, M, G, XI, XF, 1e-3, True, rk_order=4, lanczos_iter=3)
    s.set_potential(np.zeros(G))
    s.set_interaction(0.1)
    s.set_state(f, c)
    rho = oracle.onebody_dm(N, M, c) if M > 1 else np.array([[float(N)]], complex)
    x = N * 1e-9
    if M > 1:
        e, u = np.linalg.eigh(rho)
        rho = rho + (u * (x * np.exp(-e / x))) @ u.conj().T
    assert rel_err(s.get()["rinv"], np.linalg.inv(rho)) < 1e-10


def test_inverse_near_the_threshold(gpu, oracle):
    """lowest eigenvalue a little above and below 1e-9 of the highest: the
    bound cannot tell, the eigenvalues decide"""
    N, M, G = 2, 2, 33
    f = orbitals(np.random.default_rng(0), M, G, True)
    for ratio in (0.5e-9, 2e-9):
        # configurations in rank order: (2, 0), (1, 1), (0, 2); rho1 = diag(2 a^2, 2 b^2)
        b = np.sqrt(ratio / (1 + ratio))
        c = np.array([np.sqrt(1 - b * b), 0, b], np.complex128)
        s = gpu.Solver(N, M, G, XI, XF, 1e-3, True, rk_order=4, lanczos_iter=3)
        s.set_potential(np.zeros(G))
        s.set_interaction(0.1)
        s.set_state(f, c)
        lam = np.real(np.diag(oracle.onebody_dm(N, M, c))).copy()
        if lam.min() / lam.max() < 1e-9:
            x = lam.max() * 1e-9
            lam = lam + x * np.exp(-lam / x)
        assert rel_err(np.diag(s.get()["rinv"]), 1 / lam) < 1e-10, ratio

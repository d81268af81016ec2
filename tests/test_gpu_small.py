"""The one-launch path for small Fock spaces (csrc/smallsys.cuh) against the
oracle: one row in the (N-2)-space, fewer and more rows than threads, output
pairs spread over idle threads, tables too long for shared memory, the sizes on
both sides of the rule that chooses it, and a Lanczos breakdown (more vectors
than configurations).

Tolerances: the parity targets (1e-12 of the largest element for one product,
1e-10 for Lanczos steps and whole steps)."""
import numpy as np
import pytest

from helpers import phys_hint, rand_coef, rand_hint, rand_hob, rel_err

pytestmark = pytest.mark.gpu

SIZES = [(2, 2), (2, 8), (3, 7), (4, 8), (10, 4), (1500, 2), (60, 3), (24, 4), (13, 5),
         (10, 6), (11, 6), (12, 6), (5, 8), (7, 8), (8, 8)]


def dev(a):
    import torch

    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.mark.parametrize("N,M", SIZES)
def test_small_hc_vs_oracle(gpu, oracle, N, M):
    import torch

    rng = np.random.default_rng(31 * N + M)
    sp = gpu.Space(N, M)
    c, h, g = rand_coef(rng, sp.dim), rand_hob(rng, M), rand_hint(rng, M)
    sp.set_matrices(dev(h), dev(g))
    cd = dev(c)
    out = torch.empty_like(cd)
    sp.apply_hamiltonian(cd, out)
    ref = oracle.apply_hamiltonian(N, M, c, h, g)
    assert rel_err(out.cpu().numpy(), ref) < 1e-12
    sp.apply_hamiltonian(cd, cd)  # in place
    assert np.array_equal(cd.cpu().numpy(), out.cpu().numpy())


@pytest.mark.parametrize("N,M,m,imag", [(2, 2, 8, False), (2, 2, 2, True), (3, 7, 16, False),
                                        (10, 4, 5, True), (24, 4, 6, False), (10, 6, 4, False),
                                        (11, 6, 5, True), (5, 8, 3, False), (60, 3, 17, False)])
def test_small_sil_vs_oracle(gpu, oracle, N, M, m, imag):
    rng = np.random.default_rng(N * M)
    sp = gpu.Space(N, M)
    c, h, g = rand_coef(rng, sp.dim), rand_hob(rng, M), phys_hint(rng, M)
    g = g * (0.05 / np.abs(g).max())
    sp.set_matrices(dev(h), dev(g))
    cd, ref = dev(c), c
    for _ in range(2):
        sp.sil_step(cd, m, 0.01, imag)
        _, ref = oracle.sil_step(N, M, h, g, m, 0.01, imag, ref)
    assert rel_err(cd.cpu().numpy(), ref) < 1e-10


def test_small_and_large_jobs_in_one_batch(gpu, oracle):
    """slots on both paths in one step graph, small ones with the eigen-residual
    monitor; the same bits alone and together, and a stopped job leaves"""
    from oracle import hermite_orbitals

    def job(N, M, G, seed, steps, eig_tol=0.0):
        orb, _ = hermite_orbitals(M, G, -8.0, 8.0)
        return {"npar": N, "norb": M, "grid_size": G, "xi": -8.0, "xf": 8.0, "periodic": 1,
                "imagtime": 1, "rk_order": 5, "dt": 0.01, "g": 0.3, "max_steps": steps,
                "energy_tol": 1.0, "check_every": 2, "eig_tol": eig_tol,
                "pot": 0.5 * np.linspace(-8, 8, G) ** 2, "orbitals": orb,
                "coef": rand_coef(np.random.default_rng(seed), oracle.dim(N, M)),
                "der_method": 302}

    jobs = [job(10, 4, 64, 1, 6, 1e-30), job(16, 6, 64, 2, 6, 1e-30), job(9, 3, 96, 3, 6, 1e3),
            job(6, 6, 64, 4, 5, 1e-30)]
    size = sum(gpu.Batch.job_bytes(j, 5) for j in jobs)
    alone = []
    for j in jobs:
        b = gpu.Batch(2, size, 5)
        s = b.admit(j)
        b.step(6)
        alone.append((b.fetch(s), b.monitor(s)))
        b.close()
    b = gpu.Batch(6, size, 5)
    slots = [b.admit(j) for j in jobs]
    for _ in range(6):
        b.step(1)
        b.poll()  # stopped slots leave the lists
    for s, (a, mon) in zip(slots, alone):
        got = b.fetch(s)
        for k in ("orb", "coef", "rho1", "rho2", "energy", "steps", "converged"):
            assert np.array_equal(got[k], a[k]), k
        assert b.monitor(s) == mon
    # energy_tol 1 always passes: the residual decides (1e3 at the first check)
    assert [a["steps"] for a, _ in alone] == [6, 6, 2, 5]
    assert [a["converged"] for a, _ in alone] == [False, False, True, False]
    for (a, mon), j in zip(alone, jobs):
        assert mon["eig_residual"] > 0.0
    b.close()

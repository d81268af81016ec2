"""What the autotuner times: nothing for spaces whose steps launch none of its
kernels, and the contraction of a complex W for systems in real time that start
from real orbitals (their W is complex from the first step on)."""
import numpy as np
import pytest

from helpers import rand_coef, rand_hint, rand_hob
from oracle import hermite_orbitals

pytestmark = pytest.mark.gpu


def dev(a):
    import torch

    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def solver(gpu, dim, N, M, imag, G=64, real=False):
    orb, _ = hermite_orbitals(M, G, -8.0, 8.0)
    c = rand_coef(np.random.default_rng(N), dim(N, M))
    c = c.real / np.linalg.norm(c.real) + 0j if real else c
    s = gpu.Solver(N, M, G, -8.0, 8.0, 1e-3, imag, rk_order=4, lanczos_iter=5)
    s.set_potential(0.5 * np.linspace(-8, 8, G) ** 2)
    s.set_interaction(0.1)
    s.set_state(orb, c)
    return s


def test_small_spaces_are_not_tuned(gpu, oracle):
    import torch

    N, M = 9, 4  # 220 rows; no other test uses this size
    sp = gpu.Space(N, M)
    rng = np.random.default_rng(0)
    sp.set_matrices(dev(rand_hob(rng, M)), dev(rand_hint(rng, M)))
    c = dev(rand_coef(rng, sp.dim))
    r1 = torch.empty(M * M, dtype=torch.complex128, device="cuda")
    r2 = torch.empty(M ** 4, dtype=torch.complex128, device="cuda")
    step = gpu.Step(sp, c, r1, r2, 5, 0.01, False)
    solver(gpu, oracle.dim, N, M, True).step(1)
    torch.cuda.synchronize()
    assert gpu.tune_get("hcp_y", N, M) == -1
    step.close()
    # more vectors than the cluster path takes: the general one, tuned
    step = gpu.Step(sp, c, r1, r2, 17, 0.01, False)
    assert gpu.tune_get("hcp_y", N, M) >= 0
    step.close()


@pytest.mark.parametrize("N,imag", [(22, False), (23, True)])
def test_tuned_for_the_complex_w_that_comes(gpu, oracle, N, imag):
    """8 orbitals: variant 3 is 8 % ahead with a complex W, variant 0 4 % with a
    real one.  Real time, and imaginary time with complex coefficients"""
    s = solver(gpu, oracle.dim, N, 8, imag)
    assert gpu.tune_get("hcp_y", N, 8) == 3
    s.step(1)
    assert np.isfinite(s.get()["coef"]).all()


def test_all_real_stays_real(gpu, oracle):
    """imaginary time from real orbitals and coefficients: both stay real, and the
    contraction is tuned with the real W it runs with"""
    s = solver(gpu, oracle.dim, 21, 8, True, real=True)
    assert gpu.tune_get("hcp_y", 21, 8) in (0, 2, 3)
    s.step(2)
    got = s.get()
    assert not got["orb"].imag.any() and not got["coef"].imag.any()


def test_batch_in_real_time_keeps_its_bits(gpu, oracle):
    """the tuner's pass over real-time jobs leaves nothing behind: the same bits
    with the variant given"""
    N, M, G = 14, 6, 64
    orb, _ = hermite_orbitals(M, G, -8.0, 8.0)
    job = {"npar": N, "norb": M, "grid_size": G, "xi": -8.0, "xf": 8.0, "periodic": 1,
           "imagtime": 0, "rk_order": 4, "dt": 1e-3, "g": 0.2, "max_steps": 9,
           "energy_tol": 0.0, "check_every": 0, "pot": 0.5 * np.linspace(-8, 8, G) ** 2,
           "orbitals": orb, "coef": rand_coef(np.random.default_rng(1), oracle.dim(N, M)),
           "der_method": 302}
    out = []
    for v in (None, 0, 3):
        b = gpu.Batch(2, 2 * gpu.Batch.job_bytes(job, 5), 5)
        s = b.admit(job)
        if v is not None:
            b.set_variant(M, v)
        b.step(3)
        out.append(b.fetch(s))
        b.close()
    for o in out[1:]:
        for k in ("orb", "coef", "rho1", "rho2", "energy"):
            assert np.array_equal(o[k], out[0][k]), k

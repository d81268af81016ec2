"""The Lanczos recurrence with its row work in the gather-back of H.C
(csrc/lanczos.cu, kernels.h): spaces of one block to many, more dots than one
pass takes, the copied and the in-place start vector, wide spaces; and a batch
slot's results read in one launch or by the copy engine (csrc/batch.cu)."""
import numpy as np
import pytest

from helpers import phys_hint, rand_coef, rand_hint, rand_hob, rel_err
from oracle import hermite_orbitals

pytestmark = pytest.mark.gpu


def system(gpu, N, M, hint=rand_hint):
    import torch

    rng = np.random.default_rng(7 * N + M)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    sp = gpu.Space(N, M)
    c, h, g = rand_coef(rng, sp.dim), rand_hob(rng, M), hint(rng, M)
    sp.set_matrices(dev(h), dev(g))
    return sp, c, h, g, dev(c)


# (14, 4): 680 rows, small enough for a cluster but for m > 16; (22, 3): 276
# rows, a second block of 20; (60, 3) and on: many blocks; M > 8: 64-row blocks
@pytest.mark.parametrize("N,M,m", [(22, 3, 20), (14, 4, 18), (12, 6, 5), (11, 7, 3), (8, 8, 4),
                                   (60, 4, 6), (3, 10, 5), (4, 12, 4)])
@pytest.mark.parametrize("imag", [False, True])
def test_step_vs_oracle(gpu, oracle, N, M, m, imag):
    sp, c, h, g, cd = system(gpu, N, M, phys_hint)
    ref = c
    for _ in range(2):
        sp.sil_step(cd, m, 0.002, imag)
        ref = oracle.sil_step(N, M, h, g, m, 0.002, imag, ref)[1]
    got = cd.cpu().numpy()
    if np.isfinite(ref).all():
        assert rel_err(got, ref) < 1e-10
    else:  # the oracle's exp(-E dt) overflows before it normalises
        assert imag and abs(np.vdot(got, got) - 1) < 1e-12


def test_breakdown_stops_the_recurrence(gpu, oracle):
    """an eigenvector to start from: beta_0 is rounding, the step a phase"""
    N, M = 12, 6
    sp, c, h, g, cd = system(gpu, N, M)
    h = np.diag(np.arange(1.0, M + 1.0)) + 0j
    g = np.zeros_like(g)
    import torch

    sp.set_matrices(torch.from_numpy(h).cuda(), torch.from_numpy(g).cuda())
    c = np.zeros(sp.dim, np.complex128)
    c[0] = 1.0
    cd = torch.from_numpy(c).cuda()
    sp.sil_step(cd, 5, 0.01, False)
    assert rel_err(cd.cpu().numpy(), oracle.sil_step(N, M, h, g, 5, 0.01, False, c)[1]) < 1e-12


def test_fetch_both_ways(gpu, oracle):
    """20349 coefficients are above the pinned words, 84 are not; the arrays
    left out of a call are not written and the others are the same bytes"""
    import ctypes as C

    for N, M, G in [(3, 7, 64), (16, 6, 64), (5, 2, 128)]:
        dim = oracle.dim(N, M)
        orb, _ = hermite_orbitals(M, G, -8.0, 8.0)
        job = {"npar": N, "norb": M, "grid_size": G, "xi": -8.0, "xf": 8.0, "periodic": 1,
               "imagtime": 1, "rk_order": 4, "dt": 0.005, "g": 0.02, "max_steps": 9,
               "energy_tol": 0.0, "check_every": 0,
               "pot": 0.5 * np.linspace(-8, 8, G) ** 2, "orbitals": orb,
               "coef": rand_coef(np.random.default_rng(N), dim), "der_method": 302}
        b = gpu.Batch(1, gpu.Batch.job_bytes(job, 4), 4)
        s = b.admit(job)
        b.step(2)
        out = b.fetch(s)
        assert out["steps"] == 2 and not out["converged"] and np.isfinite(out["energy"])
        assert abs(np.vdot(out["coef"], out["coef"]) - 1) < 1e-12
        e, n, cv = C.c_double(), C.c_uint32(), C.c_int()
        lib = gpu.load()
        for k in range(4):  # one array at a time
            buf = [np.full(a.size, np.nan + 0j) for a in
                   (out["orb"], out["coef"], out["rho1"], out["rho2"])]
            ptr = [x.ctypes.data if i == k else None for i, x in enumerate(buf)]
            assert lib.mctdhb_batch_fetch(b.h, s, *ptr, C.byref(e), C.byref(n), C.byref(cv)) == 0
            for i, key in enumerate(("orb", "coef", "rho1", "rho2")):
                if i == k:
                    assert np.array_equal(buf[i], out[key].reshape(-1))
                else:
                    assert np.isnan(buf[i]).all()
            assert (e.value, n.value, cv.value) == (out["energy"], 2, 0)
        assert lib.mctdhb_batch_fetch(b.h, s, None, None, None, None, None, None, None) == 0
        b.close()

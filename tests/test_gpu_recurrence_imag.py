"""Imaginary-time Lanczos steps of many blocks (csrc/lanczos.cu: the sums by the
last block, the shifted exponents, the fused |C|^2), with an interaction small
enough that the oracle's exp(-E dt) stays finite, so that every element is
compared: 1e-10 of the largest, as for Lanczos steps elsewhere.  (60, 4): 39,711
rows in 156 blocks; (11, 7): 12,376; (22, 3) with more dots than one pass
takes."""
import numpy as np
import pytest

from helpers import phys_hint, rand_coef, rand_hob, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,M,m", [(60, 4, 6), (11, 7, 3), (12, 6, 5), (22, 3, 20), (20, 6, 8),
                                   (9, 8, 4), (4, 12, 4)])
@pytest.mark.parametrize("dt", [0.002, 0.02])
def test_imaginary_step_vs_oracle(gpu, oracle, N, M, m, dt):
    import torch

    rng = np.random.default_rng(7 * N + M)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    sp = gpu.Space(N, M)
    c, h, g = rand_coef(rng, sp.dim), rand_hob(rng, M), phys_hint(rng, M)
    g = g * (0.05 / np.abs(g).max())
    sp.set_matrices(dev(h), dev(g))
    cd, ref = dev(c), c
    for _ in range(2):
        sp.sil_step(cd, m, dt, True)
        ref = oracle.sil_step(N, M, h, g, m, dt, True, ref)[1]
    assert np.isfinite(ref).all()
    got = cd.cpu().numpy()
    assert rel_err(got, ref) < 1e-10
    assert abs(np.vdot(got, got) - 1) < 1e-12


def test_exponents_that_overflow_unshifted(gpu, oracle):
    """exp(-E dt) with |E| dt beyond 709: the shifted exponents against a step of
    the oracle with h lowered by a constant, which moves E alone"""
    import torch

    N, M, m, dt = 30, 4, 5, 0.05
    rng = np.random.default_rng(3)
    h, g = rand_hob(rng, M), phys_hint(rng, M)
    g = g * (0.05 / np.abs(g).max())
    shift = -1000.0 / (N * dt)  # N shift dt = -1000
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    sp = gpu.Space(N, M)
    c = rand_coef(rng, sp.dim)
    sp.set_matrices(dev(h + shift * np.eye(M)), dev(g))
    cd = dev(c)
    sp.sil_step(cd, m, dt, True)
    ref = oracle.sil_step(N, M, h, g, m, dt, True, c)[1]
    # E is 2e4 where |H| alone is 1e2: its rounding, 2e4 eps dt on the exponents
    # and 2e4 eps on the products, is far below
    assert rel_err(cd.cpu().numpy(), ref) < 1e-8

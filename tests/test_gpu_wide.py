"""H.C, densities and the short iterative Lanczos step above 8 orbitals
(csrc/wide.cu: 16- or 32-row contraction tiles, 64-pair Gram super-tiles)
against the oracle, at the edges of their tiles: one row in the (N-2)-space,
rows just above and below a tile, 45 / 66 / 136 pairs around the super-tile of
64, one- and two-strip contraction (20 / 21 orbitals), the most orbitals.

Tolerances: the parity targets of the other sizes (1e-12 of the largest
element for one product or Gram sum, 1e-10 for a Lanczos step)."""
import numpy as np
import pytest

from helpers import phys_hint, rand_coef, rand_hint, rand_hob, rel_err

pytestmark = pytest.mark.gpu

SIZES = [(2, 9), (3, 9), (5, 9), (4, 11), (3, 16), (3, 20), (4, 21), (2, 30), (3, 30)]


def space(gpu, N, M, seed, hint):
    import torch

    rng = np.random.default_rng(seed)
    sp = gpu.Space(N, M)
    c, h, g = rand_coef(rng, sp.dim), rand_hob(rng, M), hint(rng, M)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    sp.set_matrices(dev(h), dev(g))
    return sp, c, h, g, dev(c)


@pytest.mark.parametrize("N,M", SIZES)
def test_wide_hc_and_densities_vs_oracle(gpu, oracle, N, M):
    import torch

    sp, c, h, g, cd = space(gpu, N, M, 100 * N + M, rand_hint)
    out = torch.empty_like(cd)
    sp.apply_hamiltonian(cd, out)
    r1 = torch.empty(M, M, dtype=torch.complex128, device="cuda")
    r2 = torch.empty(M ** 4, dtype=torch.complex128, device="cuda")
    sp.density_matrices(cd, r1, r2)
    assert rel_err(out.cpu().numpy(), oracle.apply_hamiltonian(N, M, c, h, g)) < 1e-12
    assert rel_err(r1.cpu().numpy(), oracle.onebody_dm(N, M, c)) < 1e-12
    assert rel_err(r2.cpu().numpy(), oracle.twobody_dm(N, M, c)) < 1e-12


@pytest.mark.parametrize("N,M,imag", [(4, 9, False), (3, 21, True)])
def test_wide_sil_step_vs_oracle(gpu, oracle, N, M, imag):
    sp, c, h, g, cd = space(gpu, N, M, 7, phys_hint)
    sp.sil_step(cd, 5, 0.01, imag)
    assert rel_err(cd.cpu().numpy(), oracle.sil_step(N, M, h, g, 5, 0.01, imag, c)[1]) < 1e-10

"""The kernels above 8 orbitals (csrc/wide.cu) in spaces where their blocks go
round more than once: the gather-back has 8 blocks an SM of 64 rows (75,776 rows
on 148 SMs), the Gram kernel 296 blocks over the super-tiles of 64 x 64 pairs.
(8, 12): 75,582 and (7, 13) 50,388 rows are within one pass of the first,
(9, 12) 167,960 and (13, 9) 203,490 take three; (7, 16): 15,504 rows of the
(N-2)-space are 485 tiles on 49 blocks a super-tile, (13, 9): 75,582 are 2,362
on 296.  Against the oracle: 1e-12 of the largest element for a product or a
Gram sum, 1e-10 for a Lanczos step."""
import numpy as np
import pytest

from helpers import phys_hint, rand_coef, rand_hint, rand_hob, rel_err

pytestmark = pytest.mark.gpu


def space(gpu, N, M, hint):
    import torch

    rng = np.random.default_rng(100 * N + M)
    sp = gpu.Space(N, M)
    c, h, g = rand_coef(rng, sp.dim), rand_hob(rng, M), hint(rng, M)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    sp.set_matrices(dev(h), dev(g))
    return sp, c, h, g, dev(c)


@pytest.mark.parametrize("N,M", [(9, 12), (13, 9), (7, 16)])
def test_products_and_densities(gpu, oracle, N, M):
    import torch

    sp, c, h, g, cd = space(gpu, N, M, rand_hint)
    out = torch.empty_like(cd)
    sp.apply_hamiltonian(cd, out)
    r1 = torch.empty(M, M, dtype=torch.complex128, device="cuda")
    r2 = torch.empty(M ** 4, dtype=torch.complex128, device="cuda")
    sp.density_matrices(cd, r1, r2)
    assert rel_err(out.cpu().numpy(), oracle.apply_hamiltonian(N, M, c, h, g)) < 1e-12
    assert rel_err(r1.cpu().numpy(), oracle.onebody_dm(N, M, c)) < 1e-12
    assert rel_err(r2.cpu().numpy(), oracle.twobody_dm(N, M, c)) < 1e-12


def test_lanczos_step(gpu, oracle):
    """the gather-back with the recurrence's row work, three passes a block"""
    N, M = 13, 9
    sp, c, h, g, cd = space(gpu, N, M, phys_hint)
    g = g * (0.05 / np.abs(g).max())
    import torch

    sp.set_matrices(torch.from_numpy(h).cuda(), torch.from_numpy(g).cuda())
    sp.sil_step(cd, 4, 0.01, False)
    assert rel_err(cd.cpu().numpy(), oracle.sil_step(N, M, h, g, 4, 0.01, False, c)[1]) < 1e-10

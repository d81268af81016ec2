"""The contraction with a real pair matrix (real orbitals): at five and six
orbitals it keeps the registers as launched (csrc/pairhc_tmpl.cuh, hcp_y_kernel).
Every variant gives the same bits, at one row, remainders of a chunk of 32 rows
and several chunks a warp; against the oracle 1e-12 of the largest element; and
a lost handover leaves NaN here too."""
import numpy as np
import pytest

from helpers import rand_coef, rel_err

pytestmark = pytest.mark.gpu

VARIANTS = {4: [0, 1, 3], 5: [0, 1, 3], 6: [0, 1, 2, 3], 7: [0, 2, 3], 8: [0, 2, 3]}



@pytest.mark.parametrize("N,M", [(29, 4), (14, 5), (17, 5), (30, 5), (10, 6), (20, 6), (10, 7),
                                 (9, 8), (8, 8)])
def test_real_w(gpu, oracle, N, M):
    import torch

    rng = np.random.default_rng(N * M)
    h = rng.normal(size=(M, M))
    h = (h + h.T) / 2 + 0j
    g = rng.normal(size=M ** 4) + 0j
    sp = gpu.Space(N, M)
    c = rand_coef(rng, sp.dim)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    sp.set_matrices(dev(h), dev(g))
    cd = dev(c)
    before = gpu.tune_get("hcp_y", N, M)
    out = {}
    for v in VARIANTS[M]:
        gpu.tune_set("hcp_y", N, M, v)
        out[v] = torch.full_like(cd, float("nan"))
        sp.apply_hamiltonian(cd, out[v])
    assert rel_err(out[0].cpu().numpy(), oracle.apply_hamiltonian(N, M, c, h, g)) < 1e-12
    for v in VARIANTS[M][1:]:
        assert torch.equal(out[v], out[0]), v
    sp.set_nowait(True)
    gpu.tune_set("hcp_y", N, M, 3)
    lost = torch.zeros_like(cd)
    sp.apply_hamiltonian(cd, lost)
    assert torch.isnan(lost.real).all()
    sp.set_nowait(False)
    sp.apply_hamiltonian(cd, lost)
    assert torch.equal(lost, out[0])
    gpu.tune_set("hcp_y", N, M, max(before, 0))

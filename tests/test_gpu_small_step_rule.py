"""Which step of one system runs on one cluster of blocks (csrc/smallsys.h): up
to 2,048 configurations, one a thread, and up to twice that where the product
is small; more take the general path, which is faster from there.  The routes differ in their launches, 2 an iteration on the
cluster (product, orthogonalisation) and 4 beside it.  Both against the oracle
at the edge; 1e-10 of the largest element, as for Lanczos steps elsewhere."""
import numpy as np
import pytest

from helpers import phys_hint, rand_coef, rand_hob, rel_err

pytestmark = pytest.mark.gpu


# 2,048, 2,049, 4,096 and 4,097; 2,016, 2,080, 4,095 and 4,186; 2,600 (0.20 M
# multiply-adds a product) and 2,925 (0.23 M); 2,002 and 2,380; 1,716 and 3,003 rows
@pytest.mark.parametrize("N,M,cluster", [(2047, 2, True), (2048, 2, True), (4095, 2, True),
                                         (4096, 2, False), (62, 3, True), (63, 3, True),
                                         (89, 3, True), (90, 3, False), (23, 4, True),
                                         (24, 4, False), (9, 6, True), (13, 5, False),
                                         (6, 8, True), (8, 7, False)])
@pytest.mark.parametrize("imag", [False, True])
def test_step_at_the_edge(gpu, oracle, N, M, cluster, imag):
    import torch

    rng = np.random.default_rng(N + M)
    sp = gpu.Space(N, M)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    c, h, g = rand_coef(rng, sp.dim), rand_hob(rng, M), phys_hint(rng, M)
    g = g * (0.05 / np.abs(g).max())
    sp.set_matrices(dev(h), dev(g))
    cd = dev(c)
    r1 = torch.empty(M * M, dtype=torch.complex128, device="cuda")
    r2 = torch.empty(M ** 4, dtype=torch.complex128, device="cuda")
    dt = 0.01 / max(1.0, N / 20)  # |H| dt stays small with many bosons
    m = 5
    step = gpu.Step(sp, cd, r1, r2, m, dt, imag)
    densities = 3
    if cluster:
        assert step.kernels == m + (m - 1) + 1 + densities
    else:
        assert step.kernels == 2 * m + 2 * (m - 1) + 2 + (1 if imag else 0) + densities
    step.launch()
    torch.cuda.synchronize()
    ref = oracle.sil_step(N, M, h, g, m, dt, imag, c)[1]
    assert rel_err(cd.cpu().numpy(), ref) < 1e-10
    assert rel_err(r2.cpu().numpy(), oracle.twobody_dm(N, M, ref)) < 1e-10
    step.close()


def test_dimensions_are_checked_on_both_routes(gpu):
    import torch

    for N, M in ((4, 3), (13, 5)):
        sp = gpu.Space(N, M)
        c = torch.zeros(sp.dim, dtype=torch.complex128, device="cuda")
        for m in (0, 1, 65):
            with pytest.raises(gpu.MctdhbError):
                sp.sil_step(c, m, 0.01, False)

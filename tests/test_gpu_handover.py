"""Waits of the contraction's handover that run out (csrc/pairhc_tmpl.cuh,
batch_tmpl.cuh): without the waits no consumer warp finds its first rows ready,
so every handover of a launch is lost.  H.C then comes out NaN, every job with
rows in the launch is aborted, jobs on other kernels go on, and the context
stays usable."""
import numpy as np
import pytest

from helpers import rand_coef, rand_hint, rand_hob, rel_err
from oracle import hermite_orbitals

pytestmark = pytest.mark.gpu

# one and two consumer warps a producer warp, with and without the register
# split; fewer chunks than warps, and several chunks a warp
@pytest.mark.parametrize("N,M", [(8, 4), (30, 5), (24, 6), (14, 7), (12, 8)])
def test_lost_product_is_nan_everywhere(gpu, oracle, N, M):
    import torch

    rng = np.random.default_rng(N + M)
    sp = gpu.Space(N, M)
    c, h, g = rand_coef(rng, sp.dim), rand_hob(rng, M), rand_hint(rng, M)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    sp.set_matrices(dev(h), dev(g))
    cd = dev(c)
    before = gpu.tune_get("hcp_y", N, M)
    gpu.tune_set("hcp_y", N, M, 3)
    out = torch.zeros_like(cd)
    sp.set_nowait(True)
    sp.apply_hamiltonian(cd, out)
    torch.cuda.synchronize()
    # small spaces run on one cluster of blocks and hand nothing over
    small = oracle.dim(N - 2, M) * (M * (M + 1) // 2) ** 2 <= 250_000
    if not small:
        assert torch.isnan(out.real).all() and torch.isnan(out.imag).all()
        state = cd.clone()
        sp.sil_step(state, 17, 0.01, False)
        torch.cuda.synchronize()
        assert torch.isnan(state.real).any()
    sp.set_nowait(False)
    sp.apply_hamiltonian(cd, out)
    assert rel_err(out.cpu().numpy(), oracle.apply_hamiltonian(N, M, c, h, g)) < 1e-12
    if before >= 0:
        gpu.tune_set("hcp_y", N, M, before)


def job(dim, N, M, seed, G=64):
    orb, _ = hermite_orbitals(M, G, -8.0, 8.0)
    return {"npar": N, "norb": M, "grid_size": G, "xi": -8.0, "xf": 8.0, "periodic": 1,
            "imagtime": 1, "rk_order": 4, "dt": 0.01, "g": 0.2, "max_steps": 1 << 20,
            "energy_tol": 0.0, "check_every": 0, "pot": 0.5 * np.linspace(-8, 8, G) ** 2,
            "orbitals": orb, "coef": rand_coef(np.random.default_rng(seed), dim(N, M)),
            "der_method": 302}


def test_every_job_that_missed_rows_is_aborted(gpu, oracle):
    """three jobs of 5 orbitals with 139 tiles of 256 rows each: with one block
    an SM a block's list goes over two or three of them; and the same with two
    consumer warps a producer (8 orbitals).  A small job and jobs on the
    block-barrier variant are not touched."""
    jobs = [job(oracle.dim, 30, 5, 1), job(oracle.dim, 30, 5, 2), job(oracle.dim, 30, 5, 3),
            job(oracle.dim, 10, 8, 4), job(oracle.dim, 10, 8, 5),
            job(oracle.dim, 14, 6, 6), job(oracle.dim, 8, 3, 7)]
    b = gpu.Batch(len(jobs), sum(gpu.Batch.job_bytes(j, 4) for j in jobs), 4)
    slots = [b.admit(j) for j in jobs]
    for m, v in ((5, 3), (8, 3), (6, 0)):
        b.set_variant(m, v)
    b.step(1)
    assert list(b.poll()[1][slots]) == [1] * 7
    b.set_nowait(True)
    b.step(1)
    b.sync()
    _, state, steps, _ = b.poll()
    assert list(state[slots]) == [3, 3, 3, 3, 3, 1, 1]
    assert list(steps[slots]) == [1, 1, 1, 1, 1, 2, 2]
    # slots are given back and taken again; a fresh job steps
    for s in slots[:5]:
        b.release(s)
    b.set_nowait(False)
    s = b.admit(jobs[0])
    b.step(1)
    out = b.fetch(s)
    assert out["steps"] == 1 and abs(np.vdot(out["coef"], out["coef"]) - 1) < 1e-12
    b.close()

"""The pair contraction's 32-row pipeline (variant 3, csrc/pairhc_tmpl.cuh and
batch_tmpl.cuh): chunks of a row to a few hundred rows against the oracle, and
in the batched engine, where every change of slot in a block's tile list stages
another W and other tables, the same bits as variant 0 and as each job alone."""
import numpy as np
import pytest

from helpers import rand_coef, rand_hint, rand_hob, rel_err
from oracle import hermite_orbitals

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,M", [(250, 3), (300, 3), (41, 4), (18, 5), (12, 6), (9, 7), (8, 8),
                                 (700, 3)])
@pytest.mark.parametrize("real", [False, True])
def test_contraction_vs_oracle(gpu, oracle, N, M, real):
    """general-path sizes with ragged last chunks; real W takes two products"""
    import torch

    rng = np.random.default_rng(N + M)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    sp = gpu.Space(N, M)
    c, h, g = rand_coef(rng, sp.dim), rand_hob(rng, M), rand_hint(rng, M)
    if real:
        h, g = np.ascontiguousarray(h.real + 0j), np.ascontiguousarray(g.real + 0j)
    sp.set_matrices(dev(h), dev(g))
    cd = dev(c)
    ref = oracle.apply_hamiltonian(N, M, c, h, g)
    got = {}
    for v in (0, 3):
        gpu.tune_set("hcp_y", N, M, v)
        out = torch.empty_like(cd)
        sp.apply_hamiltonian(cd, out)
        got[v] = out.cpu().numpy()
    assert rel_err(got[3], ref) < 1e-12
    assert np.array_equal(got[0], got[3])


def test_batched_pipeline_over_many_slots(gpu, oracle):
    def job(N, M, seed):
        orb, _ = hermite_orbitals(M, 64, -8.0, 8.0)
        return {"npar": N, "norb": M, "grid_size": 64, "xi": -8.0, "xf": 8.0, "periodic": 1,
                "imagtime": seed % 2, "rk_order": 4, "dt": 0.005, "g": 0.02, "max_steps": 100,
                "energy_tol": 0.0, "check_every": 0,
                "pot": 0.5 * np.linspace(-8, 8, 64) ** 2, "orbitals": orb,
                "coef": rand_coef(np.random.default_rng(seed), oracle.dim(N, M)),
                "der_method": 302}

    sizes = [(210, 3), (12, 6), (230, 3), (13, 6), (250, 3), (12, 6), (8, 8), (16, 6), (9, 8),
             (36, 4), (40, 4), (700, 3)]
    jobs = [job(N, M, i) for i, (N, M) in enumerate(sizes)]
    total = sum(gpu.Batch.job_bytes(j, 4) for j in jobs)

    def run(jobs, v):
        b = gpu.Batch(len(jobs), total, 4)
        slots = [b.admit(j) for j in jobs]
        for M in (3, 4, 6, 8):
            b.set_variant(M, v)
        b.step(2)
        out = [b.fetch(s) for s in slots]
        assert all(st == 1 for st in b.poll()[1])  # running: no handover was lost
        b.close()
        return out

    mix = {v: run(jobs, v) for v in (0, 3)}
    for i, j in enumerate(jobs):
        alone = run([j], 3)[0]
        for k in ("orb", "coef", "rho1", "rho2"):
            assert np.array_equal(mix[3][i][k], mix[0][i][k]), (i, k)
            assert np.array_equal(mix[3][i][k], alone[k]), (i, k)

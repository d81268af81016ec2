"""Batches of one to many slots: the orbital side of a slot and the step of a
small one run on clusters of 8, 4, 2 or 1 blocks by how many slots run
(csrc/batch.h, cluster_blocks), and a job's bits do not depend on it.  Jobs on
both paths, 2 to 8 orbitals, real and imaginary time, full and split step, the
robust projector, and vectors above the rows that one block takes."""
import numpy as np
import pytest

from helpers import rand_coef
from oracle import hermite_orbitals

pytestmark = pytest.mark.gpu


def job(dim, N, M, G, seed, steps=1 << 20, imag=1, split=0, robust=0, eig_tol=0.0):
    orb, _ = hermite_orbitals(M, G, -8.0, 8.0)
    return {"npar": N, "norb": M, "grid_size": G, "xi": -8.0, "xf": 8.0, "periodic": 1,
            "imagtime": imag, "rk_order": 4, "dt": 0.004, "g": 0.3, "max_steps": steps,
            "energy_tol": 1.0 if eig_tol else 0.0, "check_every": 1 if eig_tol else 0,
            "eig_tol": eig_tol, "pot": 0.5 * np.linspace(-8, 8, G) ** 2, "orbitals": orb,
            "coef": rand_coef(np.random.default_rng(seed), dim(N, M)), "der_method": 302,
            "orb_method": 31 if split else 30, "impr_ortho": robust}


KEYS = ("orb", "coef", "rho1", "rho2", "energy", "steps", "converged")


def run(gpu, jobs, count, steps):
    """the jobs in the first slots, copies of the first one behind them"""
    room = sum(gpu.Batch.job_bytes(j, 4) for j in jobs)
    fill = gpu.Batch.job_bytes(jobs[0], 4)
    b = gpu.Batch(count, room + max(0, count - len(jobs)) * fill, 4)
    slots = [b.admit(j) for j in jobs]
    extra = [b.admit(jobs[0]) for _ in range(count - len(jobs))]
    b.step(steps)
    out = [b.fetch(s) for s in slots]
    out += [b.fetch(s) for s in extra[-1:]]
    mon = [b.monitor(s) for s in slots]
    b.close()
    return out, mon


# a slot by itself, and counts past the waves of 8, 4, 2 and 1 blocks of 148 SMs
@pytest.mark.parametrize("count", [8, 20, 60, 100, 300])
def test_bits_do_not_depend_on_the_slots(gpu, oracle, count):
    d = oracle.dim
    jobs = [job(d, 8, 3, 96, 1, eig_tol=1e-30), job(d, 10, 4, 130, 2, imag=0),
            job(d, 120, 2, 64, 3), job(d, 14, 5, 257, 4, robust=1),
            job(d, 9, 6, 64, 5, imag=0, split=1), job(d, 4, 7, 65, 6), job(d, 4, 8, 64, 7)]
    alone, mon1 = zip(*[(o[0], m[0]) for o, m in (run(gpu, [j], 1, 3) for j in jobs)])
    out, mon = run(gpu, jobs, count, 3)
    for i, want in enumerate(alone):
        for k in KEYS:
            assert np.array_equal(out[i][k], want[k]), (i, k)
        assert mon[i] == mon1[i]
    if count > len(jobs):
        for k in KEYS:
            assert np.array_equal(out[-1][k], alone[0][k]), k


def test_long_vectors_of_few_orbitals(gpu, oracle):
    """9,001 and 18,336 rows: more than one block a slot however many there are"""
    jobs = [job(oracle.dim, 190, 3, 64, 1), job(oracle.dim, 9000, 2, 64, 2)]
    alone = [run(gpu, [j], 1, 2)[0][0] for j in jobs]
    out, _ = run(gpu, jobs, 160, 2)
    for got, want in zip(out, alone):
        for k in KEYS:
            assert np.array_equal(got[k], want[k]), k


def test_fewer_slots_as_jobs_stop(gpu, oracle):
    """40 jobs that stop after 1 to 5 steps: the cluster size changes under the
    others, whose bits stay"""
    jobs = [job(oracle.dim, 8, 3, 64, i, steps=1 + i % 5) for i in range(40)]
    alone = [run(gpu, [j], 1, 6)[0][0] for j in jobs[:5]]
    b = gpu.Batch(40, sum(gpu.Batch.job_bytes(j, 4) for j in jobs), 4)
    slots = [b.admit(j) for j in jobs]
    for _ in range(6):
        b.step(1)
        b.poll()
    for i in range(5):
        got = b.fetch(slots[i])
        for k in KEYS:
            assert np.array_equal(got[k], alone[i][k]), (i, k)
    b.close()

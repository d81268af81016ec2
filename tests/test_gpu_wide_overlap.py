"""H.C above 8 orbitals on one Space from several streams and threads at once,
beside a Lanczos step of the same Space, and inside a stream capture: products
have a scratch apart from the steps' and wait for one another (csrc/capi.cu), so
overlapping calls give the doubles of calls one after another.

Tolerance against the oracle: 1e-12 of the largest element, as for one product
elsewhere; overlapping calls are compared bit for bit."""
import threading

import numpy as np
import pytest

from helpers import phys_hint, rand_coef, rand_hint, rand_hob, rel_err

pytestmark = pytest.mark.gpu


def setup(gpu, N, M, hint=rand_hint, count=4):
    import torch

    rng = np.random.default_rng(10 * N + M)
    sp = gpu.Space(N, M)
    h, g = rand_hob(rng, M), hint(rng, M)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    sp.set_matrices(dev(h), dev(g))
    c = [rand_coef(rng, sp.dim) for _ in range(count)]
    return sp, h, g, c, [dev(x) for x in c]


def one_after_another(sp, vectors):
    import torch

    out = [torch.empty_like(v) for v in vectors]
    for v, o in zip(vectors, out):
        sp.apply_hamiltonian(v, o)
    torch.cuda.synchronize()
    return out


@pytest.mark.parametrize("N,M", [(6, 10), (8, 9)])
def test_streams_overlap(gpu, oracle, N, M):
    import torch

    sp, h, g, c, dc = setup(gpu, N, M)
    want = one_after_another(sp, dc)
    assert rel_err(want[0].cpu().numpy(), oracle.apply_hamiltonian(N, M, c[0], h, g)) < 1e-12
    streams = [torch.cuda.Stream() for _ in dc]
    out = [[torch.full_like(v, float("nan")) for v in dc] for _ in range(32)]
    torch.cuda.synchronize()
    for row in out:
        for s, v, o in zip(streams, dc, row):
            sp.apply_hamiltonian(v, o, s)
    torch.cuda.synchronize()
    for row in out:
        for o, w in zip(row, want):
            assert torch.equal(o, w)


def test_threads_overlap(gpu):
    import torch

    sp, _, _, _, dc = setup(gpu, 7, 10)
    want = one_after_another(sp, dc)
    out = [[torch.full_like(v, float("nan")) for _ in range(32)] for v in dc]
    torch.cuda.synchronize()

    def work(v, outs):
        s = torch.cuda.Stream()
        for o in outs:
            sp.apply_hamiltonian(v, o, s)
        s.synchronize()

    ts = [threading.Thread(target=work, args=a) for a in zip(dc, out)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for outs, w in zip(out, want):
        assert all(torch.equal(o, w) for o in outs)


def test_products_beside_a_step(gpu):
    import torch

    N, M = 7, 10
    sp, _, _, _, dc = setup(gpu, N, M, phys_hint)
    want = one_after_another(sp, dc[:1])[0]
    r1 = torch.empty(M * M, dtype=torch.complex128, device="cuda")
    r2 = torch.empty(M ** 4, dtype=torch.complex128, device="cuda")
    state, alone = dc[1].clone(), dc[1].clone()
    step = gpu.Step(sp, alone, r1, r2, 5, 0.002, False)
    for _ in range(8):
        step.launch()
    torch.cuda.synchronize()
    want_rho = r2.clone()
    step.close()
    step = gpu.Step(sp, state, r1, r2, 5, 0.002, False)
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    out = [torch.full_like(want, float("nan")) for _ in range(64)]
    torch.cuda.synchronize()
    for i in range(8):
        step.launch(a)
        for o in out[8 * i:8 * i + 8]:
            sp.apply_hamiltonian(dc[0], o, b)
    torch.cuda.synchronize()
    assert torch.equal(state, alone) and torch.equal(r2, want_rho)
    assert all(torch.equal(o, want) for o in out)
    step.close()


@pytest.mark.parametrize("N,M", [(5, 9), (3, 21)])
def test_captured_product(gpu, oracle, N, M):
    """row by row, without scratch: replays beside eager products"""
    import torch

    sp, h, g, c, dc = setup(gpu, N, M)
    want = one_after_another(sp, dc)
    captured = torch.full_like(dc[0], float("nan"))
    inplace = dc[2].clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        sp.apply_hamiltonian(dc[0], captured, torch.cuda.current_stream())
    other = torch.cuda.Stream()
    out = [torch.full_like(dc[1], float("nan")) for _ in range(32)]
    torch.cuda.synchronize()
    graph.replay()
    for o in out:
        sp.apply_hamiltonian(dc[1], o, other)
    torch.cuda.synchronize()
    assert rel_err(captured.cpu().numpy(), oracle.apply_hamiltonian(N, M, c[0], h, g)) < 1e-12
    assert all(torch.equal(o, want[1]) for o in out)
    graph2 = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph2):
        sp.apply_hamiltonian(inplace, inplace, torch.cuda.current_stream())
    graph2.replay()
    torch.cuda.synchronize()
    assert torch.equal(inplace, want[2])


def test_solver_above_eight_orbitals(gpu, oracle):
    """its own Space forms the pair matrix alone"""
    from oracle import hermite_orbitals

    N, M, G = 3, 9, 96
    orb, _ = hermite_orbitals(M, G, -9.0, 9.0)
    c = rand_coef(np.random.default_rng(1), oracle.dim(N, M))
    pot = 0.5 * np.linspace(-9, 9, G) ** 2
    dx, dt, gi = 18.0 / (G - 1), 1e-3, 0.2
    s = gpu.Solver(N, M, G, -9.0, 9.0, dt, True, rk_order=4, lanczos_iter=4)
    s.set_potential(pot)
    s.set_interaction(gi)
    s.set_state(orb, c)
    r1, r2, ri = oracle.sync_density_matrices(N, M, c)
    st = {"orb": orb.copy(), "coef": c.copy(), "hob": np.zeros((M, M), complex),
          "hint": np.zeros(M ** 4, complex), "rho1": np.ascontiguousarray(r1),
          "rho2": np.ascontiguousarray(r2), "rinv": np.ascontiguousarray(ri)}
    for _ in range(2):
        s.step(1)
        oracle.propagate_step(st, N, dx, dt, -0.5, 0.0, gi, True, True, 4, 4, pot)
    got = s.get()
    for k in ("orb", "coef", "rho1"):
        assert rel_err(got[k], st[k]) < 1e-10, k

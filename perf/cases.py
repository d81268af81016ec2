"""Measured cases: what a user of the framework has it do, through its public entry points.

A case names a kind of call and its sizes:

  hc       Space.apply_hamiltonian: one H.C product on device vectors.  What a
           caller with an eigensolver or integrator of its own calls, and what
           the short iterative Lanczos step is made of.
  dens     Space.density_matrices: rho1 and rho2 of one coefficient vector.
  step     Step.launch: one configurational step (Lanczos + rho1 + rho2) as a
           replayed CUDA graph, real or imaginary time.
  solver   Solver.step: whole MCTDHB steps (orbitals, matrices, coefficients,
           densities) of one system, `steps` of them between two looks.
  batch    Batch.step + Batch.fetch: a mix of systems of uneven size advanced
           `steps` steps together, and every result read back to host memory.
  dropin   DropIn.propagate_coef_sil: the reference's own C entry point on host
           buffers.

Sizes follow the workloads of bench.py (N=10 M=4 relaxation, N=30 M=8 quench,
N=100 M=6 at the memory edge, the mix N in 10..60, M in 3..6), the tests' sizes
(M up to 12) and generic ones between them.  All arithmetic is complex128.
`exact` restates every path in plain torch, from the formulas.
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "1d-mctdhb_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

C128 = torch.complex128


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # the smallest product a user calls: one small system in a loop of its own
        {"name": "hc_n10_m4", "kind": "hc", "n": 10, "m": 4},
        # an ordinary product, an odd number of orbitals
        {"name": "hc_n25_m7", "kind": "hc", "n": 25, "m": 7},
        # the product of the large quench, 10.3 M configurations
        {"name": "hc_n30_m8", "kind": "hc", "n": 30, "m": 8},
        # the largest product: 96.6 M configurations, 1.5 GB a vector
        {"name": "hc_n100_m6", "kind": "hc", "n": 100, "m": 6},
        # densities of the largest system of the mix
        {"name": "dens_n60_m6", "kind": "dens", "n": 60, "m": 6},
        # few bosons in many orbitals: strongly correlated systems
        {"name": "step_n8_m10", "kind": "step", "n": 8, "m": 10, "lanczos": 5, "imag": False},
        # one coefficient step of the large quench
        {"name": "step_n30_m8", "kind": "step", "n": 30, "m": 8, "lanczos": 6, "imag": False},
        # the plain relaxation: a small system, where latency counts
        {"name": "relax_n10_m4", "kind": "solver", "n": 10, "m": 4, "grid": 256, "imag": True,
         "rk": 5, "lanczos": 5, "der": 302, "split": False, "steps": 4},
        # a quench with the reference's default derivatives and the split step
        {"name": "quench_n16_m6", "kind": "solver", "n": 16, "m": 6, "grid": 1024, "imag": False,
         "rk": 4, "lanczos": 6, "der": 300, "split": True, "steps": 2},
        # many small systems together: a parameter scan of few-boson traps
        {"name": "batch_small", "kind": "batch", "jobs": 32, "nmin": 10, "nmax": 24, "mmin": 3,
         "mmax": 4, "real": 0.3, "lanczos": 5, "steps": 4},
        # the mix of uneven relaxations and quenches that the engine serves
        {"name": "batch_mix", "kind": "batch", "jobs": 48, "nmin": 10, "nmax": 60, "mmin": 3,
         "mmax": 6, "real": 0.3, "lanczos": 5, "steps": 4},
        # a program of the reference that links this library: host buffers
        {"name": "dropin_n20_m6", "kind": "dropin", "n": 20, "m": 6, "lanczos": 5, "imag": True},
    ]


def dim(n, m):
    return math.comb(n + m - 1, m - 1)


def draw(rng):
    kind = rng.choice(["hc", "hc", "dens", "step", "solver", "batch", "dropin"])
    imag = rng.random() < 0.6
    if kind in ("hc", "dens", "step"):
        # orbitals 2..8, now and then 9..12; the size spread over its logarithm
        m = rng.randint(2, 8) if rng.random() < 0.8 else rng.randint(9, 12)
        top = {"hc": 2.0e7, "dens": 2.0e7, "step": 6.0e6}[kind] if m <= 8 else 6.0e4
        want = math.exp(rng.uniform(math.log(60.0), math.log(top)))
        n = 3
        while n < 400 and dim(n + 1, m) <= want:
            n += 1
        case = {"kind": kind, "n": n, "m": m}
        if kind == "step":
            case.update(lanczos=rng.randint(3, 8), imag=imag)
        return case
    if kind == "solver":
        m = rng.randint(2, 7)
        want = math.exp(rng.uniform(math.log(30.0), math.log(1.0e5)))
        n = 2
        while n < 200 and dim(n + 1, m) <= want:
            n += 1
        der = rng.choice([300, 301, 302])
        # explicit Runge-Kutta of the whole orbital equation is for relaxations
        # with finite differences; the other derivatives come with the split step
        split = der != 302 or rng.random() < 0.3
        return {"kind": kind, "n": n, "m": m, "grid": rng.randint(101, 1025), "imag": imag,
                "rk": rng.choice([4, 5]), "lanczos": rng.randint(3, 8), "der": der,
                "split": split, "steps": rng.randint(1, 4)}
    if kind == "batch":
        mmin = rng.randint(2, 4)
        nmin = rng.randint(4, 12)
        return {"kind": kind, "jobs": rng.randint(3, 40), "nmin": nmin,
                "nmax": nmin + rng.randint(2, 30), "mmin": mmin, "mmax": mmin + rng.randint(0, 2),
                "real": rng.choice([0.0, 0.3, 1.0]), "lanczos": rng.randint(4, 6),
                "steps": rng.randint(1, 5)}
    m = rng.randint(3, 6)
    want = math.exp(rng.uniform(math.log(100.0), math.log(6.0e4)))
    n = 3
    while n < 80 and dim(n + 1, m) <= want:
        n += 1
    return {"kind": kind, "n": n, "m": m, "lanczos": rng.randint(3, 8), "imag": imag}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def simpson(n, h):
    """composite Simpson weights, 3/8 rule on the last four points for an even n"""
    w = np.zeros(n)
    odd = n if n % 2 else n - 3
    for i in range(0, odd - 2, 2):
        w[i:i + 3] += np.array([1.0, 4.0, 1.0]) * h / 3
    if n % 2 == 0:
        w[n - 4:] += np.array([1.0, 3.0, 3.0, 1.0]) * 3 * h / 8
    return w


def oscillator_orbitals(m, grid, xi, xf):
    """the m lowest harmonic-oscillator functions, orthonormal in the Simpson metric"""
    x = np.linspace(xi, xf, grid)
    w = simpson(grid, x[1] - x[0])
    f = np.zeros((m, grid), np.complex128)
    prev, cur = np.zeros(grid), np.exp(-x ** 2 / 2)
    for k in range(m):
        f[k] = cur
        prev, cur = cur, (math.sqrt(2.0) * x * cur - math.sqrt(k) * prev) / math.sqrt(k + 1)
    for i in range(m):
        for j in range(i):
            f[i] -= np.sum(w * f[j].conj() * f[i]) * f[j]
        f[i] /= math.sqrt(np.sum(w * np.abs(f[i]) ** 2))
    return f


def trap(double_well, grid, xi, xf):
    x = np.linspace(xi, xf, grid)
    return 0.5 * x ** 2 + (4.0 * np.exp(-x ** 2 / 0.5) if double_well else 0.0)


def orbital_matrices(rng, m, g):
    """h_kl and g_ksql of m oscillator functions in a random unitary basis, as
    complex orbitals have them in a running propagation"""
    grid, xi, xf = 161, -9.0, 9.0
    q, r = np.linalg.qr(rng.normal(size=(m, m)) + 1j * rng.normal(size=(m, m)))
    u = q * (np.diag(r) / np.abs(np.diag(r)))
    f = u @ oscillator_orbitals(m, grid, xi, xf)
    w = simpson(grid, (xf - xi) / (grid - 1))
    levels = np.arange(m) + 0.5
    h = u.conj() @ np.diag(levels) @ u.T
    h = (h + h.conj().T) / 2
    pair = (f[:, None, :] * f[None, :, :]).reshape(m * m, grid)  # symmetric in its indices
    t = g * (pair.conj() * w) @ pair.T  # [k s][q l]
    hint = t.reshape(m, m, m, m).transpose(3, 2, 1, 0).reshape(-1)  # k + sM + qM^2 + lM^3
    return h, np.ascontiguousarray(hint)


def coefficients(count, seed, device):
    gen = torch.Generator(device=device)
    gen.manual_seed(seed)
    c = torch.randn(count, 2, dtype=torch.float64, device=device, generator=gen)
    return torch.view_as_complex(c)


def space_inputs(case, seed):
    n, m = case["n"], case["m"]
    rng = np.random.default_rng([seed, n, m])
    h, hint = orbital_matrices(rng, m, 0.1)
    c = coefficients(dim(n, m), seed, _device())
    c /= torch.linalg.vector_norm(c)
    return h, hint, c


def time_step(case):
    return 0.01 if case["imag"] else 0.005


def system(rng, m, grid, imag, der, split):
    """trap, interaction and time step of one system on [-10, 10]; with finite
    differences and explicit Runge-Kutta dt stays in the stability region"""
    xi, xf = -10.0, 10.0
    pot = trap(rng.random() < 0.5, grid, xi, xf)
    g = float(rng.uniform(0.01, 1.0))
    dt = 0.01 if imag else 0.005
    if not split:
        dx = (xf - xi) / (grid - 1)
        dt = min(dt, 1.5 / (2.0 / dx ** 2 + float(np.max(pot))))
    return {"xi": xi, "xf": xf, "pot": pot, "g": g, "dt": dt,
            "orbitals": oscillator_orbitals(m, grid, xi, xf)}


def solver_inputs(case, seed):
    rng = np.random.default_rng([seed, case["n"], case["m"]])
    s = system(rng, case["m"], case["grid"], case["imag"], case["der"], case["split"])
    c = rng.normal(size=(dim(case["n"], case["m"]), 2)) @ np.array([1.0, 1.0j])
    s["coef"] = c / np.linalg.norm(c)
    s.update(n=case["n"], m=case["m"], grid=case["grid"], imag=case["imag"], rk=case["rk"],
             lanczos=case["lanczos"], der=case["der"], split=case["split"])
    return s


def batch_inputs(case, seed):
    """the systems of a mix: sizes from the case alone, states from the seed"""
    sizes = np.random.default_rng([case["jobs"], case["nmin"], case["nmax"], case["mmin"],
                                   case["mmax"]])
    rng = np.random.default_rng(seed)
    jobs = []
    for _ in range(case["jobs"]):
        n = int(sizes.integers(case["nmin"], case["nmax"] + 1))
        m = int(sizes.integers(case["mmin"], case["mmax"] + 1))
        grid = int(sizes.choice([256, 512, 1024]))
        imag = bool(sizes.random() >= case["real"])
        s = system(rng, m, grid, imag, 302, False)
        s.update(n=n, m=m, grid=grid, imag=imag, rk=5, lanczos=case["lanczos"], der=302,
                 split=False)
        jobs.append(s)
    total = sum(dim(s["n"], s["m"]) for s in jobs)
    c = coefficients(total, seed, _device()).cpu().numpy()
    at = 0
    for s in jobs:
        k = dim(s["n"], s["m"])
        s["coef"] = c[at:at + k] / np.linalg.norm(c[at:at + k])
        at += k
    return jobs


# ---------------------------------------------------------------------------
# the framework's calls
# ---------------------------------------------------------------------------
class _Multiconf:
    """the index tables of the drop-in entry points, given back at the end"""

    def __init__(self, dropin, n, m):
        self.dropin, self.mc = dropin, dropin.multiconf(n, m)

    def __del__(self):
        self.dropin.destroy(self.mc)


class _DeviceArray:
    """complex128 device memory that a handle owns, for torch.as_tensor"""

    def __init__(self, owner, ptr, shape):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": tuple(shape) + (2,), "typestr": "<f8",
                                         "data": (int(ptr), False), "version": 3}


def _view(owner, ptr, shape):
    return torch.view_as_complex(torch.as_tensor(_DeviceArray(owner, ptr, shape), device="cuda"))


def prepare(case, seed):
    import mctdhb_b200 as mb

    kind = case["kind"]
    if kind in ("hc", "dens", "step"):
        n, m = case["n"], case["m"]
        h, hint, c = space_inputs(case, seed)
        sp = mb.Space(n, m)
        sp.set_matrices(torch.from_numpy(h).cuda(), torch.from_numpy(hint).cuda())
        s = {"kind": kind, "space": sp, "coef": c}
        if kind == "hc":
            s["out"] = torch.empty_like(c)
        else:
            s["rho1"] = torch.empty(m, m, dtype=C128, device="cuda")
            s["rho2"] = torch.empty(m ** 4, dtype=C128, device="cuda")
        torch.cuda.synchronize()
        if kind == "step":
            s["step"] = mb.Step(sp, c, s["rho1"], s["rho2"], case["lanczos"], time_step(case),
                                case["imag"])
        return s
    if kind == "solver":
        d = solver_inputs(case, seed)
        sv = mb.Solver(d["n"], d["m"], d["grid"], d["xi"], d["xf"], d["dt"], d["imag"],
                       rk_order=d["rk"], lanczos_iter=d["lanczos"])
        sv.set_derivative(d["der"])
        sv.set_orb_method(31 if d["split"] else 30)
        sv.set_potential(d["pot"])
        sv.set_interaction(d["g"])
        sv.set_state(d["orbitals"], d["coef"])
        lib = mb.load()
        return {"kind": kind, "solver": sv, "steps": case["steps"],
                "coef": _view(sv, lib.mctdhb_solver_device_coef(sv.h), (sv.dim,)),
                "orb": _view(sv, lib.mctdhb_solver_device_orbitals(sv.h), (d["m"], d["grid"]))}
    if kind == "batch":
        jobs = []
        for d in batch_inputs(case, seed):
            jobs.append({"npar": d["n"], "norb": d["m"], "grid_size": d["grid"], "xi": d["xi"],
                         "xf": d["xf"], "periodic": 1, "imagtime": int(d["imag"]),
                         "rk_order": d["rk"], "dt": d["dt"], "g": d["g"],
                         "max_steps": 1 << 30, "energy_tol": 0.0,
                         "check_every": 1 if d["imag"] else 0, "pot": d["pot"],
                         "orbitals": d["orbitals"], "coef": d["coef"]})
        room = sum(mb.Batch.job_bytes(j, case["lanczos"]) for j in jobs)
        b = mb.Batch(len(jobs), room, case["lanczos"])
        slots = [b.admit(j) for j in jobs]
        # results go to pinned host memory, one buffer per field
        sizes = {"orb": [j["norb"] * j["grid_size"] for j in jobs],
                 "coef": [dim(j["npar"], j["norb"]) for j in jobs],
                 "rho1": [j["norb"] ** 2 for j in jobs], "rho2": [j["norb"] ** 4 for j in jobs]}
        host = {k: torch.zeros(sum(v), dtype=C128, pin_memory=True) for k, v in sizes.items()}
        outs = [{} for _ in jobs]
        for k, v in sizes.items():
            at = 0
            for out, count in zip(outs, v):
                out[k] = host[k][at:at + count].numpy()
                at += count
        return {"kind": kind, "batch": b, "slots": slots, "outs": outs, "host": host,
                "steps": case["steps"]}
    d = mb.DropIn()
    h, hint, c = space_inputs(case, seed)
    return {"kind": kind, "dropin": d, "mc": _Multiconf(d, case["n"], case["m"]), "hob": h,
            "hint": hint, "coef": c.cpu().numpy(), "lanczos": case["lanczos"],
            "dt": time_step(case), "imag": case["imag"]}


def run(state):
    kind = state["kind"]
    if kind == "hc":
        state["space"].apply_hamiltonian(state["coef"], state["out"])
        return state["out"]
    if kind == "dens":
        state["space"].density_matrices(state["coef"], state["rho1"], state["rho2"])
        return {"rho1": state["rho1"], "rho2": state["rho2"]}
    if kind == "step":
        state["step"].launch()
        return {k: state[k] for k in ("coef", "rho1", "rho2")}
    if kind == "solver":
        state["solver"].step(state["steps"])
        return {"orb": state["orb"], "coef": state["coef"]}
    if kind == "batch":
        b = state["batch"]
        b.step(state["steps"])
        energy = np.zeros(len(state["slots"]))
        for i, (slot, out) in enumerate(zip(state["slots"], state["outs"])):
            energy[i] = b.fetch(slot, out)["energy"]
        return dict(state["host"], energy=energy)
    cnext, coef, diag, offd = state["dropin"].propagate_coef_sil(
        state["mc"].mc, state["hob"], state["hint"], state["coef"], state["lanczos"], state["dt"],
        state["imag"])
    return {"cnext": cnext, "coef": coef, "diag": diag, "offd": offd}


# ---------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------
def _hc_flops(n, m):
    """one complex multiply-add (8) per entry of the pair operator and row of
    the (N-2)-boson space, and one real-by-complex one (4) per pair and row
    each way"""
    p = m * (m + 1) / 2
    return 8.0 * dim(n - 2, m) * p * p + 4.0 * p * (dim(n - 2, m) + dim(n, m))


def _dens_flops(n, m):
    p = m * (m + 1) / 2
    return 8.0 * dim(n - 2, m) * p * (p + 1) / 2


def _lanczos_work(n, m, k):
    """k products, full reorthogonalisation, the combination; the coefficients
    are read and written once"""
    nc = dim(n, m)
    flops = k * _hc_flops(n, m) + nc * (8.0 * k + 8.0 * k * (k - 1) + 8.0 * k)
    return {"bytes": 32.0 * nc, "flops": flops}


def _orbital_flops(m, grid, rk, der, split):
    stages = {2: 2, 4: 4, 5: 6}[rk]
    rhs = grid * (8.0 * m * (m ** 3 + m ** 2 + m) + 16.0 * m * m)
    lin = 40.0 * m * grid * math.log2(grid) if der != 302 else 20.0 * m * grid
    linear = 2 * lin if split else stages * lin
    return stages * (rhs + 16.0 * m * grid) + linear + 8.0 * grid * m ** 4


def _system_work(n, m, grid, rk, lanczos, der, split):
    w = _lanczos_work(n, m, lanczos)
    return {"bytes": w["bytes"] + 32.0 * m * grid,
            "flops": w["flops"] + _dens_flops(n, m) + _orbital_flops(m, grid, rk, der, split)}


def work(case):
    kind = case["kind"]
    if kind == "batch":
        total = {"bytes": 0.0, "flops": 0.0}
        for d in _batch_sizes(case):
            w = _system_work(d["n"], d["m"], d["grid"], 5, case["lanczos"], 302, False)
            total["bytes"] += w["bytes"]
            total["flops"] += w["flops"] * case["steps"]
        return total
    n, m = case["n"], case["m"]
    if kind == "hc":
        return {"bytes": 32.0 * dim(n, m) + 16.0 * m ** 4, "flops": _hc_flops(n, m)}
    if kind == "dens":
        return {"bytes": 16.0 * dim(n, m) + 16.0 * m ** 4, "flops": _dens_flops(n, m)}
    if kind == "solver":
        w = _system_work(n, m, case["grid"], case["rk"], case["lanczos"], case["der"],
                         case["split"])
        return {"bytes": w["bytes"], "flops": w["flops"] * case["steps"]}
    w = _lanczos_work(n, m, case["lanczos"])
    if kind == "step":
        w["flops"] += _dens_flops(n, m)
        w["bytes"] += 16.0 * m ** 4
    return w


def _batch_sizes(case):
    sizes = np.random.default_rng([case["jobs"], case["nmin"], case["nmax"], case["mmin"],
                                   case["mmax"]])
    out = []
    for _ in range(case["jobs"]):
        n = int(sizes.integers(case["nmin"], case["nmax"] + 1))
        m = int(sizes.integers(case["mmin"], case["mmax"] + 1))
        grid = int(sizes.choice([256, 512, 1024]))
        sizes.random()
        out.append({"n": n, "m": m, "grid": grid})
    return out


# ---------------------------------------------------------------------------
# the same values in plain torch
# ---------------------------------------------------------------------------
class PairSpace:
    """N bosons in M orbitals through the states with two bosons removed: row r
    of the (N-2)-boson space and pair (q, l) hold
    A_r(q, l) = <r|a_q a_l|C> = sqrt((n_q + 1)(n_l + 1 + [q = l])) C[rank(n + e_q + e_l)],
    configurations ranked as D - 1 - sum_x binom(L_x + x, x + 1) with
    L_x = n_0 + ... + n_x."""

    CHUNK = 1 << 21

    def __init__(self, n, m, device):
        self.n, self.m, self.device = n, m, device
        self.dim, self.dim2 = dim(n, m), dim(n - 2, m)
        self.pairs = [(q, l) for q in range(m) for l in range(q, m)]
        self.table = torch.tensor([[math.comb(L + x, x + 1) for L in range(n + 1)]
                                   for x in range(m - 1)], dtype=torch.int64, device=device)

    def chunks(self):
        return [(a, min(a + self.CHUNK, self.dim2)) for a in range(0, self.dim2, self.CHUNK)]

    def rows(self, a, b):
        """occupations and cumulative occupations of the rows a..b-1"""
        rest = self.dim2 - 1 - torch.arange(a, b, device=self.device)
        above = torch.full_like(rest, self.n - 2)
        occ, cum = [None] * self.m, [None] * (self.m - 1)
        for x in range(self.m - 2, -1, -1):
            level = torch.searchsorted(self.table[x], rest, right=True) - 1
            # binom(x, x + 1) = 0 at L = 0 only, so the largest level is unique
            level = torch.minimum(level, above)
            rest = rest - self.table[x][level]
            occ[x + 1], cum[x], above = above - level, level, level
        occ[0] = above
        # weights of each orbital's level with 0, 1 and 2 bosons more
        weight = [[self.table[x][cum[x] + d] for d in range(3)] for x in range(self.m - 1)]
        return occ, weight

    def target(self, occ, weight, q, l):
        """rank of the row with a boson more in q and in l, and the factor"""
        s = 0
        for x in range(self.m - 1):
            s = s + weight[x][int(x >= q) + int(x >= l)]
        f = (occ[q] + 1) * (occ[l] + 1 + int(q == l))
        return self.dim - 1 - s, f.to(torch.float64).sqrt()

    def removed(self, c, a, b):
        """A for the rows a..b-1 (pairs x rows), with its targets and factors"""
        occ, weight = self.rows(a, b)
        to, fac, amp = [], [], []
        for q, l in self.pairs:
            j, f = self.target(occ, weight, q, l)
            to.append(j)
            fac.append(f)
            amp.append(c[j] * f)
        return torch.stack(amp), to, fac

    def operator(self, h, hint):
        """H = sum W[P][Q] a+_P a_Q: the interaction with the multiplicities of
        the pairs, the one-body part spread over a spectator boson"""
        m, at = self.m, {p: i for i, p in enumerate(self.pairs)}
        g = hint.reshape(m, m, m, m)  # [l][q][s][k]
        w = np.zeros((len(self.pairs),) * 2, np.complex128)
        for i, (k, s) in enumerate(self.pairs):
            for j, (q, l) in enumerate(self.pairs):
                w[i, j] = 0.5 * (1 + (k != s)) * (1 + (q != l)) * g[l, q, s, k]
        for k in range(m):
            for q in range(m):
                for x in range(m):
                    w[at[tuple(sorted((k, x)))], at[tuple(sorted((q, x)))]] += h[k, q] / (self.n - 1)
        return torch.from_numpy(w).to(self.device)

    def apply(self, w, c):
        out = torch.zeros_like(c)
        for a, b in self.chunks():
            amp, to, fac = self.removed(c, a, b)
            y = w @ amp
            for p in range(len(self.pairs)):
                out[to[p]] += y[p] * fac[p]
        return out

    def densities(self, c):
        m = self.m
        gram = 0
        for a, b in self.chunks():
            amp, _, _ = self.removed(c, a, b)
            gram = gram + amp.conj() @ amp.T
        at = {p: i for i, p in enumerate(self.pairs)}
        idx = torch.tensor([[at[tuple(sorted((k, s)))] for s in range(m)] for k in range(m)],
                           device=self.device)
        full = gram[idx.reshape(-1)][:, idx.reshape(-1)].reshape(m, m, m, m)  # [k][s][q][l]
        rho1 = torch.einsum("kssl->kl", full) / (self.n - 1)
        return rho1, full.permute(3, 2, 1, 0).reshape(-1).contiguous()

    def lanczos_step(self, w, c, count, dt, imag):
        """short iterative Lanczos with full reorthogonalisation: the
        combination before any renormalisation, and the recurrence's numbers"""
        vec, diag, offd = [c], [], []
        out = self.apply(w, c)
        diag.append(torch.vdot(c, out))
        biggest = 0.0
        for i in range(count - 1):
            out = out - diag[i] * vec[i]
            over = [torch.vdot(v, out) for v in vec]
            for v, o in zip(vec, over):
                out = out - o * v
            beta = float(torch.linalg.vector_norm(out))
            biggest = max(biggest, beta)
            offd.append(beta)
            if beta == 0.0 or beta / biggest < 1e-14:
                break
            vec.append(out / beta)
            out = self.apply(w, vec[-1]) - beta * vec[i]
            diag.append(torch.vdot(vec[-1], out))
        k = len(vec)
        d = np.array([complex(x) for x in diag])
        t = np.diag(d[:k].real) + np.diag(offd[:k - 1], 1) + np.diag(offd[:k - 1], -1)
        e, u = np.linalg.eigh(t)
        y = u @ (np.exp((-dt if imag else -1j * dt) * e) * u[0])
        new = sum(complex(yk) * v for yk, v in zip(y, vec))
        return new, d, np.array(offd)


class PlainSystem:
    """one MCTDHB system: orbitals, coefficients and their matrices"""

    def __init__(self, d, device):
        self.d, self.device = d, device
        self.sp = PairSpace(d["n"], d["m"], device)
        to = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(device)  # noqa: E731
        self.orb, self.coef, self.pot = to(d["orbitals"]), to(d["coef"]), to(d["pot"])
        self.dx = (d["xf"] - d["xi"]) / (d["grid"] - 1)
        self.w = to(simpson(d["grid"], self.dx))
        self.tf = -1j if d["imag"] else 1.0
        self.sync_densities()

    def sync_densities(self):
        r1, self.rho2 = self.sp.densities(self.coef)
        e, u = torch.linalg.eigh(r1)
        if float(e[0] / e[-1]) < 1e-9:  # regularisation
            x = float(e[-1]) * 1e-9
            r1 = r1 + (u * (x * torch.exp(-e / x))) @ u.conj().T
        self.rho1, self.rinv = r1, torch.linalg.inv(r1)

    def matrices(self, f):
        """h_kl (fourth-order periodic first derivative) and g_ksql"""
        p = f[:, :-1]
        r = 1.0 / (12 * self.dx)
        df = (torch.roll(p, 2, 1) - torch.roll(p, -2, 1)
              + 8 * (torch.roll(p, -1, 1) - torch.roll(p, 1, 1))) * r
        df = torch.cat([df, df[:, :1]], 1)
        h = 0.5 * (df.conj() * self.w) @ df.T + (f.conj() * (self.w * self.pot)) @ f.T
        h = (h + h.conj().T) / 2
        m = f.shape[0]
        pair = (f[:, None] * f[None]).reshape(m * m, -1)
        g = self.d["g"] * (pair.conj() * self.w) @ pair.T
        return h.cpu().numpy(), g.reshape(m, m, m, m).permute(3, 2, 1, 0).reshape(-1).cpu().numpy()

    def interacting(self, q, f):
        """sum_s conj(f_s) sum_{q,l} Q[k][s, q, l] f_q f_l"""
        m = f.shape[0]
        t = (q.reshape(-1, m) @ f).reshape(m, m, m, -1)  # [k][l][s]
        return torch.einsum("klsx,lx,sx->kx", t, f, f.conj())

    def freq2(self):
        n = self.d["grid"] - 1
        k = torch.fft.fftfreq(n, self.dx, dtype=torch.float64).to(self.device)
        return (2 * math.pi * k) ** 2

    def linear(self, f):
        if self.d["der"] == 302:
            p = f[:, :-1]
            lap = (torch.roll(p, 1, 1) + torch.roll(p, -1, 1) - 2 * p) / self.dx ** 2
        else:
            lap = -torch.fft.ifft(self.freq2() * torch.fft.fft(f[:, :-1]))
        lin = -0.5 * lap + self.pot[:-1] * f[:, :-1]
        return torch.cat([lin, lin[:, :1]], 1)

    def rhs(self, q, f):
        hf = self.linear(f) + self.interacting(q, f)
        p = (f.conj() * self.w) @ hf.T  # [s][k]
        return -1j * self.tf * (hf - p.T @ f)

    def split_rhs(self, q, hb, f):
        return -1j * self.tf * (self.interacting(q, f) - hb @ f + self.pot * f)

    def half(self, f):
        dth = 0.5 * self.d["dt"] * self.tf
        if self.d["der"] == 302:
            n = self.d["grid"] - 1
            c = torch.cos(2 * math.pi * torch.arange(n, device=self.device, dtype=torch.float64) / n)
            t = -0.5 * dth / self.dx ** 2
            mul = (1j - t * (1 - c)) / (1j + t * (1 - c))
        else:
            mul = torch.exp(-1j * dth * 0.5 * self.freq2())
        out = torch.fft.ifft(mul * torch.fft.fft(f[:, :-1]))
        return torch.cat([out, out[:, :1]], 1)

    def runge_kutta(self, rhs, y):
        if self.d["rk"] == 4:
            a = [[], [0.5], [0, 0.5], [0, 0, 1.0]]
            b = [1 / 6, 2 / 6, 2 / 6, 1 / 6]
        else:
            a = [[], [0.25], [0.125, 0.125], [0, -0.5, 1.0], [3 / 16, 0, 0, 9 / 16],
                 [-3 / 7, 2 / 7, 12 / 7, -12 / 7, 8 / 7]]
            b = [7 / 90, 0, 32 / 90, 12 / 90, 32 / 90, 7 / 90]
        k = []
        for row in a:
            k.append(rhs(y + self.d["dt"] * sum(c * s for c, s in zip(row, k) if c)
                         if row else y))
        return y + self.d["dt"] * sum(c * s for c, s in zip(b, k) if c)

    def gram_schmidt(self, f):
        """the overlap is followed point by point as the orbital is updated"""
        f = f.clone()
        norm = lambda v: v * torch.rsqrt(torch.sum(self.w * v.abs() ** 2))  # noqa: E731
        f[0] = norm(f[0])
        for i in range(1, f.shape[0]):
            for j in range(i):
                over = torch.sum(self.w * f[j].conj() * f[i])
                fac = torch.cumprod(1 - self.w * f[j].abs() ** 2, 0)
                fac = torch.cat([torch.ones_like(fac[:1]), fac[:-1]])
                f[i] = f[i] - over * fac * f[j]
            f[i] = norm(f[i])
        return f

    def wrap(self, f):
        return torch.cat([f[:, :-1], f[:, :1]], 1)

    def step(self):
        d, m = self.d, self.d["m"]
        f = self.wrap(self.orb)
        rho2 = self.rho2.reshape(m, m, m, m)  # [l][q][s][k]
        # as [k][l][s][q], contracted over q first
        q = d["g"] * torch.einsum("ka,lqsa->klsq", self.rinv, rho2)
        q = q.contiguous()
        if d["split"]:
            f = self.half(f)
            h, hint = (torch.from_numpy(x).to(self.device) for x in self.matrices(f))
            g = hint.reshape(m, m, m, m)  # g(j, s, l, q) at j + sM + lM^2 + qM^3
            b = torch.einsum("ka,lqsa,qlsj->kj", self.rinv, rho2, g)
            hb = h.T + b
            f = self.half(self.runge_kutta(lambda y: self.split_rhs(q, hb, y), f))
        else:
            f = self.runge_kutta(lambda y: self.rhs(q, y), f)
        if d["imag"]:
            f = self.gram_schmidt(f)
        self.orb = f = self.wrap(f)
        h, hint = self.matrices(f)
        self.hob, self.hint = h, hint
        c, _, _ = self.sp.lanczos_step(self.sp.operator(h, hint), self.coef, d["lanczos"],
                                       d["dt"], d["imag"])
        self.coef = c / torch.linalg.vector_norm(c) if d["imag"] else c
        self.sync_densities()

    def energy(self):
        m = self.d["m"]
        h = torch.from_numpy(self.hob).to(self.device)
        g = torch.from_numpy(self.hint).to(self.device).reshape(m, m, m, m)
        e = torch.sum(self.rho1 * h)
        # rho2(k, l, s, q) g(k, l, q, s)
        e = e + 0.5 * torch.einsum("qslk,sqlk->", self.rho2.reshape(m, m, m, m), g)
        return float(e.real)


def exact(case, seed):
    kind, device = case["kind"], _device()
    if kind == "solver":
        s = PlainSystem(solver_inputs(case, seed), device)
        for _ in range(case["steps"]):
            s.step()
        return {"orb": s.orb, "coef": s.coef}
    if kind == "batch":
        got = {"orb": [], "coef": [], "rho1": [], "rho2": []}
        energy = []
        for d in batch_inputs(case, seed):
            s = PlainSystem(d, device)
            for _ in range(case["steps"]):
                s.step()
            for k, v in (("orb", s.orb), ("coef", s.coef), ("rho1", s.rho1), ("rho2", s.rho2)):
                got[k].append(v.reshape(-1).cpu())
            energy.append(s.energy())
        return dict({k: torch.cat(v) for k, v in got.items()}, energy=np.array(energy))
    h, hint, c = space_inputs(case, seed)
    sp = PairSpace(case["n"], case["m"], device)
    w = sp.operator(h, hint)
    if kind == "hc":
        return sp.apply(w, c)
    if kind == "dens":
        rho1, rho2 = sp.densities(c)
        return {"rho1": rho1, "rho2": rho2}
    new, diag, offd = sp.lanczos_step(w, c, case["lanczos"], time_step(case), case["imag"])
    if kind == "dropin":
        coef = new / torch.linalg.vector_norm(new) if case["imag"] else new
        pad = lambda v: np.concatenate([v, np.zeros(case["lanczos"] - len(v))])  # noqa: E731
        return {"cnext": new, "coef": coef, "diag": pad(diag), "offd": pad(offd).astype(complex)}
    if case["imag"]:
        new = new / torch.linalg.vector_norm(new)
    rho1, rho2 = sp.densities(new)
    return {"coef": new, "rho1": rho1, "rho2": rho2}

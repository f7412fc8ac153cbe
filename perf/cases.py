"""Performance cases: the work a user of this framework has it do, through its public entry points.

  run     a single run (``Run.run``): a few implicit time steps from a state in hand, with the invariants of every
          step, in FP64 or mixed precision, kinetic or potential preconditioner
  sweep   many uneven runs advanced together (``Batch.step``), the seeded instance table of the benchmark
  apply   one call of the solver class, as an outside Krylov driver makes them: the preconditioned residual
          (``function``) or Jacobian (``jacobian``), or the residual and its norm (``function_norm``)
  gmres   one preconditioned linear solve of a Picard pass (``PETScVlasovSolver.gmres``)
  fields  moments of a distribution, the Poisson solve and the Hamiltonian profile (``Toolbox``, ``PETScPoissonSolver``)
  adjoint the gradient of a loss through one converged step (``Adjoint.step``), the backward direction

Grids are those of the workloads, the tests and the reference's example configurations (64 x 256, 100 x 201,
50 x 101, 201 x 401, 256 x 512, 512 x 1024, 1024 x 2048, 2048 x 8192).  ``draw`` takes sizes from the same ranges,
odd ones among them.  A run or sweep pass starts from the same saved state every time, as a trajectory restarted from
a checkpoint does, so that every pass does the same work.
"""
import math

import numpy as np
import torch

from vivlasov1d_b200 import workloads
from vivlasov1d_b200.adjoint import Adjoint
from vivlasov1d_b200.batch import Batch
from vivlasov1d_b200.run import Run
from vivlasov1d_b200.solver import Grid, PETScPoissonSolver, PETScVlasovSolver, Toolbox

CHARGE = -1.0
TRACED = ("mass", "L2", "energy", "entropy", "field_energy")   # momentum is zero to round-off here


def listed():
    return [
        # linear Landau damping, the smallest workload: many short kernels, latency and launches
        {"name": "run_64x256", "kind": "run", "nx": 64, "nv": 256, "family": "landau", "amp": 0.01, "k": 0.5,
         "vmax": 10.0, "ht": 0.1, "atol": 1e-12, "precision": "fp64", "pc": "tensor_kinetic", "steps": 4},
        # the reference's example grid for Landau damping: neither size a power of two
        {"name": "run_100x201", "kind": "run", "nx": 100, "nv": 201, "family": "landau", "amp": 0.05, "k": 0.5,
         "vmax": 10.0, "ht": 0.1, "atol": 1e-12, "precision": "fp64", "pc": "tensor_kinetic", "steps": 4},
        # a small run with the potential preconditioner, as the reference's weak Jeans example chooses it
        {"name": "run_potential_50x101", "kind": "run", "nx": 50, "nv": 101, "family": "landau", "amp": 0.05,
         "k": 0.5, "vmax": 10.0, "ht": 0.1, "atol": 1e-11, "precision": "fp64", "pc": "tensor_potential", "steps": 2},
        # the nonlinear two-stream instability in FP64, an ordinary single run
        {"name": "run_512x1024", "kind": "run", "nx": 512, "nv": 1024, "family": "twostream", "amp": 0.05, "k": 0.5,
         "vmax": 8.0, "ht": 0.05, "atol": 1e-10, "precision": "fp64", "pc": "tensor_kinetic", "steps": 2},
        # nonlinear Landau damping in mixed precision, the largest single run
        {"name": "run_1024x2048_mixed", "kind": "run", "nx": 1024, "nv": 2048, "family": "landau", "amp": 0.5,
         "k": 0.5, "vmax": 10.0, "ht": 0.05, "atol": 1e-10, "precision": "mixed", "pc": "tensor_kinetic", "steps": 2},
        # the benchmark's sweep: 256 uneven runs, mixed precision
        {"name": "sweep_256_mixed", "kind": "sweep", "count": 256, "precision": "mixed", "steps": 3},
        # a small sweep in FP64: few instances, the slowest one sets the pace
        {"name": "sweep_24_fp64", "kind": "sweep", "count": 24, "precision": "fp64", "steps": 3},
        # the operator of an outside Krylov solver on the largest grid: everything streams through HBM
        {"name": "jacobian_2048x8192", "kind": "apply", "call": "jacobian", "nx": 2048, "nv": 8192,
         "bracket": "arakawaj4"},
        # the preconditioned residual on the reference's Jeans example grid (odd sizes)
        {"name": "function_201x401", "kind": "apply", "call": "function", "nx": 201, "nv": 401,
         "bracket": "arakawaj4"},
        # one linear solve of a medium grid
        {"name": "gmres_256x512", "kind": "gmres", "nx": 256, "nv": 512},
        # the potential of a given distribution at the size of the largest single run
        {"name": "fields_1024x2048", "kind": "fields", "nx": 1024, "nv": 2048},
        # the differentiation workload's grid: one backward step
        {"name": "adjoint_256x512", "kind": "adjoint", "nx": 256, "nv": 512},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _grid(rng, most):
    """nx, nv: half of the draws with nx a power of two (what the x-FFT likes), the others any number."""
    while True:
        if rng.random() < 0.5:
            nx = 2 ** rng.randint(4, 10)
        else:
            nx = _log(rng, 16, 400)
        nv = _log(rng, 48, 2048)
        if nx * nv <= most:
            return nx, nv


def draw(rng):
    kind = rng.choice(["run", "run", "run", "sweep", "apply", "apply", "gmres", "fields", "adjoint"])
    if kind == "run":
        mixed = rng.random() < 0.4
        potential = not mixed and rng.random() < 0.15
        nx, nv = _grid(rng, 20000 if potential else 1 << 20)
        return {"kind": "run", "nx": nx, "nv": nv, "family": rng.choice(["landau", "twostream"]),
                "amp": round(math.exp(rng.uniform(math.log(0.01), math.log(0.3))), 4), "k": 0.5,
                "vmax": 10.0, "ht": rng.choice([0.05, 0.1]), "atol": 1e-11 if nx * nv < 100000 else 1e-10,
                "precision": "mixed" if mixed else "fp64", "pc": "tensor_potential" if potential else "tensor_kinetic",
                "steps": rng.randint(2, 4)}
    if kind == "sweep":
        return {"kind": "sweep", "count": _log(rng, 4, 64), "precision": rng.choice(["mixed", "fp64"]),
                "steps": rng.randint(2, 4)}
    if kind == "apply":
        nx, nv = _grid(rng, 1 << 20)
        return {"kind": "apply", "call": rng.choice(["jacobian", "function", "function_norm"]), "nx": nx, "nv": nv,
                "bracket": rng.choice(["arakawaj4", "arakawaj4", "arakawaj1", "arakawaj2"])}
    nx, nv = _grid(rng, 1 << 18 if kind == "adjoint" else 1 << 20)
    return {"kind": kind, "nx": nx, "nv": nv}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _rand(shape, gen):
    return torch.rand(shape, generator=gen, dtype=torch.float64, device="cuda")


def _axes(nx, nv, L, vmax):
    x = torch.arange(nx, dtype=torch.float64, device="cuda") * (L / nx)
    v = -vmax + torch.arange(nv, dtype=torch.float64, device="cuda") * (2 * vmax / (nv - 1))
    return x, v


def _profile(nx, L, k, amp, gen):
    """1 + amp cos(k x + p1) and a few weaker harmonics of random phase."""
    x = torch.arange(nx, dtype=torch.float64, device="cuda") * (L / nx)
    w = torch.tensor([1.0, 0.1, 0.03], dtype=torch.float64, device="cuda") * (0.9 + 0.2 * _rand((3,), gen))
    ph = 2 * math.pi * _rand((3,), gen)
    m = torch.arange(1, 4, dtype=torch.float64, device="cuda")
    return 1.0 + amp * (w[:, None] * torch.cos(m[:, None] * k * x + ph[:, None])).sum(0)


def _distribution(family, nx, nv, L, vmax, k, amp, gen):
    """(nv, nx): a perturbed Maxwellian, two-stream or bump-on-tail equilibrium, zero on the two rows at each v end."""
    _, v = _axes(nx, nv, L, vmax)
    m = torch.exp(-v ** 2 / 2) / math.sqrt(2 * math.pi)
    if family == "twostream":
        m = v ** 2 * m
    elif family == "bump_on_tail":
        m = 0.9 * m + 0.2 * torch.exp(-(v - 4.5) ** 2 / 0.5) / math.sqrt(2 * math.pi)
    f = m[:, None] * _profile(nx, L, k, amp, gen)[None, :]
    f[:2] = 0.0
    f[-2:] = 0.0
    return f


def _length(k):
    return 2 * math.pi / k


def _run_config(nx, nv, L, vmax, ht, atol, pc="tensor_kinetic", rtol=1e-4):
    cfg = workloads.config(nx, nv, L, -vmax, vmax, ht, ksp_rtol=rtol, snes_atol=atol)
    cfg["solver"]["preconditioner_scheme"] = pc
    return cfg


def _sweep_specs(case):
    return workloads.sweep_specs(case["count"])


def _sweep_field(s, gen):
    return _distribution(s["family"], s["nx"], s["nv"], s["L"], 10.0, s["k"], s["amp"], gen)


def _apply_fields(case, seed):
    """F, Fh and the h1 profiles of the current and the previous level; X a Krylov vector."""
    nx, nv, gen = case["nx"], case["nv"], _gen(seed)
    L = 4 * math.pi
    F = _distribution("landau", nx, nv, L, 8.0, 0.5, 0.2, gen)
    Fh = F * (1.0 + 0.01 * (_rand((nv, nx), gen) - 0.5))
    X = 2.0 * _rand((nv, nx), gen) - 1.0
    h1p, h1h = (0.1 * (_profile(nx, L, 0.5, 1.0, gen) - 1.0) for _ in range(2))
    return F, Fh, X, h1p, h1h


def prepare(case, seed):
    kind = case["kind"]
    gen = _gen(seed)
    if kind == "run":
        L = _length(case["k"])
        f0 = _distribution(case["family"], case["nx"], case["nv"], L, case["vmax"], case["k"], case["amp"], gen)
        run = Run(_run_config(case["nx"], case["nv"], L, case["vmax"], case["ht"], case["atol"], case["pc"]), f0=f0,
                  precision=case["precision"])
        return {"case": case, "run": run, "start": run.fc.clone()}
    if kind == "sweep":
        runs = []
        for s in _sweep_specs(case):
            runs.append(Run(_run_config(s["nx"], s["nv"], s["L"], 10.0, 0.1, 1e-12), f0=_sweep_field(s, gen),
                            precision=case["precision"]))
        live = [t for r in runs for t in (r.fc, r.pc_int, r.h1c)]
        return {"case": case, "runs": runs, "batch": Batch(runs), "live": live, "start": [t.clone() for t in live]}
    if kind == "fields":
        grid = Grid(case["nx"], case["nv"], 4 * math.pi, 10.0, ht=0.05)
        F = _distribution("bump_on_tail", case["nx"], case["nv"], 4 * math.pi, 10.0, 0.5, 0.5, gen)
        out = [grid.xvec() for _ in range(6)]
        return {"case": case, "toolbox": Toolbox(grid), "poisson": PETScPoissonSolver(None, grid=grid, charge=CHARGE),
                "F": F, "out": out}
    if kind == "adjoint":
        L = 4 * math.pi
        f0 = _distribution("landau", case["nx"], case["nv"], L, 10.0, 0.5, 0.1, gen)
        run = Run(_run_config(case["nx"], case["nv"], L, 10.0, 0.1, 1e-11, rtol=1e-8), f0=f0)
        f = run.fc.clone()
        run.step()
        gF = 2.0 * _rand((case["nv"], case["nx"]), gen) - 1.0
        return {"case": case, "adjoint": Adjoint(run), "F": run.fc.clone(), "f": f, "gF": gF}
    F, Fh, X, h1p, h1h = _apply_fields(case, seed)
    grid = Grid(case["nx"], case["nv"], 4 * math.pi, 8.0, ht=0.05)
    config = {"poisson_bracket": case.get("bracket", "arakawaj4"), "preconditioner": "tensor_kinetic"}
    solver = PETScVlasovSolver(config, None, None, grid, None, h1p, h1h, None, None, None, charge=CHARGE)
    solver.update_history(Fh)
    solver.update_previous()
    return {"case": case, "solver": solver, "F": F, "X": X, "Y": grid.field()}


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _state(run):
    return {"f": run.fc, "phi": run.pc_int, "n": run.N, "u": run.U, "e": run.E}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "run":
        r = state["run"]
        r.fc.copy_(state["start"])
        r.calculate_moments()
        hist = r.run(case["steps"], invariants=True)
        r.reports.clear()
        out = _state(r)
        for name in TRACED:
            out[name] = np.array([h["invariants"][name] for h in hist])
        return out
    if kind == "sweep":
        torch._foreach_copy_(state["live"], state["start"])
        for _ in range(case["steps"]):
            state["batch"].step()
        return {"f": torch.cat([r.fc.view(-1) for r in state["runs"]]),
                "phi": torch.cat([r.pc_int for r in state["runs"]])}
    if kind == "fields":
        n, u, e, a, phi, h1 = state["out"]
        state["toolbox"].compute_moments(state["F"], n, u, e, a)
        state["poisson"].solve(n, phi)
        state["toolbox"].potential_to_hamiltonian(phi, h1)
        return {"n": n, "u": u, "e": e, "a": a, "phi": phi, "h1": h1}
    if kind == "adjoint":
        return state["adjoint"].step(state["F"], state["f"], state["gF"])
    s, Y = state["solver"], state["Y"]
    if kind == "gmres":
        s.gmres(state["X"], Y, rtol=1e-10)
        return Y
    if case["call"] == "jacobian":
        s.jacobian(state["X"], Y)
        return Y
    if case["call"] == "function":
        s.function(state["F"], Y)
        return Y
    return {"norm": s.function_norm(state["F"], Y), "Y": Y}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    """Inputs read once and outputs written once; flops of one bracket residual, and of one FFT pair and tridiagonal
    solve where the path preconditions (an iterative path needs them at least once a step)."""
    kind = case["kind"]
    if kind == "sweep":
        sizes, steps = [(s["nx"], s["nv"]) for s in _sweep_specs(case)], case["steps"]
    else:
        sizes, steps = [(case["nx"], case["nv"])], case.get("steps", 1)
    byts = flops = 0.0
    for nx, nv in sizes:
        c = nx * nv
        pc = c * (5.0 * math.log2(nx) + 10.0)
        if kind in ("run", "sweep"):
            byts += 16.0 * c
            flops += steps * (c * 2 * 25.0 + pc)
        elif kind == "fields":
            byts += 8.0 * c
            flops += 6.0 * c
        elif kind == "adjoint":
            byts += 32.0 * c
            flops += c * 2 * 25.0 + pc
        elif kind == "gmres":
            byts += 16.0 * c
            flops += c * 25.0 + pc
        elif case["call"] == "jacobian":
            byts += 16.0 * c
            flops += c * 25.0 + pc
        else:
            byts += 24.0 * c
            flops += c * 25.0 + (pc if case["call"] == "function" else 0.0)
    return {"bytes": byts, "flops": flops}


# ---------------------------------------------------------------------------
# the same in plain 64-bit torch
# ---------------------------------------------------------------------------
class _Model:
    """The discrete equations on (nv, nx) tensors: Arakawa brackets, moments, the CFD4 Poisson solve."""

    def __init__(self, nx, nv, L, vmax, ht, bracket="arakawaj4"):
        self.nx, self.nv, self.ht, self.bracket = nx, nv, ht, bracket
        self.hx, self.hv = L / nx, 2 * vmax / (nv - 1)
        _, self.v = _axes(nx, nv, L, vmax)
        self.h0 = 0.5 * self.v ** 2

    def brk(self, f, h):
        """[f, h] on the rows 2 <= j < nv-2, zero on the others."""
        nv = self.nv

        def s(a, i, j):
            return torch.roll(a, -i, 1)[2 + j:nv - 2 + j]

        j1 = (s(f, 1, 0) - s(f, -1, 0)) * (s(h, 0, 1) - s(h, 0, -1)) \
            - (s(f, 0, 1) - s(f, 0, -1)) * (s(h, 1, 0) - s(h, -1, 0)) \
            + s(f, 1, 0) * (s(h, 1, 1) - s(h, 1, -1)) - s(f, -1, 0) * (s(h, -1, 1) - s(h, -1, -1)) \
            - s(f, 0, 1) * (s(h, 1, 1) - s(h, -1, 1)) + s(f, 0, -1) * (s(h, 1, -1) - s(h, -1, -1)) \
            + s(f, 1, 1) * (s(h, 0, 1) - s(h, 1, 0)) - s(f, -1, -1) * (s(h, -1, 0) - s(h, 0, -1)) \
            - s(f, -1, 1) * (s(h, 0, 1) - s(h, -1, 0)) + s(f, 1, -1) * (s(h, 1, 0) - s(h, 0, -1))
        j2 = (s(f, 1, 1) - s(f, -1, -1)) * (s(h, -1, 1) - s(h, 1, -1)) \
            - (s(f, -1, 1) - s(f, 1, -1)) * (s(h, 1, 1) - s(h, -1, -1)) \
            + s(f, 2, 0) * (s(h, 1, 1) - s(h, 1, -1)) - s(f, -2, 0) * (s(h, -1, 1) - s(h, -1, -1)) \
            - s(f, 0, 2) * (s(h, 1, 1) - s(h, -1, 1)) + s(f, 0, -2) * (s(h, 1, -1) - s(h, -1, -1)) \
            + s(f, 1, 1) * (s(h, 0, 2) - s(h, 2, 0)) - s(f, -1, -1) * (s(h, -2, 0) - s(h, 0, -2)) \
            - s(f, -1, 1) * (s(h, 0, 2) - s(h, -2, 0)) + s(f, 1, -1) * (s(h, 2, 0) - s(h, 0, -2))
        c = 1.0 / (self.hx * self.hv)
        y = {"arakawaj1": j1 * (c / 12), "arakawaj2": j2 * (c / 24)}.get(self.bracket, j1 * (c / 6) - j2 * (c / 24))
        return torch.nn.functional.pad(y, (0, 0, 2, 2))

    def moments(self, f):
        n, u, e = (self.hv * (f * w[:, None]).sum(0) for w in (torch.ones_like(self.v), self.v, self.v ** 2))
        return n, u, e, n * n / (n * e - u * u)

    def phi(self, n):
        t = 2 * math.pi * torch.arange(self.nx // 2 + 1, dtype=torch.float64, device=n.device) / self.nx
        sym = (54 - 64 * torch.cos(t) + 10 * torch.cos(2 * t)) / (12 * self.hx ** 2)
        sym[0] = 1.0
        spec = torch.fft.rfft(-(n - n.mean()) * CHARGE) / sym
        return torch.fft.irfft(torch.cat([torch.zeros_like(spec[:1]), spec[1:]]), n=self.nx)

    def h1(self, f):
        p = self.phi(self.hv * f.sum(0))
        return p - p.mean()

    def have(self, h1p, h1h):
        return self.h0[:, None] + (0.5 * (h1p + h1h))[None, :]

    def residual(self, F, f, H):
        return (F - f) / self.ht + self.brk(0.5 * (F + f), H)

    def jvp(self, X, H):
        return X / self.ht + 0.5 * self.brk(X, H)

    def bands(self):
        """The v-tridiagonal matrix of every x mode, (nv, modes) each: sub, main and super diagonal."""
        nx, hv = self.nx, self.hv
        z = 2j * math.pi * torch.arange(nx, dtype=torch.float64, device=self.v.device) / nx
        lam = torch.fft.ifftshift(torch.exp(z * (nx - 1)) - torch.exp(z))[:nx // 2 + 1]
        c, v = 0.5 / (self.hx * hv * 12), self.v
        return ((0.5 * (2 * hv * v - hv * hv) * c)[:, None] * lam, (4 * hv * v * c)[:, None] * lam + 1.0 / self.ht,
                (0.5 * (2 * hv * v + hv * hv) * c)[:, None] * lam)

    def tridiagonal(self, X):
        """P X: the matrices themselves."""
        lo, di, up = self.bands()
        d = torch.fft.rfft(X, dim=1)
        y = di * d
        y[1:] += lo[1:] * d[:-1]
        y[:-1] += up[:-1] * d[1:]
        return torch.fft.irfft(y, n=self.nx, dim=1)

    def precondition(self, X):
        """P^-1 X: irFFT_x o (v-tridiagonal solve per mode) o rFFT_x with the averaged kinetic bracket."""
        nx, nv = self.nx, self.nv
        lo, di, up = self.bands()
        d = torch.fft.rfft(X, dim=1)
        for j in range(1, nv):          # row j: lo[j] x[j-1] + di[j] x[j] + up[j] x[j+1]
            m = lo[j] / di[j - 1]
            di[j] -= m * up[j - 1]
            d[j] -= m * d[j - 1]
        d[nv - 1] /= di[nv - 1]
        for j in range(nv - 2, -1, -1):
            d[j] = (d[j] - up[j] * d[j + 1]) / di[j]
        return torch.fft.irfft(d, n=nx, dim=1)


def _solve(A, b, rtol, most=600):
    """GMRES without restart, twice orthogonalised; A acts on fields shaped like b."""
    beta = b.norm()
    if beta == 0:
        return torch.zeros_like(b)
    V = torch.empty(most + 1, b.numel(), dtype=b.dtype, device=b.device)
    V[0] = b.reshape(-1) / beta
    H = np.zeros((most + 1, most))
    for k in range(most):
        w = A(V[k].view(b.shape)).reshape(-1)
        h = V[:k + 1] @ w
        w = w - V[:k + 1].T @ h
        g = V[:k + 1] @ w
        w = w - V[:k + 1].T @ g
        H[:k + 1, k] = (h + g).cpu().numpy()
        H[k + 1, k] = float(w.norm())
        V[k + 1] = w / H[k + 1, k]
        if k % 8 == 7 or k + 1 == most or H[k + 1, k] < 1e-14 * abs(H[:k + 1, k]).max():
            e = np.zeros(k + 2)
            e[0] = float(beta)
            y = np.linalg.lstsq(H[:k + 2, :k + 1], e, rcond=None)[0]
            if np.linalg.norm(e - H[:k + 2, :k + 1] @ y) <= rtol * float(beta):
                break
    return (torch.from_numpy(y).to(b.device) @ V[:k + 1]).view(b.shape)


def _step(m, f, h1h):
    """F of one implicit midpoint step from f: Picard over h1 with the linear system solved each time."""
    F, h1, last = f.clone(), h1h.clone(), math.inf
    for _ in range(30):
        H = m.have(h1, h1h)
        r = m.residual(F, f, H)
        now = float(r.norm())
        if now < 1e-14 * float(f.norm()) / m.ht or now >= last:
            break
        last = now
        F = F - _solve(lambda x: m.jvp(x, H), r, 1e-4)
        h1 = m.h1(F)
    return F, h1


def _invariants(m, f, phi):
    hh = m.hx * m.hv
    fp = torch.roll(f, -1, 1)
    h1 = phi - phi.mean()
    pos = torch.where(f > 0, f, torch.full_like(f, 1e-15))[:-1]
    kin, pot = (f * m.h0[:, None]).sum() * hh, (f * h1).sum() * hh
    d = torch.roll(phi, -1) - phi
    return {"mass": (f[:-1] + fp[:-1] + fp[1:] + f[1:]).sum() * 0.25 * hh, "L2": hh * (f[:-1] ** 2).sum(),
            "energy": kin + 0.5 * pot, "entropy": -hh * (pos * pos.log()).sum(),
            "field_energy": 0.5 * CHARGE * (d * d).sum() / m.hx}


def exact(case, seed):
    kind = case["kind"]
    gen = _gen(seed)
    if kind == "run":
        L = _length(case["k"])
        m = _Model(case["nx"], case["nv"], L, case["vmax"], case["ht"])
        f = _distribution(case["family"], case["nx"], case["nv"], L, case["vmax"], case["k"], case["amp"], gen)
        f = f / (f.sum() * m.hv / m.nx)
        h1, trace = m.h1(f), []
        for _ in range(case["steps"]):
            f, h1 = _step(m, f, h1)
            trace.append(_invariants(m, f, m.phi(m.hv * f.sum(0))))
        n, u, e, _ = m.moments(f)
        out = {"f": f, "phi": m.phi(n), "n": n, "u": u, "e": e}
        for name in TRACED:
            out[name] = np.array([float(t[name]) for t in trace])
        return out
    if kind == "sweep":
        if case["count"] > 24:     # a minute and more
            return None
        fs, phis = [], []
        for s in _sweep_specs(case):
            m = _Model(s["nx"], s["nv"], s["L"], 10.0, 0.1)
            f = _sweep_field(s, gen)
            f = f / (f.sum() * m.hv / m.nx)
            h1 = m.h1(f)
            for _ in range(case["steps"]):
                f, h1 = _step(m, f, h1)
            fs.append(f.view(-1))
            phis.append(m.phi(m.hv * f.sum(0)))
        return {"f": torch.cat(fs), "phi": torch.cat(phis)}
    if kind == "fields":
        m = _Model(case["nx"], case["nv"], 4 * math.pi, 10.0, 0.05)
        F = _distribution("bump_on_tail", case["nx"], case["nv"], 4 * math.pi, 10.0, 0.5, 0.5, gen)
        n, u, e, a = m.moments(F)
        phi = m.phi(n)
        return {"n": n, "u": u, "e": e, "a": a, "phi": phi, "h1": phi - phi.mean()}
    if kind == "adjoint":
        L = 4 * math.pi
        m = _Model(case["nx"], case["nv"], L, 10.0, 0.1)
        f = _distribution("landau", case["nx"], case["nv"], L, 10.0, 0.5, 0.1, gen)
        f = f / (f.sum() * m.hv / m.nx)
        gF = 2.0 * _rand((case["nv"], case["nx"]), gen) - 1.0
        h1h = m.h1(f)
        F, _ = _step(m, f, h1h)
        F.requires_grad_(True)
        with torch.enable_grad():
            G = m.residual(F, f, m.have(m.h1(F), h1h))
        lam = _solve(lambda y: torch.autograd.grad(G, F, y, retain_graph=True)[0], gF, 1e-13)
        return -gF + (2.0 / m.ht) * lam
    F, Fh, X, h1p, h1h = _apply_fields(case, seed)
    m = _Model(case["nx"], case["nv"], 4 * math.pi, 8.0, 0.05, case.get("bracket", "arakawaj4"))
    H = m.have(h1p, h1h)
    if kind == "gmres":          # (P^-1 J) y = X; an even nx has P^-1 invertible, so J y = P X
        if case["nx"] % 2:
            return None
        return _solve(lambda y: m.jvp(y, H), m.tridiagonal(X), 1e-13)
    if case["call"] == "jacobian":
        return m.precondition(m.jvp(X, H))
    R = m.residual(F, Fh, H)
    if case["call"] == "function":
        return m.precondition(R)
    return {"norm": float(R.norm()), "Y": R}

"""What is timed: calls of the solver as its users make them, over the sizes they make them at.

The sizes are those of ``bench.py`` (the plain 40x20 solve, the 100x50 ELBO batch, the
400x200 single solve, the uneven batch of orders 3 to 5, the serving stream) and of the
tests, with fewer time steps where a full run would only repeat the same step.  A user
keeps the plan of a mesh and the batch object from call to call, and brings new velocities
and observations.
"""
import functools
import math

import numpy as np
import torch

from mun_b200 import Batch, SEMPlan, SolveSpec
from mun_b200.autograd import GridLikelihood, GridModel
from mun_b200.mesh import create_global_mesh
from mun_b200.sem_waveform import SEMSimulation
from mun_b200.serving import Engine

DEV = "cuda"
F64 = torch.float64
INTERFACES, LAYERS = (300.0, 650.0), (1500.0, 2200.0, 3000.0)  # three layers over 1 km depth
CMAX = 3600.0                                                  # velocities are clipped here
SIGMA = 1e-10                                                  # noise level of the data
INV_SIGMA2 = 1.0 / (SIGMA ** 2 + 1e-24)                        # as the drivers form it
ANOMALY = ((880.0, 140.0), (1000.0, 110.0), (1120.0, 140.0), (1140.0, 210.0), (1000.0, 250.0), (860.0, 210.0))


def listed():
    def solve(name, **kw):
        c = dict(kind="solve", models=1, nelx=100, nelz=50, npol=4, nt=1000, nrec=100, mode="gradient",
                 boundary="sponge", exact=False, ckpt=0, it0=0, it1=0, decim=1)
        c.update(kw)
        return dict(c, name=name)

    return [
        # one likelihood on the smallest mesh, receivers read before the update: all latency
        solve("forward 20x10", nelx=20, nelz=10, nt=500, nrec=20, mode="forward"),
        # the plain method: one gradient on the 40x20 mesh (bench.py's plain run)
        solve("gradient 40x20", nelx=40, nelz=20, nt=2000, nrec=50),
        # a proposal of one MCMC chain: forward with the misfit summed on the device
        solve("likelihood 91x45", nelx=91, nelz=45, nt=1500, nrec=50, mode="likelihood"),
        # one sample's gradient on the mesh of the ELBO batch
        solve("gradient 100x50", nt=3000),
        # an ELBO step's batch of samples
        solve("gradient 100x50 x128", models=128),
        # the same physics with Stacey edges and a free surface, a smaller batch
        solve("stacey 100x50 x32", models=32, nt=800, boundary="stacey"),
        # one large survey model
        solve("gradient 400x200", nelx=400, nelz=200, nt=2000, nrec=400),
        # order 5, windowed and decimated data, few checkpoints kept (memory-bound users)
        solve("order 5, replay", nelx=37, nelz=31, npol=5, nt=1200, nrec=24, exact=True, ckpt=150, it0=60,
              it1=1100, decim=4),
        # uneven meshes, orders and step counts in one call
        dict(kind="mixed", name="mixed 12", models=12, lo=40, hi=200, nt=1200, nrec=100, shapes=3),
        # the flow trainer's step through autograd: theta in, log-likelihoods and d/dtheta out
        dict(kind="flow", name="flow 16", models=16, nelx=100, nelz=50, npol=4, nt=1000, nrec=100),
        # the drop-in class on the layered model: control points in, likelihood and gradient out
        dict(kind="dropin", name="drop-in 48x28", nelx=48, nelz=28, npol=4, nt=800, nrec=50),
        # requests of four chains and one flow batch through the serving engine
        dict(kind="serving", name="serving 24", chains=4, each=4, flow=8, nelx=80, nt=600, nrec=50),
    ]


def draw(rng):
    """Meshes of 20 to 400 elements across (about two to one), orders 3 to 5, single solves
    and batches, forward and gradient, sponge and Stacey edges, windows and checkpoints."""
    kind = rng.choice(["solve"] * 9 + ["mixed", "flow", "dropin", "serving"])
    log = lambda a, b: int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))  # noqa: E731
    if kind == "mixed":
        return dict(kind=kind, models=rng.randint(4, 12), lo=40, hi=200, nt=rng.randint(400, 1200), nrec=100,
                    shapes=rng.randint(0, 10**6))
    if kind == "flow":
        nelx = rng.randint(60, 120)
        return dict(kind=kind, models=rng.randint(4, 24), nelx=nelx, nelz=nelx // 2, npol=4,
                    nt=rng.randint(400, 1200), nrec=100)
    if kind == "dropin":
        return dict(kind=kind, nelx=rng.randint(30, 72), nelz=rng.randint(18, 42), npol=rng.choice([4, 4, 5]),
                    nt=rng.randint(300, 1500), nrec=50)
    if kind == "serving":
        return dict(kind=kind, chains=rng.randint(2, 6), each=rng.randint(2, 5), flow=rng.randint(2, 10),
                    nelx=rng.randint(60, 120), nt=rng.randint(300, 800), nrec=50)
    c = dict(kind="solve", models=rng.choice([1, 1, log(2, 128)]), nelx=log(20, 400), npol=rng.choice([3, 4, 4, 4, 5]),
             mode=rng.choice(["forward", "likelihood", "gradient", "gradient"]),
             boundary=rng.choice(["sponge"] * 4 + ["stacey"]), exact=rng.random() < 0.5, ckpt=0, it0=0, it1=0, decim=1)
    c["nelz"] = max(8, int(c["nelx"] * rng.uniform(0.4, 0.8)))
    c["nrec"] = max(10, min(400, int(c["nelx"] * rng.uniform(0.5, 1.5))))
    # node steps at most half the largest listed case's, whatever the mode
    nodes = c["nelx"] * c["nelz"] * c["npol"] ** 2
    c["models"] = max(1, min(c["models"], 320_000_000 // (nodes * 300)))
    c["nt"] = min(log(300, 3000), max(300, 320_000_000 // (nodes * c["models"])))
    if c["mode"] == "gradient" and c["boundary"] == "sponge" and rng.random() < 0.3:
        c["it0"], c["it1"], c["decim"] = c["nt"] // 20, c["nt"] - c["nt"] // 12, rng.randint(1, 6)
    if c["mode"] == "gradient" and rng.random() < 0.25:
        c["ckpt"] = max(40, c["nt"] // rng.randint(3, 9))
    return c


# ------------------------------------------------------------------ meshes and inputs


def _extent(nelx, nelz):
    return 20.0 * nelx, 20.0 * nelz  # 20 m elements: about 6 to a wavelength at 10 Hz


def _dt(npol, cmax=CMAX, h=20.0):
    return 0.35 * (h / (npol + 1)) / (cmax * (npol + 1) * math.sqrt(2.0))


def _receivers(nelx, nelz, nrec):
    X, _ = _extent(nelx, nelz)
    return np.stack([np.linspace(0.0, X, nrec), np.full(nrec, 10.0)], 1)


@functools.lru_cache(maxsize=64)
def _plan(nelx, nelz, npol, nt, nrec, boundary="sponge"):
    """(plan, node coordinates, node_grid on the device): kept by a user for all calls on this mesh."""
    X, Z = _extent(nelx, nelz)
    coords, _, node_grid = create_global_mesh(0.0, X, 0.0, Z, nelx, nelz, npol)
    plan = SEMPlan(xmin=0.0, xmax=X, zmin=0.0, zmax=Z, nelx=nelx, nelz=nelz, npol=npol, dt=_dt(npol), nt=nt,
                   src_xz=(0.5 * X + 0.5, 20.0), f0=10.0, amp=1.0, receivers=_receivers(nelx, nelz, nrec),
                   pml_thickness=0.1 * X, sponge_cmax=3000.0, coords=coords, node_grid=node_grid, boundary=boundary)
    return plan, coords, torch.as_tensor(node_grid, device=DEV)


@functools.lru_cache(maxsize=1)
def _batch():
    return Batch()


@functools.lru_cache(maxsize=1)
def _engine():
    return Engine(max_solves=256, memory_cap_bytes=24 << 30)


def _hat_basis(x, n):
    """Cubic B-spline values (len(x), n) on a uniform grid over [0, 1], one node beyond each end."""
    s = (x[:, None] * (n - 3) - (torch.arange(n, dtype=F64, device=x.device) - 1.0)[None, :]).abs()
    return torch.where(s < 1, 2 / 3 - s * s + 0.5 * s ** 3, torch.where(s < 2, (2 - s) ** 3 / 6, torch.zeros_like(s)))


def _layers(nelx, nelz, npol):
    """(nz, nx): the three layers stretched over the depth."""
    z = _lines(nelz, npol) * 1000.0
    base = torch.full_like(z, LAYERS[0])
    for zi, vi in zip(INTERFACES, LAYERS[1:]):
        base = torch.where(z >= zi, torch.full_like(z, vi), base)
    return base[:, None].expand(-1, nelx * npol + 1).contiguous()


def _grid_velocity(nelx, nelz, npol, models, gen):
    """(models, nz, nx): the layers with B-spline node perturbations of 100 m/s as the flow draws them."""
    gx, gz = _lines(nelx, npol), _lines(nelz, npol)
    theta = 100.0 * torch.randn(models, 6, 10, generator=gen, dtype=F64).to(DEV)
    pert = torch.einsum("za,mab,xb->mzx", _hat_basis(gz, 6), theta, _hat_basis(gx, 10))
    return (_layers(nelx, nelz, npol) + pert).clamp(1200.0, CMAX)


def _data(nelx, nelz, nrec, nt, dt, gen, first=0):
    """(nt, nrec) recorded traces: the direct wave and two reflections of a 2-D medium, with noise."""
    X, Z = _extent(nelx, nelz)
    rec = torch.as_tensor(_receivers(nelx, nelz, nrec), device=DEV)
    t = torch.arange(nt, dtype=F64, device=DEV) * dt
    a = (math.pi * 10.0 * (t - 0.1)) ** 2
    wave = (1 - 2 * a) * torch.exp(-a)
    half = 1 / torch.sqrt(t + 0.5 * dt)
    n = 2 * nt
    src = torch.fft.irfft(torch.fft.rfft(wave, n) * torch.fft.rfft(half, n), n)[:nt] * dt
    c = LAYERS[0] * (1 + 0.03 * float(torch.randn(1, generator=gen, dtype=F64)))
    out = torch.zeros(nt, nrec, dtype=F64, device=DEV)
    for depth, amp in ((0.0, 1.0), (0.3 * Z, 0.2), (0.65 * Z, 0.15)):
        r = torch.sqrt((rec[:, 0] - 0.5 * X) ** 2 + (2 * depth + 10.0) ** 2).clamp_min(10.0)
        at = t[:, None] - (r / c)[None, :]
        i = (at / dt).clamp(0, nt - 2)
        k = i.long()
        w = torch.where(at > 0, src[k] * (1 - (i - k)) + src[k + 1] * (i - k), torch.zeros_like(at))
        out += amp / (2 * math.pi * c * c) * torch.sqrt(c / (2 * r))[None, :] * w
    return out + SIGMA * torch.randn(nt, nrec, generator=gen, dtype=F64).to(DEV)


def _window(case):
    it1 = case["it1"] or case["nt"]
    return case["it0"], it1, case["decim"]


def _inputs(case, seed):
    """Velocities (models, nz, nx) and observations on the misfit grid, from the seed alone."""
    gen = torch.Generator().manual_seed(seed)
    v = _grid_velocity(case["nelx"], case["nelz"], case["npol"], case["models"], gen)
    y = _data(case["nelx"], case["nelz"], case["nrec"], case["nt"], _dt(case["npol"]), gen)
    it0, it1, decim = _window(case)
    return v, y[it0:it1:decim].contiguous()


def _mixed(case):
    """The cases of an uneven batch's solves."""
    rng = np.random.default_rng(case["shapes"])
    out = []
    for _ in range(case["models"]):
        nelx, npol = int(rng.integers(case["lo"], case["hi"] + 1)), int(rng.choice([3, 4, 5]))
        nt = int(case["nt"] * rng.uniform(0.3, 1.0))
        out.append(dict(models=1, nelx=nelx, nelz=nelx // 2, npol=npol, nt=nt, nrec=case["nrec"], mode="gradient",
                        boundary="sponge", exact=False, ckpt=0, it0=0, it1=0, decim=1))
    return out


def _serving(case):
    """(chains' cases, flow batch's case): forward likelihoods on several meshes, gradients on one."""
    base = dict(npol=4, nrec=case["nrec"], boundary="sponge", exact=False, ckpt=case["nt"], it0=0, it1=0, decim=1)
    chains = [dict(base, models=case["each"], nelx=case["nelx"] - 7 * i, nelz=(case["nelx"] - 7 * i) // 2,
                   nt=case["nt"] + 40 * i, mode="likelihood") for i in range(case["chains"])]
    return chains, dict(base, models=case["flow"], nelx=case["nelx"], nelz=case["nelx"] // 2, nt=case["nt"],
                        mode="gradient")


def _solve_state(case, seed):
    plan, _, node_grid = _plan(case["nelx"], case["nelz"], case["npol"], case["nt"], case["nrec"], case["boundary"])
    v, y = _inputs(case, seed)
    m, grad = case["models"], case["mode"] == "gradient"
    st = {"case": case, "plan": plan, "v": v.reshape(m, -1)[:, node_grid].contiguous(), "y": y}
    st["rec"] = torch.empty(m, case["nt"], case["nrec"], dtype=torch.float32, device=DEV)
    st["loglik"] = torch.empty(m, 1, dtype=F64, device=DEV) if case["mode"] != "forward" else None
    st["grad"] = torch.empty(m, plan.npoints, dtype=F64, device=DEV) if grad else None
    return st


def _specs(st):
    c, out = st["case"], []
    for i in range(c["models"]):
        s = SolveSpec(st["plan"], st["v"][i], rec=st["rec"][i])
        if c["mode"] != "forward":
            s.misfit, s.y_obs, s.inv_sigma2, s.loglik = True, st["y"], INV_SIGMA2, st["loglik"][i]
            s.window = _window(c)
        if c["mode"] == "gradient":
            s.adjoint, s.exact, s.grad, s.ckpt_k = True, c["exact"], st["grad"][i], c["ckpt"]
        out.append(s)
    return out


def _answers(st):
    return {k: st[k] for k in ("rec", "loglik", "grad")}


def prepare(case, seed):
    kind = case["kind"]
    if kind == "solve":
        return {"kind": kind, "batch": _batch(), "solves": [_solve_state(case, seed)]}
    if kind == "mixed":
        return {"kind": kind, "batch": _batch(),
                "solves": [_solve_state(c, seed * 1009 + i) for i, c in enumerate(_mixed(case))]}
    if kind == "serving":
        chains, flow = _serving(case)
        return {"kind": kind, "engine": _engine(),
                "solves": [_solve_state(c, seed * 1009 + i) for i, c in enumerate(chains + [flow])]}
    if kind == "flow":
        theta, y = _flow_inputs(case, seed)
        model = _grid_model(case["nelx"], case["nelz"], case["npol"], case["nt"], case["nrec"])
        return {"kind": kind, "batch": _batch(), "model": model, "theta": theta.requires_grad_(True), "y": y,
                "up": _upstream(case, seed)}
    ctrl, y = _dropin_inputs(case, seed)
    sim = SEMSimulation(_dropin_config(case))
    return {"kind": kind, "sim": sim, "params": {"bspline_ctrl": ctrl, "y_obs": y, "obs_dt": _dt(case["npol"], 3000.0),
                                                 "obs_nt": case["nt"], "noise_std": SIGMA}}


def run(state):
    kind = state["kind"]
    if kind in ("solve", "mixed"):
        state["batch"].run([s for st in state["solves"] for s in _specs(st)])
        return [_answers(st) for st in state["solves"]]
    if kind == "serving":
        eng = state["engine"]
        tickets = [eng.submit(s) for st in state["solves"] for s in _engine_specs(st)]
        eng.run_until_done(tickets)
        done = [eng.release(t) for t in tickets]
        out, at = [], 0
        for st in state["solves"]:
            m = st["case"]["models"]
            got, at = done[at:at + m], at + m
            out.append({"rec": torch.stack([s.rec for s in got]), "loglik": torch.cat([s.loglik for s in got]),
                        "grad": torch.stack([s.grad for s in got]) if got[0].grad is not None else None})
        return out
    if kind == "flow":
        theta = state["theta"]
        theta.grad = None
        ll = GridLikelihood.apply(theta, state["model"], state["y"], SIGMA, True, state["batch"])
        ll.backward(state["up"])
        return {"loglik": ll.detach(), "grad": theta.grad}
    return state["sim"].run_forward_and_adjoint(state["params"])


def _engine_specs(st):
    """The engine allocates a request's outputs when it is submitted."""
    c = st["case"]
    return [SolveSpec(st["plan"], st["v"][i], misfit=True, y_obs=st["y"], inv_sigma2=INV_SIGMA2,
                      adjoint=c["mode"] == "gradient", exact=False, ckpt_k=c["nt"] if c["mode"] == "gradient" else 0)
            for i in range(c["models"])]


# ------------------------------------------------------------------ flow trainer


@functools.lru_cache(maxsize=8)
def _grid_model(nelx, nelz, npol, nt, nrec):
    plan, coords, node_grid = _plan(nelx, nelz, npol, nt, nrec)
    X, Z = _extent(nelx, nelz)
    base = _layers(nelx, nelz, npol).reshape(-1)[node_grid]
    return GridModel(plan, coords, base.cpu().numpy(), ((0.0, X), (0.0, Z)), 10, 6, device=DEV)


def _flow_inputs(case, seed):
    gen = torch.Generator().manual_seed(seed)
    theta = (100.0 * torch.randn(case["models"], 60, generator=gen, dtype=F64)).clamp(-400, 400).to(DEV)
    y = _data(case["nelx"], case["nelz"], case["nrec"], case["nt"], _dt(case["npol"]), gen)
    return theta, y


def _upstream(case, seed):
    gen = torch.Generator().manual_seed(seed + 77)
    return (torch.rand(case["models"], generator=gen, dtype=F64) + 0.5).to(DEV)


# ------------------------------------------------------------------ drop-in class


def _dropin_config(case):
    dt = _dt(case["npol"], 3000.0)
    X, Z = _extent(case["nelx"], case["nelz"])
    return {
        "domain": {"xmin": 0.0, "xmax": X, "zmin": 0.0, "zmax": Z, "nelem_x": case["nelx"], "nelem_z": case["nelz"]},
        "time": {"total_time": (case["nt"] - 0.5) * dt, "dt": 1.0},
        "source": {"position": (0.5 * X + 0.5, 20.0), "frequency": 10.0, "amplitude": 1.0},
        "receivers": {"positions": _receivers(case["nelx"], case["nelz"], case["nrec"]).tolist()},
        "method": {"polynomial_order": case["npol"], "pml_thickness": 0.1 * X},
        "velocity": {"vmin": 1500.0, "vmax": 3000.0, "control_points": _anomaly(case).tolist(), "tau": 10.0,
                     "spline_samples": 400, "layers": {"interfaces_z": [0.3 * Z + 0.5, 0.65 * Z + 0.5], "velocities": list(LAYERS)},
                     "anomaly": {"v_inside": 2400.0, "blend": "smooth"}},
        "output": {"visualize": False, "save_wavefield": False},
    }


def _anomaly(case):
    X, Z = _extent(case["nelx"], case["nelz"])
    a = np.asarray(ANOMALY)
    return np.stack([a[:, 0] / 2000.0 * X, a[:, 1] / 600.0 * Z], 1)


def _dropin_inputs(case, seed):
    gen = torch.Generator().manual_seed(seed)
    ctrl = _anomaly(case) + 0.01 * case["nelx"] * torch.randn(6, 2, generator=gen, dtype=F64).numpy()
    y = _data(case["nelx"], case["nelz"], case["nrec"], case["nt"], _dt(case["npol"], 3000.0), gen)
    return ctrl, y.cpu().numpy()


# ------------------------------------------------------------------ work


def _march_work(c):
    """Bytes and operations of one solve case: velocities in, traces and gradients out, and
    the wavefield of every step written and read back where a gradient needs it."""
    n, N, NP = c["nelx"] * c["nelz"] * c["npol"] ** 2, c["npol"], c["npol"] + 1
    grad = c["mode"] == "gradient"
    line = 2 * (4 * NP * NP + 2 * NP) / N           # both directions' D^T (beta c^2 (D u)), per node
    step = line + 16
    flops = n * c["nt"] * (step + (step + 2 * (2 * NP * NP + 2 * NP) / N + 6 if grad else 0))
    by = n * 8 + 4 * c["nt"] * c["nrec"] + (8 * c["nt"] * c["nrec"] if c["mode"] != "forward" else 0)
    if grad:
        by += 8 * n + 8.0 * n * c["nt"]
    return c["models"] * by, c["models"] * flops


def _as_solves(case):
    base = dict(models=1, mode="gradient", boundary="sponge", exact=False, ckpt=0, it0=0, it1=0, decim=1)
    if case["kind"] == "solve":
        return [case]
    if case["kind"] == "mixed":
        return _mixed(case)
    if case["kind"] == "serving":
        chains, flow = _serving(case)
        return chains + [flow]
    return [dict(base, **{k: v for k, v in case.items() if k not in ("kind", "name")})]


def work(case):
    got = [_march_work(c) for c in _as_solves(case)]
    return {"bytes": sum(g[0] for g in got), "flops": sum(g[1] for g in got)}


# ------------------------------------------------------------------ the same in 64 bits, plain torch


@functools.lru_cache(maxsize=None)
def _gll(N):
    """Gauss-Lobatto-Legendre points, weights and the differentiation matrix D[a, b] = l_b'(x_a)."""
    P = np.polynomial.legendre.Legendre.basis(N)
    x = np.concatenate([[-1.0], np.sort(P.deriv().roots().real), [1.0]])
    w = 2.0 / (N * (N + 1) * P(x) ** 2)
    bw = np.array([1.0 / np.prod([x[j] - x[k] for k in range(N + 1) if k != j]) for j in range(N + 1)])
    D = np.array([[0.0 if i == j else bw[j] / (bw[i] * (x[i] - x[j])) for j in range(N + 1)] for i in range(N + 1)])
    np.fill_diagonal(D, -D.sum(1))
    return x, w, D


def _lines(nel, N):
    """Coordinates in [0, 1] of the grid lines along one axis."""
    x = _gll(N)[0]
    e = (np.arange(nel)[:, None] + 0.5 * (1 + x[None, :N])).reshape(-1) / nel
    return torch.as_tensor(np.append(e, 1.0), device=DEV)


def _assembled(nel, N, vals):
    out = np.zeros(nel * N + 1)
    for e in range(nel):
        out[e * N:(e + 1) * N + 1] += vals
    return out


def _node_order(nelx, nelz, N):
    """Grid index of each node in first-seen order of the sweep over elements (row by row, and
    row by row inside an element)."""
    gz, gx = np.divmod(np.arange((nelx * N + 1) * (nelz * N + 1)), nelx * N + 1)
    ex, ez = np.maximum(0, -(-gx // N) - 1), np.maximum(0, -(-gz // N) - 1)
    return torch.as_tensor(np.lexsort((gx - ex * N, gz - ez * N, ex, ez)), device=DEV)


class _March:
    """The wave equation on one mesh in float64, models along the first axis."""

    def __init__(self, c, v, cmax_sponge=3000.0, dt=None):
        self.c, self.N, self.dt = c, c["npol"], dt or _dt(c["npol"])
        nelx, nelz, N = c["nelx"], c["nelz"], self.N
        x, w, D = _gll(N)
        X, Z = _extent(nelx, nelz)
        dx, dz = X / nelx, Z / nelz
        J = 0.25 * dx * dz
        T = lambda a: torch.as_tensor(a, device=DEV)  # noqa: E731
        self.D, self.w = T(D), T(w)
        mx, mz = _assembled(nelx, N, w), _assembled(nelz, N, w)
        self.Rz, self.Rx = T(J * (2 / dx) ** 2 * mz)[:, None], T(J * (2 / dz) ** 2 * mx)[None, :]
        M = T(J * mz[:, None] * mx[None, :])
        self.P = self.dt ** 2 / M
        self.v, c2 = v, v * v
        self.cx = self._ux(c2) * self.w
        self.cz = self._ux(c2.transpose(1, 2)) * self.w
        self.stacey = c["boundary"] == "stacey"
        if self.stacey:
            beta = np.zeros((nelz * N + 1, nelx * N + 1))
            beta[:, 0] += mz * dz / 2
            beta[:, -1] += mz * dz / 2
            beta[-1] += mx * dx / 2
            beta[0] = 0
            self.beta = T(beta)
            self.a = 0.5 * self.dt * v * self.beta / M
        else:
            th = 0.1 * X

            def sig(n, L):
                s = _lines(n, N).cpu().numpy() * L
                d = np.maximum(np.maximum(th - s, s - (L - th)), 0.0) / th
                return T(-4.0 * cmax_sponge * math.log(1e-8) / (2 * th) * d ** 3)
            self.d = torch.exp(-sig(nelz, Z) * self.dt)[:, None] * torch.exp(-sig(nelx, X) * self.dt)[None, :]
        t = np.arange(c["nt"]) * self.dt
        a = (np.pi * 10.0 * (t - 0.1)) ** 2
        s = (1 - 2 * a) * np.exp(-a)
        s = s - np.trapezoid(s, t) / (t[-1] - t[0])
        s[t >= 0.3] = 0.0
        self.src = [float(q) for q in self.dt ** 2 * s]
        gx, gz = _lines(nelx, N).cpu().numpy() * X, _lines(nelz, N).cpu().numpy() * Z
        self.at = int(np.argmin(np.abs(gz - 20.0))), int(np.argmin(np.abs(gx - 0.5 * X - 0.5)))
        pos = _receivers(nelx, nelz, c["nrec"])
        idx, wr = [], []
        for rx, rz in pos:
            ex, ez = min(max(int(rx / dx), 0), nelx - 1), min(max(int(rz / dz), 0), nelz - 1)
            xi, eta = 2 * (rx - ex * dx) / dx - 1, 2 * (rz - ez * dz) / dz - 1
            L = lambda q: np.array([np.prod([(q - x[k]) / (x[i] - x[k]) for k in range(N + 1) if k != i]) for i in range(N + 1)])  # noqa: E731
            j, i = np.meshgrid(ez * N + np.arange(N + 1), ex * N + np.arange(N + 1), indexing="ij")
            idx.append((j * (nelx * N + 1) + i).reshape(-1))
            wr.append((L(eta)[:, None] * L(xi)[None, :]).reshape(-1))
        self.ri, self.rw = T(np.array(idx)), T(np.array(wr))

    def _ux(self, u):
        return u.unfold(2, self.N + 1, self.N)

    def _sum(self, r, n):
        N = self.N
        out = torch.zeros(r.shape[0], r.shape[1], n, dtype=F64, device=DEV)
        out[:, :, :n - 1].view(r.shape[0], r.shape[1], -1, N).add_(r[..., :N])
        out[:, :, N::N].add_(r[..., N])
        return out

    def K(self, u):
        ut = u.transpose(1, 2)
        kx = self._sum((self._ux(u) @ self.D.T * self.cx) @ self.D, u.shape[2])
        kz = self._sum((self._ux(ut) @ self.D.T * self.cz) @ self.D, u.shape[1])
        return self.Rz * kx + self.Rx * kz.transpose(1, 2)

    def sens(self, u, lam):
        ut, lt = u.transpose(1, 2), lam.transpose(1, 2)
        sx = self._sum(self.w * (self._ux(u) @ self.D.T) * (self._ux(lam) @ self.D.T), u.shape[2])
        sz = self._sum(self.w * (self._ux(ut) @ self.D.T) * (self._ux(lt) @ self.D.T), u.shape[1])
        return self.Rz * sx + self.Rx * sz.transpose(1, 2)

    def step(self, b, v, force, damp):
        if self.stacey:
            w = ((1 - self.a) * v + force) / (1 + self.a)
            w[:, 0] = 0.0
            return b + w, w
        w = v + force
        return (self.d * (b + w), self.d * w) if damp else (b + w, w)

    def read(self, b):
        return (b.reshape(b.shape[0], -1)[:, self.ri] * self.rw).sum(-1)

    def solve(self, y, mode, exact, window):
        """rec, log-likelihood and d loglik / dc for every model."""
        nt, m = self.c["nt"], self.v.shape[0]
        b, v = torch.zeros_like(self.v), torch.zeros_like(self.v)
        rec = torch.empty(m, nt, self.c["nrec"], dtype=F64, device=DEV)
        it0, it1, decim = window
        hist = torch.empty(nt + 1, *self.v.shape, dtype=F64, device=DEV) if mode == "gradient" else None
        if hist is not None:
            hist[0] = 0.0
        for t in range(nt):
            if mode != "gradient":
                rec[:, t] = self.read(b)
            f = -self.P * self.K(b)
            f[:, self.at[0], self.at[1]] += self.src[t]
            b, v = self.step(b, v, f, True)
            if mode == "gradient":
                rec[:, t] = self.read(b)
                hist[t + 1] = b
        if mode == "forward":
            return rec, None, None
        res = torch.zeros_like(rec)
        res[:, it0:it1:decim] = rec[:, it0:it1:decim] - y
        ll = -0.5 * INV_SIGMA2 * (res * res).sum((1, 2))
        if mode != "gradient":
            return rec, ll[:, None], None
        lam, mu, acc = torch.zeros_like(b), torch.zeros_like(b), torch.zeros_like(b)
        for t in range(it1 - 1, it0 - 1, -1):
            inj = torch.zeros(m, lam.shape[1] * lam.shape[2], dtype=F64, device=DEV)
            inj.index_add_(1, self.ri.reshape(-1), (res[:, t, :, None] * self.rw).reshape(m, -1))
            acc += self.sens(hist[t + 1], lam)
            if self.stacey and t + 2 <= nt:
                acc += self.beta / (4 * self.dt * self.v) * lam * (hist[t + 2] - hist[t])
            lam, mu = self.step(lam, mu, self.P * (inj.view_as(lam) - self.K(lam)), exact)
        return rec, ll[:, None], 2 * self.v * acc * INV_SIGMA2


def _exact_solve(c, seed):
    v, y = _inputs(c, seed)
    per = (c["nt"] + 1 if c["mode"] == "gradient" else 8) * v[0].numel() * 8
    some = max(1, int(30e9 // per))
    order = _node_order(c["nelx"], c["nelz"], c["npol"])
    got = [_March(c, v[i:i + some]).solve(y, c["mode"], c["exact"], _window(c)) for i in range(0, len(v), some)]
    cat = lambda k: None if got[0][k] is None else torch.cat([g[k] for g in got])  # noqa: E731
    g = cat(2)
    return {"rec": cat(0), "loglik": cat(1), "grad": None if g is None else g.reshape(len(v), -1)[:, order]}


def _spline_basis(knots, deg, u):
    """Dense (len(u), n) B-spline basis values, the last span closed on the right."""
    n = len(knots) - deg - 1
    i = np.clip(np.searchsorted(knots, u, side="right") - 1, deg, n - 1)
    B = np.zeros((len(u), len(knots) - 1))
    B[np.arange(len(u)), i] = 1.0
    for k in range(1, deg + 1):
        nxt = np.zeros((len(u), len(knots) - 1 - k))
        for j in range(nxt.shape[1]):
            for a, num in ((j, u - knots[j]), (j + 1, knots[j + k + 1] - u)):
                den = knots[a + k] - knots[a]
                if den > 0:
                    nxt[:, j] += num / den * B[:, a]
        B = nxt
    return B


def _exact_dropin(case, seed):
    ctrl, y = _dropin_inputs(case, seed)
    nelx, nelz, N, K = case["nelx"], case["nelz"], case["npol"], 6
    X, Z = _extent(nelx, nelz)
    gx, gz = _lines(nelx, N).cpu().numpy() * X, _lines(nelz, N).cpu().numpy() * Z
    pts = np.stack(np.meshgrid(gx, gz), -1).reshape(-1, 2)
    cc = np.vstack([ctrl, np.tile(ctrl[0], (3, 1))])     # closed by repeating the first point
    n = len(cc)
    knots = np.concatenate([np.zeros(4), np.linspace(0, 1, n - 2)[1:-1], np.ones(4)])

    def diff(co, deg, kn):
        d = deg * (co[1:] - co[:-1]) / np.maximum(kn[deg + 1:deg + len(co)] - kn[1:len(co)], 1e-300)[:, None]
        return d, kn[1:-1]
    c1, k1 = diff(cc, 3, knots)
    c2, k2 = diff(c1, 2, k1)
    at = lambda u, d: (_spline_basis(knots, 3, u) @ cc, _spline_basis(k1, 2, u) @ c1, _spline_basis(k2, 1, u) @ c2)[:d + 1]  # noqa: E731
    u0 = np.linspace(0, 1, 400)
    poly = at(u0, 0)[0]
    u = u0[((pts[:, None] - poly[None]) ** 2).sum(-1).argmin(1)]
    for _ in range(7):
        C, C1, C2 = at(u, 2)
        r = C - pts
        f2 = (C1 * C1).sum(1) + (r * C2).sum(1)
        u = np.clip(u - (r * C1).sum(1) / np.where(np.abs(f2) < 1e-14, 1e-14, f2), 0.0, 1.0)
    rv = pts - at(u, 0)[0]
    dist = np.sqrt((rv * rv).sum(1))
    inside = np.zeros(len(pts), bool)
    for (ax, az), (bx, bz) in zip(poly, np.roll(poly, -1, 0)):
        if az != bz:
            inside ^= ((az > pts[:, 1]) != (bz > pts[:, 1])) & (pts[:, 0] < ax + (pts[:, 1] - az) * (bx - ax) / (bz - az))
    sign = np.where(inside, -1.0, 1.0)
    bg = np.asarray(LAYERS)[np.searchsorted([0.3 * Z + 0.5, 0.65 * Z + 0.5], pts[:, 1], side="right")]
    s = 1 / (1 + np.exp(np.clip(sign * dist / 10.0, -50, 50)))
    v = torch.as_tensor((bg + (2400.0 - bg) * s).reshape(1, len(gz), len(gx)), device=DEV)
    c = _as_solves(case)[0]
    rec, ll, g = _March(c, v, dt=_dt(N, 3000.0)).solve(torch.as_tensor(y, device=DEV), "gradient", False, _window(c))
    dv = (2400.0 - bg) * s * (1 - s) * (-0.1)
    w = np.where(np.abs(dv) > 1e-8 * np.maximum(1.0, np.abs(2400.0 - bg)), -g.cpu().numpy().reshape(-1) * dv, 0.0)
    B = _spline_basis(knots, 3, u)
    B[:, 0] += B[:, K:].sum(1)
    nrm = sign[:, None] * rv / (dist[:, None] + 1e-15)
    return {"loglik": float(ll), "grad_wrt_ctrl": np.einsum("p,pj,pd->jd", w, B[:, :K], nrm).reshape(-1),
            "clean_data": rec[0].cpu().numpy(), "dt": _dt(N, 3000.0), "nt": case["nt"]}


def exact(case, seed):
    kind = case["kind"]
    if kind == "solve":
        return [_exact_solve(case, seed)]
    if kind == "mixed":
        return [_exact_solve(c, seed * 1009 + i) for i, c in enumerate(_mixed(case))]
    if kind == "serving":
        chains, flow = _serving(case)
        got = [_exact_solve(c, seed * 1009 + i) for i, c in enumerate(chains + [flow])]
        return [dict(g, loglik=g["loglik"][:, 0]) for g in got]
    if kind == "dropin":
        return _exact_dropin(case, seed)
    theta, y = _flow_inputs(case, seed)
    nelx, nelz, N = case["nelx"], case["nelz"], case["npol"]

    def clamped(u, n):
        kn = np.concatenate([np.zeros(3), np.linspace(0, 1, n - 2), np.ones(3)])
        return torch.as_tensor(_spline_basis(kn, 3, u.cpu().numpy()), device=DEV)
    Bx, Bz = clamped(_lines(nelx, N), 10), clamped(_lines(nelz, N), 6)
    v = _layers(nelx, nelz, N) + torch.einsum("za,mab,xb->mzx", Bz, theta.view(-1, 6, 10), Bx)
    c = _as_solves(case)[0]
    some = max(1, int(30e9 // ((c["nt"] + 1) * v[0].numel() * 8)))
    ll, g = [], []
    for i in range(0, len(v), some):
        _, a, b = _March(c, v[i:i + some]).solve(y, "gradient", True, _window(c))
        ll.append(a[:, 0])
        g.append(torch.einsum("za,mzx,xb->mab", Bz, b, Bx).reshape(len(b), 60))
    return {"loglik": torch.cat(ll), "grad": torch.cat(g) * _upstream(case, seed)[:, None]}

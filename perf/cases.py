"""What a user of this package has it do, as timed cases.

Every case goes through the package's public Python entry points.  Three
families:

* SIMPLEC runs (`Simplec`, `Batch`): a user resumes an instance from a saved
  state, advances it some outer iterations and saves the state again.  The
  state is a developed transient (a Scarborough run from the initial guess),
  the time step is then held at the value that run reached, so that a pass
  does the same work each time.
* Linear solves: the host drop-ins of the reference's solver classes, and
  flexible GMRES on device tensors.
* The learned p' correction's network: inference and a training step.

States come from the seed: geometry, chamber conditions, coefficients and
right-hand sides all vary with it.
"""
import json
import os

# a batch keeps many streams in flight; with the default 8 hardware queues they share them
os.environ.setdefault("CUDA_DEVICE_MAX_CONNECTIONS", "32")

import numpy as np
import torch

from mach2d_b200 import unet
from mach2d_b200.simplec import Batch, Simplec, euler_cosine_case, n01_case
from mach2d_b200.solvers import fgmres, solvers_init, tdma_lines
from mach2d_b200.thermo import mixture_init

# what a host driver keeps of an instance between runs
FIELDS = ("u", "v", "p", "T", "ro", "ue", "ve", "un", "vn", "Uce", "Vcn", "roe", "ron")
STRIPS = ("uin", "vin", "pin", "Tin", "Mw", "plin", "pina")


def listed():
    return [
        # the reference's own deck: launch and latency bound, the smallest grid that is run
        {"name": "deck-n01-20x10", "kind": "run", "geom": "n01", "nxr": 20, "nyr": 10, "solver": 0, "lag": 0,
         "model": "euler", "warm": 40, "iters": 30},
        # the 80x40 Euler nozzle that users run to convergence (24,000 iterations)
        {"name": "euler-80x40", "kind": "run", "geom": "c01", "nxr": 80, "nyr": 40, "solver": 0, "lag": 0,
         "model": "euler", "warm": 40, "iters": 20},
        # the headline workload: one large nozzle, FP64 as the reference
        {"name": "euler-512x256", "kind": "run", "geom": "c01", "nxr": 512, "nyr": 256, "solver": 0, "lag": 0,
         "model": "euler", "warm": 20, "iters": 8},
        # the fastest way to a converged 512x256 nozzle: FP32 factors reused over solves
        {"name": "euler-512x256-lagged", "kind": "run", "geom": "c01", "nxr": 512, "nyr": 256, "solver": 2, "lag": 32,
         "model": "euler", "warm": 20, "iters": 8},
        # Navier-Stokes with the energy equation, MIXTURE air and Baldwin-Lomax
        {"name": "turbulent-512x256", "kind": "run", "geom": "c01", "nxr": 512, "nyr": 256, "solver": 0, "lag": 0,
         "model": "turbulent", "warm": 20, "iters": 4},
        # the reference's other solver option, on a ragged grid
        {"name": "tdma-203x77", "kind": "run", "geom": "c01", "nxr": 203, "nyr": 77, "solver": 1, "lag": 0,
         "model": "euler", "warm": 20, "iters": 4},
        # as many large nozzles as fill one GPU
        {"name": "batch-16x512x256", "kind": "batch", "n": 16, "nxr": 512, "nyr": 256, "uneven": False, "solver": 0,
         "warm": 12, "iters": 3},
        # a parameter sweep: uneven nozzles with FP32 sweeps, all in flight
        {"name": "sweep-48", "kind": "batch", "n": 48, "nxr": 512, "nyr": 128, "uneven": True, "solver": 2,
         "warm": 12, "iters": 3},
        # one routine swapped under a host driver: MSI on host arrays, copies included
        {"name": "msi9-host-258x130", "kind": "host", "nd": 9, "nx": 258, "ny": 130, "solver": "MSI", "tol": 1e-10},
        # the isolated 9-diagonal system to 1e-12 on device tensors
        {"name": "fgmres9-1026x514", "kind": "fgmres", "nd": 9, "nx": 1026, "ny": 514, "prec": 0, "tol": 1e-12},
        # the network on the pressure systems of eight 512x256 nozzles
        {"name": "unet-forward-8x256x512", "kind": "unet", "train": False, "batch": 8, "H": 256, "W": 512},
        # a training step on a minibatch of 256x128 systems
        {"name": "unet-train-8x128x256", "kind": "unet", "train": True, "batch": 8, "H": 128, "W": 256},
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["run"] * 5 + ["batch"] + ["host"] * 2 + ["lines", "fgmres", "unet", "unet"])
    if kind == "run":
        model = rng.choice(["euler", "euler", "turbulent"])
        solver = rng.choice([0, 0, 0, 1, 2, 2])
        n01 = model == "euler" and rng.random() < 0.2
        nxr, nyr = (_log_int(rng, 16, 40), _log_int(rng, 8, 24)) if n01 else (_log_int(rng, 40, 512), _log_int(rng, 20, 256))
        return {"kind": "run", "geom": "n01" if n01 else "c01", "nxr": nxr, "nyr": nyr,
                "solver": solver, "lag": rng.choice([0, 32]) if solver == 2 else 0, "model": model, "warm": 20,
                "iters": rng.randint(2, 3 if solver == 1 else 8)}
    if kind == "batch":
        return {"kind": "batch", "n": rng.randint(4, 24), "nxr": _log_int(rng, 64, 320), "nyr": _log_int(rng, 32, 128),
                "uneven": rng.random() < 0.5, "solver": rng.choice([0, 2]), "warm": 12, "iters": rng.randint(1, 3)}
    if kind == "host":
        return {"kind": "host", "nd": rng.choice([5, 9]), "nx": _log_int(rng, 20, 500), "ny": _log_int(rng, 12, 250),
                "solver": rng.choice(["MSI", "MSI", "MSI_MIXED"]), "tol": 1e-10}
    if kind == "lines":
        return {"kind": "lines", "n": _log_int(rng, 30, 1024), "nlines": _log_int(rng, 20, 512)}
    if kind == "fgmres":
        return {"kind": "fgmres", "nd": rng.choice([5, 9]), "nx": _log_int(rng, 64, 1000), "ny": _log_int(rng, 32, 500),
                "prec": rng.choice([0, 1]), "tol": 1e-12}
    return {"kind": "unet", "train": rng.random() < 0.4, "batch": rng.randint(1, 8), "H": 8 * rng.randint(2, 20),
            "W": 8 * rng.randint(4, 48)}


# ------------------------------------------------------------------ SIMPLEC
def _air():
    path = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tests", "golden",
                        "air_species.json")
    with open(path) as fh:
        d = json.load(fh)
    return mixture_init(d["base"], d["fractions"], d["Mi"], d["cpi"], d["mui"], d["kpi"])


def _nozzle(case, rng):
    if case["geom"] == "n01":
        return n01_case(case["nxr"], case["nyr"], solver=case["solver"], p0=rng.uniform(0.9e6, 1.2e6),
                        T0=rng.uniform(780.0, 900.0))
    over = dict(solver=case["solver"], msi_lag=case["lag"], Rin=rng.uniform(1.9, 2.1), Rout=rng.uniform(1.7, 1.9))
    if case["model"] == "turbulent":
        over.update(modvis=1, kg=2, a1=1e-6, p0=rng.uniform(1.9e6, 2.1e6), T0=rng.uniform(1450.0, 1550.0), Twall=-1.0,
                    ktm=1, mix=_air(), modtur=1, prt=0.9)
    else:
        over.update(p0=rng.uniform(0.8e6, 1.2e6), T0=rng.uniform(900.0, 1100.0))
    return euler_cosine_case(case["nxr"], case["nyr"], **over)


def _sweep(case, rng):
    cases, sizes = [], np.random.default_rng(case["n"])      # the sizes belong to the case, the flow to the seed
    for _ in range(case["n"]):
        nxr, nyr = case["nxr"], case["nyr"]
        if case["uneven"]:
            nxr, nyr = int(sizes.integers(nxr // 2, nxr + 1)), int(sizes.integers(nyr // 2, nyr + 1))
        cases.append(euler_cosine_case(nxr, nyr, Rin=rng.uniform(1.7, 2.3), Rout=rng.uniform(1.5, 2.0),
                                       Lc=rng.uniform(1.5, 2.5), Ld=rng.uniform(3, 5), p0=rng.uniform(5e5, 3e6),
                                       T0=rng.uniform(600, 1500), solver=case["solver"]))
    return cases


def _pinned(sim, names):
    out = {}
    for f in names:
        t = torch.empty(sim.ny if f in STRIPS else sim.nx * sim.ny, dtype=torch.float64, pin_memory=True)
        out[f] = t.numpy()
    return out


def _saved(sim):
    """The instance's state as a host driver would save it, in pinned memory."""
    host = _pinned(sim, FIELDS + STRIPS)
    sim.get_fields(host)
    return host


def _held(c, dt):
    """The case with its time step held at dt (the ramp model between equal ends)."""
    d = type(c).from_buffer_copy(c)
    d.dtmodel, d.dt1, d.dt2 = 0, dt, dt
    return d


def _prepare_run(case, seed):
    c = _nozzle(case, np.random.default_rng(seed))
    first = Simplec(c)
    first.set_graph(True)
    first.run(case["warm"])
    saved, dt = _saved(first), first.scalar("dt")
    first.close()
    sim = Simplec(_held(c, dt))
    sim.set_graph(True)
    sim.set_fields(saved)
    sim.iterate()            # captures the iteration once, as any program's first iteration does
    return {"sim": sim, "in": saved, "out": _pinned(sim, FIELDS)}


def _run_run(case, s):
    s["sim"].set_fields(s["in"])
    rep = s["sim"].run(case["iters"])
    s["sim"].get_fields(s["out"])
    return [rep.norm, rep.normpl, rep.rmass, rep.fmi, rep.fme, rep.Fd, s["out"]]


def _prepare_batch(case, seed):
    cases = _sweep(case, np.random.default_rng(seed))
    first = Batch(cases)
    for sim in first.instances:
        sim.set_graph(True)
    first.iterate(case["warm"])
    saved = [_saved(sim) for sim in first.instances]
    held = [_held(c, sim.scalar("dt")) for c, sim in zip(cases, first.instances)]
    first.close()
    batch = Batch(held)
    for sim, state in zip(batch.instances, saved):
        sim.set_graph(True)
        sim.set_fields(state)
    batch.iterate(1)
    return {"batch": batch, "in": saved, "out": [_pinned(sim, ("u", "v", "p")) for sim in batch.instances]}


def _run_batch(case, s):
    b = s["batch"]
    for sim, state in zip(b.instances, s["in"]):
        sim.set_fields(state)
    reps = b.iterate(case["iters"])
    for sim, out in zip(b.instances, s["out"]):
        sim.get_fields(out)
    # one output per field over all instances
    return [[r.fmi for r in reps][:8], [np.concatenate([o[f] for o in s["out"]]) for f in ("u", "v", "p")]]


# -------------------------------------------------------------- linear solves
OFF9 = ((-1, -1), (0, -1), (1, -1), (-1, 0), (0, 0), (1, 0), (-1, 1), (0, 1), (1, 1))
OFF5 = ((0, -1), (-1, 0), (0, 0), (1, 0), (0, 1))


def _system(nd, nx, ny, seed):
    """The isolated-system workload: couplings U[-1, 0] between real cells,
    aP = 1.05 sum|a_nb|, a zero-Dirichlet ghost ring.  The right-hand side
    belongs to a solution that is drawn first (N(0, 1) on the real cells)."""
    rng = np.random.default_rng(seed)
    off = OFF9 if nd == 9 else OFF5
    inner = np.zeros((ny, nx), bool)
    inner[1:-1, 1:-1] = True
    xs = np.where(inner, rng.standard_normal((ny, nx)), 0.0)
    a, kp = np.zeros((nd, ny, nx)), off.index((0, 0))
    pad = np.pad(inner, 1)
    for k, (di, dj) in enumerate(off):
        if k != kp:
            nb = pad[1 + dj:1 + dj + ny, 1 + di:1 + di + nx]
            a[k] = np.where(inner & nb, -rng.random((ny, nx)), 0.0)
    s = np.abs(a).sum(axis=0)
    a[kp] = np.where(inner, np.where(s > 0, 1.05 * s, 1.0), 1.0)
    xp, b = np.pad(xs, 1), np.zeros((ny, nx))
    for k, (di, dj) in enumerate(off):
        b += a[k] * xp[1 + dj:1 + dj + ny, 1 + di:1 + di + nx]
    return a.reshape(nd, -1), b.reshape(-1), xs.reshape(-1)


def _lines(n, nlines, seed):
    rng = np.random.default_rng(seed)
    aw, ae = -rng.random((nlines, n)), -rng.random((nlines, n))
    aw[:, 0] = 0.0
    ae[:, -1] = 0.0
    ap = 1.05 * (np.abs(aw) + np.abs(ae)) + 1e-3
    return aw, ap, ae, rng.standard_normal((nlines, n))


# -------------------------------------------------------------------- network
def _images(case, seed):
    """Feature planes, targets and masks as harvested p' systems have them:
    a normalised residual, coefficients over aP (unit diagonal, empty corner
    planes), a standardised log-Jacobian."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    n, H, W = case["batch"], case["H"], case["W"]
    f = torch.zeros(n, 11, H, W, device="cuda")
    f[:, 0] = torch.randn(n, H, W, device="cuda", generator=g)
    for k in (2, 4, 6, 8):
        f[:, k] = -0.25 * (0.5 + torch.rand(n, H, W, device="cuda", generator=g))
    f[:, 5] = 1.0
    f[:, 10] = torch.randn(n, H, W, device="cuda", generator=g)
    t = 1.5 * f[:, 0] + 0.25 * torch.randn(n, H, W, device="cuda", generator=g)
    m = torch.ones(n, H, W, device="cuda")
    m[:, H - H // 16:] = 0.0
    return f, t, m


def _layers(p):
    """[(weights [cout, cin, 3, 3], bias)] of the 14 convolutions, then the head."""
    out, at = [], 0
    for ci, co in unet.LAYERS:
        w = p[at:at + co * 9 * ci].view(co, 3, 3, ci).permute(0, 3, 1, 2)
        at += co * 9 * ci
        out.append((w, p[at:at + co]))
        at += co
    return out, p[at:at + 16], p[at + 16]


def _network64(p, f):
    F = torch.nn.functional
    conv, wh, bh = _layers(p)
    x = torch.cat([f, torch.zeros_like(f[:, :5])], 1)

    def pair(k, h):
        for w, b in conv[k:k + 2]:
            h = F.gelu(F.conv2d(h, w, b, padding=1), approximate="tanh")
        return h
    s = []
    for lv in range(3):
        x = pair(2 * lv, x)
        s.append(x)
        x = F.avg_pool2d(x, 2)
    x = pair(6, x)
    for k, skip in ((8, s[2]), (10, s[1]), (12, s[0])):
        x = pair(k, torch.cat([x.repeat_interleave(2, 2).repeat_interleave(2, 3), skip], 1))
    return (x * wh.view(1, -1, 1, 1)).sum(1) + bh


# ------------------------------------------------------------------- the cases
def prepare(case, seed):
    k = case["kind"]
    if k == "run":
        s = _prepare_run(case, seed)
    elif k == "batch":
        s = _prepare_batch(case, seed)
    elif k == "host":
        a, b, _ = _system(case["nd"], case["nx"], case["ny"], seed)
        five, nine = solvers_init(case["nx"], case["ny"], case["solver"], 400, 400, case["tol"], case["tol"])
        s = {"solver": nine if case["nd"] == 9 else five, "a": a, "b": b}
    elif k == "lines":
        s = {"lines": _lines(case["n"], case["nlines"], seed)}
    elif k == "fgmres":
        a, b, _ = _system(case["nd"], case["nx"], case["ny"], seed)
        s = {"a": torch.from_numpy(a).cuda(), "b": torch.from_numpy(b).cuda()}
    else:
        f, t, m = _images(case, seed)
        net = unet.UNet(case["batch"], case["H"], case["W"], seed=seed)
        s = {"net": net, "f": f, "t": t, "m": m, "scale": 1.0 / float(m.sum()), "out": torch.empty_like(t)}
    s["case"] = case
    return s


def run(s):
    case = s["case"]
    k = case["kind"]
    if k == "run":
        return _run_run(case, s)
    if k == "batch":
        return _run_batch(case, s)
    if k == "host":
        x = np.zeros(case["nx"] * case["ny"])
        s["solver"].solve(s["a"], s["b"], x)
        return x
    if k == "lines":
        return tdma_lines(*s["lines"])
    if k == "fgmres":
        x = torch.zeros_like(s["b"])
        fgmres(case["nd"], case["nx"], case["ny"], s["a"], s["b"], x, case["tol"], prec=case["prec"])
        return x
    if not case["train"]:
        s["net"].forward(s["f"], s["out"])
        return s["out"]
    loss = s["net"].loss_grad(s["f"], s["t"], s["m"], scale=s["scale"])
    s["net"].adam(1e-4)
    return [loss, s["net"].grads()]


def exact(case, seed):
    k = case["kind"]
    if k in ("host", "fgmres"):
        return _system(case["nd"], case["nx"], case["ny"], seed)[2]
    if k == "lines":
        aw, ap, ae, d = _lines(case["n"], case["nlines"], seed)
        n = case["n"]
        P, Q, x = np.zeros_like(ap), np.zeros_like(ap), np.zeros_like(ap)
        for i in range(n):
            den = ap[:, i] + (aw[:, i] * P[:, i - 1] if i else 0.0)
            P[:, i] = -ae[:, i] / den
            Q[:, i] = (d[:, i] - (aw[:, i] * Q[:, i - 1] if i else 0.0)) / den
        x[:, n - 1] = Q[:, n - 1]
        for i in range(n - 2, -1, -1):
            x[:, i] = P[:, i] * x[:, i + 1] + Q[:, i]
        return x
    if k == "unet":
        f, t, m = _images(case, seed)
        p = torch.from_numpy(unet.init_params(seed)).cuda().double().requires_grad_(case["train"])
        grad = torch.zeros_like(p)
        outs, loss = [], 0.0
        for q in range(case["batch"]):
            y = _network64(p, f[q:q + 1].double())
            if case["train"]:
                part = (m[q:q + 1].double() * (y - t[q:q + 1].double()) ** 2).sum() / float(m.sum())
                grad += torch.autograd.grad(part, p)[0]
                loss += float(part)
            else:
                outs.append(y)
        return [loss, grad] if case["train"] else torch.cat(outs)
    return None      # a whole outer iteration has no short restatement


def _cells(case):
    if case["kind"] == "batch" and case["uneven"]:
        return case["n"] * 9 * case["nxr"] * case["nyr"] // 16     # the mean of the drawn sizes
    return case.get("n", 1) * (case["nxr"] + 2) * (case["nyr"] + 2)


def work(case):
    """Inputs read once and outputs written once.  An outer iteration reads
    the state and the grid metrics (41 planes), assembles and solves three
    systems and writes the state (13 planes)."""
    k = case["kind"]
    if k in ("run", "batch"):
        return {"bytes": 8.0 * 54 * _cells(case) * case["iters"], "flops": 600.0 * _cells(case) * case["iters"]}
    if k in ("host", "fgmres"):
        n = case["nx"] * case["ny"]
        return {"bytes": 8.0 * (case["nd"] + 2) * n, "flops": 15 * 6.0 * case["nd"] * n}
    if k == "lines":
        n = case["n"] * case["nlines"]
        return {"bytes": 40.0 * n, "flops": 8.0 * n}
    H, W = case["H"], case["W"]
    lv = (0, 0, 1, 1, 2, 2, 3, 3, 2, 2, 1, 1, 0, 0)
    fl = case["batch"] * sum(18.0 * (H >> q) * (W >> q) * ci * co for (ci, co), q in zip(unet.LAYERS, lv))
    planes = 4.0 * case["batch"] * H * W
    par = 4.0 * unet.param_count()
    if case["train"]:
        return {"bytes": planes * 13 + 8 * par, "flops": 3 * fl}
    return {"bytes": planes * 12 + par, "flops": fl}

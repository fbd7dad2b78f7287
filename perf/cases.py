"""The work that users of this library have it do, as cases that can be timed.

Every case goes through the public entry points of sodecl_b200: `Integrator`
(device buffers through `launch`, host arrays through `upload` and `run`), the
reference's `sodecl.sodecl()` call, `fit.trajectory_mse` with its backward
pass, and `Batch`.  The systems are the two that ship with the package: the
6-state oculomotor model and the Kuramoto model of N phases.  Sizes are those
of the package's workloads and tests, over their range: from a call on two
orbits to a sweep of a million.

Steps are small enough for every orbit to stay finite and well conditioned
(oculomotor: 1e-6 to 2e-6 explicit, 1e-4 to 1e-3 implicit; Kuramoto: 0.01 to
0.05), as a user's are.

`exact` integrates the same inputs with plain torch operations in 64 bits.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from sodecl_b200 import Integrator, system_path
from sodecl_b200.batch import Batch
from sodecl_b200.fit import Adjoint, trajectory_mse
from sodecl_b200.sodecl import sodecl

NOMINAL = (120.0, 1.5, 0.0045, 0.05, 600.0, 9.0)
OCULOMOTOR_Y0 = (0.0, 0.0, 0.0, 0.0, 0.0, 2.0)
SOLVER_ID = {"se": 0, "euler": 1, "rk4": 2, "ie": 3, "im": 4}

# the classes of an uneven sweep: (system, solver, equations, parameters, dt)
BATCH_CLASSES = tuple(("kuramoto", solver, N, N + 1, 0.01) for N in (4, 16, 64) for solver in ("euler", "rk4", "ie")) + \
    (("oculomotor", "euler", 6, 6, 1e-6), ("oculomotor", "rk4", 6, 6, 1e-6), ("oculomotor", "ie", 6, 6, 1e-3))


def _launch(name, system, solver, orbits, steps, ksteps, dt, neq=6, precision="fp64", lanes=1):
    return dict(name=name, kind="launch", system=system, solver=solver, orbits=orbits, steps=steps, ksteps=ksteps,
                dt=dt, neq=neq, precision=precision, lanes=lanes)


def listed():
    return [
        # One call of the reference's Python function, as its README's example makes it: two orbits of a
        # three-oscillator stochastic Kuramoto model.  All latency: a new manager, one thousand dependent steps.
        dict(name="readme_sde_call", kind="call", system="kuramoto", solver="se", orbits=2, steps=1000, ksteps=40,
             dt=0.05, neq=3),
        # A small deterministic sweep: 1024 orbits of eight phases leave most of the GPU idle.
        _launch("small_kuramoto_euler", "kuramoto", "euler", 1024, 1000, 10, 0.05, neq=8),
        # The large parameter sweep that the library is for, device to device.
        _launch("rk4_sweep_2p20", "oculomotor", "rk4", 1 << 20, 2000, 400, 1e-6),
        # The same sweep at an ordinary, odd size with numpy arrays in and all records out.
        dict(name="rk4_host_records", kind="host", system="oculomotor", solver="rk4", orbits=65553, steps=2000,
             ksteps=20, dt=1e-6, neq=6),
        # In single precision, records as float.
        _launch("rk4_fp32", "oculomotor", "rk4", (1 << 18) + 3, 2000, 400, 1e-6, precision="fp32"),
        # Implicit midpoint at the reference's Newton settings.
        _launch("implicit_midpoint", "oculomotor", "im", 1 << 17, 200, 50, 1e-4),
        # Implicit Euler at a coarse step (about forty Newton passes a step), an odd number of orbits.
        _launch("implicit_euler", "oculomotor", "ie", 16411, 100, 50, 1e-3),
        # Stochastic Kuramoto of 32 phases with sixteen lanes per orbit: wide systems and the noise stream.
        _launch("sde_kuramoto32", "kuramoto", "se", 1 << 16, 200, 100, 0.01, neq=32, lanes=16),
        # Every step recorded: the run of a user who plots or post-processes whole trajectories.
        _launch("euler_dense_records", "oculomotor", "euler", 1 << 18, 128, 1, 1e-6),
        # The adaptive solver at its default tolerances.
        _launch("adaptive", "oculomotor", "dp45", 1 << 17, 200, 20, 1e-4),
        # One iteration of model fitting: loss and its gradient with respect to parameters and initial values.
        dict(name="fit_gradient", kind="fit", system="oculomotor", solver="rk4", orbits=1 << 15, steps=1000,
             ksteps=100, dt=2e-6, neq=6),
        # An uneven sweep in one persistent launch: twelve system x solver classes, step counts from 100 to 1000.
        dict(name="uneven_batch", kind="batch", orbits=4099, least=100, most=1000),
    ]


def draw(rng):
    """One more case of the same ranges, its size log-uniform and mostly odd."""
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["call", "kuramoto", "kuramoto", "rk4", "fp32", "host", "implicit", "dense", "adaptive", "fit",
                       "batch"])
    if kind == "call":
        if rng.random() < 0.5:
            return dict(kind="call", system="kuramoto", solver=rng.choice(["se", "euler", "rk4"]), orbits=size(1, 64),
                        steps=40 * size(5, 25), ksteps=40, dt=0.05, neq=size(2, 8))
        return dict(kind="call", system="oculomotor", solver=rng.choice(["se", "euler", "rk4"]), orbits=size(1, 256),
                    steps=100 * size(5, 20), ksteps=100, dt=1e-6, neq=6)
    if kind == "kuramoto":
        neq = size(3, 64)
        lanes = rng.choice([1, 2 ** min(5, max(1, (neq - 1).bit_length() - 1))])
        solver = rng.choice(["se", "se", "euler", "rk4", "ie"])
        steps = 20 * size(5, 20)
        cost = neq * neq * steps * {"se": 1, "euler": 1, "rk4": 4, "ie": 8}[solver]
        c = _launch(None, "kuramoto", solver, size(64, max(65, min(1 << 16, 2e9 / cost))), steps, 20, 0.01, neq=neq,
                    precision="fp64" if solver == "ie" else rng.choice(["fp64", "fp64", "fp32"]), lanes=lanes)
    elif kind == "rk4":
        c = _launch(None, "oculomotor", rng.choice(["rk4", "rk4", "se"]), size(64, 1 << 19), 100 * size(2, 20), 100,
                    1e-6)
    elif kind == "fp32":
        c = _launch(None, "oculomotor", rng.choice(["rk4", "euler"]), size(1024, 1 << 19), 100 * size(2, 20), 100,
                    1e-6, precision="fp32")
    elif kind == "host":
        ksteps = rng.choice([10, 25, 50])
        return dict(kind="host", system="oculomotor", solver=rng.choice(["euler", "rk4"]), orbits=size(256, 1 << 16),
                    steps=ksteps * size(5, 80), ksteps=ksteps, dt=1e-6, neq=6)
    elif kind == "implicit":
        solver = rng.choice(["im", "ie"])
        c = _launch(None, "oculomotor", solver, size(64, 1 << 16 if solver == "im" else 1 << 14), 20 * size(2, 6), 20,
                    rng.choice([1e-4, 2e-4]) if solver == "im" else rng.choice([5e-4, 1e-3]))
    elif kind == "dense":
        c = _launch(None, "oculomotor", rng.choice(["euler", "rk4"]), size(256, 1 << 18), size(16, 100), 1, 1e-6)
    elif kind == "adaptive":
        c = _launch(None, "oculomotor", "dp45", size(64, 1 << 17), 20 * size(2, 10), 20, 1e-4)
    elif kind == "fit":
        return dict(kind="fit", system="oculomotor", solver=rng.choice(["rk4", "rk4", "euler"]), orbits=size(64, 1 << 15),
                    steps=50 * size(2, 16), ksteps=50, dt=2e-6, neq=6)
    else:
        return dict(kind="batch", orbits=size(100, 4000), least=20, most=size(100, 900))
    del c["name"]
    return c


# ---------------------------------------------------------------------------
# Inputs

def _inputs(case, seed):
    """(t0, y0[n, neq], params[n, npar], counters or None) on the GPU."""
    n, neq = case["orbits"], case["neq"]
    g = torch.Generator("cuda").manual_seed(seed)

    def uniform(lo, hi, *shape):
        return lo + (hi - lo) * torch.rand(*shape, dtype=torch.float64, device="cuda", generator=g)

    noisy = case["solver"] == "se"
    t0 = torch.zeros(n, dtype=torch.float64, device="cuda")
    if case["system"] == "oculomotor":
        p = torch.tensor(NOMINAL, dtype=torch.float64, device="cuda") * uniform(0.5, 1.5, n, 6)
        y0 = torch.tensor(OCULOMOTOR_Y0, dtype=torch.float64, device="cuda").repeat(n, 1)
        # other starting points than the nominal one, so that orbits differ at once
        y0[:, 5] *= uniform(0.5, 1.5, n)
        if noisy:
            p = torch.cat([p, uniform(0.0, 0.1, n, 2)], dim=1)
    else:
        omega = torch.randn(1, neq, dtype=torch.float64, device="cuda", generator=g)
        cols = [uniform(0.0, 5.0, n, 1), omega.expand(n, neq)]
        if noisy:
            cols.append(uniform(0.0, 0.5, n, 1).expand(n, neq))
        p = torch.cat(cols, dim=1).contiguous()
        y0 = uniform(0.0, 2 * math.pi, n, neq)
    counters = None
    if noisy:
        counters = (torch.arange(n, dtype=torch.float64, device="cuda") * 2.0 ** 20 + float(seed % 1000)).contiguous()
    return t0, y0, p.contiguous(), counters


def _npar(case):
    noisy = case["solver"] == "se"
    if case["system"] == "oculomotor":
        return 6 + (2 if noisy else 0)
    return case["neq"] + 1 + (case["neq"] if noisy else 0)


def _nnoi(case):
    if case["solver"] != "se":
        return 0
    return 2 if case["system"] == "oculomotor" else case["neq"]


@functools.lru_cache(maxsize=32)
def _integrator(system, solver, orbits, steps, ksteps, dt, neq, npar, nnoi, precision, lanes):
    """A configured program; a user's program keeps it while its inputs change."""
    return Integrator(system_path(system), solver, dt=dt, tspan=(steps - 0.5) * dt, ksteps=ksteps, neq=neq, npar=npar,
                      nnoi=nnoi, orbits=orbits, precision=precision, record_f32=precision == "fp32", lanes=lanes)


def _handle(case):
    return _integrator(case["system"], case["solver"], case["orbits"], case["steps"], case["ksteps"], case["dt"],
                       case["neq"], _npar(case), _nnoi(case), case.get("precision", "fp64"), case.get("lanes", 1))


@functools.lru_cache(maxsize=4)
def _batch():
    b = Batch()
    for system, solver, neq, npar, dt in BATCH_CLASSES:
        b.add_class(system_path(system), solver, neq=neq, npar=npar, dt=dt)
    return b.compile()


def _batch_items(case, seed):
    """(class, steps, y0 per class, params per class) of an uneven sweep."""
    rng = np.random.default_rng(seed)
    n = case["orbits"]
    cls = rng.permutation(np.arange(n) % len(BATCH_CLASSES)).astype(np.int32)
    steps = np.exp(rng.uniform(np.log(case["least"]), np.log(case["most"]), n)).astype(np.int64)
    y0, p = [], []
    for c in cls:
        system, _, neq, _, _ = BATCH_CLASSES[c]
        if system == "oculomotor":
            y0.append(np.array(OCULOMOTOR_Y0))
            p.append(np.array(NOMINAL) * rng.uniform(0.5, 1.5, 6))
        else:
            y0.append(rng.uniform(0, 2 * np.pi, neq))
            p.append(np.concatenate([[rng.uniform(0, 5)], rng.normal(size=neq)]))
    return cls, steps, y0, p


def _targets(case, y0, p, seed):
    """Noisy observations to fit: trajectories of other parameters (integrated
    at a coarser step, which is far below the noise) plus N(0, 1e-2)."""
    g = torch.Generator("cuda").manual_seed(seed + 1)
    true_p = p * (0.95 + 0.1 * torch.rand(p.shape, dtype=torch.float64, device="cuda", generator=g))
    h = case["dt"] * case["ksteps"] / 10
    y = y0
    out = [y0.T]
    for _ in range(case["steps"] // case["ksteps"]):
        for _ in range(10):
            y = torch.stack(_rk4(_oculomotor, list(y.unbind(1)), list(true_p.unbind(1)), h), dim=1)
        out.append(y.T)
    rec = torch.stack(out)
    return (rec + 1e-2 * torch.randn(rec.shape, dtype=torch.float64, device="cuda", generator=g)).contiguous()


def prepare(case, seed):
    if case["kind"] == "batch":
        cls, steps, y0, p = _batch_items(case, seed)
        return dict(case=case, batch=_batch(), cls=cls, steps=steps, t0=np.zeros(len(cls)), y0=np.concatenate(y0),
                    p=np.concatenate(p), by_class=[np.flatnonzero(cls == k) for k in range(len(BATCH_CLASSES))])
    t0, y0, p, counters = _inputs(case, seed)
    s = dict(case=case)
    if case["kind"] in ("call", "host"):
        s.update(t0=t0.cpu().numpy(), y0=y0.cpu().numpy(), p=p.cpu().numpy(),
                 counters=None if counters is None else counters.cpu().numpy())
        if case["kind"] == "host":
            s["sim"] = _handle(case)
        return s
    s["sim"] = _handle(case)
    if case["kind"] == "fit":
        s.update(t0=t0, y0=y0, p=p, targets=_targets(case, y0, p, seed), adjoint=Adjoint(s["sim"]))
        return s
    n, neq = case["orbits"], case["neq"]
    s.update(t0=t0, y0=y0, p=p, counters0=counters, t=torch.empty_like(t0), y=torch.empty_like(y0))
    s["records"] = torch.empty((s["sim"].num_records, neq, n), device="cuda",
                               dtype=torch.float32 if case["precision"] == "fp32" else torch.float64)
    s["counters"] = None if counters is None else torch.empty_like(counters)
    s["steps_h"] = torch.empty(n, dtype=torch.float64, device="cuda") if case["solver"] == "dp45" else None
    s["passes"] = torch.empty(n, dtype=torch.int64, device="cuda") if case["solver"] in ("ie", "im", "dp45") else None
    return s


# ---------------------------------------------------------------------------
# One pass

def run(s):
    return _RUN[s["case"]["kind"]](s)


def _run_call(s):
    c = s["case"]
    _, records = sodecl(0, 0, system_path(c["system"]), s["y0"], s["p"], SOLVER_ID[c["solver"]], c["orbits"],
                        c["neq"], _nnoi(c), c["dt"], (c["steps"] - 0.5) * c["dt"], c["ksteps"], 0,
                        counters=s["counters"])
    return records


def _run_host(s):
    sim = s["sim"]
    sim.upload(s["t0"], s["y0"], s["p"], s["counters"])
    return sim.run()


def _run_launch(s):
    sim, c = s["sim"], s["case"]
    s["t"].copy_(s["t0"])
    s["y"].copy_(s["y0"])
    counters = s["counters"]
    if counters is not None:
        counters.copy_(s["counters0"])
    elif s["steps_h"] is not None:  # the adaptive solver's step sizes: none yet
        counters = s["steps_h"].zero_()
    passes = None if s["passes"] is None else s["passes"].zero_()
    sim.launch(t=s["t"].data_ptr(), y=s["y"].data_ptr(), params=s["p"].data_ptr(),
               counters=None if counters is None else counters.data_ptr(), records=s["records"].data_ptr(),
               newton_passes=None if passes is None else passes.data_ptr(),
               stream=torch.cuda.current_stream().cuda_stream)
    out = dict(records=s["records"], t=s["t"])
    if c["precision"] == "fp64":  # in single precision the last record is the state
        out["y"] = s["y"]
    if s["counters"] is not None:
        out["counters"] = counters
    if passes is not None:
        out["passes"] = passes
    return out


def _run_fit(s):
    p = s["p"].requires_grad_(True)
    y0 = s["y0"].requires_grad_(True)
    p.grad = y0.grad = None
    loss = trajectory_mse(p, y0, s["t0"], s["targets"], s["adjoint"])
    loss.sum().backward()
    return dict(loss=loss.detach(), grad_params=p.grad, grad_y0=y0.grad)


def _run_batch(s):
    b = s["batch"]
    b.set_items(s["cls"], s["steps"], s["t0"], s["y0"], s["p"])
    b.run()
    t, y, _, passes, _ = b.results()
    return dict(t=t, passes=passes,
                y=[np.stack([y[i] for i in items]) if len(items) else np.zeros(1) for items in s["by_class"]])


_RUN = {"call": _run_call, "host": _run_host, "launch": _run_launch, "fit": _run_fit, "batch": _run_batch}


# ---------------------------------------------------------------------------
# The work a pass cannot do without

def _rhs_flops(system, neq):
    return 33 if system == "oculomotor" else 3 * neq * neq + 3 * neq


def _step_flops(system, solver, neq, nnoi=0):
    f = _rhs_flops(system, neq)
    if solver == "rk4":
        return 4 * f + 14 * neq
    if solver == "dp45":
        return 7 * f + 84 * neq
    if solver in ("ie", "im"):  # at least two Newton passes: one that moves, one that stops
        return 2 * f + 12 * neq
    return f + 3 * neq + 10 * nnoi


def work(case):
    if case["kind"] == "batch":
        mean = (case["most"] - case["least"]) / math.log(case["most"] / case["least"])
        each = case["orbits"] / len(BATCH_CLASSES)
        return dict(bytes=sum(each * (8 * (2 * neq + npar) + 32) for _, _, neq, npar, _ in BATCH_CLASSES),
                    flops=sum(each * mean * _step_flops(system, solver, neq)
                              for system, solver, neq, _, _ in BATCH_CLASSES))
    n, neq = case["orbits"], case["neq"]
    steps = -(-case["steps"] // case["ksteps"]) * case["ksteps"]
    records = steps // case["ksteps"] + 1
    state = 8 * n * (2 * neq + 2 + _npar(case))
    flops = n * steps * _step_flops(case["system"], case["solver"], neq, _nnoi(case))
    if case["kind"] == "fit":  # the reverse sweep: one vector-Jacobian product per stage, about twice a right-hand side
        return dict(bytes=8 * n * (records * neq + 2 * neq + 2 * _npar(case) + 1), flops=3 * flops)
    if case["solver"] == "dp45":  # at least one attempt an interval
        flops = n * (records - 1) * _step_flops(case["system"], "dp45", neq)
    size = 4 if case.get("precision") == "fp32" else 8
    return dict(bytes=state + size * n * neq * records, flops=flops)


# ---------------------------------------------------------------------------
# The same in plain 64-bit torch

def _oculomotor(y, p):
    def burst(x):
        return torch.where(x > 0, p[4] * (1.0 - torch.exp(-torch.clamp(x, min=0.0) / p[5])),
                           -(p[0] / p[1]) * x * torch.exp(torch.clamp(x, max=0.0) / p[1]))

    pos, vel = 1.0 / (0.15 * 0.012), 1.0 / 0.15 + 1.0 / 0.012
    drive = y[3] - y[4]
    it = 1.0 / p[2]
    return [y[1], -(vel * y[1]) - pos * y[0] + pos * y[2] + vel * drive, -(y[2] / 25.0) + drive,
            it * (-y[3] - p[3] * y[3] * y[4] * y[4] + burst(y[5])),
            it * (-y[4] - p[3] * y[4] * y[3] * y[3] + burst(-y[5])), -drive]


def _rk4(f, y, p, h):
    k1 = f(y, p)
    k2 = f([a + 0.5 * h * k for a, k in zip(y, k1)], p)
    k3 = f([a + 0.5 * h * k for a, k in zip(y, k2)], p)
    k4 = f([a + h * k for a, k in zip(y, k3)], p)
    return [a + (q1 + 2.0 * q2 + 2.0 * q3 + q4) * h / 6.0 for a, q1, q2, q3, q4 in zip(y, k1, k2, k3, k4)]


def _kuramoto(y, p):
    """y [n, N]; p [n, 1 + N ...]"""
    N = y.shape[1]
    return torch.sin(y[:, None, :] - y[:, :, None]).sum(2) * (p[:, :1] / N) + p[:, 1:N + 1]


def _kuramoto_rk4(y, p, h):
    k1 = _kuramoto(y, p)
    k2 = _kuramoto(y + 0.5 * h * k1, p)
    k3 = _kuramoto(y + 0.5 * h * k2, p)
    k4 = _kuramoto(y + h * k3, p)
    return y + (k1 + 2.0 * k2 + 2.0 * k3 + k4) * h / 6.0


def _shr(x, k):
    """Logical right shift of 64-bit words held in int64."""
    return (x >> k) & ((1 << (64 - k)) - 1)


def _threefry(c0, c1):
    """Threefry-2x64, 20 rounds, key {0, 0xf00dcafe}."""
    def wrap(v):
        v &= (1 << 64) - 1
        return v - (1 << 64) if v >> 63 else v

    key = [0, 0xf00dcafe]
    key.append(0x1BD11BDAA9FC1A22 ^ key[0] ^ key[1])
    rot = (16, 42, 12, 31, 16, 32, 24, 21)
    x0, x1 = c0 + wrap(key[0]), c1 + wrap(key[1])
    for r in range(20):
        x0 = x0 + x1
        k = rot[r % 8]
        x1 = ((x1 << k) | _shr(x1, 64 - k)) ^ x0
        if r % 4 == 3:
            j = r // 4 + 1
            x0 = x0 + wrap(key[j % 3])
            x1 = x1 + wrap(key[(j + 1) % 3] + j)
    return x0, x1


def _normals(counters, nnoi, h):
    """One step's Gaussian increments [n, nnoi], and the counters after it."""
    n, pairs = counters.numel(), (nnoi + 1) // 2
    c1 = counters.to(torch.int64)[:, None] + torch.arange(pairs, device=counters.device)
    c0 = torch.arange(n, device=counters.device, dtype=torch.int64)[:, None].expand(n, pairs)
    w0, w1 = _threefry(c0, c1)
    u0, u1 = ((1 + _shr(w, 11)).double() * float.fromhex("0x1.fffffffffffffp-54") for w in (w0, w1))
    rad, ang = torch.sqrt(-2.0 * torch.log(u0)), 2.0 * math.pi * u1
    z = torch.stack([rad * torch.cos(ang), rad * torch.sin(ang)], dim=2).reshape(n, 2 * pairs) * math.sqrt(h)
    return z[:, :nnoi], counters + pairs


def _band_solve(up, lo, d, v):
    """The reference's elimination: up[i] row i's super-diagonal (zero for the
    last two rows), lo[i] row i+1's sub-diagonal, d the diagonal; lists."""
    d, v, n = list(d), list(v), len(d)
    for i in range(1, n):
        if i < n - 2:
            f = up[i] / d[i - 1]
            d[i] = d[i] - f * lo[i - 1]
            v[i] = v[i] - f * v[i - 1]
    x = [None] * n
    x[n - 1] = v[n - 1] / d[n - 1]
    for i in range(n - 2, -1, -1):
        x[i] = (v[i] - lo[i] * x[i + 1]) / d[i]
    return x


def _oculomotor_bands(y, p):
    one = torch.ones_like(y[0])
    pos, vel = 1.0 / (0.15 * 0.012), 1.0 / 0.15 + 1.0 / 0.012
    up = [one, pos * one, one, -(2.0 * p[3] * y[4] * y[3]) / p[2], None, None]
    lo = [-pos * one, 0.0 * one, 0.0 * one, -(2.0 * p[3] * y[4] * y[3]) / p[2], one]
    d = [0.0 * one, -vel * one, -one / 25.0, -(p[3] * y[4] * y[4] + 1.0) / p[2], -(p[3] * y[3] * y[3] + 1.0) / p[2],
         0.0 * one]
    return up, lo, d


def _kuramoto_bands(y, p):
    N = len(y)
    Y = torch.stack(y, dim=1)
    c = torch.cos(Y[:, None, :] - Y[:, :, None]) * (p[:, :1, None] / N)
    up = [c[:, i, i + 1] if i < N - 2 else None for i in range(N)]
    lo = [c[:, i + 1, i] for i in range(N - 1)]
    diag = torch.diagonal(c, dim1=1, dim2=2) - c.sum(2)
    return up, lo, list(diag.unbind(1))


def _newton_step(solver, f, bands, y, p, h, tol=1e-7, limit=1000):
    """One implicit step of the list-of-equations state y."""
    x = list(y)
    live = torch.ones_like(y[0], dtype=torch.bool)
    w = 0.5 if solver == "im" else 1.0
    for _ in range(limit):
        at = [(a + b) * 0.5 for a, b in zip(y, x)] if solver == "im" else x
        r = [b - a - k * h for a, b, k in zip(y, x, f(at, p))]
        norm = torch.sqrt(sum(v * v for v in r)) if solver == "im" else sum(v.abs() for v in r)
        live = live & ~(norm < tol)
        if not bool(live.any()):
            break
        up, lo, d = bands(at, p)
        dx = _band_solve([None if u is None else -w * h * u for u in up], [-w * h * v for v in lo],
                         [1.0 - w * h * v for v in d], r)
        x = [torch.where(live, b - e, b) for b, e in zip(x, dx)]
    return x


def _dp_records(y, p, dt, ksteps, chunks, rtol=1e-6, atol=1e-9):
    """Dormand-Prince 5(4) on the record grid, every orbit with its own steps;
    None where an interval takes too many attempts to be worth waiting for."""
    A = ((), (1 / 5,), (3 / 40, 9 / 40), (44 / 45, -56 / 15, 32 / 9),
         (19372 / 6561, -25360 / 2187, 64448 / 6561, -212 / 729),
         (9017 / 3168, -355 / 33, 46732 / 5247, 49 / 176, -5103 / 18656),
         (35 / 384, 0.0, 500 / 1113, 125 / 192, -2187 / 6784, 11 / 84))
    E = (71 / 57600, 0.0, -71 / 16695, 71 / 1920, -17253 / 339200, 22 / 525, -1 / 40)
    t = torch.zeros_like(y[0])
    h = torch.full_like(t, dt)
    out, total = [torch.stack(y)], 0
    for _ in range(chunks):
        end = t + ksteps * dt
        rejected = torch.zeros_like(t, dtype=torch.bool)
        while bool((t < end).any()):
            total += 1
            if total > 4000:
                return None
            live = t < end
            last = t + h >= end
            hh = torch.where(last, end - t, h)
            k = []
            for row in A:
                k.append(_oculomotor([a + hh * sum(c * q[e] for c, q in zip(row, k) if c) if row else a
                                      for e, a in enumerate(y)], p))
            y5 = [a + hh * sum(c * q[e] for c, q in zip(A[6], k) if c) for e, a in enumerate(y)]
            acc = 0.0
            for e, a in enumerate(y):
                err = hh * sum(c * q[e] for c, q in zip(E, k) if c)
                acc = acc + (err / (atol + rtol * torch.maximum(a.abs(), y5[e].abs()))) ** 2
            err = torch.sqrt(acc / len(y))
            fac = torch.clamp(torch.where(err > 0, 0.9 * torch.exp(-0.2 * torch.log(err)), 5.0), 0.2, 5.0)
            ok = live & (err <= 1)
            t = torch.where(ok, torch.where(last, end, t + hh), t)
            y = [torch.where(ok, b, a) for a, b in zip(y, y5)]
            grown = hh * torch.where(rejected, torch.clamp(fac, max=1.0), fac)
            h = torch.where(ok, torch.where(last, h, grown), torch.where(live, hh * torch.clamp(fac, max=1.0), h))
            rejected = torch.where(live, ~ok, rejected)
        out.append(torch.stack(y))
    return t, torch.stack(out)


def _integrate(case, t, y, p, counters):
    """(t, y[n, neq], records[record, neq, n], counters)."""
    h = float("%g" % case["dt"])
    steps, ksteps, solver, neq = case["steps"], case["ksteps"], case["solver"], case["neq"]
    chunks = math.ceil((steps - 0.5) * case["dt"] / (case["dt"] * ksteps))
    ocm = case["system"] == "oculomotor"
    cols = [c.contiguous() for c in p.unbind(1)]
    out = [y.T]
    pos = 1.0 / 0.15 + 1.0 / 0.012
    for _ in range(chunks):
        for _ in range(ksteps):
            if solver in ("ie", "im"):
                if ocm:
                    x = _newton_step(solver, _oculomotor, _oculomotor_bands, list(y.unbind(1)), cols, h)
                else:
                    x = _newton_step(solver, lambda a, q: list(_kuramoto(torch.stack(a, dim=1), q).unbind(1)),
                                     _kuramoto_bands, list(y.unbind(1)), p, h)
                y = torch.stack(x, dim=1)
            elif solver == "rk4":
                y = torch.stack(_rk4(_oculomotor, list(y.unbind(1)), cols, h), dim=1) if ocm else _kuramoto_rk4(y, p, h)
            else:
                f = torch.stack(_oculomotor(list(y.unbind(1)), cols), dim=1) if ocm else _kuramoto(y, p)
                new = y + f * h
                if solver == "se":
                    z, counters = _normals(counters, _nnoi(case), h)
                    if ocm:
                        new[:, 1] += pos * (y[:, 3] - y[:, 4]) * p[:, 6] * z[:, 0] + p[:, 7] * z[:, 1]
                    else:
                        new = new + p[:, neq + 1:] * z
                y = new
            t = t + h
        out.append(y.T)
    return t, y, torch.stack(out), counters


def _exact_fit(case, seed):
    from torch.utils.checkpoint import checkpoint

    t0, y0, p, _ = _inputs(case, seed)
    targets = _targets(case, y0, p, seed)
    h, rk4 = float("%g" % case["dt"]), case["solver"] == "rk4"
    p.requires_grad_(True)
    y0.requires_grad_(True)

    def ten(*a):
        y, q = list(a[:6]), list(a[6:])
        for _ in range(10):
            y = _rk4(_oculomotor, y, q, h) if rk4 else [u + k * h for u, k in zip(y, _oculomotor(y, q))]
        return tuple(y)

    y, q = tuple(y0.unbind(1)), tuple(p.unbind(1))
    loss = ((torch.stack(y) - targets[0]) ** 2).sum(0)
    chunks = case["steps"] // case["ksteps"]
    for r in range(chunks):
        for _ in range(case["ksteps"] // 10):
            y = checkpoint(ten, *y, *q, use_reentrant=False)
        loss = loss + ((torch.stack(y) - targets[r + 1]) ** 2).sum(0)
    loss = loss / ((chunks + 1) * 6)
    loss.sum().backward()
    return dict(loss=loss.detach(), grad_params=p.grad, grad_y0=y0.grad)


def _exact_batch(case, seed):
    """The classes of the explicit solvers; the implicit ones would take minutes."""
    cls, steps, y0, p = _batch_items(case, seed)
    out, t = [], np.zeros(len(cls))
    for k, (system, solver, neq, _, dt) in enumerate(BATCH_CLASSES):
        items = np.flatnonzero(cls == k)
        for i in items:  # the time, one addition a step
            t[i] = np.cumsum(np.full(steps[i], dt))[-1] if steps[i] > 0 else 0.0
        if solver == "ie" or not len(items):
            out.append(None)
            continue
        y = torch.tensor(np.stack([y0[i] for i in items]), device="cuda")
        q = torch.tensor(np.stack([p[i] for i in items]), device="cuda")
        left = torch.tensor(steps[items], device="cuda")[:, None]
        for s in range(int(steps[items].max())):
            if system == "oculomotor":
                a, b = list(y.unbind(1)), list(q.unbind(1))
                new = _rk4(_oculomotor, a, b, dt) if solver == "rk4" else [u + v * dt for u, v in zip(a, _oculomotor(a, b))]
                new = torch.stack(new, dim=1)
            else:
                new = _kuramoto_rk4(y, q, dt) if solver == "rk4" else y + _kuramoto(y, q) * dt
            y = torch.where(left > s, new, y)
        out.append(y.cpu().numpy())
    return dict(t=t, passes=None, y=out)


def exact(case, seed):
    if case["kind"] == "batch":
        return _exact_batch(case, seed)
    if case["kind"] == "fit":
        return _exact_fit(case, seed)
    t, y, p, counters = _inputs(case, seed)
    if case["solver"] == "dp45":
        got = _dp_records(list(y.unbind(1)), [c.contiguous() for c in p.unbind(1)], case["dt"], case["ksteps"],
                          math.ceil((case["steps"] - 0.5) / case["ksteps"]))
        return None if got is None else dict(records=got[1], t=got[0], y=got[1][-1].T, passes=None)
    t, y, records, counters = _integrate(case, t, y, p, counters)
    if case["kind"] == "call":  # (orbits * neq, records): row equation * orbits + orbit
        return records.reshape(records.shape[0], -1).T
    if case["kind"] == "host":
        return records
    out = dict(records=records, t=t)
    if case["precision"] == "fp64":
        out["y"] = y
    if counters is not None:
        out["counters"] = counters
    if case["solver"] in ("ie", "im"):
        out["passes"] = None
    return out

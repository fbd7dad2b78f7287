"""Speculative steps on the GPU against the programs without them (a file that
mentions printf gets none)."""
import numpy as np
import pytest

from sodecl_b200 import Integrator, system_path
from sodecl_b200.batch import Batch
from test_device_math import pairs

pytestmark = pytest.mark.gpu

HEAD = "void sode_system(double t, double y[_numeq_], double yout[_numeq_], double p[_numpar_])\n{\n"
NONE = "/* printf */\n"


def run(source, solver, y0, p, **kw):
    """(records, status) with speculative steps and without."""
    out = []
    for text in (source, NONE + source):
        args = dict(dt=0.01, tspan=0.095, ksteps=2, neq=y0.shape[1], npar=p.shape[1], orbits=len(y0), fmad=False)
        with Integrator(None, solver, system_src=text, **{**args, **kw}) as sim:
            assert ("#define SODECL_SPECULATE 1" in sim.program_source) == (text is source)
            sim.upload(np.zeros(len(y0)), y0, p)
            out.append((sim.run(), *sim.status()))
    return out


@pytest.mark.parametrize("solver", ["dp45"])
def test_quotients_keep_a_zeros_sign(solver):
    """The direction of every state hangs on the sign of a zero quotient."""
    source = HEAD + "\tfor (int i = 0; i < _numeq_; i++) yout[i] = copysign(1.0, p[i] / p[4]);\n}\n"
    zeros = np.array([[0.0, -0.0, 0.0, -0.0]])
    p = np.concatenate([np.repeat(zeros, 4, axis=0), np.array([[3.0], [-3.0], [1e-20], [-1e20]])], axis=1)
    got, plain = run(source, solver, np.ones((4, 4)), p)
    want = 1 + np.sign(p[:, 4:5]) * np.array([1.0, -1.0, 1.0, -1.0]) * got[0].shape[0] * 0.02
    for a, b in zip(got, plain):
        np.testing.assert_array_equal(a, b)
    assert np.all(np.sign(got[0][-1].T - 1) == np.sign(want - 1))


@pytest.mark.parametrize("lanes", [1, 2])
@pytest.mark.parametrize("precision,division", [("fp64", "reciprocal"), ("fp64", "ieee"), ("fp32", "reciprocal"), ("fp32", "ieee")])
def test_quotients_are_ieee_in_every_mode(precision, division, lanes):
    """One Euler step of size 1 from -0 is the quotient itself: random pairs, pairs
    whose quotient lies next to the middle between two numbers, and specials."""
    a, b = pairs(53 if precision == "fp64" else 24, 200000, 6)
    np.nan_to_num(a, copy=False, nan=np.nan, posinf=np.inf, neginf=-np.inf)  # (quiet NaNs alone)
    np.nan_to_num(b, copy=False, nan=np.nan, posinf=np.inf, neginf=-np.inf)
    if precision == "fp32":
        a = np.concatenate([a, np.float32([float.fromhex("0x1.d074d8p+0")])])
        b = np.concatenate([b, np.float32([float.fromhex("0x1.527e7cp+0")])])
    source = "double sode_system_row(int i, double t, double y[_numeq_], double p[_numpar_]) { return p[0] / p[1]; }\n" + HEAD + \
        "\tfor (int i = 0; i < _numeq_; i++) yout[i] = sode_system_row(i, t, y, p);\n}\n"
    n = a.size
    with Integrator(None, "euler", system_src=source, dt=1.0, tspan=0.5, ksteps=1, neq=2, npar=2, orbits=n, lanes=lanes,
                    precision=precision, division=division) as sim:
        assert sim.division == division
        sim.upload(np.zeros(n), np.full((n, 2), -0.0), np.stack([a, b], axis=1).astype(np.float64))
        got = sim.run()[1].astype(a.dtype)
    with np.errstate(all="ignore"):
        want = a / b
    word = np.int64 if precision == "fp64" else np.int32
    nan = np.isnan(want)
    for row in got:
        assert np.isnan(row[nan]).all()
        np.testing.assert_array_equal(row[~nan].view(word), want[~nan].view(word))


# grows through 2^30 within a run; products beside every function and quotient
GROW = "double sode_system_row(int i, double t, double y[_numeq_], double p[_numpar_])\n{\n" \
    "\treturn p[0] * y[i] + p[1] * sin(y[i]) * y[i] - p[2] * y[i] / (3.0 + p[1] * exp(-p[2] * y[i] * y[i]));\n}\n" + HEAD + \
    "\tfor (int i = 0; i < _numeq_; i++) yout[i] = sode_system_row(i, t, y, p);\n}\n"


@pytest.mark.parametrize("fmad", [False, True])
@pytest.mark.parametrize("solver,lanes,precision", [("euler", 1, "fp64"), ("rk4", 1, "fp64"), ("euler", 4, "fp64"), ("rk4", 4, "fp64"),
                                                    ("rk4", 1, "fp32")])
def test_results_do_not_depend_on_where_a_run_begins(solver, lanes, precision, fmad):
    """Orbits that leave the range at different steps: the same last state for
    every record interval, in one launch and in many, alone and side by side,
    and in a batch."""
    n, neq, steps, h = 45, 5, 48, 0.01
    rng = np.random.default_rng(7)
    p = np.stack([rng.uniform(10, 120, n), rng.uniform(0, 3, n), rng.uniform(0.5, 2, n)], axis=1)
    if precision == "fp32":  # past 2^102 instead of 2^30, and to infinity
        p[:, 0] *= 5
    y0 = rng.uniform(0.5, 3.0, (n, neq))
    kw = dict(system_src=GROW, dt=h, neq=neq, npar=3, lanes=lanes, precision=precision, fmad=fmad)

    def run(ksteps, sel=slice(None)):
        m = len(y0[sel])
        with Integrator(None, solver, orbits=m, tspan=(steps - 0.5) * h, ksteps=ksteps, **kw) as sim:
            assert "#define SODECL_SPECULATE 1" in sim.program_source
            sim.upload(np.zeros(m), y0[sel], p[sel])
            return sim.run()[-1]

    want = run(48)
    if precision == "fp64":
        assert (np.abs(want).max(axis=0) > 2.0 ** 31).sum() > n // 3 and (np.abs(want).max(axis=0) < 2.0 ** 29).any()
    for ksteps in (1, 3, 8, 16):
        np.testing.assert_array_equal(run(ksteps), want)
    np.testing.assert_array_equal(run(6, slice(3, 4)), want[:, 3:4])
    if precision == "fp64":
        b = Batch(fmad=fmad)
        b.add_class(None, solver, neq=neq, npar=3, dt=h, lanes=lanes, system_src=GROW)
        b.compile()
        b.set_items(np.zeros(n, np.int32), np.full(n, steps), np.zeros(n), y0.ravel(), p.ravel())
        b.run()
        np.testing.assert_array_equal(np.stack(b.results()[1], axis=1), want)


@pytest.mark.parametrize("solver,lanes", [("euler", 1), ("rk4", 1), ("rk4", 2), ("se", 1), ("dp45", 1)])
def test_orbits_that_stay_outside_or_come_back(solver, lanes):
    """Dividends below 2^-900 for good, divisors of zero, arguments of exp and
    sine beyond their ranges that return: the plain program's bits."""
    source = "double sode_system_row(int i, double t, double y[_numeq_], double p[_numpar_])\n{\n" \
        "\treturn %s - y[i] / p[1] + p[2] / p[3];\n}\n" % ("p[0] * y[i]" if solver == "dp45" else "p[0] * sin(y[i]) * exp(-y[i] * p[1])") + \
        HEAD + "\tfor (int i = 0; i < _numeq_; i++) yout[i] = sode_system_row(i, t, y, p);\n}\n" \
        "double sode_system_stoch_row(int i, double t, double y[_numeq_], double p[_numpar_], double noise[_numnoi_])\n{\n" \
        "\treturn 0.1 * noise[i];\n}\n" \
        "void sode_system_stoch(double t, double y[_numeq_], double stoch[_numeq_], double p[_numpar_], double noise[_numnoi_])\n{\n" \
        "\tfor (int i = 0; i < _numeq_; i++) stoch[i] = sode_system_stoch_row(i, t, y, p, noise);\n}\n"
    y0 = np.array([[1.0, 2.0], [1e-290, 1e-280], [710.0, -720.0], [2.0 ** 31, 5.0], [1e300, 1.0], [1.0, 1.0], [np.nan, np.nan],
                   [np.nan, 1.0], [0.0, -0.0], [740.0, 741.0]])
    p = np.tile([0.5, 0.4, 1.0, 2.0], (len(y0), 1))
    p[1] = [0.0, 0.4, 0.0, 1.0]
    p[5] = [0.5, 0.4, 1.0, 0.0]
    p[4, 1] = p[3, 1] = 0.02  # decays quickly, back into the range
    noisy = {"nnoi": 2, "fmad": False} if solver == "se" else {}
    out = []
    for text in (source, NONE + source):
        with Integrator(None, solver, system_src=text, dt=0.01, tspan=0.995, ksteps=4, neq=2, npar=4, orbits=len(y0),
                        **{"fmad": False, "lanes": lanes, **noisy}) as sim:
            assert ("#define SODECL_SPECULATE 1" in sim.program_source) == (text is source)
            sim.upload(np.zeros(len(y0)), y0, p, np.zeros(len(y0)) if solver == "se" else None)
            out.append(sim.run())
    got, plain = out
    np.testing.assert_array_equal(np.isnan(got), np.isnan(plain))
    if solver == "dp45":
        np.testing.assert_array_equal(got, plain)
    else:  # the library's sin and exp differ in the last bits
        with np.errstate(all="ignore"):
            off = np.abs(got - plain) / np.maximum(np.abs(plain), 1e-300)
        assert np.nanmax(np.where(np.isfinite(plain), off, 0)) <= 1e-12
        np.testing.assert_array_equal(got[~np.isfinite(plain)], plain[~np.isfinite(plain)])


@pytest.mark.parametrize("solver", ["ie", "im"])
def test_implicit_steps_beyond_the_sines_range(solver):
    """Phases past 2^30 from the start, or from some step on: passes and states of
    one thread per orbit, whose sines have no speculative copy."""
    n, neq = 9, 6
    rng = np.random.default_rng(8)
    y0 = rng.uniform(0, 6, (n, neq))
    y0[3:6, 0] += 2.0 ** 31
    p = np.concatenate([np.full((n, 1), 2.0), rng.normal(size=(n, neq))], axis=1)
    p[6:, 1] = 4e9  # one phase runs away: 2^30 after some 27 steps
    out = []
    for lanes in (1, 4):
        with Integrator(system_path("kuramoto"), solver, dt=0.01, tspan=0.395, ksteps=5, neq=neq, npar=neq + 1, orbits=n,
                        lanes=lanes, fmad=False, newton_max_iter=40) as sim:
            sim.upload(np.zeros(n), y0, p)
            out.append((sim.run(), *sim.status()))
    for one, many in zip(*out):
        np.testing.assert_array_equal(many, one)


def test_one_thread_and_lanes_agree_beyond_256_equations():
    n, neq = 3, 260
    rng = np.random.default_rng(9)
    y0, p = rng.uniform(0, 6, (n, neq)), np.concatenate([np.full((n, 1), 2.0), rng.normal(size=(n, neq))], axis=1)
    out = []
    for lanes in (1, 32):
        with Integrator(system_path("kuramoto"), "euler", dt=0.01, tspan=0.045, ksteps=2, neq=neq, npar=neq + 1, orbits=n,
                        lanes=lanes, fmad=False) as sim:
            sim.upload(np.zeros(n), y0, p)
            out.append(sim.run())
    np.testing.assert_array_equal(*out)


@pytest.mark.parametrize("system,neq,dt", [("kuramoto", 5, 0.01), ("oculomotor", 6, 1e-4)])
def test_adaptive_steps_with_contraction(system, neq, dt):
    """Few orbits take the speculative program, many the plain one: the same
    attempts and records with FMA contraction too."""
    with open(system_path(system)) as f:
        source = f.read()
    n = 777 if system == "oculomotor" else 60
    rng = np.random.default_rng(neq)
    if system == "kuramoto":
        p = np.concatenate([rng.uniform(0, 5, (n, 1)), rng.normal(size=(n, neq))], axis=1)
        y0 = rng.uniform(0, 2 * np.pi, (n, neq))
    else:
        p = np.array([120.0, 1.5, 0.0045, 0.05, 600.0, 9.0]) * rng.uniform(0.5, 1.5, (n, 6))
        y0 = np.tile([0.0, 0.0, 0.0, 0.0, 0.0, 2.0], (n, 1)) * rng.uniform(0.5, 1.5, (n, 1))
    got, plain = run(source, "dp45", y0, p, dt=dt, tspan=199.5 * dt, ksteps=20, fmad=True)
    for a, b in zip(got, plain):
        np.testing.assert_array_equal(a, b)

"""The branch-free sin, cos, exp and quotient of the explicit and stochastic
solvers (csrc/device/fastmath.cuh) at the edges of the ranges they cover, and
the repetition of a run of steps that leaves them.

Values: one Euler step of size 1 from y = -0 gives the right-hand side itself
(-0 + f keeps f's sign of zero), compared with numpy.  Tolerances: sin, cos and
exp are within 1.7, 1.7 and 0.9 ulp of the true value, CUDA's (outside the
ranges) within 2, 2 and 1, numpy's within 1, so 3 ulp covers either; quotients
are numpy's, bit for bit, but for results below 2^-960, which may be one ulp
off."""
import numpy as np
import pytest

from sodecl_b200 import Integrator, system_path

pytestmark = pytest.mark.gpu

VALUES = """
void sode_system(double t, double y[_numeq_], double yout[_numeq_], double p[_numpar_])
{
	yout[0] = sin(p[0]);
	yout[1] = cos(p[0]);
	yout[2] = exp(p[0]);
	yout[3] = p[0] / p[1];
}
"""
# phases that grow past 2^30 in the middle of a run of steps
DRIFT = """
double sode_system_row(int i, double t, double y[_numeq_], double p[_numpar_])
{
	return p[0] + sin(y[i]) + cos(y[i]) / p[1];
}
void sode_system(double t, double y[_numeq_], double yout[_numeq_], double p[_numpar_])
{
	for (int i = 0; i < _numeq_; i++)
	{
		yout[i] = sode_system_row(i, t, y, p);
	}
}
"""


def edges():
    pi = np.pi * np.arange(0, 9) / 4
    lim = [2.0 ** 30, 708.0, 709.0, 709.78, 709.79, 745.0, 745.13, 746.0]
    a = np.concatenate([[0.0, 1e-320, 1e-310, 5e-300, 1e-200, 1e-20, 1.0, 1e22, 1e200, 1.7e308, np.inf, np.nan], pi,
                        np.nextafter(pi, 10), 1e6 + pi, lim, np.nextafter(lim, 0), np.nextafter(lim, 1e30)])
    a = np.concatenate([a, -a])
    b = np.array([1.0, 3.0, 6.0, 0.0045, 1e-30, 1e30, 2.0 ** -1000, np.nextafter(2.0 ** -1000, 0), 2.0 ** 960,
                  np.nextafter(2.0 ** 960, 0), 1e-310, 1.7e308, 0.0, np.inf, np.nan])
    b = np.concatenate([b, -b])
    return np.repeat(a, b.size), np.tile(b, a.size)


@pytest.mark.parametrize("fmad", [0, 1])
def test_values_at_the_edges_of_the_ranges(fmad):
    a, b = edges()
    n = a.size
    with Integrator(None, "euler", system_src=VALUES, dt=1.0, tspan=0.5, ksteps=1, neq=4, npar=2, orbits=n,
                    fmad=bool(fmad)) as sim:
        assert "#define SODECL_SPECULATE 1" in sim.program_source and sim.division == "reciprocal"
        sim.upload(np.zeros(n), np.full((n, 4), -0.0), np.stack([a, b], axis=1))
        got = sim.run()[1]
    with np.errstate(all="ignore"):
        want = np.stack([np.sin(a), np.cos(a), np.exp(a), a / b])
        ulps = np.abs(got - want) / np.spacing(np.abs(want))
    finite = np.isfinite(want)
    np.testing.assert_array_equal(np.isnan(got), np.isnan(want))
    np.testing.assert_array_equal(got[~finite], want[~finite])

    np.testing.assert_array_equal(np.signbit(got[~np.isnan(want)]), np.signbit(want[~np.isnan(want)]))
    assert ulps[:3][finite[:3]].max() <= 3
    q, w = got[3], want[3]
    normal = finite[3] & ((np.abs(w) >= 2.0 ** -960) | (w == 0))
    np.testing.assert_array_equal(q[normal], w[normal])
    assert ulps[3][finite[3]].max() <= 1


@pytest.mark.parametrize("division", ["ieee", "reciprocal"])
def test_float_quotients_at_the_edges_of_the_range(division):
    """Correctly rounded, but within 2^-19 of an ulp of the middle between two
    floats and below 2^-100, where they may be one ulp off."""
    a = np.array([0.0, 1e-45, 1e-40, 1.2e-38, 1e-30, 1e-8, 0.3, 1.0, 2.5, 7.0, 1e8, 1e30, 3.4e38, np.inf, np.nan], np.float32)
    lim = np.array([2.0 ** -100, 2.0 ** 100, 2.0, 4.0], np.float32)
    b = np.concatenate([lim, np.nextafter(lim, np.float32(0)), np.nextafter(lim, np.float32(np.inf)),
                        (lim * (1 - 65 * 2.0 ** -24)).astype(np.float32), (lim * (1 - 64 * 2.0 ** -24)).astype(np.float32),
                        np.array([1.0, 3.0, 6.0, 25.0, 0.0045, 1e-30, 1e30, 1e-45, 1e-38, 3.4e38, 0.0, np.inf, np.nan], np.float32)])
    a, b = np.concatenate([a, -a]), np.concatenate([b, -b])
    a, b = np.repeat(a, b.size), np.tile(b, a.size)
    n = a.size
    src = VALUES.replace("sin(p[0])", "0").replace("cos(p[0])", "0").replace("exp(p[0])", "0")
    with Integrator(None, "euler", system_src=src, dt=1.0, tspan=0.5, ksteps=1, neq=4, npar=2, orbits=n,
                    precision="fp32", division=division) as sim:
        assert "#define SODECL_SPECULATE 1" in sim.program_source and sim.division == division
        sim.upload(np.zeros(n), np.full((n, 4), -0.0), np.stack([a, b], axis=1).astype(np.float64))
        got = sim.run()[1, 3].astype(np.float32)
    with np.errstate(all="ignore"):
        exact = a.astype(np.float64) / b.astype(np.float64)
        want = a / b
        ulp = np.spacing(np.abs(want)).astype(np.float64)
        off = np.abs(got.astype(np.float64) - want)
        middle = np.abs(np.abs(exact - want) / ulp - 0.5) < 2.0 ** -19
    finite = np.isfinite(want)
    np.testing.assert_array_equal(np.isnan(got), np.isnan(want))
    np.testing.assert_array_equal(got[~finite], want[~finite])
    np.testing.assert_array_equal(np.signbit(got[~np.isnan(want)]), np.signbit(want[~np.isnan(want)]))
    same = finite & ~middle & ((np.abs(want) >= 2.0 ** -100) | (want == 0))
    np.testing.assert_array_equal(got[same], want[same])
    assert np.all(off[finite] <= ulp[finite])


@pytest.mark.parametrize("ksteps", [1, 7, 8, 9, 40])
@pytest.mark.parametrize("lanes", [1, 4])
def test_runs_that_leave_the_range_are_repeated(ksteps, lanes):
    """Orbits that stay inside, cross 2^30 early, late or start beyond, side by
    side; each like alone, bit for bit, and like the same steps in numpy."""
    n, neq, steps, h = 67, 5, 40, 0.01
    rate = np.array([1.0, 1e10, 2e11, 3e9, 5e10])[np.arange(n) % 5]
    y0 = np.linspace(0.0, 6.0, n * neq).reshape(n, neq) + np.where(np.arange(n) % 11 == 3, 2.0 ** 31, 0.0)[:, None]
    p = np.stack([rate, np.full(n, 2.5)], axis=1)
    kw = dict(system_src=DRIFT, dt=h, tspan=(steps - 0.5) * h, ksteps=ksteps, neq=neq, npar=2, lanes=lanes)

    def run(sel):
        with Integrator(None, "euler", orbits=len(sel), **kw) as sim:
            sim.upload(np.zeros(len(sel)), y0[sel], p[sel])
            return sim.run()

    got = run(np.arange(n))
    for sel in (np.array([1]), np.array([2, 3]), np.arange(5, 30, 5)):
        np.testing.assert_array_equal(run(sel), got[:, :, sel])
    y = y0.copy()
    done = 0
    for r in range(got.shape[0]):
        # each step adds up to h (ulp of the sine + ...) and the rounding of y:
        # a few ulps of the largest |y| a step, and the sine turns an error of
        # y into one of h times it: exp(2 h steps) = 2.2 over the run
        bound = 2.2 * (done + 1) * 4 * np.spacing(np.abs(y).max(axis=1))
        assert np.all(np.abs(got[r].T - y) <= bound[:, None])
        for _ in range(min(ksteps, got.shape[0] * ksteps)):
            y = y + (p[:, :1] + np.sin(y) + np.cos(y) / 2.5) * h
        done += ksteps


@pytest.mark.parametrize("system,solver,lanes,copies", [
    ("kuramoto", "euler", 1, 2), ("kuramoto", "rk4", 4, 2), ("kuramoto", "ie", 4, 2), ("kuramoto", "im", 8, 2),
    ("kuramoto", "ie", 1, 1), ("oculomotor", "rk4", 1, 2), ("oculomotor", "ie", 1, 0)])
def test_shipped_systems_compile_with_it(system, solver, lanes, copies):
    """No compilation falls back to the plain program unnoticed."""
    neq, npar = (8, 9) if system == "kuramoto" else (6, 6)
    with Integrator(system_path(system), solver, dt=0.01, tspan=0.1, ksteps=5, neq=neq, npar=npar, orbits=4, lanes=lanes) as sim:
        text = sim.program_source
    assert text.count("#define sin(...)") == copies


@pytest.mark.parametrize("solver,neq,lanes", [("ie", 3, 2), ("ie", 16, 8), ("im", 5, 4), ("im", 33, 32)])
def test_banded_solve_of_lanes_outside_its_range(solver, neq, lanes):
    """Couplings of zero, tiny, ordinary and huge, and NaN: entries of the band
    beyond 2^-480 and 2^480 take IEEE quotients, the others the same bits."""
    coupling = np.array([2.0, 0.0, 1e-200, 1e160, 3.5, np.nan, 1e-150, 4.5])
    n = coupling.size
    rng = np.random.default_rng(neq)
    p = np.concatenate([coupling[:, None], rng.normal(size=(n, neq))], axis=1)
    y0 = rng.uniform(0, 2 * np.pi, (n, neq))
    out = []
    for many in (1, lanes):
        with Integrator(system_path("kuramoto"), solver, dt=0.01, tspan=0.095, ksteps=2, neq=neq, npar=neq + 1,
                        orbits=n, lanes=many, fmad=False, newton_max_iter=50) as sim:
            sim.upload(np.zeros(n), y0, p)
            out.append((sim.run(), *sim.status()))
    for one, many in zip(*out):
        np.testing.assert_array_equal(many, one)


@pytest.mark.parametrize("system,neq", [("kuramoto", 3), ("kuramoto", 9), ("oculomotor", 6)])
def test_adaptive_attempts_have_the_plain_programs_bits(system, neq, tmp_path):
    """Dividends inside, at and beyond the covered range, zero and NaN; a file
    that mentions printf is built without speculative attempts."""
    source = open(system_path(system)).read()
    plain = tmp_path / "plain.cl"
    plain.write_text(source + "\n/* printf */\n")
    n = 45
    rng = np.random.default_rng(neq)
    if system == "kuramoto":
        special = [2.0, 0.0, 5e-324, 1e-300, 2.0 ** -900, 2.0 ** 900, 1e280, np.nan, -3.0]
        p = np.concatenate([np.resize(special, (n, 1)), rng.normal(size=(n, neq))], axis=1)
        y0 = rng.uniform(0, 2 * np.pi, (n, neq))
        dt = 0.01
    else:
        p = np.array([600.0, 9.0, 0.0045, 0.05, 110.0, 1.5]) * rng.uniform(0.5, 1.5, (n, 6))
        p[:4, 4] = [0.0, 1e-310, 1e300, np.nan]
        p[4:7, 5] = [1e-40, 1e40, np.inf]
        y0 = np.tile([0.0, 0.0, 0.0, 0.0, 0.0, 5.0], (n, 1))
        y0[::5, 5] = 1e-280
        dt = 1e-4
    out = []
    for path in (system_path(system), str(plain)):
        with Integrator(path, "dp45", dt=dt, tspan=30 * dt, ksteps=10, neq=neq, npar=p.shape[1], orbits=n,
                        fmad=False) as sim:
            assert ("#define SODECL_SPECULATE 1" in sim.program_source) == (path != str(plain))
            sim.upload(np.zeros(n), y0, p)
            out.append((sim.run(), *sim.status()))
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)

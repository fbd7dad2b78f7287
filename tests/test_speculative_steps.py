"""Speculative steps on the GPU against the programs without them (a file that
mentions printf gets none)."""
import numpy as np
import pytest

from sodecl_b200 import Integrator
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

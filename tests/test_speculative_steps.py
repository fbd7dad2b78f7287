"""Speculative steps on the GPU against the programs without them (a file that
mentions printf gets none)."""
import numpy as np
import pytest

from sodecl_b200 import Integrator

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

"""Speculative steps never let a system file see a number its functions cannot
give, and no file whose loops or addresses hang on numbers gets them.

The functions of csrc/device are compiled for the host and evaluated here;
which program a file gets is read from the assembled text.  No such file is
run: its speculative copy could run forever or read out of range."""
import numpy as np
import pytest

from device_math import call
from sodecl_b200 import Integrator, system_path
from sodecl_b200.batch import Batch


def bounded(fn, x):
    y, outside = np.empty_like(x), np.empty(x.size, dtype=np.uint8)
    call(fn + "_bounded", x, y, outside)
    return y, outside.astype(bool)


def arguments(seed=0):
    """Every magnitude, the ends of the ranges, Inf and NaN."""
    rng = np.random.default_rng(seed)
    x = np.exp(rng.uniform(np.log(1e-320), np.log(1.7e308), 200000))
    ends = np.array([2.0 ** 30, 708.0, 709.78, 710.0, 745.2, 746.0, 748.0, 800.0, 900.0, 1e4, 1e300, np.inf, np.nan, 0.0])
    x = np.concatenate([x, rng.uniform(0, 1500, 200000), ends, np.nextafter(ends, 0), np.nextafter(ends, np.inf)])
    return np.concatenate([x, -x])


@pytest.mark.parametrize("fn", ["sin", "cos", "exp"])
def test_speculative_values_are_the_functions(fn):
    """Inside the range the value, outside it one the function can have."""
    x = arguments()
    y, outside = bounded(fn, x)
    with np.errstate(all="ignore"):
        want = getattr(np, fn)(x)
    np.testing.assert_array_equal(np.isnan(y), np.isnan(want))
    ok = ~np.isnan(want)
    low, high = (0.0, np.inf) if fn == "exp" else (-1.0, 1.0)
    assert y[ok].min() >= low and y[ok].max() <= high
    assert not outside[~ok].any()  # NaN is the value for NaN, and sin's and cos's for Inf
    inside = ok & ~outside
    np.testing.assert_array_equal(np.isinf(y[inside]), np.isinf(want[inside]))
    f = inside & np.isfinite(want)
    # the functions' 1.5 ulp (test_device_math.py) and numpy's one
    assert np.all(np.abs(y[f] - want[f]) <= 2.5 * np.spacing(np.abs(want[f])))
    if fn == "exp":
        far = ok & (np.abs(x) >= 748)
        assert not outside[far].any()
        np.testing.assert_array_equal(y[far], want[far])


HEAD = "void sode_system(double t, double y[_numeq_], double yout[_numeq_], double p[_numpar_])\n{\n"
PLAIN = "\tyout[0] = exp(-y[0] * y[0]) / p[0];\n"
HAZARDS = {
    "while": "\tdouble a = y[0];\n\twhile (a < -M_PI) a += 2.0 * M_PI;\n\tyout[0] = exp(-a * a);\n",
    "do": "\tdouble a = y[0];\n\tdo { a -= 1; } while (a > 0);\n\tyout[0] = exp(-a);\n",
    "cast in a subscript": "\tyout[0] = p[(int)(10.0 * exp(-y[0] * y[0]))];\n",
    "int from a value": "\tint k = 10.0 * exp(-y[0]);\n\tyout[0] = p[k];\n",
    "int from a function": "\tint k = rint(exp(-y[0]));\n\tyout[0] = p[k];\n",
    "unsigned assigned": "\tunsigned k;\n\tk = exp(-y[0]);\n\tyout[0] = p[k];\n",
    "int moved by a comparison": "\tint k = 3;\n\tif (exp(y[0]) < 0) k += 1000;\n\tyout[0] = p[k];\n",
    "floating loop": "\tdouble s = 0;\n\tfor (double a = 0; a < exp(y[0]); a += 1.0) s += a;\n\tyout[0] = s;\n",
    "loop bound": "\tdouble s = exp(y[0]);\n\tint i;\n\tfor (i = 0; i < s; i++) s -= 1;\n\tyout[0] = s;\n",
    "endless loop": "\tdouble s = exp(y[0]);\n\tfor (;;) { s -= 1; if (s < 0) break; }\n\tyout[0] = s;\n",
    "loop variable moved": "\tdouble s = exp(y[0]);\n\tfor (int i = 0; i < 9; i++) { if (s > 0) i--; }\n\tyout[0] = s;\n",
    "comparison in a subscript": "\tint k = exp(y[0]) > 1;\n\tyout[0] = p[k];\n",
    "goto": "\tdouble s = exp(y[0]);\nagain:\n\ts -= 1;\n\tif (s > 0) goto again;\n\tyout[0] = s;\n",
    "pointer": "\tdouble *q = y;\n\tq += lrint(exp(y[0]));\n\tyout[0] = *q;\n",
    "pointer arithmetic": "\tyout[0] = *(p + lrint(exp(y[0])));\n",
    "macro": "#define AT(x) p[(int)(x)]\n\tyout[0] = AT(exp(y[0]));\n",
    "macro loop": "#define UNTIL while\n\tdouble s = exp(y[0]);\n\tUNTIL (s > 0) s -= 1;\n\tyout[0] = s;\n",
    "static_cast": "\tyout[0] = p[static_cast<int>(exp(y[0]))];\n",
    "functional cast": "\tyout[0] = p[int(exp(y[0]))];\n",
    "out argument": "\tint k;\n\tdouble s = frexp(exp(y[0]), &k);\n\tyout[0] = s * p[k];\n",
}
HELPERS = {
    "int argument": "double at(int k, double p[]) { return p[k]; }\n" + HEAD + "\tyout[0] = at(exp(y[0]), p);\n}\n",
    "int result": "int at(double x) { return x > 0 ? 3 : 5; }\n" + HEAD + "\tyout[0] = p[at(exp(y[0]))];\n}\n",
    "two types": "double at(int k, double p[]) { return p[k]; }\ndouble sum(double k) { double s = 0; "
                 "for (int i = 0; i < k; i++) s += i; return s; }\n" + HEAD + "\tyout[0] = sum(exp(y[0])) + at(1, p);\n}\n",
    "macro argument": "#define LOOP(n) for (int i = 0; i < n; i++) s += i;\ndouble at(int n, double p[]) { return p[n]; }\n" + HEAD +
                      "\tdouble s = at(1, p);\n\tLOOP(exp(y[0]))\n\tyout[0] = s;\n}\n",
    "function as a value": "double f(double x) { double (*g)(double) = f; return x > 1 ? g(x / 2) : x; }\n" + HEAD +
                           "\tyout[0] = f(exp(y[0]));\n}\n",
    "recursion": "double f(double x) { return x > 1 ? f(x / 2) : x; }\n" + HEAD + "\tyout[0] = f(exp(y[0]));\n}\n",
    "typedef": "typedef int whole;\n" + HEAD + "\twhole k = exp(y[0]);\n\tyout[0] = p[k];\n}\n",
    "int array": "__constant int tab[3] = {0, 1, 2};\n" + HEAD + "\tyout[0] = exp(p[tab[1]]);\n}\n",
}
SAFE = {
    "plain": HEAD + PLAIN + "}\n",
    "loops": HEAD + "\tint i, j;\n\tfor (i = 0; i < _numeq_; ++i)\n\t{\n\t\tyout[i] = 0;\n\t\tfor (j = _numeq_ - 1; j >= 0; j--)"
             " yout[i] += sin(y[j] - y[i]);\n\t}\n}\n",
    "selections": HEAD + "\tint right = y[0] > 0;\n\tbool left = !right;\n\tyout[0] = right ? exp(-y[0]) : (left ? exp(y[0]) : 0);\n}\n",
    "sizes": "#define ROWS (_numeq_ - 1)\n#define LAST (ROWS + 0)\n" + HEAD +
             "\tconst int n = LAST;\n\tfor (int i = 0; i <= n; i += 1) yout[i] = exp(-y[i]) / 3;\n}\n",
    "helper": "double row(int i, const double *y) { double c; double s = sincos(y[i], &c); return s * c; }\n" + HEAD +
              "\tfor (int i = 0; i < _numeq_; i++) yout[i] = row(i, y);\n}\n",
    "sincos": HEAD + "\tdouble a, b, c;\n\tfloat d;\n\ta = sincos(y[0], &b);\n\tsincos(y[1], &a, &c);\n\tsincos(1, &b);\n"
              "\tsincos(0.5f * _numeq_, &c);\n\tsincos(0.5f, &d);\n\tyout[0] = a + b * c + d;\n}\n",
    "prototype": "double f(double x);\ndouble f(double x) { return exp(x); }\n" + HEAD + "\tyout[0] = f(y[0]);\n}\n",
    "comments": "// while (1)\n" + HEAD + "\t/* int k = exp(1); goto */\n" + PLAIN + "}\n",
    "table": "__constant double tab[3] = {1.0, 2.0, 3.0};\n" + HEAD + "\tyout[0] = exp(-tab[2] * y[0]);\n}\n",
}


def speculates(source, solver="rk4", **kw):
    args = dict(dt=0.1, tspan=1.0, ksteps=1, neq=3, npar=12, orbits=1)
    with Integrator(None, solver, system_src=source, **{**args, **kw}) as sim:
        return "#define SODECL_SPECULATE 1" in sim.program_source


@pytest.mark.parametrize("solver", ["euler", "rk4", "dp45"])
@pytest.mark.parametrize("name", list(HAZARDS) + list(HELPERS))
def test_files_that_steer_by_numbers_get_no_speculative_copy(name, solver):
    source = HELPERS[name] if name in HELPERS else HEAD + HAZARDS[name] + "}\n"
    assert not speculates(source, solver)


@pytest.mark.parametrize("name", list(SAFE))
def test_files_that_do_not_keep_it(name):
    assert speculates(SAFE[name])


def test_files_that_include_others_get_none(tmp_path):
    (tmp_path / "more.h").write_text("double twice(double x) { return 2 * x; }\n")
    assert not speculates('#include "%s"\n' % (tmp_path / "more.h") + HEAD + "\tyout[0] = exp(twice(y[0]));\n}\n")


def test_such_files_in_fp32_lanes_and_batches(tmp_path):
    row = "double sode_system_row(int i, double t, double y[_numeq_], double p[_numpar_])\n{\n\tdouble a = y[i];\n%s" \
          "\treturn sin(a) / p[0];\n}\n" + HEAD + "\tfor (int i = 0; i < _numeq_; i++) yout[i] = sode_system_row(i, t, y, p);\n}\n"
    band = "void calc_jacobian(double y[_numeq_], double jac[_numeq_][_numeq_], double p[_numpar_])\n{\n}\n" \
           "void calc_jacobian_band(int i, double y[_numeq_], double band[3], double p[_numpar_])\n{\n\tband[1] = cos(y[i]);\n}\n"
    for loop, safe in (("", True), ("\twhile (a > 6.3) a -= 6.3;\n", False)):
        source = band + row % loop
        assert speculates(source, "rk4", lanes=2) == safe
        assert speculates(source, "ie", lanes=2) == safe
        assert speculates(source, "euler", precision="fp32") == safe
        path = tmp_path / "s.cl"
        path.write_text(source)
        b = Batch()
        b.add_class(str(path), "rk4", neq=3, npar=12, dt=0.1)
        assert ("#define SODECL_SPECULATE 1" in b.compile().program_source) == safe


@pytest.mark.parametrize("system", ["kuramoto", "oculomotor"])
def test_shipped_systems_keep_it(system):
    with open(system_path(system)) as f:
        assert speculates(f.read(), neq=6, npar=7)


@pytest.mark.parametrize("neq,copies", [(256, 2), (257, 1)])
def test_wide_systems_take_the_same_functions(neq, copies):
    """One thread per orbit and lanes per orbit get the same sines, whatever the
    number of equations (one thread's steps speculate up to 256)."""
    with open(system_path("kuramoto")) as f:
        source = f.read()
    for lanes in (1, 32):
        with Integrator(None, "euler", system_src=source, dt=0.1, tspan=1.0, ksteps=1, neq=neq, npar=neq + 1, orbits=1, lanes=lanes) as sim:
            assert sim.program_source.count("#define sin(...)") == (copies if lanes == 1 else 2)


GUARDED = "/* helpers */\n#ifndef X_CL\n#define X_CL\n#ifndef M_PI\n  #  define M_PI 3.0\n#endif\n#define GAIN 2.0\n" \
    "static_assert(M_PI > 3.1);\ndouble f(double x) { return GAIN * sin(M_PI * x); }\n" + HEAD + \
    "\tyout[0] = f(y[0]) / p[0];\n}\n#endif\n"


def test_guarded_files_keep_it():
    """Neither copy, nor a second class of a batch, finds what the first one defined;
    what the program defines stays."""
    assert speculates(GUARDED)
    b = Batch()
    for solver in ("euler", "rk4"):
        b.add_class(None, solver, neq=1, npar=1, dt=0.1, system_src=GUARDED)
    text = b.compile().program_source
    assert text.count("#define SODECL_SPECULATE 1") == 2 and "no speculative copy" not in text


def test_the_reason_for_no_copy_is_in_the_program():
    def reason(source):
        with Integrator(None, "rk4", system_src=source, dt=0.1, tspan=1.0, ksteps=1, neq=3, npar=12, orbits=1) as sim:
            lines = [line for line in sim.program_source.splitlines() if line.startswith("// no speculative copy: ")]
            assert len(lines) == (0 if "#define SODECL_SPECULATE 1" in sim.program_source else 1)
            return lines[0] if lines else ""

    assert reason(SAFE["plain"]) == ""
    assert reason(HEAD + HAZARDS["while"] + "}\n").endswith(": while")
    assert "did not compile" in reason("double sin(double x) { return x; }\n" + HEAD + "\tyout[0] = sin(y[0]);\n}\n")


def test_the_adaptive_solver_speculates_for_few_orbits():
    """Up to twice the threads that its plain kernel keeps on the device (2 x 148 x
    512) where the file has a quotient for every equation, else up to two warps."""
    with open(system_path("oculomotor")) as f:
        source = f.read()
    assert speculates(source, "dp45", neq=6, npar=6, orbits=2 * 148 * 512)
    assert not speculates(source, "dp45", neq=6, npar=6, orbits=2 * 148 * 512 + 1)
    assert speculates(source, "rk4", neq=6, npar=6, orbits=1 << 20)
    with open(system_path("kuramoto")) as f:
        source = f.read()
    # one quotient for all rows
    assert speculates(source, "dp45", neq=5, npar=6, orbits=64) and not speculates(source, "dp45", neq=5, npar=6, orbits=65)

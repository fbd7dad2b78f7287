"""Small host outputs, and the scan of a system file's definitions."""
import numpy as np
import pytest

from sodecl_b200 import Integrator, system_path


@pytest.mark.gpu
@pytest.mark.parametrize("orbits,records", [(1, 1), (1, 2), (2, 26), (873, 101), (874, 101), (1300, 101)])
def test_host_records_on_both_sides_of_the_staging_line(orbits, records):
    """4 MiB of records are 873.8 orbits x 6 equations x 100 records + one: one
    plain copy below, the staging threads above; the same as records on the device."""
    import torch

    rng = np.random.default_rng(orbits)
    y0 = rng.normal(size=(orbits, 6))
    p = np.array([120.0, 1.5, 0.0045, 0.05, 600.0, 9.0]) * rng.uniform(0.5, 1.5, (orbits, 6))
    kw = dict(dt=1e-6, ksteps=3, tspan=3e-6 * (records - 1.5) if records > 1 else 0.0, neq=6, npar=6, orbits=orbits)
    with Integrator(system_path("oculomotor"), "rk4", **kw) as sim:
        assert sim.num_records == records
        sim.upload(np.zeros(orbits), y0, p)
        host = sim.run()
        t, y, q = (torch.tensor(a, device="cuda") for a in (np.zeros(orbits), y0, p))
        dev = torch.empty((records, 6, orbits), dtype=torch.float64, device="cuda")
        sim.launch(t=t.data_ptr(), y=y.data_ptr(), params=q.data_ptr(), records=dev.data_ptr(),
                   stream=torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
    np.testing.assert_array_equal(host, dev.cpu().numpy())


BODY = "{ yout[0] = -y[0]; }\n"
ARGS = "(double t, double y[_numeq_], double yout[_numeq_], double p[_numpar_])"


@pytest.mark.parametrize("source,accepted", [
    ("void sode_system" + ARGS + BODY, True),
    ("void sode_system" + ARGS + ";\nvoid sode_system\t\n" + ARGS + " \n\t" + BODY, True),
    ("void sode_system" + ARGS + ";\n", False),
    ("/* void sode_system" + ARGS + BODY + "*/\n// sode_system() {\nvoid other" + ARGS + BODY, False),
    ("void my_sode_system" + ARGS + BODY, False),
    ("void sode_system2" + ARGS + BODY, False),
    ("void sode_system" + ARGS + "/* body */ // here\n" + BODY, True),
])
def test_definitions_found(source, accepted, tmp_path):
    path = tmp_path / "s.cl"
    path.write_text(source)
    build = lambda: Integrator(str(path), "euler", dt=0.1, tspan=1.0, ksteps=1, neq=1, npar=1, orbits=1)  # noqa: E731
    if accepted:
        build().close()
    else:
        with pytest.raises(Exception, match="sode_system"):
            build()


@pytest.mark.gpu
def test_device_name_fits_any_buffer():
    import ctypes as C

    from sodecl_b200 import _native as N

    whole = C.create_string_buffer(256)
    major, minor = C.c_int(), C.c_int()
    assert N.lib.sodecl_cuda_device_describe(0, whole, 256, C.byref(major), C.byref(minor)) == N.OK
    assert len(whole.value) > 4 and major.value >= 10
    for n in (1, 2, 5, len(whole.value), len(whole.value) + 1, 1000):
        buf = C.create_string_buffer(b"x" * n, n)
        assert N.lib.sodecl_cuda_device_describe(0, buf, n, None, None) == N.OK
        assert buf.value == whole.value[:n - 1]

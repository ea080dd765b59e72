"""What the engine's dopri5 solver keeps between steps: its own code
(dust2_gb300/csrc/engine/dopri5.cuh) compiled for the host."""
import ctypes
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT


def dptr(a):
    return a.ctypes.data_as(ctypes.POINTER(ctypes.c_double))


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not shutil.which(nvcc):
        pytest.skip("nvcc not available")
    lib = tmp_path_factory.mktemp("record") / "libdopri5_record.so"
    subprocess.run(
        [nvcc, "-std=c++17", "-O2", "-shared", "-Xcompiler",
         "-fPIC,-ffp-contract=off", "-I", str(ROOT / "dust2_gb300" / "csrc"),
         "-gencode", "arch=compute_103a,code=sm_103a",
         str(ROOT / "tests" / "dopri5_record_host.cu"), "-o", str(lib)],
        check=True, capture_output=True)
    return ctypes.CDLL(str(lib))


def copies(host, n_copies, times, tol=1e-6):
    times = np.asarray(times, dtype=float)
    out = np.empty((times.size, n_copies, 4))
    c4 = np.empty((n_copies, 4))
    rc = host.host_copies(n_copies, dptr(times), times.size,
                          ctypes.c_double(tol), dptr(out), dptr(c4))
    assert rc == 0
    return out, c4


@pytest.mark.parametrize("n_copies", [8, 10])
def test_resets_of_many_variables(host, n_copies):
    """Copies of four variables, two of them reset by interpolation: 32
    variables, and 40 (a reset mask of more than one word).  The error norm
    is a mean over variables and the first step is given, so the copies take
    the single system's steps up to rounding; 1e-9 is far above what 30 steps of rounding amount to
    and far below a reset's size (about 1)."""
    times = [0.7, 1.9, 3.35, 5.45, 9.8]
    one, one_c4 = copies(host, 1, times)
    many, many_c4 = copies(host, n_copies, times)
    np.testing.assert_allclose(many, np.broadcast_to(one, many.shape),
                               rtol=1e-9, atol=1e-9)
    # the record: a reset leaves its values in the first entries of c4, two
    # per copy; the others are the coefficients
    first = 2 * n_copies
    np.testing.assert_allclose(
        many_c4.ravel()[first:],
        np.broadcast_to(one_c4, many_c4.shape).ravel()[first:],
        rtol=1e-6, atol=1e-9)


@pytest.mark.parametrize("every", [1.0, 3.3])
def test_integration_in_parts(host, every):
    """One run over several output times, and a run to each with the solver
    record stored in between (dust_system_run_to_time, or output copied in
    parts): the same bits."""
    times = every * np.arange(1.0, 31)
    for k in range(200):
        pars = np.array([10.0 + k, 1000 + 13.0 * k, 0.2 + 0.002 * k, 0.1])
        got = np.empty((2, 11))
        for parts in range(2):
            assert host.host_sirode(dptr(pars), dptr(times), times.size,
                                    parts, dptr(got[parts])) == 0
        np.testing.assert_array_equal(got[0], got[1])


def test_record_when_the_solver_gives_up(host):
    """The dense-output record after an error, with and without rejected
    steps before it."""
    seen = set()
    for max_steps, ssmin in ([(n, 2.3e-16) for n in range(0, 120)] +
                             [(10000, 10.0 ** -k) for k in range(1, 5)]):
        got, want = np.zeros(13), np.zeros(13)
        n_rejected = ctypes.c_int()
        err = host.host_give_up(max_steps, ctypes.c_double(ssmin), dptr(got),
                                dptr(want), ctypes.byref(n_rejected))
        if err == -1:
            continue
        assert err > 0
        seen.add((err, min(n_rejected.value, 2)))
        np.testing.assert_array_equal(got, want)
    assert len(seen) >= 4  # both errors; no, one and several rejections


@pytest.mark.gpu
def test_simulate_equals_runs_on_device(built):
    """As above through the public verbs, and the reported errors."""
    import dust2_gb300 as d
    pars = [{"I0": 10.0 + k, "N": 1000 + 13.0 * k, "beta": 0.2 + 0.002 * k,
             "gamma": 0.1} for k in range(200)]
    times = 3.3 * np.arange(1.0, 21)
    whole = d.dust_system_create(d.sirode(), pars, n_groups=200)
    d.dust_system_set_state_initial(whole)
    want = d.dust_system_simulate(whole, times)
    parts = d.dust_system_create(d.sirode(), pars, n_groups=200)
    d.dust_system_set_state_initial(parts)
    for i, t in enumerate(times):
        d.dust_system_run_to_time(parts, t)
        np.testing.assert_array_equal(d.dust_system_state(parts),
                                      want[..., i])
    a, b = d.dust_system_internals(whole), d.dust_system_internals(parts)
    for name in ("step_size", "error", "n_steps", "n_steps_rejected"):
        np.testing.assert_array_equal(a[name], b[name])
    assert np.all(a["error"] > 0) and np.all(a["error"] <= 1)

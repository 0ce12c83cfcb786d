"""The separable inverse with one diagonalized direction (fdm_host.cpp,
fdm_tri) against the oracle's matrix A = M Om^-1 G (operator_divergence.m:208)
and against its pseudo-inverse, for every boundary-condition kind, both mode
directions and the smallest grids."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from oracle import ins2d_ref as R
from tests.cases_common import BC_COMBOS, grid_stretched, grid_uniform, is_closed
from tests.test_host_tables import ROOT, Tables


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = tmp_path_factory.mktemp("probe") / "libprobetri.so"
    csrc, nat = os.path.join(ROOT, "ins2d_b200", "csrc"), os.path.join(ROOT, "tests", "native")
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", csrc, os.path.join(nat, "probe.cpp"),
                           os.path.join(nat, "probe_fdm_tri.cpp")] +
                          [os.path.join(csrc, f) for f in ("setup.cpp", "mg_host.cpp", "fdm_host.cpp")] + ["-o", str(out)])
    lib = ctypes.CDLL(str(out))
    lib.probe_build.restype = ctypes.c_void_p
    lib.probe_build.argtypes = [ctypes.c_int, ctypes.c_int] + [ctypes.c_void_p] * 3 + [ctypes.c_double]
    lib.probe_free.argtypes = [ctypes.c_void_p]
    lib.probe_error.restype = ctypes.c_char_p
    lib.probe_fdm_tri_apply.argtypes = [ctypes.c_void_p] * 4
    return lib


@pytest.mark.parametrize("combo", sorted(BC_COMBOS))
@pytest.mark.parametrize("shape", [(23, 17), (17, 23), (16, 16), (3, 9), (2, 4), (5, 2)])
@pytest.mark.parametrize("stretch", [False, True])
def test_fdm_tri_inverse(lib, combo, shape, stretch):
    nx, ny = shape
    x = grid_stretched(nx, 0.0, 1.7) if stretch else grid_uniform(nx, 0.0, 1.7)
    y = grid_stretched(ny, -0.5, 0.5, beta=1.3) if stretch else grid_uniform(ny, -0.5, 0.5)
    bc = BC_COMBOS[combo]
    try:
        o = R.make_options(x, y, bc, Re=100.0, poisson=1)
    except Exception:
        pytest.skip("the reference has no operators for this size")
    T = Tables(lib, x, y, bc, 100.0)
    A = o.discretization.A.toarray()
    f = o.discretization.M @ np.random.default_rng(nx).standard_normal(o.grid.NV)
    z, info = np.zeros(nx * ny), np.zeros(3, np.int32)
    lib.probe_fdm_tri_apply(T.h, np.ascontiguousarray(f).ctypes.data, z.ctypes.data, info.ctypes.data)
    assert info[0] == (nx < ny) and (info[1] == 0) == is_closed(bc)
    assert np.linalg.norm(A @ z - f) <= 1e-11 * np.linalg.norm(f)
    if is_closed(bc):  # the null mode is left out: the volume-weighted mean is zero
        vol = np.kron(np.diff(y), np.diff(x))
        assert abs(vol @ z) <= 1e-12 * vol.sum() * np.max(np.abs(z))

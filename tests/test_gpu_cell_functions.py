"""Functions of one cell's update (mp_cell.cuh) on their own, compiled from
cell_functions.cu, where an error would be too small to show in the fields."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from mpulse_b200 import build

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def cell(tmp_path_factory):
    src = os.path.join(os.path.dirname(os.path.abspath(__file__)), "cell_functions.cu")
    lib = str(tmp_path_factory.mktemp("cell") / "cell_functions.so")
    subprocess.run([build.nvcc(), *build.ARCH, *build.NVCC_FLAGS, "-shared", src, "-o", lib], check=True)
    return C.CDLL(lib)


def ptr(a):
    return a.ctypes.data_as(C.c_void_p)


@pytest.mark.parametrize("dtype,name", [(np.float32, "plasma_coef_f32"), (np.float64, "plasma_coef_f64")])
@pytest.mark.parametrize("denom,chi", [(1.7, 0.02), (0.031, -3.0), (250.0, 1e-7)])
def test_plasma_kerr_coefficient_is_the_fp64_quotient(cell, denom, chi, dtype, name):
    """chi / (denom + sigma) in FP64 to the bit, whatever the state's precision."""
    sig = np.concatenate([[0.0], np.exp(np.random.default_rng(3).uniform(-20, 8, 20000))]).astype(dtype)
    out = np.empty(sig.size)
    f = getattr(cell, name)
    f.argtypes = [C.c_double, C.c_double, C.c_void_p, C.c_void_p, C.c_int]
    assert f(denom, chi, ptr(sig), ptr(out), sig.size) == 0
    np.testing.assert_array_equal(out, chi / (denom + sig.astype(np.float64)))


def kerr_starts(cell, A, C_, E2, f32):
    out = np.empty(A.size)
    f = cell.kerr_starts
    f.argtypes = [C.c_void_p] * 4 + [C.c_int] * 2
    assert f(ptr(A), ptr(C_), ptr(E2), ptr(out), A.size, f32) == 0
    return out


@pytest.mark.parametrize("f32", [0, 1], ids=["fp64", "fp32"])
def test_kerr_start_is_the_root_to_the_series_error(cell, f32):
    """Below a = A C^2 = 0.02 the start differs from the root of E + A E^3 = C by no more
    than the first term left out, 7752 a^7 C, and rounding: 2 units of FP64 for C and
    the last sum, and in the FP32 form five single roundings of the correction a C (A,
    C^2, their product, the polynomial, the correction)."""
    rng = np.random.default_rng(4)
    a = np.concatenate([np.exp(rng.uniform(np.log(1e-12), np.log(0.0199), 20000)), [0.0]])
    c = np.exp(rng.uniform(-3, 3, a.size))
    A = a / c**2
    start = kerr_starts(cell, A, c, np.full(a.size, 9.0), f32).astype(np.longdouble)
    root = c.astype(np.longdouble)
    for _ in range(8):
        root = (2 * A * root**3 + c) / (3 * A * root**2 + 1)
    bound = c * (7752 * a**7 + 4.5e-16 + (a * 5 * 2.0**-24 if f32 else 0.0))
    assert np.all(np.abs(start - root) <= bound)


@pytest.mark.parametrize("f32,tol", [(0, 5e-16), (1, 2.0**-23)], ids=["fp64", "fp32"])
def test_kerr_start_is_the_old_field_elsewhere(cell, f32, tol):
    """From a = 0.021 on, and for every negative A, the start is |E^n|: one square root
    (FP32: after one rounding of the square)."""
    rng = np.random.default_rng(5)
    a = np.concatenate([np.exp(rng.uniform(np.log(0.021), np.log(50), 5000)),
                        -np.exp(rng.uniform(np.log(1e-9), np.log(50), 5000))])
    c = np.exp(rng.uniform(-3, 3, a.size))
    e = np.exp(rng.uniform(-3, 3, a.size))
    got = kerr_starts(cell, a / c**2, c, e * e, f32)
    assert np.all(np.abs(got - e) <= tol * e)
    assert kerr_starts(cell, np.array([-1.0]), np.array([1e-3]), np.array([0.0]), f32)[0] == 0.0

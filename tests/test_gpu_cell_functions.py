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

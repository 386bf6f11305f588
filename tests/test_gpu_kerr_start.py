"""The Kerr solves on both sides of the line where their start changes from the
reversed series to |E^n| (a = chi |E|^2 / eps around 0.02): fields from far below to
above it, zero fields, and a negative chi, against the CPU oracle (which starts
from |E^n|, as MPulse does) to the suite's bars (FP64 1e-12, FP32 1e-5 relative L2)."""
import numpy as np
import pytest

from mpulse_b200 import abi, runtime
from oracle import pyoracle
from tests.cases import make_case, random_fields, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,tol", [(abi.MP_FP64, 1e-12), (abi.MP_FP32, 1e-5)], ids=["fp64", "fp32"])
@pytest.mark.parametrize("chi,scale", [(0.02, 0.01), (0.1, 0.15), (0.3, 0.4), (-0.02, 0.3)])
@pytest.mark.parametrize("case", ["nonlin_three_poles", "nl_xy"])
def test_kerr_solve_from_either_start(case, chi, scale, precision, tol):
    cfg = make_case(case, abi.MP_FP64)
    cfg.nx, cfg.ny, cfg.nz = 34, 7, 21
    cfg.chi = chi
    init = random_fields(cfg, 5, scale=scale, smooth=True)
    for v in init.values():
        v[:, :, :3] = 0.0  # cells with no field at the start
    o = pyoracle.OracleSim(cfg)
    for n, v in init.items():
        o.upload(n, v)
    assert o.step(8) == abi.MP_OK
    E2 = sum(o.download(n) ** 2 for n in abi.FIELD_NAMES[:3])
    a = abs(chi) * E2 / cfg.eps
    assert a.min() < 0.02  # the series; at the larger fields |E^n| as well
    assert scale < 0.3 or chi < 0 or a.max() > 0.02
    cfg.precision = precision
    with runtime.Simulation(cfg) as g:
        for n, v in init.items():
            g.upload(n, v)
        g.step(8)
        for n in abi.FIELD_NAMES:
            got = g.download(n)
            assert np.isfinite(got).all()
            assert rel_l2(got, o.download(n)) <= tol, n

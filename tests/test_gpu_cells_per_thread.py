"""The FP32 E half's forms with two cells per thread that other tests do not reach: a
linear medium with no or one pole and CPML on all faces (the faces loaded early), and
the Kerr medium in states above 1 GB."""
import numpy as np
import pytest

from mpulse_b200 import abi, configs, runtime
from oracle import pyoracle
from tests.cases import make_case, random_fields, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("poles", [0, 1])
@pytest.mark.parametrize("shape", [(4, 5, 9), (34, 9, 10), (66, 7, 37), (130, 33, 20)], ids=lambda s: "x".join(map(str, s)))
def test_linear_fp32_with_layers_matches_oracle(shape, poles):
    cfg = make_case("lin_all_wave_periodic", abi.MP_FP64)
    cfg.nx, cfg.ny, cfg.nz = shape
    cfg.cpml_d = min(cfg.cpml_d, min(shape))
    for q in range(poles, abi.MP_MAX_POLES):
        cfg.poles[q].eps = 0.0
    cfg.medium_z0, cfg.medium_z1 = 3, cfg.nz + 1
    cfg.sources[0].distance = min(cfg.sources[0].distance, cfg.nz - 1)
    init = random_fields(cfg, 3 + sum(shape), smooth=True)
    o = pyoracle.OracleSim(cfg)
    for n, v in init.items():
        o.upload(n, v)
    assert o.step(12) == abi.MP_OK
    cfg.precision = abi.MP_FP32
    with runtime.Simulation(cfg) as g:
        for n, v in init.items():
            g.upload(n, v)
        g.step(12)
        for n in abi.FIELD_NAMES:
            assert rel_l2(g.download(n), o.download(n)) <= 1e-5, n


@pytest.mark.parametrize("nx,ny,nz,poles,cpml", [
    (256, 250, 270, 2, abi.MP_CPML_ALL),   # 1.01 GiB
    (258, 256, 390, 1, abi.MP_CPML_ALL),   # 1.06 GiB
    (256, 256, 740, 0, abi.MP_CPML_ALL),   # 1.08 GiB
    (130, 126, 1050, 2, abi.MP_CPML_Z),    # 1.05 GiB
    (256, 258, 200, 3, abi.MP_CPML_ALL),   # 1.09 GiB: three poles keep one cell per thread
], ids=["2poles", "1pole", "vacuum", "zlayers", "3poles"])
def test_kerr_fp32_above_1_gb_matches_fp64(nx, ny, nz, poles, cpml):
    """Six steps from smooth fields that reach into all layers, against the FP64 form
    (which test_gpu_rows and test_gpu_parity compare with the oracle): the FP32 bar
    of 1e-5."""
    cfg = configs.c3_plrc_kerr(abi.MP_FP64, nx, ny, nz, medium_z0=16, focus_z=nz // 2, chi=0.2)
    three = configs.SILICA_POLES + (configs.lorentz_pole(0.3, 0.3, 0.01),)
    for q in range(abi.MP_MAX_POLES):
        cfg.poles[q].eps, cfg.poles[q].delta, cfg.poles[q].om2 = three[q] if q < poles else (0.0, 0.0, 1.0)
    cfg.cpml = cpml
    # the state's fields and accumulators, as the library counts them
    assert 4 * nx * ny * (6 * (nz + 2) + 6 * poles * (nz - 15)) > 1 << 30
    z, y, x = np.meshgrid(np.arange(nz + 2.0), np.arange(float(ny)), np.arange(float(nx)), indexing="ij", sparse=True)
    fields = {}
    for precision in (abi.MP_FP64, abi.MP_FP32):
        cfg.precision = precision
        with runtime.Simulation(cfg) as g:
            for q, n in enumerate(abi.FIELD_NAMES):
                g.upload(n, 0.3 * np.cos(0.11 * z + q) * np.cos(2 * np.pi * y / ny + 2 * q) *
                         np.cos(4 * np.pi * x / nx + 3 * q))
            g.step(6)
            for n in abi.FIELD_NAMES:
                if precision == abi.MP_FP64:
                    fields[n] = g.download(n)
                else:
                    assert rel_l2(g.download(n), fields.pop(n)) <= 1e-5, n

"""The half-step kernels where their mapping of cells to threads has its edges:
rows of 2 to 5 cells, odd and even row lengths on both sides of a warp, row
counts that leave a partial group of four, chunks of one plane and chunks with a
shorter last one, CPML layers that meet or overlap, with an injection plane; against
the CPU oracle, to the suite's bars (FP64 1e-12, FP32 1e-5 relative L2)."""
import pytest

from mpulse_b200 import abi, configs, runtime
from oracle import pyoracle
from tests.cases import make_case, random_fields, rel_l2

pytestmark = pytest.mark.gpu

SHAPES = [(2, 2, 7), (3, 5, 9), (4, 4, 8), (5, 3, 11), (31, 6, 9), (34, 9, 10), (66, 7, 37), (129, 5, 6), (130, 33, 65)]


@pytest.mark.parametrize("precision,tol", [(abi.MP_FP64, 1e-12), (abi.MP_FP32, 1e-5)], ids=["fp64", "fp32"])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("case", ["plain_periodic", "nl_xy", "lin_all_wave_periodic", "nonlin_all_short",
                                  "plasma_nonlin_all_short"])
def test_rows_match_oracle(case, shape, precision, tol):
    cfg = make_case(case, abi.MP_FP64)
    cfg.nx, cfg.ny, cfg.nz = shape
    cfg.medium_z0, cfg.medium_z1 = 3, cfg.nz + 1
    cfg.cpml_d = min(cfg.cpml_d, min(shape))
    for q in range(cfg.n_sources):
        cfg.sources[q].distance = min(cfg.sources[q].distance, cfg.nz - 1)
    init = random_fields(cfg, sum(shape), smooth=True)
    o = pyoracle.OracleSim(cfg)
    for n, v in init.items():
        o.upload(n, v)
    assert o.step(12) == abi.MP_OK
    cfg.precision = precision
    with runtime.Simulation(cfg) as g:
        for n, v in init.items():
            g.upload(n, v)
        g.step(12)
        for n in abi.FIELD_NAMES:
            assert rel_l2(g.download(n), o.download(n)) <= tol, n


def test_large_kerr_state_fp32_matches_fp64():
    """A state above 1 GB in FP32 (its E half runs two cells per thread, and both
    halves prefetch the next plane) against the FP64 form, on the workload's grid cut
    to 240 planes: eight steps from a pulse in the Kerr medium, the FP32 bar of
    1e-5."""
    fields = {}
    for precision in (abi.MP_FP64, abi.MP_FP32):
        cfg = configs.c3_plrc_kerr(precision, nz=240, focus_z=120)
        init = abi.default_init(abi.MP_INIT_PULSE)
        init.k[:] = (0.0, 0.0, 2 * 3.141592653589793 / 0.8)
        init.B[:] = (0.3, 1.0, 0.0)
        init.r0, init.z0, init.zc, init.C = 2.0, 2.5, 150 * cfg.dz, 0.0
        with runtime.Simulation(cfg) as g:
            g.initialize(init)
            g.step(8)
            fields[precision] = {n: g.download(n) for n in abi.FIELD_NAMES}
    for n in abi.FIELD_NAMES:
        assert rel_l2(fields[abi.MP_FP32][n], fields[abi.MP_FP64][n]) <= 1e-5, n

"""The objective over boxes of more than one block of 1024 cells: a step's term is
then several partial sums (up to 148, rows dealt to blocks, odd extents), and the
partial sums of all steps may exceed the context's own buffer of 32768.  Against the
same sums over the downloaded fields, and the adjoint against its CPU restatement."""
import numpy as np
import pytest

from mpulse_b200 import abi, runtime
from oracle import pyadjoint
from tests.cases import make_case, random_fields, rel_l2
from tests.test_adjoint_oracle import clean_init, design_case, design_maps
from tests.test_gpu_adjoint import gpu_sim

pytestmark = pytest.mark.gpu

E2, SZ = abi.MP_OBJ_E2_BOX, abi.MP_OBJ_SZ_PLANE


def summed_objective(cfg, init, adj):
    """J from the fields of every step, summed in FP64 on the host."""
    x0, x1, y0, y1, z0, z1 = adj.box
    J = 0.0
    with runtime.Simulation(cfg) as g:
        for n, v in init.items():
            g.upload(n, v)
        for _ in range(adj.steps):
            g.step(1)
            if adj.kind == E2:
                box = np.s_[z0:z1 + 1, y0 - 1:y1, x0 - 1:x1]
                J += cfg.dt * sum(np.sum(g.download(n)[box] ** 2) for n in ("Ex", "Ey", "Ez"))
            else:
                box = np.s_[z0, y0 - 1:y1, x0 - 1:x1]
                ex, ey, bx, by = (g.download(n)[box] for n in ("Ex", "Ey", "Bx", "By"))
                J += cfg.dt * cfg.dx * cfg.dy * np.sum(ex * by - ey * bx)
    return J


@pytest.mark.parametrize("precision", [abi.MP_FP64, abi.MP_FP32], ids=["fp64", "fp32"])
@pytest.mark.parametrize("kind,box,steps", [
    (E2, (4, 16, 5, 13, 6, 16), 3),        # 1287 cells: two blocks, rows of 13
    (E2, (1, 32, 1, 32, 3, 4), 3),         # 2048: two full blocks
    (E2, (3, 3, 2, 59, 1, 63), 2),         # rows of one cell
    (E2, (3, 63, 4, 56, 2, 54), 3),        # 171 349: the cap of 148 blocks
    (E2, (3, 63, 4, 56, 2, 54), 222),      # 32 856 partial sums: an allocation of their own
    (SZ, (2, 66, 1, 59, 31, 31), 3),       # 3835 cells of a plane: four blocks
    (SZ, (1, 67, 3, 3, 40, 40), 2),        # one row
], ids=["2blocks", "2full", "thin", "cap", "alloc", "plane", "row"])
def test_objective_over_large_boxes(kind, box, steps, precision):
    """Both sums add the same FP64 terms, up to 222 x 171 349 of them in blocks of a
    few hundred: 1e-12 of the sum of |terms| (the plane flux has either sign)."""
    cfg = make_case("lin_vacuum_cpmlz", precision)
    cfg.nx, cfg.ny, cfg.nz = 67, 59, 63
    init = random_fields(cfg, 21, smooth=True)
    adj = abi.adjoint_config(kind, box, steps)
    want = summed_objective(cfg, init, adj)
    with gpu_sim(cfg, init, {}) as g:
        got = g.objective(adj)
        again = g.objective(adj)  # goes on from there, through the same buffer
        assert g.time == 2 * steps
    assert abs(got - want) <= 1e-12 * max(abs(want), cfg.dt * cfg.dx * cfg.dy * steps)
    assert again != got


@pytest.mark.parametrize("kind,box", [(E2, (4, 34, 3, 29, 5, 7)), (SZ, (1, 36, 1, 31, 12, 12))], ids=["box", "plane"])
@pytest.mark.parametrize("every", [0, 4])
def test_adjoint_over_large_boxes(kind, box, every):
    """2511 cells of a box and 1116 of a plane (three and two partial sums a step)."""
    cfg = design_case(abi.MP_SOLVER_PLRC_NONLIN, abi.MP_CPML_ALL, n=(36, 31, 14), source=True)
    des = design_maps(cfg, 51)
    init = clean_init(cfg, 52, smooth=True, scale=0.2)
    adj = abi.adjoint_config(kind, box, 9, checkpoint_every=every)
    J_ref, g_ref = pyadjoint.adjoint_gradient(cfg, adj, init, des)
    with gpu_sim(cfg, init, des) as g:
        Jo = g.objective(adj)
    with gpu_sim(cfg, init, des) as g:
        J, grads = g.adjoint(adj)
    with gpu_sim(cfg, init, des) as g:
        Jr = g.objective_record(adj)
        Jv, grev = g.adjoint_reverse()
    assert Jo == J == Jr == Jv
    assert abs(J - J_ref) <= 1e-12 * abs(J_ref)
    for name, key in (("DesignEps", "eps"), ("DesignDepsScale", "s"), ("DesignChiScale", "u")):
        assert rel_l2(grads[name], g_ref[key]) <= 1e-10, name
        np.testing.assert_array_equal(grev[name], grads[name])

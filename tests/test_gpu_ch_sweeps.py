"""The Cahn-Hilliard PCG swept by many CTAs (dn_wch.cuh) where its layout has edges: block boundaries (32 lines),
odd column counts, one block and several, the smallest box, and with periodic x the wrap inside one block, the wrap
between blocks, and the extents (33 = 32 + 1 lines, fewer than 17) that take the other path.

Both sides solve to a relative residual of 1e-12.  The operator alpha0 I - beta1 L + beta2 L^2 with this test's
alpha0 = 1.5e4 and the largest eigenvalue of -L, 8 * 100^2, has a condition number below 1 + 2e-4 * (8e4)^2 / 1.5e4,
about 90, so two converged solutions agree to 2e-10.  The preconditioner shows in the iteration count, which is the
oracle's up to one where the residual meets the tolerance within rounding.
"""
import numpy as np
import pytest

from test_gpu_parity import interior, rel_l2, seeded_pair, unit

pytestmark = pytest.mark.gpu

BOUND = 2e-10
SHAPES = [(8, 8, 0), (31, 17, 0), (32, 40, 0), (33, 33, 0), (64, 9, 0), (65, 64, 0), (97, 50, 0), (40, 99, 0),
          (16, 40, 1), (17, 40, 1), (18, 21, 1), (32, 33, 1), (33, 40, 1), (34, 41, 1), (63, 24, 1), (64, 47, 1), (65, 30, 1),
          (98, 40, 1)]


@pytest.fixture(scope="module")
def dn():
    import ding_nsch_core_solver_b200 as m

    m.load()
    return m


@pytest.mark.parametrize("nx,ny,px", SHAPES)
def test_ch_solve_matches_the_oracle_on_edge_shapes(dn, nx, ny, px):
    cfg = unit(nx=nx, ny=ny, periodic_x=bool(px), periodic_y=False, pressure_scheme="icpcg", dt=1e-4,
               ch_tolerance=1e-12, ch_inner_iterations=2000)
    orc, gpu = seeded_pair(dn, cfg, seed=nx + 3 * ny)
    try:
        rng = np.random.default_rng(ny)
        c = gpu.get_field("c")
        alpha0 = 1.5 / cfg["dt"]
        rhs = alpha0 * (c + 0.05 * rng.standard_normal(c.shape))
        got, _, eq, its = gpu.ch_linear_solve(rhs, alpha0, c)
        want, _, eq_o = orc.ch_linear_solve(rhs, alpha0, c)
        assert rel_l2(interior(got, 3), interior(want, 3)) <= BOUND, (its, eq, eq_o)
        rep = gpu.step(0)  # and inside a step, where the oracle reports its iterations
        orc.step(0)
        assert abs(rep["ch_iterations"] - orc.report()["ch_iterations"]) <= 1
        assert rel_l2(interior(gpu.get_field("c"), 3), interior(orc.field("c"), 3)) <= BOUND
    finally:
        gpu.close()
        orc.close()

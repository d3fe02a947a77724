"""The Cahn-Hilliard sweeps of a box periodic in y (apply_seq13), where the factor's rows are one chain: line lengths
from the smallest box's (8), every remainder of its chunks of 4 rows, lines longer than the CTA's
threads, few lines, and with periodic x the wrap between the first and last two lines.

Both sides solve to a relative residual of 1e-12 and, with cells of 1/100 whatever the shape, the operator's condition
number is below 1 + 2e-4 * (8e4)^2 / 1.5e4, about 90 (alpha0 = 1.5e4, largest eigenvalue of -L 8 * 100^2), so two converged solutions agree to 2e-10.  The
preconditioner shows in the iteration count, which is the oracle's up to one where the residual meets the tolerance
within rounding.
"""
import numpy as np
import pytest

from test_gpu_parity import interior, rel_l2, seeded_pair, unit

pytestmark = pytest.mark.gpu

BOUND = 2e-10
SHAPES = [(8, 8, 0), (8, 8, 1), (8, 9, 1), (9, 10, 0), (9, 11, 1), (12, 13, 1), (40, 11, 0), (33, 64, 1), (64, 33, 0),
          (16, 230, 1), (10, 290, 0), (8, 520, 1)]


@pytest.fixture(scope="module")
def dn():
    import ding_nsch_core_solver_b200 as m

    m.load()
    return m


@pytest.mark.parametrize("nx,ny,px", SHAPES)
def test_ch_solve_with_periodic_y_matches_the_oracle(dn, nx, ny, px):
    cfg = unit(nx=nx, ny=ny, lx=nx / 100.0, ly=ny / 100.0, periodic_x=bool(px), periodic_y=True, pressure_scheme="icpcg", dt=1e-4,
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
        gpu.begin_step(0)
        rep = gpu.phase(0)  # and inside a step, where the oracle reports its iterations
        orc.step(0)
        assert abs(rep["ch_iterations"] - orc.report()["ch_iterations"]) <= 1
    finally:
        gpu.close()
        orc.close()

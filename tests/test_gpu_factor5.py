"""The 5-point incomplete factor (k_factor5) where its walk has edges: the smallest box (its loads run 5 levels
ahead, a periodic side's d is 7 levels old), level counts of every remainder of its groups of 3, more lines than its
512 threads, and every periodicity.

The pressure solve stops after one iteration on both sides, so that p shows the preconditioner itself, applied twice,
and not what the iteration makes of it.  Forward and backward substitution over at most 610 levels of two terms, in
FP64 with growth below 10 per application, leave under 2 * 2 * 610 * 10 * 1.1e-16 = 3e-12 of relative error between
two orders of summation; 1e-11 is asked for.
"""
import pytest

from test_gpu_parity import interior, rel_l2, seeded_pair, unit

pytestmark = pytest.mark.gpu

BOUND = 1e-11
SHAPES = [(8, 8, 1, 1), (9, 8, 1, 0), (8, 11, 0, 1), (10, 9, 0, 0), (31, 45, 0, 0), (40, 33, 1, 1), (513, 9, 0, 0),
          (600, 10, 1, 0), (520, 8, 1, 1), (10, 600, 1, 1)]


@pytest.fixture(scope="module")
def dn():
    import ding_nsch_core_solver_b200 as m

    m.load()
    return m


@pytest.mark.parametrize("scheme", ["icpcg", "ildlt_pcg"])
@pytest.mark.parametrize("nx,ny,px,py", SHAPES)
def test_one_iteration_with_the_factor_matches_the_oracle(dn, nx, ny, px, py, scheme):
    cfg = unit(nx=nx, ny=ny, lx=nx / 100.0, ly=ny / 100.0, periodic_x=bool(px), periodic_y=bool(py),
               pressure_scheme=scheme, dt=1e-4, density_ratio=10.0, poisson_iterations=1)
    orc, gpu = seeded_pair(dn, cfg, seed=nx + 7 * ny)
    try:
        orc.begin_step(1)
        orc.phase(1)
        orc.momentum(1)
        orc.pressure()
        got, its, _ = gpu.pressure_solve(1, *(orc.field(n) for n in ("u_star", "v_star", "rho_mid", "p", "p_prev")))
        assert its == orc.report()["pressure_iterations"] == 1
        assert rel_l2(interior(got, 3), interior(orc.field("p_corr"), 3)) <= BOUND
    finally:
        gpu.close()
        orc.close()

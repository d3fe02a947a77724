"""The pressure PCG in sweep order (dn_wpcg.cuh) where its layout has edges: block boundaries (32 lines), odd
column counts, lines as short as it takes them, one block, several blocks, more blocks than one CTA sweeps, and
the extents just below which another path is taken, with every periodicity and operator.

The systems are solved to a relative residual of 1e-12 by both sides.  p then carries at most cond(A) 1e-12 of
relative error in its slowest modes; cond(A) of the largest grid here (150 x 40 cells) is below 4 (150 / pi)^2
times the density ratio 10, under 1e5, so two converged solutions agree to 2e-7.  The preconditioner shows in the
iteration count: with the reference's factors exactly applied it is the oracle's, up to one iteration where the
residual meets the tolerance within rounding.
"""
import numpy as np
import pytest

from test_gpu_parity import interior, rel_l2, seeded_pair, unit

pytestmark = pytest.mark.gpu

BOUND = 2e-7
WALLS, PX, PY, PXY = (False, False), (True, False), (False, True), (True, True)
SHAPES = [
    # nx, ny, periodicity
    (8, 8, WALLS), (31, 17, WALLS), (32, 18, WALLS), (33, 33, WALLS), (64, 9, WALLS), (65, 40, WALLS),
    (150, 40, WALLS), (40, 131, WALLS),
    (16, 20, PX), (17, 20, PX), (32, 21, PX), (33, 16, PX), (64, 30, PX), (97, 31, PX),
    (20, 32, PY), (20, 33, PY), (20, 34, PY), (33, 47, PY), (65, 36, PY),
    (17, 33, PXY), (18, 34, PXY), (32, 35, PXY), (33, 64, PXY), (70, 41, PXY),
]


@pytest.fixture(scope="module")
def dn():
    import ding_nsch_core_solver_b200 as m

    m.load()
    return m


@pytest.mark.parametrize("scheme", ["icpcg", "split_icpcg", "split_ildlt_pcg"])
@pytest.mark.parametrize("nx,ny,per", SHAPES)
def test_pressure_solve_matches_the_oracle_on_edge_shapes(dn, nx, ny, per, scheme):
    cfg = unit(nx=nx, ny=ny, periodic_x=per[0], periodic_y=per[1], pressure_scheme=scheme, dt=1e-4,
               density_ratio=10.0, pressure_tolerance=1e-12, poisson_iterations=2000)
    orc, gpu = seeded_pair(dn, cfg, seed=nx + 7 * ny)
    try:
        rep = gpu.step(0)
        orc.step(0)
        ro = orc.report()
        g = cfg["ghost"]
        err = rel_l2(interior(gpu.get_field("p"), g), interior(orc.field("p"), g))
        assert err <= BOUND, (err, rep, ro)
        assert abs(rep["pressure_iterations"] - ro["pressure_iterations"]) <= 1, (rep, ro)
    finally:
        gpu.close()
        orc.close()


@pytest.mark.parametrize("per", [WALLS, PX, PXY])
@pytest.mark.parametrize("warps", [1, 2])
def test_blocks_of_one_cta_and_of_several_agree(dn, per, warps):
    """The same solve with one and two blocks per CTA (lines handed over in global and in shared memory) and on
    few CTAs: the same operations in the same order per cell, so only the reductions' order differs."""
    base = unit(nx=100, ny=70, periodic_x=per[0], periodic_y=per[1], pressure_scheme="icpcg", dt=1e-4,
                density_ratio=10.0, pressure_tolerance=1e-12, poisson_iterations=2000)
    orc, ref = seeded_pair(dn, base, seed=3)
    other = dn.Solver(dict(base, sweep_warps_per_cta=warps, pcg_rows_per_cta=4096))
    try:
        for n in ("c", "c_prev", "c_prev2", "p", "p_prev", "u", "v", "u_prev", "v_prev", "e_prev", "hu_prev",
                  "hv_prev"):
            other.set_field(n, ref.get_field(n))
        other.refresh_derived()
        ref.refresh_derived()
        a, b = ref.step(0), other.step(0)
        assert abs(a["pressure_iterations"] - b["pressure_iterations"]) <= 1
        assert rel_l2(interior(other.get_field("p"), 3), interior(ref.get_field("p"), 3)) <= BOUND
    finally:
        for s in (ref, other):
            s.close()
        orc.close()

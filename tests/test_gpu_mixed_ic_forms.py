"""The mixed form's IC inner solver on periodic-y grids whose lines (32 columns or fewer) are too short for the sweep order:
the staged wavefront in FP32, with every wrap, operator and factor, one sweep warp and several.

The solve ends on the FP64 residual of the FP64 operator, which is asked for, and the inner solves gain on it at the rate
of the FP64 solve, in cycles of 1e5 or so: all cycles together take no more than three times its iterations (the wavefront
on global memory takes up to six times as many).
"""
import numpy as np
import pytest

from test_gpu_parity import unit

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dn():
    import ding_nsch_core_solver_b200 as m

    m.load()
    return m


@pytest.mark.parametrize("scheme", ["split_icpcg", "icpcg", "split_ildlt_pcg"])
@pytest.mark.parametrize("nx,ny,px", [(20, 24, 0), (64, 24, 0), (64, 24, 1), (130, 24, 0), (130, 25, 1), (97, 32, 0)])
def test_short_periodic_lines_take_the_staged_wavefront(dn, nx, ny, px, scheme):
    cfg = unit(nx=nx, ny=ny, lx=nx / 64.0, ly=ny / 64.0, interface_center_x=nx / 128.0, interface_center_y=ny / 128.0,
               interface_radius=0.1, periodic_x=bool(px), periodic_y=True, pressure_scheme=scheme, dt=1e-4, density_ratio=10.0)
    plain = dn.Solver(cfg)
    mixed = dn.Solver(dict(cfg, precision="mixed", mixed_preconditioner="ic"))
    try:
        assert mixed.solver_forms()["pressure"] == plain.solver_forms()["pressure"] == "staged_wavefront"
        for s in (plain, mixed):
            s.initialize()
            rng = np.random.default_rng(nx)
            for name in ("u", "v"):
                f = s.get_field(name)
                f[3:-3, 3:-3] += 0.05 * rng.standard_normal(f[3:-3, 3:-3].shape)
                s.set_field(name, f)
            s.refresh_derived()
        for step in range(2):
            a, b = plain.step(step), mixed.step(step)
        assert not b["mixed_inner_multigrid"]
        assert b["pressure_iterations"] <= 3 * a["pressure_iterations"], (a, b)
        assert b["pressure_residual"] < 1e-10
    finally:
        plain.close()
        mixed.close()


@pytest.mark.parametrize("scheme", ["split_icpcg", "icpcg", "split_ildlt_pcg"])
@pytest.mark.parametrize("nx,ny,px,py", [(64, 24, 0, 0), (64, 24, 0, 1), (130, 24, 0, 0), (97, 32, 0, 1), (97, 32, 0, 0), (64, 64, 0, 1),
                                         (64, 64, 0, 0)])
def test_a_small_right_hand_side_is_no_breakdown(dn, nx, ny, px, py, scheme):
    """A drop at rest: a small right-hand side, whose later corrections have p.Ap under 1e-30."""
    cfg = unit(nx=nx, ny=ny, lx=nx / 64.0, ly=ny / 64.0, interface_center_x=nx / 128.0, interface_center_y=ny / 128.0,
               interface_radius=0.1, periodic_x=bool(px), periodic_y=bool(py), pressure_scheme=scheme, dt=1e-4, density_ratio=10.0)
    s = dn.Solver(dict(cfg, precision="mixed", mixed_preconditioner="ic"))
    try:
        s.initialize()
        for step in range(2):
            assert s.step(step)["pressure_residual"] < 1e-10
    finally:
        s.close()

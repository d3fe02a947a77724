"""The waits of the Cahn-Hilliard sweeps across a periodic x side (dn_wch.cuh, the wrap lines): shapes whose last step is the
last look at a wrap entry and shapes with steps to spare, with the wrap inside a block and between blocks, solved many
times over with a limit far below the default; and a limit that runs out, which ends in its status and leaves the
context usable.
"""
import numpy as np
import pytest

from ding_nsch_core_solver_b200 import capi
from test_gpu_parity import unit

pytestmark = pytest.mark.gpu

# (np + 62) % 8 == 0 for ny = 20, 36; nx % 32 == 0 puts the last line in a block's last lane
SHAPES = [(63, 24), (64, 20), (32, 36), (96, 36), (34, 41), (130, 20)]


def channel(nx, ny, **more):
    return unit(nx=nx, ny=ny, lx=nx / 100.0, ly=ny / 100.0, periodic_x=True, periodic_y=False, pressure_scheme="icpcg", dt=1e-4,
                ch_inner_iterations=2000, **more)


@pytest.mark.parametrize("nx,ny", SHAPES)
def test_many_solves_end_alike(nx, ny):
    s = capi.Solver(channel(nx, ny, device_wait_limit=1 << 18))
    try:
        assert s.solver_forms()["ch"] == "sweep_order"
        s.initialize()
        rng = np.random.default_rng(nx)
        c = s.get_field("c")
        rhs = 1.5e4 * (c + 0.05 * rng.standard_normal(c.shape))
        first = s.ch_linear_solve(rhs, 1.5e4, c)
        for _ in range(150):
            again = s.ch_linear_solve(rhs, 1.5e4, c)
            assert again[3] == first[3] and np.array_equal(again[0], first[0])
    finally:
        s.close()


def test_a_wait_that_runs_out_ends_in_its_status():
    cfg = channel(130, 20)
    short = capi.Solver(dict(cfg, device_wait_limit=1))
    try:
        short.initialize()
        c = short.get_field("c")
        with pytest.raises(capi.DnError) as e:
            short.ch_linear_solve(1.5e4 * c, 1.5e4, np.zeros_like(c))
        assert e.value.status == 8
    finally:
        short.close()
    s = capi.Solver(cfg)
    try:
        s.initialize()
        s.step(0)
    finally:
        s.close()

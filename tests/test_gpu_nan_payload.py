"""A state with a NaN ends in the same status whatever the NaN's bits are: those that mark an empty reduction slot of the
sweep-order PCGs (all ones, what memory filled with 0xff holds) or an empty hand-over entry are no exception.
"""
import numpy as np
import pytest

from ding_nsch_core_solver_b200 import capi
from test_gpu_parity import unit

pytestmark = pytest.mark.gpu

PATTERNS = [0x7FF8000000000000, 0xFFFFFFFFFFFFFFFF, 0x7FFFFFFFFFFFFFFF, 0x7FF4DEAD5EED0001, 0xFFF8000000000000]


def status(solver, call):
    try:
        call(solver)
        return 0, ""
    except capi.DnError as e:
        return e.status, str(e)
    finally:
        solver.close()


@pytest.mark.parametrize("px", [False, True])
def test_the_status_does_not_depend_on_the_nan(px):
    cfg = unit(nx=72, ny=40, periodic_x=px, periodic_y=False, pressure_scheme="split_icpcg", dt=1e-4)
    got = []
    for bits in PATTERNS:
        nan = np.array([bits], dtype=np.uint64).view(np.float64)[0]

        def step(s):
            s.initialize()
            c = s.get_field("c")
            c[3 + 20, 3 + 10] = nan
            s.set_field("c", c)
            s.step(0)

        def backend(s):
            s.initialize()
            a = {n: s.get_field(n) for n in ("u_star", "v_star", "rho_mid", "p", "p_prev")}
            a["u_star"][3 + 30, 3 + 20] = nan
            s.pressure_solve(1, a["u_star"], a["v_star"], a["rho_mid"], a["p"], a["p_prev"])

        got.append((status(capi.Solver(cfg), step), status(capi.Solver(cfg), backend)))
    assert all(g == got[0] for g in got), got
    assert got[0][0][0] == 6 and got[0][1][0] == 6  # pcg breakdown

"""Which kernels a handle's PCG solves run (dn_solver_forms): a matter of the configuration and the device, not of what
else lies in the device's memory when the handle is made; and a handle whose optional buffers cannot be had is made
all the same, runs the other form and leaves no CUDA error behind.
"""
import pytest

from test_gpu_parity import interior, rel_l2, unit

pytestmark = pytest.mark.gpu

GRID = dict(nx=512, ny=512, periodic_x=False, periodic_y=False, pressure_scheme="icpcg", dt=1e-5, ch_inner_iterations=400,
            pressure_tolerance=1e-8, poisson_iterations=3000)


@pytest.fixture(scope="module")
def dn():
    import ding_nsch_core_solver_b200 as m

    m.load()
    return m


def free_bytes():
    import torch

    return torch.cuda.mem_get_info()[0]


def fill_all_but(leave):
    """The device's memory but for about `leave` bytes, in blocks that are never touched."""
    import torch

    held = []
    for unit_bytes in (1 << 32, 1 << 28, 1 << 24):
        while free_bytes() > leave + unit_bytes:
            held.append(torch.empty(unit_bytes, dtype=torch.uint8, device="cuda"))
    return held


def one_step(dn, cfg):
    s = dn.Solver(cfg)
    try:
        s.initialize()
        s.step(0)
        return s.solver_forms(), interior(s.get_field("p"), 3).copy(), interior(s.get_field("c"), 3).copy()
    finally:
        s.close()


@pytest.mark.parametrize("spare", [1.0, -0.5], ids=["room", "no room"])
def test_forms_do_not_follow_the_free_memory(dn, spare):
    """room: the handle fits with as much again as its optional buffers to spare.  no room: half of them is missing."""
    import torch

    cfg = unit(**GRID)
    warm = dn.Solver(cfg)  # the context's own allocations
    warm.close()
    forms, p, c = one_step(dn, cfg)
    assert forms == {"ch": "sweep_order", "pressure": "sweep_order"}
    before = free_bytes()
    s = dn.Solver(cfg)
    whole = before - free_bytes()
    s.close()
    optional = 16 * 13 * 16 * 32 * (256 + 64) + 16 * 15 * 16 * 32 * (256 + 32)  # both PCGs' vectors
    held = fill_all_but(whole + int(spare * optional))
    try:
        got, p1, c1 = one_step(dn, cfg)
    finally:
        held.clear()
        torch.cuda.empty_cache()
    if spare > 0:
        assert got == forms
    else:
        assert "sweep_order" in forms.values() and got != forms
    # either form converges to 1e-10 (c) and 1e-8 (p) of the right-hand side; the operators' condition numbers are below
    # 1e5 (c) and 4 (512 / pi)^2 times the density ratio 10 (p)
    assert rel_l2(c1, c) <= 1e-5 and rel_l2(p1, p) <= 2e-2

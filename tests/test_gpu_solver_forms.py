"""Which kernels a handle's PCG solves run (dn_solver_forms): a matter of the configuration and the device, not of what
else lies in the device's memory when the handle is made; and a handle whose optional buffers cannot be had is made
all the same, runs the other form and leaves no CUDA error behind.

Each case is a process of its own: what a process has freed stays in its context's pools, where the device's count of
free memory does not show it.
"""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

GRID = dict(nx=512, ny=512, periodic_x=False, periodic_y=False, pressure_scheme="icpcg", dt=1e-5, ch_inner_iterations=400,
            pressure_tolerance=1e-8, poisson_iterations=3000)


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
    from test_gpu_parity import interior

    s = dn.Solver(cfg)
    try:
        s.initialize()
        s.step(0)
        return s.solver_forms(), interior(s.get_field("p"), 3).copy(), interior(s.get_field("c"), 3).copy()
    finally:
        s.close()


def measure(spare):
    """Forms of a handle on the empty device and beside a filled memory, and how far their steps lie apart."""
    import ding_nsch_core_solver_b200 as dn
    from test_gpu_parity import rel_l2, unit

    cfg = unit(**GRID)
    first, p, c = one_step(dn, cfg)
    before = free_bytes()
    s = dn.Solver(cfg)
    whole = before - free_bytes()
    s.close()
    optional = 16 * 13 * 16 * 32 * (256 + 64) + 16 * 15 * 16 * 32 * (256 + 32)  # both PCGs' vectors
    held = fill_all_but(whole + int(spare * optional))
    then, p1, c1 = one_step(dn, cfg)
    return dict(first=first, then=then, c=rel_l2(c1, c), p=rel_l2(p1, p), held=len(held))


def footprint(periodic_x):
    import ding_nsch_core_solver_b200 as dn
    from test_gpu_parity import unit

    cfg = unit(**dict(GRID, periodic_x=periodic_x))
    dn.Solver(cfg).close()
    before = free_bytes()
    s = dn.Solver(cfg)
    used = before - free_bytes()
    forms = s.solver_forms()
    s.close()
    return dict(forms, bytes=used)


def child(*args):
    """This file as a program; its last line."""
    here = os.path.dirname(os.path.abspath(__file__))
    env = dict(os.environ, PYTHONPATH=os.pathsep.join([os.path.dirname(here), here, os.environ.get("PYTHONPATH", "")]))
    run = subprocess.run([sys.executable, os.path.abspath(__file__), *args], capture_output=True, text=True, env=env, timeout=300)
    assert run.returncode == 0, run.stderr[-2000:]
    return json.loads(run.stdout.splitlines()[-1])


@pytest.mark.parametrize("spare", [1.0, -0.5], ids=["room", "no room"])
def test_forms_do_not_follow_the_free_memory(spare):
    """room: the handle fits with as much again as its optional buffers to spare.  no room: half of them is missing."""
    got = child("free", str(spare))
    assert got["first"] == {"ch": "sweep_order", "pressure": "sweep_order"}
    if spare > 0:
        assert got["then"] == got["first"]
    else:
        assert got["then"] != got["first"]
    # either form converges to 1e-10 (c) and 1e-8 (p) of the right-hand side; the operators' condition numbers are below
    # 1e5 (c) and 4 (512 / pi)^2 times the density ratio 10 (p)
    assert got["c"] <= 1e-5 and got["p"] <= 2e-2


def test_a_handle_holds_no_rows_of_a_form_that_it_does_not_run():
    """The ordered factor rows of the level ring (192 bytes a cell) belong to walled boxes that run it; a box swept by
    many CTAs takes what its periodic-x twin takes, which has its wrap lines on top (8 MiB for the allocator's steps)."""
    walls, channel = child("rows", "0"), child("rows", "1")
    assert walls["ch"] == channel["ch"] == "sweep_order"
    assert walls["bytes"] <= channel["bytes"] + (8 << 20)


if __name__ == "__main__":
    print(json.dumps(measure(float(sys.argv[2])) if sys.argv[1] == "free" else footprint(sys.argv[2] == "1")))

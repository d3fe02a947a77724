"""device_share: persistent launches of instances that run side by side fit the SMs together.

A block of 32 lines of the sweep-order Cahn-Hilliard PCG is a CTA that takes an SM, and one or two blocks of the pressure
PCG are.  Sixteen instances of 320 lines have 9 SMs each: ten CTAs are too many, five are not; with 32 instances
(4 SMs each) five are too many as well.  Batches through both kernels, several blocks wide, equal their instances
stepped alone bit for bit, as eager steps and replayed from a graph.
"""
import numpy as np
import pytest

from test_gpu_parity import unit

pytestmark = pytest.mark.gpu

WALLS = dict(nx=320, ny=40, periodic_x=False, periodic_y=False, pressure_scheme="split_icpcg", body_force_y=-0.98, dt=1e-4)
CHANNEL = dict(nx=100, ny=40, periodic_x=True, periodic_y=False, pressure_scheme="icpcg", top_wall_velocity_x=0.5,
               bottom_wall_velocity_x=-0.5, dt=1e-4)


@pytest.fixture(scope="module")
def dn():
    import ding_nsch_core_solver_b200 as m

    m.load()
    return m


def seeded(dn, cfg, seed, graph):
    s = dn.Solver(unit(**cfg))
    s.initialize()
    rng = np.random.default_rng(seed)
    for name, a in (("c", 0.02), ("u", 0.05), ("v", 0.05)):
        f = s.get_field(name)
        f[3:-3, 3:-3] += a * rng.standard_normal(f[3:-3, 3:-3].shape)
        s.set_field(name, f)
    s.set_initial_mass(0.0)
    s.refresh_derived()
    s.set_step_graph(graph)
    return s


@pytest.mark.parametrize("share,forms", [(1, ("sweep_order", "sweep_order")), (14, ("sweep_order", "sweep_order")),
                                         (16, ("level_ring", "sweep_order")), (32, ("level_ring", "staged_wavefront"))])
def test_forms_fit_the_share(dn, share, forms):
    import torch

    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the shares are those of 148 SMs")
    s = dn.Solver(unit(**WALLS, device_share=share))
    try:
        got = s.solver_forms()
        assert (got["ch"], got["pressure"]) == forms
    finally:
        s.close()


@pytest.mark.parametrize("graph", [False, True], ids=["eager", "graph"])
@pytest.mark.parametrize("cfg,count", [(WALLS, 16), (CHANNEL, 5)], ids=["walls", "channel"])
def test_batch_of_several_blocks_equals_each_alone(dn, cfg, count, graph):
    from ding_nsch_core_solver_b200 import capi

    cfg = dict(cfg, device_share=count)
    batch = [seeded(dn, cfg, 40 + k, graph) for k in range(count)]
    alone = [seeded(dn, cfg, 40 + k, graph) for k in range(count)]
    try:
        for step in range(4):  # the graph is recorded at step 2 and replayed at 3
            reps = capi.step_batch(batch, [step] * count)
            for k, s in enumerate(alone):
                assert s.step(step) == reps[k], (step, k)
        for k in range(count):
            for name in ("c", "mu", "u", "v", "p"):
                assert np.array_equal(batch[k].get_field(name), alone[k].get_field(name)), (k, name)
    finally:
        for s in batch + alone:
            s.close()

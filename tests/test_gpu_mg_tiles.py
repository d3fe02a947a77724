"""The multigrid V-cycle's tiles (k_mg_down, k_mg_up) and its one-CTA bottom (k_mg_bottom) where their layout has
edges: one tile and several, a last tile of a few cells, grids narrower than a tile with the region wrapped around
them several times (periodic sides), Dirichlet and Neumann walls, and every number of levels below the tiles
(none: the level-0 grid fits the bottom).

The reference is the same solve as one cluster launch (mg_cluster_cells), which runs the V-cycle phase by phase over
whole levels.  Both solves stop after one inner iteration, so that the answer is one V-cycle (pressure) or two of them
in sequence (CH) times alpha = r.z / p.q.  The V-cycles agree bit for bit; the sums in alpha are taken in another
order, in FP64 over FP32 values, so that alpha, rounded to FP32, may differ by one unit in the last place, 1.2e-7, and
each product alpha p by that and its own rounding: rel-L2 <= 2e-7.
"""
import numpy as np
import pytest

from test_gpu_parity import interior, rel_l2, seeded_pair, unit

pytestmark = pytest.mark.gpu

BOUND = 2e-7
# nx, ny, periodic x, periodic y, Dirichlet top
SHAPES = [(56, 104, 0, 0, 0), (56, 104, 1, 0, 0), (56, 104, 0, 1, 0), (104, 56, 1, 1, 0), (112, 112, 0, 0, 1),
          (16, 256, 1, 0, 0), (256, 16, 0, 1, 0), (16, 256, 0, 0, 1), (128, 64, 0, 0, 0), (64, 160, 1, 1, 0),
          (192, 96, 0, 0, 1), (32, 64, 0, 0, 0), (32, 64, 1, 1, 0), (24, 16, 0, 0, 1), (8, 16, 0, 0, 0), (10, 12, 1, 0, 0)]


@pytest.fixture(scope="module")
def dn():
    import ding_nsch_core_solver_b200 as m

    m.load()
    return m


@pytest.mark.parametrize("nx,ny,px,py,dirichlet", SHAPES)
def test_one_inner_iteration_equals_the_phase_by_phase_form(dn, nx, ny, px, py, dirichlet):
    cfg = unit(nx=nx, ny=ny, periodic_x=bool(px), periodic_y=bool(py), pressure_scheme="split_icpcg", dt=1e-4,
               precision="mixed", poisson_iterations=1, ch_inner_iterations=1)
    if dirichlet:
        cfg.update(pressure_bc_top_type="dirichlet", pressure_bc_top_value=0.3)
    got = {}
    for cells in (0, 1 << 20):
        orc, gpu = seeded_pair(dn, dict(cfg, mg_cluster_cells=cells), seed=nx + 3 * ny)
        try:
            rng = np.random.default_rng(ny)
            c = gpu.get_field("c")
            alpha0 = 1.5 / cfg["dt"]
            x, _, _, its = gpu.ch_linear_solve(alpha0 * (c + 0.05 * rng.standard_normal(c.shape)), alpha0, c)
            assert its == 1
            star = {n: orc.field(n).copy() for n in ("u_star", "v_star", "rho_mid", "p", "p_prev")}
            for n in ("u_star", "v_star"):
                star[n] += 0.1 * rng.standard_normal(star[n].shape)
            p, its, _ = gpu.pressure_solve(1, star["u_star"], star["v_star"], star["rho_mid"], star["p"], star["p_prev"])
            assert its == 1
            got[cells] = interior(x, 3) - interior(c, 3), interior(p, 3)
        finally:
            gpu.close()
            orc.close()
    for a, b in zip(got[0], got[1 << 20]):
        assert np.abs(b).max() > 0.0
        assert rel_l2(a, b) <= BOUND

"""The passes of scenes that fill the GPU a thread a row, bit for bit against the restatement.

DFSPH around 444 blocks of 256 rows (three a SM of 148), up to which the check and the push run as the
builds for few blocks a SM.
"""
import numpy as np
import pytest

from solunar_b200.abi import FluidSettings, FluidSolver

pytestmark = pytest.mark.gpu

SPACING = 0.02


def fill(worlds, n, crowd=0):
    rng = np.random.default_rng(n)
    side = np.cbrt(n) * SPACING
    pts = rng.uniform(0.02, 0.98, (n, 3)) * side
    pts[:crowd] = 0.5 * side + (pts[:crowd] - 0.5 * side) * 0.1
    vel = rng.standard_normal((n, 3)) * 0.2
    for w in worlds:
        w.add_box_container((0.0, 0.0, 0.0), (side, side + SPACING, side))
        w.add_particles(pts.astype(np.float32), vel.astype(np.float32))
    return side


def assert_same(g, o):
    assert np.array_equal(g.ids(), o.ids())
    for name in ("densities", "positions", "velocities"):
        a, b = (np.ascontiguousarray(np.asarray(getattr(w, name)(), dtype=np.float32)).view(np.uint32) for w in (g, o))
        assert np.array_equal(a, b), name


@pytest.mark.parametrize("n", [444 * 256, 444 * 256 + 1])
def test_dfsph_rows_at_the_edge_of_few_blocks(gpu_lib, oracle_lib, n):
    settings = FluidSettings(solver=FluidSolver.DFSPH, spacing=SPACING)
    g, o = gpu_lib.FluidWorld(settings), oracle_lib.OracleWorld(settings, residual_sum=1)
    fill((g, o), n)
    a, b = g.step(3e-4), o.step(3e-4)
    assert (a.substeps, a.iterations, a.held_back) == (b.substeps, b.iterations, b.held_back)
    assert_same(g, o)

"""The cell sort over boxes of odd shapes: one cell, columns and slabs without a partner in their
brick, quads cut short, and tables of one scan tile, of several, and of more than the tiles add up
themselves.  A step's densities, factors and velocities are the restatement's bits only if the walk
order names every particle once and the cell table holds.
"""
import numpy as np
import pytest

from solunar_b200.abi import FluidSettings, FluidSolver

pytestmark = pytest.mark.gpu


def bits(a):
    return np.ascontiguousarray(np.asarray(a, dtype=np.float32)).view(np.uint32)


@pytest.mark.parametrize("n,cells", [(9, (1, 1, 1)), (700, (5, 4, 7)), (700, (2, 9, 1)), (700, (1, 1, 90)),
                                     (5000, (13, 11, 10)), (33000, (33, 1, 62)), (33000, (130, 121, 303))])
def test_sort_over_odd_boxes_is_the_restatements(gpu_lib, oracle_lib, n, cells):
    rng = np.random.default_rng(11)
    settings = FluidSettings(solver=FluidSolver.DFSPH, spacing=0.02, gravity=(0.0, 0.0, 0.0))
    r = settings.radius()
    pts = (rng.uniform(0.05, 0.95, (n, 3)) * np.array(cells) - np.array([2, 0, 1])).astype(np.float32) * np.float32(r)
    vel = (rng.standard_normal(pts.shape) * 0.01).astype(np.float32)
    g, o = gpu_lib.FluidWorld(settings), oracle_lib.OracleWorld(settings, residual_sum=1)
    for w in (g, o):
        w.add_particles(pts, vel)
    for _ in range(2):
        a, b = g.step(1e-3), o.step(1e-3)
        assert (a.substeps, a.iterations) == (b.substeps, b.iterations)
    assert np.array_equal(g.ids(), o.ids())
    assert np.array_equal(bits(g.densities()), bits(o.densities()))
    assert np.array_equal(bits(g.positions()), bits(o.positions()))
    assert np.array_equal(bits(g.velocities()), bits(o.velocities()))

"""The EXACT density pass where its scan and its packed pair arithmetic can go wrong, bit for bit
against the restatement: cells of any number of points (remainders of the groups of four), particles
beside, beyond and far from a free-standing wall, lists that outgrow their room, and radii on both
sides of the range whose divisions take the reciprocal.  33,000 particles: a thread a row at supports
under 3 (smaller scenes, and larger ones at more support, give a row several lanes).
"""
import numpy as np
import pytest

from solunar_b200.abi import Arithmetic, FluidSettings, FluidSolver, Positions

pytestmark = pytest.mark.gpu


def bits(a):
    return np.ascontiguousarray(np.asarray(a, dtype=np.float32)).view(np.uint32)


@pytest.mark.parametrize("solver", [FluidSolver.WCSPH, FluidSolver.DFSPH])
@pytest.mark.parametrize("spacing,support", [(0.02, 2.0), (0.03, 1.5), (0.0166, 2.5), (2e-5, 2.0), (700.0, 2.0)])
def test_scan_and_pair_terms_are_the_restatements(gpu_lib, oracle_lib, solver, spacing, support):
    rng = np.random.default_rng(7)
    settings = FluidSettings(solver=solver, spacing=spacing, support=support, gravity=(0.0, -9.81 * spacing, 0.0))
    side = 32 * spacing * 2.0 / support
    pts = rng.uniform(-0.5, 0.5, (33000, 3)) * side
    pts[:600] *= 0.2  # a crowd past the lists' room
    pts[600:605] = 3.0 * side  # five strays in one cell, outside the walls' box
    pts[600:605] += rng.uniform(0.0, 0.3, (5, 3)) * spacing
    pts = pts.astype(np.float32)
    vel = (rng.standard_normal(pts.shape) * spacing).astype(np.float32)
    worlds = gpu_lib.FluidWorld(settings), oracle_lib.OracleWorld(settings, residual_sum=1)
    for w in worlds:
        w.add_wall((0.0, 0.0, 0.0), (5 * spacing, 7 * spacing, 6 * spacing))
        w.add_particles(pts, vel)
    g, o = worlds
    # a step's forces and solves read the kept gradient factors (and DFSPH's whole gradients)
    dt = min(0.1 * spacing, 1e-2)
    a, b = g.step(dt), o.step(dt)
    assert (a.substeps, a.iterations, a.held_back) == (b.substeps, b.iterations, b.held_back)
    assert np.array_equal(g.ids(), o.ids())
    assert np.array_equal(bits(g.positions()), bits(o.positions()))
    assert np.array_equal(bits(g.velocities()), bits(o.velocities()))
    assert np.array_equal(bits(g.densities()), bits(o.densities()))


@pytest.mark.parametrize("positions", [Positions.ABSOLUTE, Positions.CELL_RELATIVE])
@pytest.mark.parametrize("solver", [FluidSolver.WCSPH, FluidSolver.DFSPH])
def test_fast_scan_finds_the_restatements_neighbours(gpu_lib, oracle_lib, solver, positions):
    # a pair found or lost changes a density by far more than the rounding of the up to 64 terms both
    # sums hold: 64 x 2^-24 each, twice that apart.  Pairs at the very radius (which cell-relative
    # offsets may round to the other side) weigh nothing.
    rng = np.random.default_rng(9)
    settings = FluidSettings(solver=solver, spacing=0.02, arithmetic=Arithmetic.FAST, positions=positions)
    pts = (rng.uniform(-0.5, 0.5, (33000, 3)) * 0.64).astype(np.float32)
    pts[600:605] = 1.3
    pts[600:605] += (rng.uniform(0.0, 0.3, (5, 3)) * 0.02).astype(np.float32)
    worlds = gpu_lib.FluidWorld(settings), oracle_lib.OracleWorld(settings, residual_sum=1)
    for w in worlds:
        w.add_wall((0.0, 0.0, 0.0), (0.1, 0.14, 0.12))
        w.add_particles(pts)
        w.update_neighbors()
        w.compute_densities()
    g, o = worlds
    assert np.array_equal(g.ids(), o.ids())
    np.testing.assert_allclose(g.densities(), o.densities(), rtol=2 * 64 * 2.0 ** -24)

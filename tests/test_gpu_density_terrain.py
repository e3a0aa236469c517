"""The densities of worlds on terrain (mod.rs:621-675), bit for bit against the restatement: both solvers'
(a DFSPH world steps on no terrain, but its densities take the ground's share), at a size where rows
without terrain take several lanes and at one where they take a thread each.
"""
import numpy as np
import pytest

from solunar_b200.abi import FluidSettings, FluidSolver

pytestmark = pytest.mark.gpu

SPACING = 0.02
LOW, HIGH = (-0.1, -0.2, -0.1), (1.0, 0.3, 1.0)


@pytest.mark.parametrize("n", [700, 33000])
@pytest.mark.parametrize("solver", [FluidSolver.WCSPH, FluidSolver.DFSPH])
def test_densities_take_the_grounds_share(gpu_lib, oracle_lib, solver, n):
    rng = np.random.default_rng(n)
    side = np.cbrt(n) * SPACING
    pts = (rng.uniform(0.01, 0.99, (n, 3)) * side).astype(np.float32)
    settings = FluidSettings(solver=solver, spacing=SPACING)
    found = []
    for w in (gpu_lib.FluidWorld(settings), oracle_lib.OracleWorld(settings)):
        nx, ny, nz = w.terrain_nodes(LOW, HIGH)
        # ground under a slope: y below 0.2 x (distances in (y, z, x) order)
        y, _, x = np.meshgrid(*(np.arange(k) for k in (ny, nz, nx)), indexing="ij")
        step = SPACING / 2
        w.add_terrain(LOW, HIGH, ((y * step + LOW[1]) - 0.2 * (x * step + LOW[0])) / np.hypot(1.0, 0.2))
        w.add_particles(pts)
        w.update_neighbors()
        w.compute_densities()
        found.append((w.ids(), np.asarray(w.densities(), dtype=np.float32)))
    (gi, gd), (oi, od) = found
    assert np.array_equal(gi, oi)
    assert np.array_equal(gd.view(np.uint32), od.view(np.uint32))

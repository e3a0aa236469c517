"""The EXACT density pass where its scratch holds fewer rows than its grid would run, as in crowds that leave
the device no room for more: bit for bit the restatement's, with lists that outgrow their room as well.
"""
import numpy as np
import pytest

from solunar_b200.abi import FluidSettings, FluidSolver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 512, 4000])
@pytest.mark.parametrize("n", [300, 5001, 40001])
@pytest.mark.parametrize("solver", [FluidSolver.WCSPH, FluidSolver.DFSPH])
def test_a_short_scratch_strides_over_the_rows(gpu_lib, oracle_lib, solver, n, rows):
    rng = np.random.default_rng(n)
    settings = FluidSettings(solver=solver, spacing=0.02)
    side = np.cbrt(n) * 0.02
    pts = rng.uniform(0.02, 0.98, (n, 3)) * side
    pts[:100] = 0.5 * side + (pts[:100] - 0.5 * side) * 0.1
    vel = rng.standard_normal((n, 3)) * 0.2
    g, o = gpu_lib.FluidWorld(settings), oracle_lib.OracleWorld(settings, residual_sum=1)
    for w in (g, o):
        w.add_box_container((0.0, 0.0, 0.0), (side, side + 0.02, side))
        w.add_particles(pts.astype(np.float32), vel.astype(np.float32))
    g.debug_density_rows(rows)
    g.debug_list_room(8)
    a, b = g.step(3e-4), o.step(3e-4)
    assert (a.substeps, a.iterations, a.held_back) == (b.substeps, b.iterations, b.held_back)
    assert np.array_equal(g.ids(), o.ids())
    for name in ("densities", "positions", "velocities"):
        x, y = (np.asarray(getattr(w, name)(), dtype=np.float32).view(np.uint32) for w in (g, o))
        assert np.array_equal(x, y), name

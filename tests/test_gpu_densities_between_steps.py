"""compute_densities between steps, with lists that fit and with lists that outgrow their room: the steps that
follow are the restatement's bit for bit.
"""
import numpy as np
import pytest

from solunar_b200.abi import FluidSettings, FluidSolver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("room", [0, 8])
@pytest.mark.parametrize("solver", [FluidSolver.WCSPH, FluidSolver.DFSPH])
def test_a_step_after_densities(gpu_lib, oracle_lib, solver, room):
    rng = np.random.default_rng(5)
    settings = FluidSettings(solver=solver, spacing=0.02)
    pts = (rng.uniform(0.02, 0.98, (3001, 3)) * 0.3).astype(np.float32)
    vel = (rng.standard_normal(pts.shape) * 0.1).astype(np.float32)
    g, o = gpu_lib.FluidWorld(settings), oracle_lib.OracleWorld(settings, residual_sum=1)
    for w in (g, o):
        w.add_box_container((0.0, 0.0, 0.0), (0.3, 0.4, 0.3))
        w.add_particles(pts, vel)
    for before in ("update_neighbors", "step"):
        for w in (g, o):
            if before == "step":
                w.step(3e-4)
            w.update_neighbors()
        if room:
            g.debug_list_room(room)
            g.update_neighbors()
            o.update_neighbors()
        for w in (g, o):
            w.compute_densities()
        a, b = (np.asarray(w.densities(), dtype=np.float32).view(np.uint32) for w in (g, o))
        assert np.array_equal(a, b)
    # densities straight after a step, over that step's lists, then a step
    for w in (g, o):
        w.step(3e-4)
        w.compute_densities()
        w.step(3e-4)
    assert np.array_equal(g.ids(), o.ids())
    for name in ("densities", "positions", "velocities"):
        a, b = (np.asarray(getattr(w, name)(), dtype=np.float32).view(np.uint32) for w in (g, o))
        assert np.array_equal(a, b), name

"""Steps whose settings or length are so small that a zero is divided by a zero, or so large that a zero
is multiplied by an infinity: refused where the restatement refuses them, its bits where it takes them,
in the passes that give a row several lanes and in those that give it one.
"""
import numpy as np
import pytest

from solunar_b200.abi import Arithmetic, FluidSettings, FluidSolver, PhysicsError

pytestmark = pytest.mark.gpu

WCSPH, DFSPH = FluidSolver.WCSPH, FluidSolver.DFSPH
# a rest density whose square underflows, a step whose square does, a viscosity that overflows
CASES = [(dict(solver=WCSPH, rest_density=r), 1e-4) for r in (1e-22, 1e-23, 1e-25)]
CASES += [(dict(solver=DFSPH), dt) for dt in (1e-15, 1e-24, 1e-40)]
CASES += [(dict(solver=WCSPH, spacing=1e12, rest_density=1e-3, sound_speed=1e15, viscosity=v), 1e-17)
          for v in (1e-15, 1e15)]


def outcome(world, dt):
    try:
        world.step(dt)
    except PhysicsError as e:
        return e.kind
    return "ok"


@pytest.mark.parametrize("arithmetic", [Arithmetic.EXACT, Arithmetic.FAST])
@pytest.mark.parametrize("side", [6, 33])
@pytest.mark.parametrize("fields,dt", CASES)
def test_a_zero_over_a_zero_stays_refused(gpu_lib, oracle_lib, fields, dt, side, arithmetic):
    settings = FluidSettings(arithmetic=arithmetic, **fields)
    # apart enough that no particle is under pressure or asks for a push
    grid = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3)
    pts = (grid * np.float32(1.3 * settings.spacing)).astype(np.float32)
    g, o = gpu_lib.FluidWorld(settings), oracle_lib.OracleWorld(settings)
    for w in (g, o):
        w.add_particles(pts)
    expected = outcome(o, dt)
    assert outcome(g, dt) == expected
    if expected == "ok" and arithmetic == Arithmetic.EXACT:
        for name in ("densities", "positions", "velocities"):
            a, b = (np.asarray(getattr(w, name)(), dtype=np.float32).view(np.uint32) for w in (g, o))
            assert np.array_equal(a, b), name

"""Coupled steps that are refused in mid-step, while the bodies' stream may still be at work: where the next
substep's sort refuses the cells, and where a substep leaves non-finite values.  The world then steps on as
one that never met the refusal, and one that is closed at once ends cleanly.
"""
import numpy as np
import pytest

from solunar_b200.abi import BodyPose, FluidSettings, PhysicsError, Shape, body_handle

pytestmark = pytest.mark.gpu

SPACING = 0.02


@pytest.mark.parametrize("speed", [1e30, 3e38])
@pytest.mark.parametrize("n", [700, 40001])
def test_a_refused_coupled_step_leaves_nothing_behind(gpu_lib, n, speed):
    rng = np.random.default_rng(n)
    side = np.cbrt(n) * SPACING
    pts = (rng.uniform(0.02, 0.98, (n, 3)) * side).astype(np.float32)
    vel = (rng.standard_normal((n, 3)) * 0.2).astype(np.float32)
    wild = vel.copy()
    wild[n // 2] = (speed, 0.0, 0.0)
    poses = [BodyPose(body_handle(1), (side / 2,) * 3, linear_velocity=(0.3, -0.5, 0.1))]

    def world():
        w = gpu_lib.FluidWorld(FluidSettings(spacing=SPACING))
        w.add_particles(pts, vel)
        w.couple(body_handle(1), Shape.CUBOID, (0.05, 0.03, 0.04))
        return w

    calm, tried, dropped = world(), world(), world()
    for w in (tried, dropped):
        w.write_state(pts, wild)
        with pytest.raises(PhysicsError):
            w.step_with_bodies(1e-3, poses)
    dropped.close()
    order = np.argsort(tried.ids(), kind="stable")
    assert np.array_equal(tried.ids()[order], np.arange(n))
    ids = tried.ids()
    tried.write_state(pts[ids], vel[ids])
    for _ in range(2):
        assert tried.step_with_bodies(1e-3, poses) == calm.step_with_bodies(1e-3, poses)
    assert np.array_equal(tried.ids(), calm.ids())
    for name in ("densities", "positions", "velocities"):
        a, b = (np.asarray(getattr(w, name)(), dtype=np.float32).view(np.uint32) for w in (tried, calm))
        assert np.array_equal(a, b), name

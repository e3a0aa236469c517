"""A substep's status, which its last kernel writes into pinned memory where the host waits for it,
with what the coupled bodies' points take queued behind it: a substep that runs again, its lists having
outgrown their room, is taken once, and a profiled world, which waits for the stream, steps alike.
"""
import numpy as np
import pytest

from solunar_b200.abi import BodyPose, FluidSettings, Shape, body_handle

pytestmark = pytest.mark.gpu

SPACING = 0.02


def tank(world, n):
    rng = np.random.default_rng(n)
    side = np.cbrt(n) * SPACING
    pts = (rng.uniform(0.02, 0.98, (n, 3)) * side).astype(np.float32)
    vel = (rng.standard_normal((n, 3)) * 0.2).astype(np.float32)
    world.add_box_container((0.0, 0.0, 0.0), (side, side + SPACING, side))
    world.add_particles(pts, vel)
    world.couple(body_handle(1), Shape.CUBOID, (0.05, 0.03, 0.04))
    world.couple(body_handle(2), Shape.SPHERE, (0.03, 0.0, 0.0))
    return pts, vel, [BodyPose(body_handle(1), (side / 2,) * 3, linear_velocity=(0.3, -0.5, 0.1)),
                      BodyPose(body_handle(2), (side / 4, side / 2, side / 2), linear_velocity=(-0.2, 0.4, 0.0))]


def same(a, b):
    assert np.array_equal(a.ids(), b.ids())
    for name in ("densities", "positions", "velocities"):
        x, y = (np.asarray(getattr(w, name)(), dtype=np.float32).view(np.uint32) for w in (a, b))
        assert np.array_equal(x, y), name


@pytest.mark.parametrize("n", [700, 5001, 40001])
@pytest.mark.parametrize("room", [8, 0])
def test_bodies_take_each_substep_once(gpu_lib, oracle_lib, n, room):
    settings = FluidSettings(spacing=SPACING)
    g, o = gpu_lib.FluidWorld(settings), oracle_lib.OracleWorld(settings)
    for w in (g, o):
        _, _, poses = tank(w, n)
    if room:
        g.debug_list_room(room)  # the first substep's lists outgrow it: that substep runs again
    for _ in range(2):
        (a, pa), (b, pb) = g.step_with_bodies(1e-3, poses), o.step_with_bodies(1e-3, poses)
        assert (a.substeps, a.held_back) == (b.substeps, b.held_back)
        assert pa == pb
    same(g, o)


def test_a_profiled_world_waits_for_the_same_status(gpu_lib):
    g, h = (gpu_lib.FluidWorld(FluidSettings(spacing=SPACING)) for _ in range(2))
    for w in (g, h):
        _, _, poses = tank(w, 5001)
    h.profile(True)
    for _ in range(3):
        assert g.step_with_bodies(1e-3, poses) == h.step_with_bodies(1e-3, poses)
    same(g, h)

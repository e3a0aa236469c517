"""Where a step's substeps carry the bodies' points, on each side of the limits of the one-block kernel (16,384
points, 12,000 cells) and of the device's cell table, in and beside the water: bit for bit the restatement's.
"""
import numpy as np
import pytest

from solunar_b200.abi import BodyPose, FluidSettings, Shape, body_handle

pytestmark = pytest.mark.gpu

SPACING = 0.02
N = 20001
SIDE = float(np.cbrt(N)) * SPACING


def box(k, half, at, velocity=(0.3, -0.5, 0.1)):
    return k, (half,) * 3, BodyPose(body_handle(k), tuple(float(x) for x in at), linear_velocity=velocity,
                                    angular_velocity=(0.0, 0.4, 0.2))


CASES = {
    "a few points": [box(1, 0.05, (SIDE / 2,) * 3)],
    "points just under the limit": [box(1, 0.38, (SIDE / 2, SIDE + 0.36, SIDE / 2))],
    "the same, swept over more cells": [box(1, 0.38, (SIDE / 2, SIDE + 0.36, SIDE / 2), (30.0, -4.0, 10.0))],
    "points over the limit": [box(1, 0.45, (SIDE / 2, SIDE + 0.43, SIDE / 2))],
    "two far apart, more cells than a block's": [box(1, 0.05, (0.1, 0.1, 0.1)), box(2, 0.05, (1.2, 0.9, 0.9))],
    "two whose cells the host sorts": [box(1, 0.05, (0.1, 0.1, 0.1)), box(2, 0.05, (40.0, 0.3, 0.3))],
}


@pytest.mark.parametrize("name", CASES)
def test_carried_points_are_the_restatements(gpu_lib, oracle_lib, name):
    rng = np.random.default_rng(3)
    pts = (rng.uniform(0.02, 0.98, (N, 3)) * SIDE).astype(np.float32)
    vel = (rng.standard_normal((N, 3)) * 0.2).astype(np.float32)
    settings = FluidSettings(spacing=SPACING)
    g, o = gpu_lib.FluidWorld(settings), oracle_lib.OracleWorld(settings)
    for w in (g, o):
        w.add_particles(pts, vel)
        for k, half, _ in CASES[name]:
            w.couple(body_handle(k), Shape.CUBOID, half)
    poses = [pose for _, _, pose in CASES[name]]
    for _ in range(2):
        (a, pa), (b, pb) = g.step_with_bodies(4e-3, poses), o.step_with_bodies(4e-3, poses)
        assert a.substeps > 1 and (a.substeps, a.held_back, a.sound_speed) == (b.substeps, b.held_back, b.sound_speed)
        assert pa == pb
    assert np.array_equal(g.ids(), o.ids())
    for field in ("densities", "positions", "velocities"):
        x, y = (np.asarray(getattr(w, field)(), dtype=np.float32).view(np.uint32) for w in (g, o))
        assert np.array_equal(x, y), field

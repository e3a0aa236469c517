"""The passes that give a row several lanes (k_density_group, k_wcsph_force_group), bit for bit
against the restatement: at the particle counts where the number of lanes changes, on cells of few and
of many points, on crowds that outgrow the lists' room, against walls, and with a coupled body.
"""
import numpy as np
import pytest

from solunar_b200.abi import Arithmetic, BodyPose, FluidSettings, FluidSolver, Shape, body_handle

pytestmark = pytest.mark.gpu


def bits(a):
    return np.ascontiguousarray(np.asarray(a, dtype=np.float32)).view(np.uint32)


def assert_same(g, o):
    assert np.array_equal(g.ids(), o.ids())
    for name in ("densities", "positions", "velocities"):
        assert np.array_equal(bits(getattr(g, name)()), bits(getattr(o, name)())), name


def fill(worlds, n, spacing, crowd):
    rng = np.random.default_rng(n)
    side = np.cbrt(n) * spacing
    pts = rng.uniform(0.02, 0.98, (n, 3)) * side
    pts[:crowd] = 0.5 * side + (pts[:crowd] - 0.5 * side) * 0.1
    vel = rng.standard_normal((n, 3)) * 0.2
    for w in worlds:
        w.add_box_container((0.0, 0.0, 0.0), (side, side + spacing, side))
        w.add_particles(pts.astype(np.float32), vel.astype(np.float32))


@pytest.mark.parametrize("solver", [FluidSolver.WCSPH, FluidSolver.DFSPH])
@pytest.mark.parametrize("n,support", [(1, 2.0), (33, 2.0), (2048, 2.0), (2049, 2.0), (8192, 2.0), (8193, 2.0),
                                       (20481, 2.0), (32768, 2.0), (32769, 2.0), (2049, 4.0), (4097, 4.0), (9001, 4.0),
                                       (9001, 3.0), (57345, 3.0)])
def test_rows_of_any_number_of_lanes_are_the_restatements(gpu_lib, oracle_lib, solver, n, support):
    settings = FluidSettings(solver=solver, spacing=0.02, support=support)
    g, o = gpu_lib.FluidWorld(settings), oracle_lib.OracleWorld(settings, residual_sum=1)
    fill((g, o), n, 0.02, min(n // 8, 250))
    for _ in range(2 if solver == FluidSolver.WCSPH else 1):  # (the crowd bursts in DFSPH's second)
        a, b = g.step(3e-4), o.step(3e-4)
        assert (a.substeps, a.iterations, a.held_back) == (b.substeps, b.iterations, b.held_back)
    assert_same(g, o)


@pytest.mark.parametrize("n", [700, 5001, 12001, 28001, 40001])
def test_rows_with_a_body_are_the_restatements(gpu_lib, oracle_lib, n):
    settings = FluidSettings(spacing=0.02, arithmetic=Arithmetic.EXACT)
    g, o = gpu_lib.FluidWorld(settings), oracle_lib.OracleWorld(settings)
    fill((g, o), n, 0.02, 0)
    mid = 0.5 * float(np.cbrt(n)) * 0.02
    for w in (g, o):
        w.couple(body_handle(1), Shape.CUBOID, (0.05, 0.03, 0.04))
    pose = BodyPose(body_handle(1), (mid, mid, mid), linear_velocity=(0.3, -0.5, 0.1))
    (a, pa), (b, pb) = g.step_with_bodies(1e-3, [pose]), o.step_with_bodies(1e-3, [pose])
    assert (a.substeps, a.held_back, a.sound_speed) == (b.substeps, b.held_back, b.sound_speed)
    assert pa == pb
    assert_same(g, o)

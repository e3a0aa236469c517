"""The passes of scenes that fill the GPU a thread a row, bit for bit against the restatement.

DFSPH around 444 blocks of 256 rows (three a SM of 148), up to which the check and the push run as the
builds for few blocks a SM; WCSPH, with and without a body, and FAST arithmetic past what runs at once.
"""
import numpy as np
import pytest

from solunar_b200.abi import Arithmetic, BodyPose, FluidSettings, FluidSolver, Positions, Shape, body_handle

pytestmark = pytest.mark.gpu

SPACING = 0.02


def fill(worlds, n, crowd=0):
    rng = np.random.default_rng(n)
    side = np.cbrt(n) * SPACING
    pts = rng.uniform(0.02, 0.98, (n, 3)) * side
    pts[:crowd] = 0.5 * side + (pts[:crowd] - 0.5 * side) * 0.1
    vel = rng.standard_normal((n, 3)) * 0.2
    for w in worlds:
        w.add_box_container((0.0, 0.0, 0.0), (side, side + SPACING, side))
        w.add_particles(pts.astype(np.float32), vel.astype(np.float32))
    return side


def assert_same(g, o):
    assert np.array_equal(g.ids(), o.ids())
    for name in ("densities", "positions", "velocities"):
        a, b = (np.ascontiguousarray(np.asarray(getattr(w, name)(), dtype=np.float32)).view(np.uint32) for w in (g, o))
        assert np.array_equal(a, b), name


@pytest.mark.parametrize("n", [444 * 256, 444 * 256 + 1])
def test_dfsph_rows_at_the_edge_of_few_blocks(gpu_lib, oracle_lib, n):
    settings = FluidSettings(solver=FluidSolver.DFSPH, spacing=SPACING)
    g, o = gpu_lib.FluidWorld(settings), oracle_lib.OracleWorld(settings, residual_sum=1)
    fill((g, o), n)
    a, b = g.step(3e-4), o.step(3e-4)
    assert (a.substeps, a.iterations, a.held_back) == (b.substeps, b.iterations, b.held_back)
    assert_same(g, o)


# where the DFSPH density pass stops giving a row several lanes
@pytest.mark.parametrize("n,support", [(28672, 2.0), (28673, 2.0), (57344, 3.0), (57345, 3.0)])
def test_dfsph_rows_at_the_edge_of_several_lanes(gpu_lib, oracle_lib, n, support):
    settings = FluidSettings(solver=FluidSolver.DFSPH, spacing=SPACING, support=support)
    g, o = gpu_lib.FluidWorld(settings), oracle_lib.OracleWorld(settings, residual_sum=1)
    fill((g, o), n)
    a, b = g.step(3e-4), o.step(3e-4)
    assert (a.substeps, a.iterations, a.held_back) == (b.substeps, b.iterations, b.held_back)
    assert_same(g, o)


# 296 and 444 blocks of 256 rows: up to two a SM the density pass runs wide, past three the WCSPH force
# strides over its rows
@pytest.mark.parametrize("n", [296 * 256, 296 * 256 + 1, 120_001])
def test_wcsph_rows_are_the_restatements(gpu_lib, oracle_lib, n):
    settings = FluidSettings(spacing=SPACING)
    g, o = gpu_lib.FluidWorld(settings), oracle_lib.OracleWorld(settings)
    fill((g, o), n, 250)
    for _ in range(2):
        a, b = g.step(3e-4), o.step(3e-4)
        assert (a.substeps, a.held_back) == (b.substeps, b.held_back)
    assert_same(g, o)


def test_wcsph_rows_with_a_body_are_the_restatements(gpu_lib, oracle_lib):
    settings = FluidSettings(spacing=SPACING)
    g, o = gpu_lib.FluidWorld(settings), oracle_lib.OracleWorld(settings)
    side = fill((g, o), 120_001)
    for w in (g, o):
        w.couple(body_handle(1), Shape.CUBOID, (0.05, 0.03, 0.04))
    pose = BodyPose(body_handle(1), (0.5 * side,) * 3, linear_velocity=(0.3, -0.5, 0.1))
    (a, pa), (b, pb) = g.step_with_bodies(1e-3, [pose]), o.step_with_bodies(1e-3, [pose])
    assert (a.substeps, a.held_back, a.sound_speed) == (b.substeps, b.held_back, b.sound_speed)
    assert pa == pb
    assert_same(g, o)


@pytest.mark.parametrize("positions", [Positions.ABSOLUTE, Positions.CELL_RELATIVE])
@pytest.mark.parametrize("solver", [FluidSolver.WCSPH, FluidSolver.DFSPH])
def test_fast_rows_find_the_restatements_neighbours(gpu_lib, oracle_lib, solver, positions):
    # a pair found or lost changes a density by far more than the rounding of the up to 64 terms both
    # sums hold: 64 x 2^-24 each, twice that apart
    settings = FluidSettings(solver=solver, spacing=SPACING, arithmetic=Arithmetic.FAST, positions=positions)
    g, o = gpu_lib.FluidWorld(settings), oracle_lib.OracleWorld(settings)
    fill((g, o), 152_001)
    for w in (g, o):
        w.update_neighbors()
        w.compute_densities()
    assert np.array_equal(g.ids(), o.ids())
    np.testing.assert_allclose(g.densities(), o.densities(), rtol=2 * 64 * 2.0 ** -24)

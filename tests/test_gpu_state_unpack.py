"""A whole state written and read in one pass (k_unpack_state, k_pack_state): the bytes come back, a
non-finite component anywhere is refused, and the box and speed it leaves are what the next step needs."""
import numpy as np
import pytest

from solunar_b200.abi import FluidSettings, PhysicsError

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 255, 256, 257, 5000])
def test_states_round_trip_and_step_alike(gpu_lib, oracle_lib, n):
    rng = np.random.default_rng(n)
    g = gpu_lib.FluidWorld(FluidSettings(spacing=0.02))
    o = oracle_lib.OracleWorld(FluidSettings(spacing=0.02))
    pts = rng.uniform(-0.3, 0.3, (n, 3)).astype(np.float32)
    vel = (rng.standard_normal((n, 3)) * 3.0).astype(np.float32)
    g.add_particles(np.zeros((n, 3), np.float32) + np.arange(n, dtype=np.float32)[:, None] * 0.02,
                    np.zeros((n, 3), np.float32))
    g.write_state(pts, vel)
    assert np.array_equal(g.positions().view(np.uint32), pts.view(np.uint32))
    assert np.array_equal(g.velocities().view(np.uint32), vel.view(np.uint32))
    p, v = np.empty_like(pts), np.empty_like(vel)
    g.read_state_ptr(p.ctypes.data, v.ctypes.data, n)
    assert np.array_equal(p.view(np.uint32), pts.view(np.uint32))
    assert np.array_equal(v.view(np.uint32), vel.view(np.uint32))
    for where, bad in ((0, np.nan), (n - 1, np.inf)):
        for which in (0, 1):
            state = [pts.copy(), vel.copy()]
            state[which][where, 2] = bad
            with pytest.raises(PhysicsError):
                g.write_state(*state)
    o.add_particles(pts, vel)
    a, b = g.step(1e-3), o.step(1e-3)
    assert (a.substeps, a.held_back, np.float32(a.max_speed)) == (b.substeps, b.held_back, np.float32(b.max_speed))
    assert np.array_equal(g.ids(), o.ids())
    assert np.array_equal(g.positions().view(np.uint32), np.asarray(o.positions(), np.float32).view(np.uint32))

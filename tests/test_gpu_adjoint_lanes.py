"""The WCSPH adjoint at the particle counts where the lanes a row takes change, and with a thread a
row, against the exact derivative of the FP32 program (the float restatement in derivative numbers):
<d, J d> = <J^T d, d> for velocity directions d.  The tolerances are the adjoint's own FP32 rounding,
as for the small scenes: 1e-5 on the directions and 1e-4 on the viscosity.
"""
import numpy as np
import pytest

from solunar_b200 import scenes
from solunar_b200.abi import FluidSettings

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("counts,support", [((3, 5, 2), 2.0), ((20, 20, 20), 2.0), ((21, 20, 20), 2.0),
                                            ((29, 29, 30), 2.0), ((16, 16, 16), 4.0), ((17, 16, 16), 4.0),
                                            ((28, 28, 27), 4.0), ((65, 64, 64), 2.0)])
def test_gradients_match_the_fp32_programs_tangent(gpu_lib, oracle_lib, counts, support):
    spacing, dt, steps = 0.02, 2e-4, 2
    tank = tuple(float(np.float32((c + 1) * spacing)) for c in counts)
    settings = FluidSettings(spacing=spacing, support=support, viscosity=0.05)
    pos = scenes.lattice_block((0.0, 0.0, 0.0), counts, spacing)
    n = len(pos)
    rng = np.random.default_rng(n)
    pos = (pos + rng.uniform(-0.1, 0.1, pos.shape) * spacing).astype(np.float32)
    vel = rng.normal(0.0, 0.2, pos.shape).astype(np.float32)
    d = rng.normal(size=pos.shape).astype(np.float32)
    w = gpu_lib.FluidWorld(settings)
    w.add_box_container((0.0, 0.0, 0.0), tank)
    w.add_particles(pos, vel)
    w.tape_begin(0)
    for _ in range(steps):
        w.step(dt)
    dvel = d[w.ids()]
    dp, dv, params = w.step_backward(np.zeros_like(dvel), dvel)
    w.tape_end()
    zero = np.zeros(pos.shape)
    run = lambda dq, q: oracle_lib.tangent_run(settings, ((0.0, 0.0, 0.0), tank), pos, vel, zero, dq, dparams=q,  # noqa: E731
                                               steps=steps, dt=dt, precision=32)[3]
    want = float(np.sum(d.astype(np.float64) * run(d.astype(np.float64), np.zeros(5))))
    assert abs(float(np.sum(dv.astype(np.float64) * d)) - want) <= 1e-5 * abs(want)
    # viscosity, against the size of the terms it is summed from (their signs are random)
    nu = run(zero, np.array([1.0, 0.0, 0.0, 0.0, 0.0]))
    terms = d.astype(np.float64) * nu
    assert abs(params["viscosity"] - terms.sum()) <= 1e-4 * np.abs(terms).sum() / np.sqrt(terms.size)

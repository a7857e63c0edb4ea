"""The FP32 form's displacement: sum of the corners' N p/m in corner order, then times dt, per particle.

Every particle is driven at a constant velocity v, so every node's p/m is v and each step moves a particle by dt times
the corner sum.  v and dt are floats whose product lies 0.93 to 0.97 x 2^-24 off its float.  Multiplied once per
node, that is the error of every step (0.95 in those units of the displacement); multiplied after the sum, whose
last bit changes from particle to particle and from step to step, it averages to 0.5 (restated in float32 on the CPU:
0.48 to 0.52 in corner order).  The line is half-way, at 0.75.
"""
import numpy as np
import pytest

from code_mpm_gb300 import engine, scenes

pytestmark = pytest.mark.gpu

H = 1.0e-3
DT = 1.19402070453134e-08
V = np.array([1.2493528127670288, -1.2494596242904663, 1.2489298582077026])


@pytest.fixture(scope="module", autouse=True)
def _lib():
    from code_mpm_gb300 import build

    build.build()
    engine.lib()


@pytest.mark.parametrize("mode", [0, 2])
def test_rounding_of_the_displacement_is_not_taken_per_node(mode):
    rng = np.random.Generator(np.random.PCG64(4))
    cells = np.array([20, 20, 20], dtype=np.int32)
    pos = rng.uniform(2.0, 17.0, (20_000, 3)) * H
    n, steps = len(pos), 256
    st = scenes._alloc(cells * H, cells, n, DT, 1, 2, n)
    scenes._material(st, 0, scenes.ELASTIC, 2700.0, 70.0e9, 0.3)
    scenes._finish_particles(st, pos, (0.5 * H) ** 3, np.zeros(n, dtype=np.int32))
    st["vel"][:] = V
    st["pflags"][:] = scenes.PF_DC_X | scenes.PF_DC_Y | scenes.PF_DC_Z
    st["dc_list"][:] = np.arange(n)
    st["tl_time"][:] = [0.0, 1.0]
    st["tl_vel"][:] = V
    with engine.Engine.from_state(st, engine.FORM_FP32) as e:
        e.set_option(engine.OPT_GATHER, mode)
        e.advance(steps, DT, False)
        out = e.download_state(st)
    moved = steps * DT * V
    err = (out["pos"] - st["pos"] - moved) / (np.abs(moved) * 2.0 ** -24)
    assert np.all(np.abs(err.mean(axis=0)) <= 0.75), err.mean(axis=0)

"""A tuning's block size means in the engine it is handed to what ran when it was timed: 128 in the FP64 form is at
most 128, as in an engine that nobody tuned.

64 particles in one cell: blocks of 32, which so few particles take, add two partial sums to a node, one block of 128 a
single sum of 64, and the two round differently.  Two terms add to the same bits in either order.
"""
import numpy as np
import pytest

from code_mpm_gb300 import engine, scenes

pytestmark = pytest.mark.gpu

H = 1.0e-3


@pytest.fixture(scope="module", autouse=True)
def _lib():
    from code_mpm_gb300 import build

    build.build()
    engine.lib()


def test_reported_blocks_set_what_ran():
    rng = np.random.Generator(np.random.PCG64(8))
    cells = np.array([3, 3, 3], dtype=np.int32)
    pos = (1.0 + rng.uniform(0.1, 0.9, (64, 3))) * H
    st = scenes._alloc(cells * H, cells, 64, 1.0e-8, 1, 0, 0)
    scenes._material(st, 0, scenes.ELASTIC, 2700.0, 70.0e9, 0.3)
    scenes._finish_particles(st, pos, (0.2 * H) ** 3, np.zeros(64, dtype=np.int32))
    st["mass"][:] *= rng.uniform(0.5, 1.5, 64)
    st["vel"][:] = rng.normal(0.0, 1.0, (64, 3))
    out = []
    for block in (None, 128):
        with engine.Engine.from_state(st, engine.FORM_FP64) as e:
            for key in (engine.OPT_P2G_BLOCK, engine.OPT_PASS1_BLOCK, engine.OPT_PASS_BLOCK):
                if block:
                    e.set_option(key, block)
            e.advance(1, 1.0e-8, False)
            out.append(e.download_state(st))
    for k in ("g_mass", "g_mom", "vel"):
        assert np.array_equal(out[0][k], out[1][k]), k

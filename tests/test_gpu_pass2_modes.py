"""The pass-2 mode and block that the FP32 form takes by itself, on either side of the line between them (512 threads
per SM: 77,824 particles on 152 SMs), against the same kernel asked for by the options.

One particle in every third cell per axis: no two share a node, every node's sum has one term, and the runs are equal
to the bit.
"""
import numpy as np
import pytest
import torch

from code_mpm_gb300 import engine, scenes

pytestmark = pytest.mark.gpu

SMS = torch.cuda.get_device_properties(0).multi_processor_count if torch.cuda.is_available() else 152
H = 1.0e-3


@pytest.fixture(scope="module", autouse=True)
def _lib():
    from code_mpm_gb300 import build

    build.build()
    engine.lib()


def _scene(n):
    side = int(np.ceil(n ** (1.0 / 3.0)))
    cells = np.array([3 * side] * 3, dtype=np.int32)
    rng = np.random.Generator(np.random.PCG64(n))
    at = np.stack(np.unravel_index(np.arange(n), (side,) * 3), axis=1)
    pos = (3 * at + rng.uniform(0.1, 0.9, at.shape)) * H
    st = scenes._alloc(cells * H, cells, n, 1.0e-8, 1, 0, 0)
    scenes._material(st, 0, scenes.ELASTIC, 2700.0, 70.0e9, 0.3)
    scenes._finish_particles(st, pos, (0.5 * H) ** 3, np.zeros(n, dtype=np.int32))
    st["vel"][:] = rng.normal(0.0, 10.0, (n, 3))
    st["stress"][:] = rng.normal(0.0, 1.0e6, (n, 6))
    return st


def _run(st, mode, block):
    with engine.Engine.from_state(st, engine.FORM_FP32) as e:
        if mode is not None:
            e.set_option(engine.OPT_GATHER, mode)
            e.set_option(engine.OPT_PASS_BLOCK, block)
        e.advance(4, 1.0e-8, False)
        return e.download_state(st)


@pytest.mark.parametrize("n,mode,block", [(1, 2, 128), (129, 2, 128), (512 * SMS - 1, 2, 128), (512 * SMS, 0, 256),
                                          (512 * SMS + 1, 0, 256)])
def test_the_mode_taken_is_the_mode_asked_for(n, mode, block):
    st = _scene(n)
    own, asked = _run(st, None, 0), _run(st, mode, block)
    for k in ("pos", "vel", "stress", "strain", "F", "vol", "e_strain", "g_mass", "g_state"):
        assert np.array_equal(own[k], asked[k]), k
    assert not np.array_equal(own["stress"], st["stress"])

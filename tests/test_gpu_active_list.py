"""The active-node list at grid sizes that end within, at and past its tiles, on either side of the size at which a
thread takes 16 nodes instead of 4 (one block per SM: 622,592 nodes on 152 SMs).

Scattered particles in rigid motion: a node that the list missed (or a mark left over) shows in the active set, in the
node masses, and in the particles' velocity, which every step leaves as it is.  The sums are of at most a few tens of
FP64 terms (1e-13 relative); FP32 sums and cell-local coordinates give 1e-5.
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


def _scene(cells):
    cells = np.array(cells, dtype=np.int32)
    rng = np.random.Generator(np.random.PCG64(int(cells.sum())))
    at = rng.integers(0, cells, (400, 3))
    at[0], at[1] = 0, cells - 1  # the first and the last node are in the list
    pos = (at + rng.uniform(0.1, 0.9, at.shape)) * H
    st = scenes._alloc(cells * H, cells, len(pos), 1.0e-8, 1, 0, 0)
    scenes._material(st, 0, scenes.ELASTIC, 2700.0, 70.0e9, 0.3)
    scenes._finish_particles(st, pos, (0.5 * H) ** 3, np.zeros(len(pos), dtype=np.int32))
    st["vel"][:] = (3.0, -2.0, 1.0)
    return st


@pytest.mark.parametrize("form,tol", [(engine.FORM_FP64, 1e-13), (engine.FORM_FP32, 1e-5)])
@pytest.mark.parametrize("cells", [(2, 2, 2), (15, 15, 3), (14, 16, 16), (30, 7, 10), (75, 90, 89), (76, 90, 89)])
def test_every_occupied_node_is_in_the_list(cells, form, tol):
    st = _scene(cells)
    nx, ny, nz = (int(c) + 1 for c in cells)
    mass = np.zeros(nx * ny * nz)
    u = st["pos"] / H
    b = np.floor(u).astype(int)
    for k in range(8):
        o = np.array([k >> 2 & 1, k >> 1 & 1, k & 1])
        w = np.prod(1.0 - np.abs(u - b - o), axis=1)
        np.add.at(mass, (b[:, 0] + o[0]) + nx * ((b[:, 1] + o[1]) + ny * (b[:, 2] + o[2])), w * st["mass"])
    with engine.Engine.from_state(st, form) as e:
        e.advance(5, 1.0e-8, False)  # 5e-8 s: 1.5e-4 of a cell
        out = e.download_state(st)
    assert np.array_equal(out["g_state"] & 1, (mass > 0).astype(out["g_state"].dtype))
    assert np.abs(out["g_mass"] - mass).max() <= 1e-3 * mass.max()  # the particles have moved
    assert abs(out["g_mass"].sum() - st["mass"].sum()) <= max(tol, 1e-12) * st["mass"].sum()
    assert np.abs(out["vel"] - st["vel"]).max() <= 10 * tol * 3.0

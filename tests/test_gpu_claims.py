"""Displacement control's node claims: the last list entry of an axis wins, whatever the list's length and order.

A lane whose neighbour along the list claims the same cell's nodes and axes leaves the claim to it, so the lists here
end within, at and just past a warp, put many entries in one cell, alternate axes between neighbours and give every
entry its own velocity.  Against the CPU restatement, with the parity contract's 1e-9.
"""
import numpy as np
import pytest

import pyoracle
from code_mpm_gb300 import engine, scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib():
    from code_mpm_gb300 import build

    build.build()
    engine.lib()


@pytest.mark.parametrize("contact", [0, 1])
@pytest.mark.parametrize("order", ["cells", "shuffled"])
@pytest.mark.parametrize("size", [1, 31, 32, 33, 65])
def test_last_claim_wins(size, order, contact):
    st = scenes.contact_small(seed=6) if contact else scenes.mixed_small(seed=6)
    rng = np.random.Generator(np.random.PCG64(size))
    cell = np.floor(st["pos"] / (st.length / st.cells)).astype(int)
    by_cell = np.lexsort(cell.T)
    dc = by_cell[:size].copy()
    if order == "shuffled":
        rng.shuffle(dc)
    st["pflags"][st["dc_list"]] = 0
    st["pflags"][dc] = rng.choice([2, 4, 6, 6, 6, 7], size).astype(st["pflags"].dtype)  # x, y and z bits 1, 2, 4
    st["dc_mult"][dc] = rng.uniform(-1.0, 1.0, size)
    st["dc_list"] = dc.astype(np.uint32)
    ref = st.copy()
    pyoracle.advance(ref, 2, contact)
    with engine.Engine.from_state(st, engine.FORM_FP64) as e:
        e.advance(2, st.dt_max, contact)
        gpu = e.download_state(st)
    for k in ("pos", "vel", "g_vel", "g_mom"):
        scale = np.abs(ref[k]).max()
        assert np.abs(gpu[k] - ref[k]).max() <= 1e-9 * scale, k
    assert np.array_equal(gpu["g_state"], ref["g_state"])

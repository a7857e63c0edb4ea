"""P2G's cell runs sum per-axis moments of the stress (modes 2 to 4); mode 0 adds each particle's corners one by one.

Both add the same contributions, so after one step the node sums agree to the rounding of a node's sum: up to 64
particles in FP32 (64 x 2^-24 = 4e-6 of the largest entry, 1e-5 here) and 64 x 2^-53 in FP64 (1e-13).  The scenes carry
the cases the moments treat apart: external forces (none: the forces are not read), and, in FP32, particles whose
cell-local coordinate lies below 3e-8 of a cell, of which rounding leaves one gradient factor per axis.
"""
import numpy as np
import pytest

from code_mpm_gb300 import engine, scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _lib():
    from code_mpm_gb300 import build

    build.build()
    engine.lib()


def _scene(contact, planes, forces):
    st = scenes.contact_small(seed=4) if contact else scenes.mixed_small(seed=4)
    rng = np.random.Generator(np.random.PCG64(9))
    n = st.n_particles
    h = st.length / st.cells
    body = np.nonzero((st["pflags"] & 15) == 0)[0]
    st["stress"][body] = rng.normal(0.0, 30.0e6, (body.size, 6))
    if planes:  # one axis in turn: just above a node plane, exactly on one, and just below
        for j, i in enumerate(body[: 3 * (body.size // 4)]):
            a = j % 3
            k = np.rint(st["pos"][i, a] / h[a])
            st["pos"][i, a] = k * h[a] * (1.0 + (0.0, 1e-9, -1e-13)[(j // 3) % 3])
    st["fext"][:] = rng.normal(0.0, 1.0, (n, 3)) if forces else 0.0
    return st


@pytest.mark.parametrize("form,tol", [(engine.FORM_FP64, 1e-13), (engine.FORM_FP32, 1e-5)])
@pytest.mark.parametrize("contact", [0, 1])
@pytest.mark.parametrize("planes,forces", [(0, 0), (1, 0), (1, 1)])
def test_moments_sum_what_the_corners_sum(form, tol, contact, planes, forces):
    st = _scene(contact, planes, forces)
    outs = {}
    for mode, block in ((0, 128), (3, 128), (3, 512), (3, 0)):
        with engine.Engine.from_state(st, form) as e:
            e.set_option(engine.OPT_P2G_REDUCE, mode)
            if block:
                e.set_option(engine.OPT_P2G_BLOCK, block)
                e.set_option(engine.OPT_PASS1_BLOCK, block)
            e.advance(1, st.dt_max, bool(contact))
            outs[mode, block] = e.download_state(st)
    a = outs.pop((0, 128))
    for cfg, b in outs.items():
        for k in ("g_mass", "g_mom", "g_force", "g_mass_gradient"):
            scale = np.abs(a[k]).max()
            assert np.abs(a[k] - b[k]).max() <= tol * scale, (cfg, k)
        assert np.array_equal(a["g_state"] & 1, b["g_state"] & 1), cfg

"""The FP32 form's fallback return map with yield stresses next to nothing and stresses far past the surface: what the
map in pairs of floats does not cover is computed in FP64.  Finite, and near the FP64 form after a few steps: the
stresses are of the size of the trial states (the radius is nothing beside them), so FP32's rounding of a step's strain
increment (6e-8 of v dt / h, here up to 1e-3 of the increment) bounds the difference; 1e-2 of the largest value.
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


@pytest.mark.parametrize("gather", [0, 2])
@pytest.mark.parametrize("yield_", [0.0, 1e-30, 1e-12, 1.0])
def test_tiny_yield_stresses(yield_, gather):
    st = scenes.mixed_small(seed=5)
    rng = np.random.Generator(np.random.PCG64(2))
    hardening = st["materials"]["type"] == scenes.VONMISESHARDENING
    assert hardening.any()
    st["materials"]["yield_"][hardening] = yield_
    st["stress"][:] = rng.normal(0.0, 1.0e7, st["stress"].shape)
    out = {}
    for form in (engine.FORM_FP32, engine.FORM_FP64):
        with engine.Engine.from_state(st, form) as e:
            if form == engine.FORM_FP32:
                e.set_option(engine.OPT_GATHER, gather)
            e.advance(4, st.dt_max, False)
            out[form] = e.download_state(st)
    a, b = out[engine.FORM_FP32], out[engine.FORM_FP64]
    for k in ("stress", "eps_p", "backstress", "vel", "pos"):
        assert np.isfinite(a[k]).all(), k
        assert np.abs(a[k] - b[k]).max() <= 1e-2 * np.abs(b[k]).max(), k

"""Particles uploaded again into a context that keeps its displacement-control list and monitor mask.

After enough steps either form stores its particles in cell order and has turned both lists into slot numbers; an
upload is in the caller's numbering, and so are the lists again.  The same number of particles, fewer (their entries of
the list are left out) and more (past the mask's end: in no monitor), against a context that was given those lists
afresh.  The two differ by the order of the node sums: 1e-9 of a field's largest value in FP64, 1e-4 in FP32, as for
runs in another storage order.
"""
import numpy as np
import pytest

from code_mpm_gb300 import engine, scenes
from code_mpm_gb300.snapshot import PARTICLE_FIELDS

pytestmark = pytest.mark.gpu

KEYS = ("pos", "vel", "stress", "strain", "F", "e_strain")


@pytest.fixture(scope="module", autouse=True)
def _lib():
    from code_mpm_gb300 import build

    build.build()
    engine.lib()


def _scene(contact):
    """A scene whose controlled particles stand anywhere in the list of particles."""
    st = scenes.platen_block(size=(6e-3, 6e-3, 4e-3), h=1e-3, speed=20.0) if contact else scenes.mixed_small(seed=3)
    rng = np.random.Generator(np.random.PCG64(1))
    order = rng.permutation(st.n_particles)
    place = np.empty_like(order)
    place[order] = np.arange(order.size)
    for k in PARTICLE_FIELDS:
        st[k] = st[k][order]
    st["dc_list"] = place[st["dc_list"]].astype(np.uint32)
    mask = rng.integers(0, 32, st.n_particles).astype(np.uint8)
    return st, mask


def _first(st, n):
    out = st.copy()
    for k in PARTICLE_FIELDS:
        out[k] = st[k][:n]
    out["dc_list"] = st["dc_list"][st["dc_list"] < n]
    return out


@pytest.mark.parametrize("form,tol", [(engine.FORM_FP64, 1e-9), (engine.FORM_FP32, 1e-4)])
@pytest.mark.parametrize("contact", [0, 1])
@pytest.mark.parametrize("change", ["same", "fewer", "more"])
def test_lists_keep_the_callers_numbering(change, contact, form, tol):
    st, mask = _scene(contact)
    part = _first(st, 2 * st.n_particles // 3)
    before, after = {"same": (st, st), "fewer": (st, part), "more": (part, st)}[change]
    kept = np.zeros(after.n_particles, dtype=np.uint8)
    m = min(before.n_particles, after.n_particles)
    kept[:m] = mask[:m]
    want = after.copy()
    want["dc_list"] = want["dc_list"][want["dc_list"] < before.n_particles]
    got = []
    with engine.Engine.from_state(before, form) as e:
        e.upload_monitor_mask(mask[:before.n_particles])
        e.advance(10, st.dt_max, bool(contact))
        e.upload_particles({k: np.ascontiguousarray(after[k]) for k in PARTICLE_FIELDS}, after.n_particles)
        e.n_particles = after.n_particles
        e.set_sim(time=st.time, dt_max=st.dt_max, mass_min=st.mass_min, damping=st.damping)
        e.advance(12, st.dt_max, bool(contact))
        got.append((e.download_state(after), e.monitors()))
    with engine.Engine.from_state(want, form) as e:
        e.upload_monitor_mask(kept)
        e.advance(12, st.dt_max, bool(contact))
        got.append((e.download_state(after), e.monitors()))
    (a, ma), (b, mb) = got
    for k in KEYS:
        assert np.abs(a[k] - b[k]).max() <= tol * np.abs(b[k]).max(), k
    assert ma["count"] == mb["count"]
    for k in ("kinetic", "strain_energy", "stress_p_max"):
        assert abs(ma[k] - mb[k]) <= tol * abs(mb[k]), k
    for k in ("momentum", "position_mean"):
        assert np.abs(np.subtract(ma[k], mb[k])).max() <= tol * np.abs(mb[k]).max(), k

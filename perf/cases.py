"""The workloads whose speed matters to a user of this library, as callable cases.

A case is a dict of plain values.  ``listed()`` gives the standing ones, ``draw(rng)`` one more of the same ranges,
``prepare(case, seed)`` what a program holds before the call, ``run(state)`` one pass through the public entry points,
``work(case)`` the bytes and operations a pass cannot do without, and ``exact(case, seed)`` the same outputs in 64 bits
from plain torch.

Kinds of cases:

* ``steps``: a simulation in mid-run is advanced by some steps and its particle state is read back, as a driver does
  between two snapshots (``Engine.advance``, ``Engine.download_particles``), with the default launch options.  The FP64
  form hands the state over in double; the FP32 form's fields go on to the GPU as float32, what the form carries
  (positions stay double).
* ``infer``: the learned return map over device rows (``Net.infer_device``).
* ``grad``: loss and gradient of a training batch from host rows (``Net.loss_grad``).
* ``order``: the cell order of device positions (``cell_order_noalloc``).

The mid-run states are made from the seed: smooth fields of displacement, velocity, stress and strain over the scene's
particles, of the sizes a crush reaches, with about a quarter of the plastic particles on the yield surface.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from code_mpm_gb300 import engine, scenes
from code_mpm_gb300.snapshot import PF_DC_SKIP

STEEL = dict(E=200.0e9, nu=0.3, yield_=250.0e6, C0=2.0e-3, C1=1.0e12)

# particle fields a step changes and a driver reads back; the two below only on the path that writes them
FIELDS = {"pos": 3, "vel": 3, "vol": 1, "F": 9, "stress": 6, "strain": 6, "eps_p": 6, "e_strain": 1, "e_plastic": 1,
          "backstress": 1}
NONCONTACT_FIELDS = {"e_strain_max": 1, "e_strain_ti": 1}
CONTACT_FP64_FIELDS = {"strain_rate": 6, "mp_mass_gradient": 3}


def listed():
    return [
        # the smallest call: a few thousand particles of three materials with a platen, a frictional wall and a
        # fixed floor, plain form; latency and launches are all there is
        dict(name="mixed_fp64_3k", kind="steps", scene="mixed", fp32=False, contact=False, nx=8, ny=10, nz=6, steps=20),
        # the classic vibrating elastic bar (40,000 particles), both forms
        dict(name="bar_fp32_40k", kind="steps", scene="bar", fp32=True, contact=False, nx=50, ny=10, nz=10, steps=100),
        dict(name="bar_fp64_40k", kind="steps", scene="bar", fp32=False, contact=False, nx=50, ny=10, nz=10, steps=40),
        # three plastic and elastic materials mixed at random, non-contact loop, ragged grid
        dict(name="mixed_fp32_300k", kind="steps", scene="mixed", fp32=True, contact=False, nx=61, ny=47, nz=21,
             steps=60),
        # a solid J2 block crushed by a platen on a frictional floor (contact loop): the chosen form at an ordinary
        # size, the plain form at an odd one
        dict(name="block_fp32_1m", kind="steps", scene="block", fp32=True, contact=True, nx=64, ny=64, nz=32,
             steps=60),
        dict(name="block_fp64_280k", kind="steps", scene="block", fp32=False, contact=True, nx=41, ny=37, nz=23,
             steps=12),
        # a batch of square honeycombs of uneven size, one grid each, advanced together (the headline workload):
        # the chosen form at the largest size here, the plain form on a small batch
        dict(name="cells_fp32_5m", kind="steps", scene="cells", fp32=True, contact=True, nx=32, ny=4, nz=5_000_000,
             steps=60),
        dict(name="cells_fp64_400k", kind="steps", scene="cells", fp32=False, contact=True, nx=5, ny=9, nz=400_000,
             steps=12),
        # a graded foam in a large, mostly empty grid (33 million nodes)
        dict(name="foam_fp32_2m", kind="steps", scene="foam", fp32=True, contact=True, nx=3, ny=400, nz=200, steps=60),
        # the learned return map alone: inference over a large set, and one training batch's loss and gradient
        dict(name="infer_8m", kind="infer", n=8_000_000),
        dict(name="grad_64k", kind="grad", n=65_536),
        # the cell order for callers that cannot allocate
        dict(name="order_700k", kind="order", n=700_001, nx=160, ny=120, nz=90),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    pick = rng.choice(["mixed", "bar", "block", "block", "cells", "cells", "foam", "infer", "grad", "order"])
    if pick == "infer":
        return dict(kind="infer", n=_log(rng, 20_000, 8_000_000))
    if pick == "grad":
        return dict(kind="grad", n=_log(rng, 1_000, 65_000))
    if pick == "order":
        return dict(kind="order", n=_log(rng, 2_000, 1_000_000), nx=rng.randint(20, 200), ny=rng.randint(20, 200),
                    nz=rng.randint(20, 200))
    fp32 = rng.random() < 0.6
    case = dict(kind="steps", scene=pick, fp32=fp32, contact=pick not in ("mixed", "bar"))
    if pick == "mixed":
        case.update(nx=rng.randint(8, 60 if fp32 else 30), ny=rng.randint(9, 48 if fp32 else 30), nz=rng.randint(6, 24),
                    steps=rng.randint(10, 60 if fp32 else 20))
    elif pick == "bar":
        case.update(nx=rng.randint(20, 120), ny=rng.choice([6, 8, 10, 12, 14]), nz=0,
                    steps=rng.randint(20, 120 if fp32 else 40))
        case["nz"] = case["ny"]
    elif pick == "block":
        top = 64 if fp32 else 40
        case.update(nx=rng.randint(9, top), ny=rng.randint(9, top), nz=rng.randint(6, top // 2),
                    steps=rng.randint(15, 60) if fp32 else rng.randint(4, 12))
    elif pick == "cells":
        case.update(nx=rng.randint(2, 16 if fp32 else 5), ny=rng.randint(1, 99),
                    steps=rng.randint(15, 60) if fp32 else rng.randint(4, 12))
        case["nz"] = case["nx"] * _log(rng, 20_000, 200_000 if fp32 else 90_000)
    else:
        case.update(fp32=True, nx=rng.randint(1, 2), ny=rng.randint(100, 260), nz=rng.randint(60, 150),
                    steps=rng.randint(15, 40))
    return case


# ---------------------------------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------------------------------
def _scenes(case, seed):
    """The case's scene as a list of States (one per specimen) in their undeformed configuration."""
    h = 1.0e-3
    if case["scene"] == "mixed":
        sts = [scenes.mixed_small(seed=seed, h=h, ncell=(case["nx"], case["ny"], case["nz"]))]
    elif case["scene"] == "bar":
        sts = [scenes.bar(case["nx"], case["ny"], h, seed=seed, v0=0.5 + (seed % 97) / 97.0)]
    elif case["scene"] == "block":
        sts = [scenes.platen_block(size=(case["nx"] * h, case["ny"] * h, case["nz"] * h), h=h)]
    elif case["scene"] == "cells":
        sts = scenes.honeycomb_batch(case["nx"], seed=case["ny"], total=float(case["nz"]))
    else:
        h = 0.25e-3
        sts = [scenes.graded_foam(ncell=case["nx"], block=(case["ny"] * h, case["ny"] * h, case["nz"] * h), h=h)]
    for st in sts:  # the nodes' boundary conditions only: the other node fields start at zero
        for k in ("g_mass", "g_mom", "g_vel", "g_force", "g_force_temp", "g_mass_gradient", "g_state"):
            st[k] = st[k][:0]
    return sts


def _waves(rng, y, comps, amp):
    """Smooth random fields over the unit-box coordinates y (n x 3): comps columns of amplitude amp."""
    out = torch.zeros((y.shape[0], comps), dtype=torch.float64, device=y.device)
    for c in range(comps):
        for _ in range(2):
            f = torch.tensor(rng.uniform(-1.6, 1.6, 3), device=y.device)
            out[:, c] += torch.sin(2.0 * math.pi * (y @ f) + float(rng.uniform(0.0, 2.0 * math.pi)))
    return out * (0.5 * amp)


def _mid_run(st, rng):
    """Fields of a crush in progress on the scene's own particles (not the platen, not strays outside the body)."""
    dev = "cuda"
    own = ((st["pflags"] & (PF_DC_SKIP | 7)) == 0)
    idx = np.nonzero(own)[0]
    h = float((st.length / st.cells).min())
    x = torch.from_numpy(st["pos"]).to(dev)
    ii = torch.from_numpy(idx).to(dev)
    xb = x[ii]
    lo, hi = xb.min(0).values, xb.max(0).values
    y = (xb - lo) / (hi - lo).max()
    m = st["materials"]
    mat = st["material"][idx]
    col = lambda k: torch.from_numpy(np.ascontiguousarray(m[k][mat].astype(np.float64))).to(dev)  # noqa: E731
    typ, E, nu, Y, C0, C1 = (col(k) for k in ("type", "E", "nu", "yield_", "C0", "C1"))
    k0 = Y / math.sqrt(3.0)
    sig = _waves(rng, y, 6, 1.0)
    p = sig[:, :3].mean(1, keepdim=True)
    d = sig.clone()
    d[:, :3] -= p
    j = torch.sqrt(0.5 * (d[:, :3] ** 2).sum(1) + (d[:, 3:] ** 2).sum(1))
    q = torch.quantile(j[:: max(1, j.numel() // 100_000)], 0.75)
    ratio = j / q  # above 1: has yielded
    scale = torch.where(typ == 0, torch.full_like(k0, 60.0e6), k0)
    eb = torch.where(typ == 0, torch.zeros_like(ratio), 0.01 * torch.clamp(ratio - 1.0, min=0.0))
    R = torch.where(typ == 4, math.sqrt(2.0 / 3.0) * C1 * -torch.expm1(-C0 * eb), torch.zeros_like(eb))
    rad = scale + R / math.sqrt(2.0)
    want = torch.where((ratio > 1.0) & (typ != 0), rad, ratio * scale)
    d *= (want / torch.clamp(j, min=1e-30))[:, None]
    n = d / torch.sqrt((d[:, :3] ** 2).sum(1) + 2.0 * (d[:, 3:] ** 2).sum(1) + 1e-30)[:, None]
    ep = math.sqrt(1.5) * eb[:, None] * n
    sig = d.clone()
    sig[:, :3] += 0.4 * scale[:, None] * p / q
    el = (1.0 + nu)[:, None] * sig / E[:, None]
    el[:, :3] -= (nu / E)[:, None] * sig[:, :3].sum(1, keepdim=True)
    t = el + ep  # tensor strain
    F = torch.zeros((t.shape[0], 9), dtype=torch.float64, device=dev)
    F[:, 0], F[:, 4], F[:, 8] = 1.0 + t[:, 0], 1.0 + t[:, 1], 1.0 + t[:, 2]
    F[:, 1] = F[:, 3] = t[:, 3]
    F[:, 5] = F[:, 7] = t[:, 4]
    F[:, 2] = F[:, 6] = t[:, 5]
    V0 = torch.from_numpy(st["vol0"][idx]).to(dev)
    V = V0 * _det(F)
    eng = torch.tensor([1.0, 1.0, 1.0, 2.0, 2.0, 2.0], dtype=torch.float64, device=dev)
    new = {"pos": xb + _waves(rng, y, 3, 0.4 * h), "vel": _waves(rng, y, 3, 4.0), "stress": sig, "backstress": R,
           "F": F, "vol": V, "strain": t * eng, "eps_p": ep * eng,
           "e_strain": 0.5 * (sig * el * eng).sum(1) * V0 + 0.9 * rad * math.sqrt(3.0) * eb * V0,
           "e_plastic": 0.9 * rad * math.sqrt(3.0) * eb * V0}
    new["e_strain_max"] = new["e_strain"] * 1.01
    new["e_strain_ti"] = new["e_strain"] * (200.0 * st.dt_max)
    for k, v in new.items():
        st[k][idx] = v.cpu().numpy()
    st["fext"][:] = 0.0


def _det(F):
    """Determinants of 3 x 3 matrices given as n x 9 (rows or columns in turn)."""
    a = F.unbind(1)
    return (a[0] * (a[4] * a[8] - a[5] * a[7]) - a[1] * (a[3] * a[8] - a[5] * a[6]) +
            a[2] * (a[3] * a[7] - a[4] * a[6]))


def _states(case, seed):
    rng = np.random.Generator(np.random.PCG64([seed, 77]))
    sts = _scenes(case, seed)
    if case["scene"] != "bar":
        for st in sts:
            _mid_run(st, rng)
    return sts


def _fields(case):
    f = dict(FIELDS)
    if not case["contact"]:
        f.update(NONCONTACT_FIELDS)
    elif not case["fp32"]:
        f.update(CONTACT_FP64_FIELDS)
    return f


def _net_weights(seed, last=1.0):
    rng = np.random.Generator(np.random.PCG64([seed, 5]))
    out = []
    for rows, cols, used_rows, used_cols in ((128, 16, 128, 13), (128, 128, 128, 128), (128, 128, 128, 128),
                                             (8, 128, 7, 128)):
        W = np.zeros((rows, cols))
        W[:used_rows, :used_cols] = rng.uniform(-1.0, 1.0, (used_rows, used_cols)) * math.sqrt(6.0 / used_cols)
        b = np.zeros(rows)
        b[:used_rows] = rng.uniform(-0.1, 0.1, used_rows)
        if rows == 8:
            W, b = W * last, b * last
        out += [W.ravel(), b]
    return np.concatenate(out).astype(np.float32)


def _map_rows(n, seed):
    """Return-map inputs (stress, R, strain increment) as the training distribution has them."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    x = torch.empty((n, 13), dtype=torch.float32, device="cuda")
    x[:, :6] = (torch.rand((n, 6), generator=g, device="cuda") * 3.0 - 1.5) * STEEL["yield_"]
    ep = torch.rand((n,), generator=g, device="cuda") * 0.2
    x[:, 6] = math.sqrt(2.0 / 3.0) * STEEL["C1"] * -torch.expm1(-STEEL["C0"] * ep)
    x[:, 7:] = torch.randn((n, 6), generator=g, device="cuda") * 2.0e-4
    return x


def _batch_rows(n, seed):
    rng = np.random.Generator(np.random.PCG64([seed, 9]))
    x = np.zeros((n, 16), dtype=np.float32)
    x[:, :13] = rng.uniform(-1.5, 1.5, (n, 13))
    t = np.zeros((n, 8), dtype=np.float32)
    t[:, :7] = rng.normal(0.0, 1.0, (n, 7))
    return x, t


def _positions(case, seed):
    """Structure-of-arrays positions in and a little around a grid of 1 mm cells, in clumps as a scene's are."""
    n = case["n"]
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    ext = torch.tensor([case["nx"], case["ny"], case["nz"]], dtype=torch.float64, device="cuda") * 1.0e-3
    run = 64
    at = torch.rand(((n + run - 1) // run, 3), generator=g, dtype=torch.float64, device="cuda") * ext * 1.02 - 0.01 * ext
    x = at.repeat_interleave(run, 0)[:n] + torch.rand((n, 3), generator=g, dtype=torch.float64, device="cuda") * 2.0e-3
    return x.t().contiguous()


def prepare(case, seed):
    if case["kind"] == "infer":
        net = engine.Net(n_samples=1000, **STEEL)
        net.set_params(_net_weights(seed, 3.0e7))  # outputs of the size of a plastic correction (Pa)
        x = _map_rows(case["n"], seed)
        return dict(case=case, net=net, x=x, out=torch.empty((case["n"], 7), dtype=torch.float32, device="cuda"))
    if case["kind"] == "grad":
        net = engine.Net(n_samples=1000, **STEEL)
        net.set_params(_net_weights(seed))
        x, t = _batch_rows(case["n"], seed)
        return dict(case=case, net=net, x=x, t=t)
    if case["kind"] == "order":
        n = case["n"]
        cells = (case["nx"], case["ny"], case["nz"])
        return dict(case=case, pos=_positions(case, seed), cells=cells, length=tuple(c * 1.0e-3 for c in cells),
                    keys=torch.empty(n, dtype=torch.int32, device="cuda"),
                    order=torch.empty(n, dtype=torch.int32, device="cuda"))
    sts = _states(case, seed)
    form = engine.FORM_FP32 if case["fp32"] else engine.FORM_FP64
    e = engine.Engine.from_batch(sts, form) if case["scene"] == "cells" else engine.Engine.from_state(sts[0], form)
    if case["contact"]:
        e.set_option(engine.OPT_FLOOR_FRICTION, 1)
    n = e.n_particles
    host = {k: torch.empty((n,) if c == 1 else (n, c), dtype=torch.float64, pin_memory=True)
            for k, c in _fields(case).items()}
    return dict(case=case, engine=e, host=host, views={k: v.numpy() for k, v in host.items()}, dt=sts[0].dt_max)


def run(state):
    case = state["case"]
    if case["kind"] == "infer":
        state["net"].infer_device(state["x"].data_ptr(), state["out"].data_ptr(), case["n"], engine.INFER_TC)
        return {"rows": state["out"]}
    if case["kind"] == "grad":
        loss, g = state["net"].loss_grad(state["x"], state["t"])
        return {"loss": loss, "grad": g}
    if case["kind"] == "order":
        rc = engine.cell_order_noalloc(state["length"], state["cells"], state["pos"].data_ptr(), case["n"],
                                       state["keys"].data_ptr(), state["order"].data_ptr())
        if rc != 0:
            raise RuntimeError(f"cell_order_noalloc returned {rc}")
        return {"keys": state["keys"], "order": state["order"]}
    e = state["engine"]
    e.advance(case["steps"], state["dt"], case["contact"])
    e.download_particles(state["views"])
    if not case["fp32"]:
        return state["host"]
    out = {k: v.to("cuda", non_blocking=True) for k, v in state["host"].items()}
    return {k: v if k == "pos" else v.float() for k, v in out.items()}


def work(case):
    if case["kind"] == "infer":
        return {"bytes": case["n"] * 20 * 4, "flops": case["n"] * 2 * (13 * 128 + 2 * 128 * 128 + 128 * 7)}
    if case["kind"] == "grad":
        per = 2 * (13 * 128 + 2 * 128 * 128 + 128 * 7)
        return {"bytes": case["n"] * 24 * 4, "flops": case["n"] * (3 * per - 2 * 13 * 128)}
    if case["kind"] == "order":
        return {"bytes": case["n"] * (24 + 8), "flops": case["n"] * 12}
    n = sum(st.n_particles for st in _scenes(case, 1))
    # per particle and step: the state read and the changed state written once (mass, V0, material, flags read;
    # position, velocity, V, F, stress, strain, plastic strain, back stress, energies read and written), in the
    # form's types; then the fields handed over
    r = 4 if case["fp32"] else 8
    e = 2 if case["contact"] else 4
    both = 24 + 8 * e + r * (3 + 1 + 9 + 6 + 6 + 6 + 1)
    step = 2 * both + 2 * r + 5
    return {"bytes": n * (step * case["steps"] + 8 * sum(_fields(case).values())), "flops": n * 900 * case["steps"]}


# ---------------------------------------------------------------------------------------------------------------------
# 64-bit values from plain torch
# ---------------------------------------------------------------------------------------------------------------------
class _Sim:
    """The classic double-pass step in float64 torch on the GPU, all specimens at once."""

    def __init__(self, sts, case):
        dev = "cuda"
        self.contact = case["contact"]
        cat = lambda k: torch.from_numpy(np.concatenate([st[k] for st in sts])).to(dev)  # noqa: E731
        self.P = {k: cat(k) for k in ("pos", "vel", "fext", "mass", "vol", "vol0", "F", "stress", "strain", "eps_p",
                                      "e_strain", "e_strain_max", "e_strain_ti", "e_plastic", "backstress")}
        n = self.n = self.P["pos"].shape[0]
        self.flags = cat("pflags").to(torch.int64)
        self.mult = cat("dc_mult").double()
        sid = np.concatenate([np.full(st.n_particles, i) for i, st in enumerate(sts)])
        self.sid = torch.from_numpy(sid).to(dev)
        grid = np.array([st.cells for st in sts], dtype=np.int64)
        self.nodes = torch.from_numpy(grid + 1).to(dev)[self.sid]
        self.h = torch.from_numpy(np.array([st.length / st.cells for st in sts])).to(dev)[self.sid]
        off = np.cumsum([0] + [st.n_nodes for st in sts])
        self.off = torch.from_numpy(off[:-1]).to(dev)[self.sid]
        self.nn = int(off[-1])
        self.fixed = cat("fixed").to(torch.int64)
        self.friction = cat("friction")
        mats = np.concatenate([st["materials"] for st in sts])
        moff = np.cumsum([0] + [len(st["materials"]) for st in sts])
        mi = np.concatenate([st["material"] + moff[i] for i, st in enumerate(sts)])
        col = lambda k: torch.from_numpy(np.ascontiguousarray(mats[k][mi].astype(np.float64))).to(dev)  # noqa: E731
        self.M = {k: col(k) for k in ("type", "E", "nu", "yield_", "C0", "C1")}
        poff = np.cumsum([0] + [st.n_particles for st in sts])
        dc = np.concatenate([st["dc_list"].astype(np.int64) + poff[i] for i, st in enumerate(sts)])
        self.dc = torch.from_numpy(dc).to(dev)
        self.tl_t, self.tl_v = sts[0]["tl_time"], sts[0]["tl_vel"]
        self.dt, self.time = sts[0].dt_max, sts[0].time
        self.skip = ((self.flags & 8) != 0) if self.contact else torch.zeros(n, dtype=torch.bool, device=dev)

    def corners(self):
        """Per corner: node index (nn when out of range), weight and gradient columns."""
        q = self.P["pos"] / self.h
        b = torch.floor(q)
        u = q - b
        b = b.to(torch.int64)
        N = [torch.stack([1.0 - u[:, a], u[:, a]]) for a in range(3)]
        inside = (u > 1.0e-12).double()
        G = [torch.stack([-inside[:, a] / self.h[:, a], inside[:, a] / self.h[:, a]]) for a in range(3)]
        for k in range(8):
            o = ((k >> 2) & 1, (k >> 1) & 1, k & 1)
            c = [b[:, a] + o[a] for a in range(3)]
            ok = torch.ones(self.n, dtype=torch.bool, device=q.device)
            for a in range(3):
                ok &= (c[a] >= 0) & (c[a] < self.nodes[:, a])
            i = self.off + c[0] + self.nodes[:, 0] * (c[1] + self.nodes[:, 1] * c[2])
            i = torch.where(ok, i, torch.full_like(i, self.nn))
            n = [N[a][o[a]] for a in range(3)]
            g = torch.stack([G[0][o[0]] * n[1] * n[2], n[0] * G[1][o[1]] * n[2], n[0] * n[1] * G[2][o[2]]], 1)
            yield i, n[0] * n[1] * n[2], g

    def timeline(self):
        out = np.zeros(3)
        for k in range(len(self.tl_t) - 1):
            if self.tl_t[k] <= self.time < self.tl_t[k + 1]:
                s = (self.time - self.tl_t[k]) / (self.tl_t[k + 1] - self.tl_t[k])
                out = (1.0 - s) * self.tl_v[k] + s * self.tl_v[k + 1]
        return out

    def claims(self, cs):
        """Per axis: the nodes taken by displacement control and the particle that has the last word on each."""
        out = []
        rank = torch.arange(1, len(self.dc) + 1, dtype=torch.int64, device=self.sid.device)
        for a in range(3):
            own = torch.zeros(self.nn + 1, dtype=torch.int64, device=rank.device)
            on = torch.ones_like(rank, dtype=torch.bool) if self.contact else (self.flags[self.dc] >> a) & 1 != 0
            for i, _, _ in cs:
                own.scatter_reduce_(0, i[self.dc][on], rank[on], "amax")
            own[self.nn] = 0
            at = own.nonzero()[:, 0]
            out.append((at, self.dc[own[at] - 1]))
        return out

    def step(self):
        P, dt, nn = self.P, self.dt, self.nn
        dev = P["pos"].device
        cs = list(self.corners())
        s, V, m = P["stress"], P["vol"], P["mass"]
        acc = torch.zeros((nn + 1, 7), dtype=torch.float64, device=dev)
        mv = m[:, None] * P["vel"]
        for i, N, G in cs:
            f = torch.stack([G[:, 0] * s[:, 0] + G[:, 1] * s[:, 3] + G[:, 2] * s[:, 5],
                             G[:, 1] * s[:, 1] + G[:, 0] * s[:, 3] + G[:, 2] * s[:, 4],
                             G[:, 2] * s[:, 2] + G[:, 0] * s[:, 5] + G[:, 1] * s[:, 4]], 1)
            f = N[:, None] * P["fext"] - V[:, None] * f
            acc.index_add_(0, i, torch.cat([(N * m)[:, None], N[:, None] * mv, f], 1))
        act = (acc[:nn, 0] > 0).nonzero()[:, 0]
        slot = torch.full((nn + 1,), act.numel(), dtype=torch.int64, device=dev)
        slot[act] = torch.arange(act.numel(), device=dev)
        a = acc[act]
        del acc
        mass, p, f = a[:, 0], a[:, 1:4].clone(), a[:, 4:7].clone()
        v = torch.zeros_like(p)
        fx, mu = self.fixed[act], self.friction[act]
        own = [(slot[at], who) for at, who in self.claims(cs)]

        def control():
            for c, (at, who) in enumerate(own):
                vp = P["vel"][who, c]
                v[at, c] = vp
                p[at, c] = mass[at] * vp
                f[at, c] = 0.0

        def coulomb(t, fn, on):
            trial = p[:, t] + f[:, t] * dt
            ff = -mu * torch.sign(trial) * fn.abs()
            cap = (trial / dt).abs()
            ff = torch.where((ff * dt).abs() > trial.abs(), torch.sign(ff) * cap, ff)
            on = on & ((trial * dt).abs() > 1.0e-24)
            f[:, t] = torch.where(on, f[:, t] + ff, f[:, t])

        fix = [(fx >> c) & 1 != 0 for c in range(3)]
        if not self.contact:
            control()
            coulomb(1, f[:, 0].clone(), fix[0] & (f[:, 0] > 0))
            for c in range(3):
                for z in (v, p, f):
                    z[fix[c], c] = 0.0
            p += f * dt
        else:
            fz = f[:, 2].clone()
            on = fix[2] & (mu > 0) & (fz < 0)
            coulomb(0, fz, on)
            coulomb(1, fz, on)
            p += f * dt
            for c in range(3):
                for z in (v, p, f):
                    z[fix[c], c] = 0.0
            control()
        pad = lambda z: torch.cat([z, torch.zeros((1, 3), dtype=torch.float64, device=dev)])  # noqa: E731
        r = pad(f / mass[:, None])
        cs = [(slot[i], N, G) for i, N, G in cs]
        live = (~self.skip).double()[:, None]
        dv = torch.zeros_like(P["vel"])
        for i, N, G in cs:
            dv += N[:, None] * r[i]
        P["vel"] = P["vel"] + dv * dt * live
        mv = m[:, None] * P["vel"] * live
        qn = torch.zeros((act.numel() + 1, 3), dtype=torch.float64, device=dev)
        for i, N, G in cs:
            qn.index_add_(0, i, N[:, None] * mv)
        v += qn[:-1] / mass[:, None]

        def boundary():
            for c in range(3):
                v[fix[c], c] = 0.0
                p[fix[c], c] = 0.0

        if self.contact:
            boundary()
            control()
        else:
            control()
            boundary()
        r, v = pad(p / mass[:, None]), pad(v)
        L = torch.zeros((self.n, 3, 3), dtype=torch.float64, device=dev)  # [row r, column c] = dv_r/dx_c
        dx = torch.zeros_like(P["pos"])
        for i, N, G in cs:
            dx += N[:, None] * r[i]
            L += v[i][:, :, None] * G[:, None, :]
        self.update(dx * dt * live, L * live[:, :, None])
        tv = self.timeline()
        d = self.dc
        for c in range(3):
            if self.contact:
                vel = self.mult[d] * tv[c]
                P["vel"][d, c] = vel
                P["pos"][d, c] += vel * dt
            else:
                on = d[(self.flags[d] >> c) & 1 != 0]
                P["vel"][on, c] = self.mult[on] * tv[c]
        self.time += dt

    def update(self, dx, L):
        P, M, dt = self.P, self.M, self.dt
        go = ~self.skip
        P["pos"] = P["pos"] + dx
        D = L * dt
        e = torch.stack([D[:, 0, 0], D[:, 1, 1], D[:, 2, 2], D[:, 0, 1] + D[:, 1, 0], D[:, 1, 2] + D[:, 2, 1],
                         D[:, 2, 0] + D[:, 0, 2]], 1)
        self.rate = e / dt
        F = P["F"].view(-1, 3, 3).transpose(1, 2)  # stored column by column
        F = F + (D @ F if self.contact else F @ D)
        V = torch.where(go, _det(F.reshape(-1, 9)) * P["vol0"], P["vol"])
        P["F"] = F.transpose(1, 2).reshape(-1, 9)
        E, nu, R, s = M["E"], M["nu"], P["backstress"], P["stress"]
        G = 0.5 * E / (1.0 + nu)
        lam = E * nu / (1.0 + nu) / (1.0 - 2.0 * nu)
        tr = G[:, None] * e
        tr[:, :3] = 2.0 * tr[:, :3] + lam[:, None] * e[:, :3].sum(1, keepdim=True)
        t = s + tr
        hyd = t[:, :3].mean(1, keepdim=True)
        dev = t.clone()
        dev[:, :3] -= hyd
        J = torch.sqrt(0.5 * (dev[:, :3] ** 2).sum(1) + (dev[:, 3:] ** 2).sum(1))
        rad = M["yield_"] / math.sqrt(3.0) + torch.where(M["type"] == 4, R / math.sqrt(2.0), torch.zeros_like(R))
        plastic = (M["type"] != 0) & (J > rad) & go
        cut = torch.where(plastic, 1.0 - rad / torch.clamp(J, min=1.0e-300), torch.zeros_like(J))
        back = dev * cut[:, None]  # the plastic correction of the stress
        ds = tr - back
        ep = back / G[:, None]
        ep[:, :3] *= 0.5
        eq = torch.sqrt((ep ** 2).sum(1) * (2.0 / 3.0))
        sat = math.sqrt(2.0 / 3.0) * M["C1"] - R
        dR = torch.where(plastic & (M["type"] == 4) & (sat > 0), M["C0"] * sat * eq, torch.zeros_like(R))
        sn = s + ds
        mid = sn if self.contact else sn - 0.5 * ds
        P["stress"], P["strain"], P["eps_p"] = sn, P["strain"] + e, P["eps_p"] + ep
        P["e_strain"] = P["e_strain"] + (mid * e).sum(1) * V
        P["e_plastic"] = P["e_plastic"] + (mid * ep).sum(1) * V
        if not self.contact:
            P["e_strain_ti"] = P["e_strain_ti"] + P["e_strain"] * dt
            P["e_strain_max"] = torch.maximum(P["e_strain_max"], P["e_strain"])
        P["vol"], P["backstress"] = V, R + dR


def exact(case, seed):
    if case["kind"] == "infer":
        w = torch.from_numpy(_net_weights(seed, 3.0e7)).double().cuda()
        x = _map_rows(case["n"], seed)
        G = 0.5 * STEEL["E"] / (1.0 + STEEL["nu"])
        lam = STEEL["E"] * STEEL["nu"] / (1.0 + STEEL["nu"]) / (1.0 - 2.0 * STEEL["nu"])
        shapes, at, p = [(128, 16), (128,), (128, 128), (128,), (128, 128), (128,), (8, 128), (8,)], 0, []
        for s in shapes:
            k = int(np.prod(s))
            p.append(w[at:at + k].view(s))
            at += k
        scale = torch.tensor([1.0 / STEEL["yield_"]] * 7 + [1.0 / 2.0e-4] * 6, dtype=torch.float64, device="cuda")
        out = torch.empty((case["n"], 7), dtype=torch.float64, device="cuda")
        for o in range(0, case["n"], 1 << 20):
            r = x[o:o + (1 << 20)].double()
            hid = r * scale
            hid = torch.relu(hid @ p[0][:, :13].t() + p[1])
            hid = torch.relu(hid @ p[2].t() + p[3])
            hid = torch.relu(hid @ p[4].t() + p[5])
            y = (hid @ p[6].t() + p[7])[:, :7]
            e = r[:, 7:]
            y[:, :6] += G * e
            y[:, :3] += G * e[:, :3] + lam * e[:, :3].sum(1, keepdim=True)
            out[o:o + (1 << 20)] = y
        return {"rows": out}
    if case["kind"] == "grad":
        x, t = (torch.from_numpy(a).double().cuda() for a in _batch_rows(case["n"], seed))
        w = torch.from_numpy(_net_weights(seed)).double().cuda().requires_grad_()
        shapes, at, p = [(128, 16), (128,), (128, 128), (128,), (128, 128), (128,), (8, 128), (8,)], 0, []
        for s in shapes:
            k = int(np.prod(s))
            p.append(w[at:at + k].view(s))
            at += k
        hid = torch.relu(x @ p[0].t() + p[1])
        hid = torch.relu(hid @ p[2].t() + p[3])
        hid = torch.relu(hid @ p[4].t() + p[5])
        y = hid @ p[6].t() + p[7]
        loss = ((y - t)[:, :7] ** 2).sum() / (7.0 * case["n"])
        loss.backward()
        return {"loss": float(loss.detach()), "grad": w.grad.cpu().numpy()}
    if case["kind"] == "order":
        return None
    sts = _states(case, seed)
    sim = _Sim(sts, case)
    if sim.n * case["steps"] > 80_000_000:
        return None  # over about 20 seconds
    for _ in range(case["steps"]):
        sim.step()
    out = {k: (None if k == "mp_mass_gradient" else sim.rate if k == "strain_rate" else sim.P[k])
           for k in _fields(case)}
    if "strain_rate" in out:
        out["strain_rate"] = torch.where(sim.skip[:, None], torch.zeros_like(sim.rate), sim.rate)
    return out

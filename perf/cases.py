"""Cases that the solver's performance is measured on: the work that a program using this
package has it do, through its public entry points.

Kinds:
  step    a water block dropped onto snow, advanced by one call (world.Simulation.step): a
          frame of four substeps replayed from a CUDA graph, or the drop-in call of a host
          that steps once per call and wants the set sizes back
  batch   many scenes stepped as one (batch.BatchSimulation.step)
  adjoint forward rollout and its gradient (adjoint.rollout, backward)
  fluid   the screen-space fluid view of a scene (render.render_fluid)
  points  the point-sprite view with temperature colours (render.render)
  setup   hash, sort, reorder and volume of the boundary, then the initial interlinks
          (world.Simulation.setup)

A stepping pass starts from a saved state, as a parameter study, a checkpointed run or the
adjoint restarts one (adjoint.restore does the same copy): every pass is the same work.
`frames` says how many frames the scene has already run when the state is saved: 0 is the
water in the air above a resting block, about 8 the impact, beyond that the melt.
"""
import math
import random

import numpy as np
import torch

from snowsimulation_b200 import adjoint, batch, render, scene, world
from snowsimulation_b200.abi import QUIRKS_FIXED, QUIRKS_REFERENCE
from snowsimulation_b200.params import make_sim_params

SPACING = 0.02
FRAME = 4   # substeps of a frame (dt = 1/240 s)
# what a substep rewrites, a phase change included
STATE = ("positions", "predict_positions", "new_positions", "velocity", "force", "correction", "mass", "massInv",
         "density", "C", "lambda_", "T", "new_T", "contrib", "predicate", "scan_index", "new_end", "connect_record",
         "connect_length", "iter_end", "new_index", "trackId")
# what a program reads after it
RESULT = ("positions", "predict_positions", "velocity", "density", "C", "lambda_", "T", "contrib", "connect_record",
          "connect_length", "iter_end", "trackId")


def _step(name, water, snow, drop, frames, graph=True, substeps=FRAME, fixed=False, sph_sph=False, dynamic=False,
          large=False):
    c = dict(kind="step", wx=water[0], wy=water[1], wz=water[2], sx=snow[0], sy=snow[1], sz=snow[2], drop=drop,
             frames=frames, graph=graph, substeps=substeps, fixed=fixed, sph_sph=sph_sph, dynamic=dynamic,
             large=large)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest call: 64 water + 144 snow particles, one substep, no graph, sizes read
        # back -- a host's time step in an interactive scene; launches and latency
        _step("tiny substep", (4, 4, 4), (6, 4, 6), 0.06, 2, graph=False, substeps=1),
        # a frame of a small scene around the impact (5,096 particles)
        _step("small frame", (10, 10, 10), (16, 16, 16), 0.1, 8),
        # odd sizes, the corrected physics, water self-contact on, eight substeps a call
        _step("odd fixed", (13, 17, 11), (37, 13, 29), 0.05, 6, substeps=8, fixed=True, sph_sph=True),
        # the README-scale scene (5,888 + 147,928): falling water above a resting block ...
        _step("readme rest", (8, 92, 8), (82, 22, 82), 0.1, 2),
        # ... the melt, water between the snow particles ...
        _step("readme melt", (8, 92, 8), (82, 22, 82), 0.1, 20),
        # ... and the drop-in call of the reference's host loop, one substep each
        _step("readme substep", (8, 92, 8), (82, 22, 82), 0.1, 9, graph=False, substeps=1),
        # 1,048,576 snow + 131,072 water in a wider box, the largest scene
        _step("large frame", (0, 64, 0), (128, 64, 128), 0.3, 10, large=True),
        # 32 independent scenes of 2k-40k particles as one batch (a data-generation run)
        dict(name="batch 32", kind="batch", scenes=32, lo=2000, hi=40000, layout=1, frames=4),
        # gradient of a loss on the final snow state: 1,024 + 8,192 particles, 20 substeps
        dict(name="adjoint", kind="adjoint", wx=8, wy=16, wz=8, sx=32, sy=8, sz=32, drop=0.005, substeps=20,
             every=10),
        # the default view of the README-scale scene at the application's window size
        dict(name="fluid view", kind="fluid", wx=8, wy=92, wz=8, sx=82, sy=22, sz=82, drop=0.1, frames=12,
             width=1600, height=900),
        # the particle view of the same scene, coloured by temperature
        dict(name="point view", kind="points", wx=8, wy=92, wz=8, sx=82, sy=22, sz=82, drop=0.1, frames=12,
             width=1280, height=720),
        # what a program runs once per scene before its first step
        dict(name="setup", kind="setup", wx=8, wy=92, wz=8, sx=82, sy=22, sz=82, drop=0.1),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _block(rng, n, most):
    """Lattice counts of about n particles, each axis at most most[k]."""
    a, b = _log(rng, 0.5, 2.0), _log(rng, 0.35, 1.2)
    e = n ** (1.0 / 3.0) / (b ** (1.0 / 3.0))
    c = [int(round(e * a ** 0.5)), int(round(e * b)), int(round(e / a ** 0.5))]
    return tuple(max(2, min(c[k], most[k])) for k in range(3))


def draw(rng):
    kind = rng.choices(("step", "batch", "adjoint", "fluid", "points", "setup"), (10, 2, 3, 2, 2, 2))[0]
    n = _log(rng, 150, 9000 if kind == "adjoint" else 200000)
    snow = _block(rng, n, (90, 60, 90))
    water = _block(rng, max(8.0, n * _log(rng, 0.02, 0.4)), (60, 90, 60))
    blocks = dict(wx=water[0], wy=water[1], wz=water[2], sx=snow[0], sy=snow[1], sz=snow[2],
                  drop=round(_log(rng, 0.005, 0.3), 4))
    if kind == "step":
        graph = rng.random() < 0.7
        return _step(None, water, snow, blocks["drop"], rng.randint(0, 24), graph=graph,
                     substeps=rng.choice((2, 4, 4, 8)) if graph else 1, fixed=rng.random() < 0.35,
                     sph_sph=rng.random() < 0.2, dynamic=n < 3000 and rng.random() < 0.2)
    if kind == "batch":
        lo = int(_log(rng, 300, 3000))
        return dict(kind="batch", scenes=rng.randint(2, 24), lo=lo, hi=int(lo * _log(rng, 2, 20)),
                    layout=rng.randint(2, 1 << 20), frames=rng.randint(0, 10))
    if kind == "adjoint":
        k = rng.randint(4, 20)
        return dict(kind="adjoint", **{**blocks, "drop": round(_log(rng, 0.002, 0.1), 4)}, substeps=k,
                    every=rng.randint(2, 12))
    if kind == "setup":
        return dict(kind="setup", **blocks)
    w = rng.randint(320, 1920)
    return dict(kind=kind, **blocks, frames=rng.randint(0, 16), width=w, height=int(w * rng.uniform(0.5, 0.8)))


# --------------------------------------------------------------------------- scenes
def _host(case, seed):
    if case.get("large"):
        return scene.config4(seed=seed)
    w = scene.scene_drop((case["wx"], case["wy"], case["wz"]), (case["sx"], case["sy"], case["sz"]), seed=seed,
                         water_jitter=0.002, snow_jitter=0.002, drop_height=case["drop"], init_links=True)
    if case["kind"] == "adjoint":
        w.flags["change_phase"] = False
    w.flags["sph_sph_correction"] = bool(case.get("sph_sph", False))
    w.flags["dynamic_max_connections"] = bool(case.get("dynamic", False))
    return w


def _batch_hosts(case, seed):
    """Scenes as config2 draws them, the sizes of a case fixed by its layout."""
    rng = random.Random(case["layout"])
    p = make_sim_params()
    hosts = []
    for s in range(case["scenes"]):
        n, frac = _log(rng, case["lo"], case["hi"]), rng.uniform(0.02, 0.3)
        kw, ks = max(1, round((n * frac) ** (1 / 3))), max(1, round((n * (1 - frac)) ** (1 / 3)))
        hosts.append(scene.scene_drop((kw, kw, kw), (ks, ks, ks), seed=seed * 1000 + s, water_jitter=0.002,
                                      snow_jitter=0.002, drop_height=rng.uniform(0.02, 0.5),
                                      T_snow=float(np.float32(rng.uniform(-20, -2))), params=p, init_links=True))
    return hosts


class _Saved:
    """A saved state of a Simulation or BatchSimulation, put back with one copy launch per type."""

    def __init__(self, sim):
        self.sim = sim
        self.n = (sim.n_sph, sim.n_dem)
        self.time = sim.scene.current_time
        live = [getattr(sim, s).t[k] for s in ("sph", "dem") for k in STATE]
        live += [t for s in ("scd", "dcd") for t in getattr(sim, s).t.values()]
        if hasattr(sim, "sid"):
            live += [sim.sid["sph"], sim.sid["dem"]]
        self.by_type = []
        for dt in (torch.float32, torch.int32):
            dst = [t for t in live if t.dtype == dt]
            self.by_type.append((dst, [t.clone() for t in dst]))

    def put_back(self):
        self.sim.n_sph, self.sim.n_dem = self.n
        self.sim.scene.current_time = self.time
        for dst, src in self.by_type:
            torch._foreach_copy_(dst, src)


def _simulation(case, seed):
    fixed = case.get("fixed", False) or case["kind"] == "adjoint"
    sim = world.Simulation(_host(case, seed), quirks=QUIRKS_FIXED if fixed else QUIRKS_REFERENCE)
    return sim.setup()


def _advance(sim, frames):
    for _ in range(frames):
        sim.step(substeps=FRAME, use_graph=True)
    return sim


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        sim = _advance(batch.BatchSimulation(_batch_hosts(case, seed)).setup(), case["frames"])
        return dict(case=case, sim=sim, saved=_Saved(sim))
    if kind == "setup":
        return dict(case=case, sim=world.Simulation(_host(case, seed)))
    sim = _simulation(case, seed)
    if kind == "adjoint":
        g = torch.Generator().manual_seed(seed)
        nd = sim.n_dem
        target = sim.dem.t["positions"][:nd] + 0.005 * torch.rand((nd, 3), generator=g).to(sim.device)
        return dict(case=case, sim=sim, saved=_Saved(sim), theta=adjoint.params_of(sim),
                    v0=sim.sph.t["velocity"][:sim.n_sph].clone(), target=target,
                    target_T=sim.dem.t["T"][:nd] + 1.0)
    _advance(sim, case["frames"])
    if kind == "step":
        return dict(case=case, sim=sim, saved=_Saved(sim))
    if kind == "fluid":
        cam = render.reference_camera(case["width"], case["height"])
    else:   # sprites of a particle's diameter (0.02 m) under the default 0.8 rad field of view
        cam = render.camera(width=case["width"], height=case["height"],
                            point_size=0.02 * case["height"] / (2.0 * math.tan(0.4)))
    return dict(case=case, sim=sim, cam=cam)


# --------------------------------------------------------------------------- passes
def _result(sim):
    out = {"water": sim.n_sph, "snow": sim.n_dem}
    for s in ("sph", "dem"):
        t = getattr(sim, s).t
        fields = RESULT if s == "dem" else [k for k in RESULT if k not in ("connect_record", "connect_length",
                                                                           "iter_end")]
        out.update({s + "." + k: t[k] for k in fields})
    out["bnd.density"] = sim.bnd.t["density"]
    out["bnd.lambda_"] = sim.bnd.t["lambda_"]
    return out


def run(state):
    case, sim = state["case"], state["sim"]
    kind = case["kind"]
    if kind == "step":
        state["saved"].put_back()
        sim.step(substeps=case["substeps"], use_graph=case["graph"])
        return _result(sim)
    if kind == "batch":
        state["saved"].put_back()
        sim.step(substeps=FRAME, use_graph=True)
        return _result(sim)
    if kind == "adjoint":
        state["saved"].put_back()
        v = state["v0"].clone().requires_grad_(True)
        th = state["theta"].clone().requires_grad_(True)
        xs, xd, Ts, Td = adjoint.rollout(sim, v, th, case["substeps"], case["every"])
        loss = adjoint.loss_fn(xd, Td, state["target"], state["target_T"], 1e-4)
        loss.backward()
        return {"loss": loss.detach(), "grad_v": v.grad, "grad_theta": th.grad, "x_sph": xs.detach(),
                "x_dem": xd.detach(), "T_sph": Ts.detach(), "T_dem": Td.detach()}
    if kind == "fluid":
        return render.render_fluid(sim, state["cam"])
    if kind == "points":
        return render.render(sim, state["cam"], ((0.2, 0.4, 1.0), (1.0, 0.3, 0.1), -10.0, 100.0))
    # setup: no links yet, as the scene was made
    d = sim.dem.t
    d["connect_record"].fill_(-1)
    d["connect_length"].zero_()
    torch.arange(0, d["iter_end"].numel() * sim.w.maxc, sim.w.maxc, out=d["iter_end"])
    sim.setup()
    return {"volume": sim.bnd.t["volume"], "b_hash": sim.bcd.t["grid_hash"], "b_index": sim.bcd.t["grid_index"],
            "b_start": sim.bcd.t["cell_start"], "d_index": sim.dcd.t["grid_index"][:sim.n_dem],
            "connect_record": d["connect_record"], "connect_length": d["connect_length"], "iter_end": d["iter_end"]}


# --------------------------------------------------------------------------- work
def _counts(case):
    if case.get("large"):
        return 131072, 1048576, 115516
    if case["kind"] == "batch":
        rng = random.Random(case["layout"])
        w = s = 0
        for _ in range(case["scenes"]):
            n, frac = _log(rng, case["lo"], case["hi"]), rng.uniform(0.02, 0.3)
            w += max(1, round((n * frac) ** (1 / 3))) ** 3
            s += max(1, round((n * (1 - frac)) ** (1 / 3))) ** 3
            rng.uniform(0.02, 0.5), rng.uniform(-20, -2)
        return w, s, 52016 * case["scenes"]
    return case["wx"] * case["wy"] * case["wz"], case["sx"] * case["sy"] * case["sz"], 52016


def work(case):
    w, s, b = _counts(case)
    kind = case["kind"]
    # state of a particle: positions, velocity, T, contrib, density, C, lambda, the masses;
    # snow also 25 link slots (record, length) and their count
    pb, lb = 12 + 12 + 4 * 7, 25 * 8 + 4
    if kind in ("fluid", "points"):
        px = case["width"] * case["height"]
        return {"bytes": (w + s) * (12 if kind == "fluid" else 16) + px * 16,
                "flops": (w + s) * 60 + px * (900 if kind == "fluid" else 40)}
    if kind == "setup":
        return {"bytes": b * (12 + 4 + 4 + 20) + s * (12 + 20 + lb), "flops": b * 20 * 15 + s * 33 * 15}
    # pair terms within the support: about 30 neighbours for the densities, the heat and
    # the PBF and contact terms, 11 links and a few contacts
    per_it = (w + s) * 30 * (14 + 20 + 9) + s * 11 * 45 + s * 4 * 60 + b * 9 * 34
    per_sub = (w + s) * 30 * (14 + 12) + w * 30 * 20 * 2 + s * 30 * 9 + 3 * per_it
    n = FRAME if kind == "batch" else case["substeps"]
    if kind == "adjoint":   # forward, the recorded forward again, and about twice its terms in reverse
        return {"bytes": 2 * (w + s) * pb + s * lb + b * 20, "flops": 4 * n * per_sub}
    return {"bytes": 2 * ((w + s) * pb + s * lb) + b * 32, "flops": n * per_sub}


# --------------------------------------------------------------------------- 64 bits
def exact(case, seed):
    """The boundary volumes of the set-up in 64 bits (Akinci: V = m / (m W(0) + sum m W(d))).
    A whole call of the solver has no such value here: its interlink topology follows from
    single roundings, and the rest from it."""
    if case["kind"] != "setup":
        return None
    w = _host(case, seed)
    x = torch.from_numpy(np.asarray(w.bnd["positions"], np.float64))
    h, m = float(w.params.effective_radius), float(w.bnd["mass"][0])
    poly6 = float(w.params.poly6)
    # cells of h: a particle's neighbours lie in the 27 cells around its own
    c = torch.floor(x / h).long()
    c -= c.min(0).values - 1
    ext = c.max(0).values + 2
    key = (c[:, 0] * ext[1] + c[:, 1]) * ext[2] + c[:, 2]
    key, order = torch.sort(key, stable=True)
    xs = x[order]
    starts = torch.searchsorted(key, torch.arange(int(ext.prod()) + 1))
    most = int((starts[1:] - starts[:-1]).max())
    rho = torch.zeros(len(x), dtype=torch.float64)
    for dx in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dz in (-1, 0, 1):
                k = key + (dx * ext[1] + dy) * ext[2] + dz
                s, e = starts[k], starts[k + 1]
                for q in range(most):
                    j = torch.clamp(s + q, max=len(x) - 1)
                    d2 = ((xs - xs[j]) ** 2).sum(1)
                    ok = (s + q < e) & (d2 < h * h)
                    rho += torch.where(ok, m * poly6 * (h * h - d2) ** 3, torch.zeros_like(d2))
    vol = torch.empty_like(rho)
    vol[order] = m / rho
    return {"volume": vol, "b_hash": None, "b_index": None, "b_start": None, "d_index": None,
            "connect_record": None, "connect_length": None, "iter_end": None}

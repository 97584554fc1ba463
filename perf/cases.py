"""The work that users of this framework have it do, as timed cases.

Every case goes through the public entry points a program calls: the C API of the trace
(`soltrace_b200.lib`: st_sim_run, the readback calls, flux maps, st_b200_sim_run_batch) and the
flux surrogate (`soltrace_b200.surrogate`).  Scenes are the ones of `soltrace_b200.scenes`, at
the sizes of the tests and the benchmark and over the ranges between them.

A state holds a context with its scene pushed (what a front end keeps between runs), so one
pass is one st_sim_run and the readback of its results.  The trace is Monte Carlo over
per-ray streams keyed by the run's seed: the same seed gives the same counts and records.
"""
import math

import numpy as np
import torch

from soltrace_b200 import scenes, surrogate
from soltrace_b200.capi import dptr, iptr
from soltrace_b200.lib import load

DISH_MAP = (2, 1, 0, 50, 50, -0.25, 0.25, -0.25, 0.25, 1)
TROUGH_MAP = (3, 2, 1, 72, 120, 0.0, 0.035, -6.0, 6.0, 1)
FIELD_MAP = (2, 1, 1, 100, 100, 0.0, 4.0, -5.0, 5.0, 1)
MAPS = {"dish": DISH_MAP, "trough": TROUGH_MAP, "field": FIELD_MAP, "beam_down": scenes.GROUND_MAP}


def listed():
    return [
        # The smallest call a front end makes: a dish with a thousand rays, every intersection read
        # back (a check of a design while it is being edited).  Latency and launches.
        {"name": "dish 1e3 records", "kind": "dish", "hits": 1000, "mixed": False, "records": True},
        # Given rays (no sun, no errors) through the dish: ray-by-ray checks against another code,
        # measured ray sets.  An odd count; some rays miss the dish.
        {"name": "dish explicit 1e5", "kind": "explicit", "rays": 100_003, "mixed": False},
        # The dish at a million rays with the absorber's flux map: a design study's ordinary run.
        {"name": "dish flux 1e6", "kind": "dish", "hits": 1_000_000, "mixed": False, "records": False},
        # A trough with its glass envelope (refraction, three stages) at ten million rays, mixed
        # precision: an optical-efficiency run.
        {"name": "trough flux mixed 1e7", "kind": "trough", "hits": 10_000_000, "mixed": True, "records": False},
        # A small heliostat field with all records, an odd ray count: what a script over pysoltrace
        # or the GUI's ray viewer asks for.
        {"name": "field300 records 2e4", "kind": "field", "helios": 300, "hits": 20_011, "mixed": False,
         "records": True, "elevation": 45.0, "azimuth": 180.0},
        # The 2,000-heliostat field at a million hits with its records read back, low morning sun.
        {"name": "field2000 records mixed 1e6", "kind": "field", "helios": 2000, "hits": 1_000_000, "mixed": True,
         "records": True, "elevation": 25.0, "azimuth": 120.0},
        # The field in double precision with the receiver's flux map: a flux study's accurate run.
        {"name": "field2000 flux fp64 1e7", "kind": "field", "helios": 2000, "hits": 10_000_000, "mixed": False,
         "records": False, "elevation": 45.0, "azimuth": 180.0},
        # The headline run: 1e8 hits on the field in mixed precision, the receiver's flux map.
        {"name": "field2000 flux mixed 1e8", "kind": "field", "helios": 2000, "hits": 100_000_000, "mixed": True,
         "records": False, "elevation": 45.0, "azimuth": 180.0},
        # Beam-down tower (hyperboloid secondary, torus lip, ground receiver) in double precision.
        {"name": "beam-down1000 fp64 1e6", "kind": "beam_down", "helios": 1000, "hits": 1_000_000, "mixed": False,
         "records": False},
        # A day of sun positions over a tracking beam-down field in one call.
        {"name": "batch 24 suns mixed", "kind": "batch", "helios": 2000, "suns": 24, "hits": 400_000, "mixed": True},
        # Surrogate inference: the receiver maps of 64 situations of a 2,000-heliostat field.
        {"name": "surrogate maps 64x2000", "kind": "maps", "helios": 2000, "suns": 64},
        # Surrogate training: the gradients of one minibatch (forward, loss and backward passes).
        {"name": "surrogate gradients 16384", "kind": "gradients", "rows": 16384},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["dish", "trough", "field", "field", "field", "beam_down", "batch", "explicit", "maps",
                       "gradients"])
    mixed = rng.random() < 0.5
    if kind in ("dish", "trough", "field", "beam_down"):
        records = rng.random() < 0.4
        top = 1_000_000 if records or kind == "beam_down" else {"dish": 10_000_000, "trough": 10_000_000,
                                                               "field": 20_000_000}[kind]
        c = {"kind": kind, "hits": _log(rng, 1000, top), "mixed": mixed, "records": records}
        if kind == "field":
            c.update(helios=_log(rng, 200, 2000), elevation=round(rng.uniform(15.0, 80.0), 2),
                     azimuth=round(rng.uniform(100.0, 260.0), 2))
        elif kind == "beam_down":
            c.update(helios=_log(rng, 100, 2000))
        return c
    if kind == "batch":
        return {"kind": kind, "helios": _log(rng, 200, 2000), "suns": rng.randint(2, 24),
                "hits": _log(rng, 10_000, 400_000), "mixed": mixed}
    if kind == "explicit":
        return {"kind": kind, "rays": _log(rng, 1000, 100_003), "mixed": mixed}
    if kind == "maps":
        return {"kind": kind, "helios": _log(rng, 60, 2000), "suns": rng.randint(1, 64)}
    return {"kind": "gradients", "rows": _log(rng, 1000, 16384)}


class _Context:
    """A context of the trace with its scene pushed, freed with the state."""

    def __init__(self, api, scene, mixed, records, flux_map):
        self.api, self.ctx = api, api.st_create_context()
        scenes.push(api, self.ctx, scene)
        api.st_b200_set_precision(self.ctx, int(mixed))
        api.st_b200_set_records(self.ctx, int(records))
        if flux_map is not None:
            api.st_b200_add_flux_map(self.ctx, *flux_map)
        self.elements = [len(s.elements) for s in scene.stages]

    def __del__(self):
        self.api.st_free_context(self.ctx)

    def check(self, rc):
        if rc < 0:
            raise RuntimeError("; ".join(self.api.messages(self.ctx)))
        return rc


class _Records:
    """Room for a run's records (at most `room` of them), as a program that reads many runs back
    keeps it: st_locations & co. fill the same arrays after every run."""

    def __init__(self, room):
        self.room = room
        self.d = {k: np.zeros(room) for k in ("x", "y", "z", "cx", "cy", "cz")}
        self.i = {k: np.zeros(room, dtype=np.int32) for k in ("element", "stage", "raynum")}

    def read(self, api, ctx):
        n = api.st_num_intersections(ctx)
        if n > self.room:
            raise RuntimeError("more records than there is room for")
        api.st_locations(ctx, *(dptr(self.d[k]) for k in ("x", "y", "z")))
        api.st_cosines(ctx, *(dptr(self.d[k]) for k in ("cx", "cy", "cz")))
        api.st_elementmap(ctx, iptr(self.i["element"]))
        api.st_stagemap(ctx, iptr(self.i["stage"]))
        api.st_raynumbers(ctx, iptr(self.i["raynum"]))
        return {"n": n, **self.d, **self.i}


def _room(case):
    """Records that a run of a case can leave: two per ray (trough: six, field: three)."""
    per = {"trough": 6, "field": 3, "beam_down": 4}.get(case["kind"], 2)
    return per * case.get("rays", case.get("hits")) + 64


def _explicit_rays(case, seed):
    """Rays from a plane 10 m above the dish, over a square that reaches past its rim, tilted by a
    few milliradians."""
    rng = np.random.default_rng(seed)
    n = case["rays"]
    pos = np.column_stack([rng.uniform(-5.2, 5.2, n), rng.uniform(-5.2, 5.2, n), np.full(n, 10.0)])
    d = np.column_stack([rng.normal(0.0, 0.004, n), rng.normal(0.0, 0.004, n), np.full(n, -1.0)])
    return pos, d / np.linalg.norm(d, axis=1)[:, None]


def _map_features(case, seed):
    rng = np.random.default_rng(seed)
    xy = scenes.field_layout(case["helios"]).astype(np.float64)
    out = []
    for _ in range(case["suns"]):
        sun, off, sigma = surrogate.random_situation(rng, len(xy))
        out.append(surrogate.situation_features(sun, xy[:, 0], xy[:, 1], off[:, 0], off[:, 1], sigma, 150.0))
    return torch.from_numpy(np.concatenate(out).astype(np.float32)).cuda()


def _gradient_batch(case, seed):
    """Inputs and target images (a spot on a 32 x 32 receiver image) of one minibatch."""
    rows = case["rows"]
    feats = _map_features({"helios": 2000, "suns": -(-rows // 2000)}, seed)[:rows].to(torch.bfloat16).contiguous()
    g = torch.Generator(device="cuda").manual_seed(seed)
    u = torch.rand(rows, 4, device="cuda", generator=g)
    k = torch.arange(32, device="cuda", dtype=torch.float32)
    gx = torch.exp(-0.5 * ((k - 8.0 - 16.0 * u[:, :1]) / (1.0 + 3.0 * u[:, 2:3])) ** 2)
    gy = torch.exp(-0.5 * ((k - 8.0 - 16.0 * u[:, 1:2]) / (1.0 + 3.0 * u[:, 3:])) ** 2)
    return feats, (gy[:, :, None] * gx[:, None, :]).reshape(rows, 1024).contiguous()


def prepare(case, seed):
    api = load()
    kind = case["kind"]
    if kind == "maps":
        return {"kind": kind, "net": surrogate.Mlp(api, seed=seed), "feats": _map_features(case, seed),
                "helios": case["helios"]}
    if kind == "gradients":
        x, t = _gradient_batch(case, seed)
        return {"kind": kind, "net": surrogate.Mlp(api, seed=seed), "x": x, "t": t}
    s = {"kind": kind, "seed": seed & 0x7FFFFFFF, "records": case.get("records", False)}
    if kind == "explicit":
        scene = scenes.dish_scene(1000)
        for face in (scene.optics[0].front, scene.optics[0].back):
            face.refl = 1.0
        scene.sunshape_errors = scene.optical_errors = False
        s["rays"] = _explicit_rays(case, seed)
        s["records"] = True
    elif kind == "dish":
        scene = scenes.dish_scene(case["hits"])
    elif kind == "trough":
        scene = scenes.trough_scene(case["hits"])
    elif kind == "field":
        scene = scenes.field_scene(case["helios"], case["hits"], elevation_deg=case["elevation"],
                                   azimuth_deg=case["azimuth"], seed=seed)
    elif kind == "beam_down":
        el, az = np.random.default_rng(seed).uniform((20.0, 110.0), (75.0, 250.0))
        scene = scenes.beam_down_scene(case["helios"], case["hits"], sun_xyz=scenes.sun_vector(el, az))
    else:
        scene = scenes.beam_down_scene(case["helios"], case["hits"])
        s["suns"], s["hits"], _ = scenes.annual_suns(case["suns"], seed=seed, rays_per_kw=float(case["hits"]))
        s["target"] = scenes.beam_down_target()
    if s["records"]:
        s["room"] = _Records(_room(case))
    s["map"] = None if s["records"] else MAPS["beam_down" if kind == "batch" else kind]
    s["c"] = _Context(api, scene, case["mixed"], s["records"], s["map"])
    if kind in ("field", "beam_down"):  # sparse fields and low suns need more than st_sim_params' int cap
        api.st_b200_set_max_sun_rays(s["c"].ctx, 1000 * case["hits"])
    return s


def run(state):
    kind = state["kind"]
    if kind == "maps":
        return surrogate.predict_fields(state["net"], state["feats"], state["helios"], 1.7)
    if kind == "gradients":
        net = state["net"]
        loss, dy = net.loss_grad(net.forward(state["x"]), state["t"])
        dws, dbs, _ = net.backward(dy)
        return {"loss": loss, "dw": dws, "db": dbs}
    c = state["c"]
    api, ctx = c.api, c.ctx
    if kind == "batch":
        c.check(api.run_batch(ctx, state["seed"], state["suns"], state["hits"], state["target"]))
        m = state["map"]
        maps = [api.batch_flux(ctx, 0, k, m[3], m[4]).view(np.int64) for k in range(len(state["hits"]))]
        return {"maps": np.stack(maps),
                "sun_rays": [api.batch_stats(ctx, k)["sun_rays"] for k in range(len(state["hits"]))]}
    if kind == "explicit":
        api.explicit_rays(ctx, *state["rays"])
    c.check(api.run(ctx, state["seed"]))
    if state["records"]:
        return {"records": state["room"].read(api, ctx), "sun": api.sun_stats(ctx)}
    m = state["map"]
    return {"flux": api.flux(ctx, 0, m[3], m[4]).view(np.int64), "sun_rays": api.stats(ctx)["sun_rays"],
            "counts": [a.view(np.int64) for k, n in enumerate(c.elements)
                       for a in api.element_counts(ctx, k + 1, n)]}


# ------------------------------------------------------------------------------------
# what a pass cannot do without
# ------------------------------------------------------------------------------------
# per kind: sun rays generated per first-stage hit, records left per hit, stage entries per hit
# after the first stage (rounded from runs of these scenes)
_PER_HIT = {"dish": (1.28, 1.9, 0.9), "trough": (1.01, 3.8, 1.9), "field": (8.3, 1.8, 0.85),
            "beam_down": (8.3, 2.2, 1.3), "explicit": (1.0, 2.0, 1.0)}


def work(case):
    kind = case["kind"]
    widths = list(zip(surrogate.DIMS[:-1], surrogate.DIMS[1:]))
    weights = sum(a * b for a, b in widths)
    if kind == "maps":
        rows = case["helios"] * case["suns"]
        return {"bytes": 4.0 * rows * 16 + 2.0 * weights + 4.0 * 1024 * case["suns"], "flops": 2.0 * rows * weights}
    if kind == "gradients":  # the backward pass has two products per layer, one for the first
        rows = case["rows"]
        return {"bytes": rows * (2.0 * 16 + 4.0 * 1024) + weights * (2.0 + 4.0),
                "flops": 2.0 * rows * (3.0 * weights - 16 * 256)}
    sun, rec, later = _PER_HIT["beam_down" if kind == "batch" else kind]
    hits = float(case.get("rays", case.get("hits"))) * (0.65 * case["suns"] if kind == "batch" else 1.0)
    # 189 operations per generated sun ray, 501 per first-stage hit, 177 per later stage entry
    flops = hits * ((0.0 if kind == "explicit" else 189.0 * sun) + 501.0 + 177.0 * later)
    nbytes = 400.0 * case.get("helios", 3) + 8.0 * 10000 * case.get("suns", 1)
    if kind == "explicit" or case.get("records"):
        nbytes += hits * 60.0 * rec + (48.0 * hits if kind == "explicit" else 0.0)
    return {"bytes": nbytes, "flops": flops}


# ------------------------------------------------------------------------------------
# the computed numbers in 64 bits
# ------------------------------------------------------------------------------------
def _exact_explicit(case, seed):
    """The given rays through the dish (z = r^2 / 20, 10 m across) to the absorber (0.5 m across
    in the plane z = 5): the records' positions and incoming directions, in readback order."""
    pos, d = _explicit_rays(case, seed)
    a = d[:, 0] ** 2 + d[:, 1] ** 2
    b = 2.0 * (pos[:, 0] * d[:, 0] + pos[:, 1] * d[:, 1]) - 20.0 * d[:, 2]
    c = pos[:, 0] ** 2 + pos[:, 1] ** 2 - 20.0 * pos[:, 2]
    t = 2.0 * c / (-b + np.sqrt(b * b - 4.0 * a * c))  # -b > 0: the nearer root, without cancellation
    p = pos + t[:, None] * d
    hit = p[:, 0] ** 2 + p[:, 1] ** 2 <= 25.0
    p, d = p[hit], d[hit]
    n = np.column_stack([-p[:, 0] / 10.0, -p[:, 1] / 10.0, np.ones(len(p))])
    n /= np.linalg.norm(n, axis=1)[:, None]
    out = d - 2.0 * np.sum(d * n, axis=1)[:, None] * n
    q = p + ((5.0 - p[:, 2]) / out[:, 2])[:, None] * out
    miss = q[:, 0] ** 2 + q[:, 1] ** 2 > 0.0625
    q[miss] = p[miss]  # a miss is recorded where the ray entered the stage
    # the reference's merge: both stages' full blocks of 8192 records, then the rest of each
    full = len(p) // 8192 * 8192

    def merged(u, v):
        return np.concatenate([u[:full], v[:full], u[full:], v[full:]])

    def roomy(u):
        return np.concatenate([u, np.zeros((_room(case) - len(u), 3))])

    pp, dd = roomy(merged(p, q)), roomy(merged(d, out))
    rec = {"n": None, "x": pp[:, 0], "y": pp[:, 1], "z": pp[:, 2], "cx": dd[:, 0], "cy": dd[:, 1], "cz": dd[:, 2],
           "element": None, "stage": None, "raynum": None}
    return {"records": rec, "sun": None}


def _exact_net(seed):
    g = torch.Generator(device="cpu").manual_seed(seed)
    ws = [(torch.randn(o, i, generator=g) * math.sqrt(2.0 / i)).float().to(torch.bfloat16).double().cuda()
          for i, o in zip(surrogate.DIMS[:-1], surrogate.DIMS[1:])]
    return ws, [torch.zeros(w.shape[0], dtype=torch.float64, device="cuda") for w in ws]


def _exact_forward(ws, bs, x):
    for k, (w, b) in enumerate(zip(ws, bs)):
        x = torch.nn.functional.linear(x, w, b)
        if k + 1 < len(ws):
            x = torch.relu(x)
    return x


def exact(case, seed):
    if case["kind"] == "explicit":
        return _exact_explicit(case, seed)
    if case["kind"] == "maps":
        ws, bs = _exact_net(seed)
        x = _map_features(case, seed).to(torch.bfloat16).double()
        return torch.stack([torch.clamp(_exact_forward(ws, bs, part) * 1.7, min=0.0).sum(0)
                            for part in x.split(case["helios"])])
    if case["kind"] == "gradients":
        ws, bs = _exact_net(seed)
        x, t = _gradient_batch(case, seed)
        for v in ws + bs:
            v.requires_grad_(True)
        loss = ((_exact_forward(ws, bs, x.double()) - t.double()) ** 2).mean()
        loss.backward()
        return {"loss": loss.detach().reshape(1), "dw": [w.grad for w in ws], "db": [b.grad for b in bs]}
    return None  # sampled rays: records have no value apart from the streams they draw from

"""The workloads whose speed is followed, each through the package's public entry points.

Five families: `walk` (a model resident on the GPU, Transport.run and its integer tallies), `launch` (the
LaunchOMP replacement with every tally and map of an OutputInfo), `batch` (many planar instances in one
launch), `forward` (network inference on host rows) and `train` (Adam steps on a resident data set).
Photon numbers, meshes, detectors and network sizes are those of the package's scenes, tests and benchmark,
from the smallest calls a user makes to the largest that a second holds.
"""
import ctypes
import math
import os
import tempfile

import numpy as np
import torch

from xmcml_b200 import _lib, api, batch, scenes, surrogate
from xmcml_b200 import structs as S

# Operations of one walk step: about 48 of FP32 arithmetic and 45 integer operations of the random numbers.
STEP_OPS = 93
# Walk steps of a photon, by scene, with the weight cut at 1e-4 and photons lost at the Area's faces / with
# roulette and without that loss.
STEPS = {"planar": (276, 1137), "cover": (266, 300), "heightfield": (552, 1217), "ellipsoid": (550, 1300), "biased": (145, 145)}
BATCH_STEPS = 760
# Counters of a run that are results of the walk (the others count its queries or its milliseconds).
LEDGER = ("photons_launched", "photons_terminated", "steps", "n_escaped_top", "n_escaped_bottom", "n_area", "n_cut",
          "n_roulette", "n_glass", "n_budget", "n_invalid", "n_detected", "absorbed_target_fx", "bias_gained_fx",
          "bias_lost_fx") + tuple(k + "_fx" for k in S.LEDGER_TERMS)


def listed():
    return [
        # A quick look at a layer stack: few photons, so the launch, the longest walk and the read-back count.
        {"name": "planar_look", "kind": "walk", "scene": "planar", "photons": 20_000, "roulette": False, "rings": 50,
         "bins": 1, "mesh": 0, "beam": 0.0},
        # The plain 3-layer run with roulette and the full energy balance, 1e6 photons.
        {"name": "planar_roulette", "kind": "walk", "scene": "planar", "photons": 1_000_000, "roulette": True, "rings": 50,
         "bins": 1, "mesh": 0, "beam": 0.0},
        # A stack under a glass cover with cube and ring detectors, layer filters, angles, target layers, time bins
        # and a wide beam; an odd number of photons.
        {"name": "cover_detectors", "kind": "walk", "scene": "cover", "photons": 300_007, "roulette": False, "rings": 5,
         "bins": 12, "mesh": 0, "beam": 0.3},
        # Triangulated height fields (2 x 130,050 triangles), the tallies without maps.
        {"name": "heightfield", "kind": "walk", "scene": "heightfield", "photons": 1_000_000, "roulette": True, "rings": 50,
         "bins": 200, "mesh": 256, "beam": 0.0},
        # An embedded triangulated target on the large absorption grid, 100 rings x 200 time bins.
        {"name": "ellipsoid", "kind": "walk", "scene": "ellipsoid", "photons": 1_000_000, "roulette": False, "rings": 100,
         "bins": 200, "mesh": 6, "beam": 0.0},
        # The biased walk towards an attractive point (64-bit weights, weight-integral tables).
        {"name": "biased", "kind": "walk", "scene": "biased", "photons": 50_000, "roulette": False, "rings": 50, "bins": 20,
         "mesh": 0, "beam": 0.0},
        # What a program built on the reference's LaunchOMP calls again and again: every tally, the scattering map
        # and one trajectory map per detector, added into its OutputInfo.
        {"name": "launch_heightfield", "kind": "launch", "scene": "heightfield", "photons": 3_000_000, "rings": 50, "bins": 200,
         "mesh": 256},
        # The sweep of 1,024 layered models with budgets over two decades.
        {"name": "batch_sweep", "kind": "batch", "instances": 1024, "photons": 20_000_000, "spread": 2.0, "rings": 50,
         "bins": 20, "beam": 0.0},
        # The candidates that an inverse fit hands to the Monte Carlo, or the queries outside the network's hull.
        {"name": "batch_candidates", "kind": "batch", "instances": 17, "photons": 1_700_000, "spread": 0.0, "rings": 50,
         "bins": 20, "beam": 0.5},
        # One query of the network.
        {"name": "forward_query", "kind": "forward", "rows": 1, "hidden": 256, "layers": 4, "outputs": 1000},
        # The network's inference batch.
        {"name": "forward_batch", "kind": "forward", "rows": 65_536, "hidden": 256, "layers": 4, "outputs": 1000},
        # Adam steps on minibatches drawn from a resident data set, and the new parameters.
        {"name": "train", "kind": "train", "steps": 50, "batch": 4096, "rows": 20_000, "hidden": 256, "layers": 4,
         "outputs": 1000, "weighted": True},
    ]


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("walk", "walk", "walk", "launch", "batch", "forward", "train"))
    if kind == "walk":
        scene = rng.choice(("planar", "cover", "heightfield", "ellipsoid", "biased"))
        case = {"kind": kind, "scene": scene, "photons": _spread(rng, 10_000, 60_000 if scene == "biased" else 1_000_000),
                "roulette": scene != "biased" and rng.random() < 0.5, "rings": 5, "bins": 12, "mesh": 0,
                "beam": rng.choice((0.0, round(rng.uniform(0.05, 0.5), 3)))}
        if scene != "cover":
            case["rings"], case["bins"] = rng.randint(10, 100), rng.choice((1, rng.randint(2, 200)))
        if scene == "heightfield":
            case["mesh"], case["beam"] = 2 * rng.randint(16, 127) + 1, 0.0
        elif scene == "ellipsoid":
            case["mesh"] = rng.randint(4, 6)
        return case
    if kind == "launch":
        scene = rng.choice(("planar", "heightfield"))
        return {"kind": kind, "scene": scene, "photons": _spread(rng, 50_000, 2_000_000), "rings": rng.randint(5, 50),
                "bins": rng.randint(1, 200), "mesh": 2 * rng.randint(16, 127) + 1 if scene == "heightfield" else 0}
    if kind == "batch":
        n = _spread(rng, 3, 1024)
        return {"kind": kind, "instances": n, "photons": _spread(rng, max(200_000, 2_000 * n), 15_000_000),
                "spread": rng.choice((0.0, 1.0, 2.0)), "rings": rng.choice((50, rng.randint(20, 100))),
                "bins": rng.randint(1, 40), "beam": rng.choice((0.0, 0.5))}
    net = {"hidden": rng.choice((128, 256, 256)), "layers": rng.randint(2, 5), "outputs": rng.choice((1000, rng.randint(30, 1000)))}
    if kind == "forward":
        return {"kind": kind, "rows": _spread(rng, 1, 60_000), **net}
    return {"kind": kind, "steps": rng.randint(10, 50), "batch": 128 * rng.randint(4, 32), "rows": _spread(rng, 2_000, 20_000),
            "weighted": rng.random() < 0.5, **net}


# ---- scenes ----------------------------------------------------------------------------------------------

_FILES = tempfile.TemporaryDirectory(prefix="xmc_cases_")  # model files, written once for each scene


def _cover(photons, bins):
    props = [(0.2, 0.0, 0.0, 0.0, 1.5)] + list(scenes.THREE_LAYER)
    sc = scenes.planar(props, photons=photons, n_rings=0)
    sc.rings = [scenes.Ring(0.0, 0.3, filter=[1, 2, 3, 4]), scenes.Ring(0.3, 0.6, filter=[3]),
                scenes.Ring(0.6, 1.0, angle=60.0), scenes.Ring(1.0, 2.0), scenes.Ring(2.0, 4.0, filter=[4], angle=80.0)]
    sc.cubes = [scenes.Cube((0.5, 0.5, 0.0), (0.4, 0.4, 0.01)),
                scenes.Cube((-1.0, 0.0, 0.0), (1.0, 1.0, 0.01), filter=[2, 3])]
    sc.time_start, sc.time_finish, sc.time_bins = 1.0, 30.0, bins
    sc.target_layers = [2, 3]
    sc.min_weight = 1e-3
    return sc


def _scene(case):
    kind, n, rings, bins = case["scene"], case["photons"], case["rings"], case["bins"]
    width = 5.0 / rings
    if kind == "cover":
        return _cover(n, bins)
    if kind == "heightfield":
        return scenes.height_field_tissue(photons=n, grid=case["mesh"], n_rings=rings, ring_width=width, time_bins=bins)
    if kind == "ellipsoid":
        return scenes.ellipsoid_target(photons=n, subdiv=case["mesh"], n_rings=rings, ring_width=10.0 / rings, time_bins=bins)
    sc = scenes.planar(photons=n, n_rings=rings, ring_width=width, time_bins=bins, time_finish=bins * 5.0 * scenes.C_MM_PER_PS)
    if kind == "biased":
        sc.bias_target, sc.bias_factor = (0, 0, 2), 1.0
        sc.bias_integral_precision, sc.bias_table_precision = 128, 4096
    return sc


def _model(case):
    stem = "_".join(str(case[k]) for k in ("scene", "photons", "rings", "bins", "mesh"))
    paths = [os.path.join(_FILES.name, stem + e) for e in (".xml", ".surface")]
    if not os.path.exists(paths[1]):
        _scene(case).write(_FILES.name, stem)
    return api.Model(*paths)


# ---- states ----------------------------------------------------------------------------------------------

class _Launch:
    """A caller of the LaunchOMP replacement: its model with the prebuilt tree, its OutputInfo and generator."""

    def __init__(self, case, seed):
        self.model = _model(case)
        info = self.model.info
        info.numberOfPhotons = case["photons"]
        self.lib = _lib.load()
        self.tree = self.lib.xmc_generate_bvh_tree(info.surface, info.numberOfSurfaces)
        info.bvhTree = self.tree
        self.rng = api.mcg59_init(seed, 0, 1)
        n, bins, grid = self.model.n_detectors, info.timeScaleSize, int(np.prod(self.model.grid_shape))
        self.absorption, self.scattering = np.zeros(grid), np.zeros(grid)
        self.trajectory = np.zeros((n, grid), dtype=np.uint64)
        self.dets, self.times = (S.DetectorInfo * n)(), (S.TimeInfo * (n * bins))()
        at = lambda array, kind: array.ctypes.data_as(ctypes.POINTER(kind))  # noqa: E731
        for d in range(n):
            self.dets[d].trajectory, self.dets[d].trajectorySize = at(self.trajectory[d], ctypes.c_uint64), grid
            self.dets[d].timeScale = ctypes.cast(ctypes.byref(self.times, d * bins * ctypes.sizeof(S.TimeInfo)), ctypes.POINTER(S.TimeInfo))
            self.dets[d].timeScaleSize = bins
        self.info = S.OutputInfo(0, 0.0, at(self.absorption, ctypes.c_double), at(self.scattering, ctypes.c_double), grid, self.dets, n)

    def results(self):
        out = {"absorption": self.absorption, "scattering": self.scattering, "trajectory": self.trajectory}
        for what, rows, cls in (("detector", self.dets, S.DetectorInfo), ("time", self.times, S.TimeInfo)):
            for name, kind in (("numberOfPhotons", "u8"), ("weight", "f8"), ("targetWeight", "f8")):
                dt = np.dtype({"names": [name], "formats": [kind], "offsets": [getattr(cls, name).offset],
                               "itemsize": ctypes.sizeof(cls)})
                out[what + "_" + name] = np.frombuffer(rows, dtype=dt)[name]
        return out

    def __del__(self):
        self.model.info.bvhTree = None
        self.lib.xmc_free_bvh_tree(self.tree)


def _instances(case, seed):
    inst = batch.sample_instances(seed, case["instances"], budget=(1.0, 2.0), beam_radius=(0.0, case["beam"]))
    share = 10.0 ** np.random.default_rng(seed + 1).uniform(0.0, max(case["spread"], 1e-9), case["instances"])
    inst.photons = np.maximum(1, np.round(share * (case["photons"] / share.sum()))).astype(np.uint64)
    return inst


def _net(case, rng):
    """He-uniform weights and small biases in the flat layout (per layer W [out, in] row-major, then b)."""
    dims = [15] + [case["hidden"]] * case["layers"] + [case["outputs"]]
    parts = []
    for i in range(len(dims) - 1):
        lim = math.sqrt(6.0 / dims[i])
        parts += [rng.uniform(-lim, lim, dims[i + 1] * dims[i]), 0.1 * rng.standard_normal(dims[i + 1])]
    return dims, np.concatenate(parts).astype(np.float32)


def _data(case, rng, rows):
    """Standardised inputs, and targets that depend smoothly on them with a little noise."""
    x = rng.standard_normal((rows, 15)).astype(np.float32)
    a = rng.standard_normal((15, 24)).astype(np.float32) / math.sqrt(15.0)
    b = rng.standard_normal((24, case["outputs"])).astype(np.float32) / 4.0
    t = np.tanh(x @ a) @ b + 0.05 * rng.standard_normal((rows, 1)).astype(np.float32)
    return x, t.astype(np.float32)


def _weights(case, rng):
    w = rng.uniform(0.05, 2.0, case["outputs"])
    return (w / w.mean()).astype(np.float32) if case["weighted"] else None


LR, B1, B2, EPS = 2e-3, 0.9, 0.999, 1e-8


def prepare(case, seed):
    kind = case["kind"]
    if kind == "walk":
        model = _model(case)
        opts = {"roulette": case["roulette"], "area_kill": not case["roulette"], "beam_radius": case["beam"]}
        return {"case": case, "t": api.Transport(model, **opts), "model": model, "seed": seed}
    if kind == "launch":
        return {"case": case, "launch": _Launch(case, seed)}
    if kind == "batch":
        b = batch.Batch(n_rings=case["rings"], ring_width=5.0 / case["rings"], n_time=case["bins"], max_instances=case["instances"])
        return {"case": case, "b": b, "inst": _instances(case, seed)}
    rng = np.random.default_rng(seed)
    rows = case["rows"] if kind == "forward" else case["batch"]
    net = surrogate.MLP(15, case["outputs"], case["hidden"], case["layers"], max_rows=(rows + 127) // 128 * 128)
    net.set_params(_net(case, rng)[1])
    if kind == "forward":
        return {"case": case, "net": net, "x": rng.standard_normal((rows, 15)).astype(np.float32)}
    x, t = _data(case, rng, case["rows"])
    net.set_output_weights(_weights(case, rng))
    net.set_dataset(x, t)
    return {"case": case, "net": net, "seed": seed}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "walk":
        led = state["t"].run(case["photons"], seed=state["seed"])
        out = state["t"].tallies()
        out["ledger"] = [led[k] for k in LEDGER]
        return out
    if kind == "launch":
        s = state["launch"]
        api.launch_omp(s.model, s, s.rng)
        return s.results()
    if kind == "batch":
        out = state["b"].run(state["inst"])
        return {k: v for k, v in out.items() if k not in ("kernel_ms", "status")}
    if kind == "forward":
        return state["net"].forward(state["x"])[0]
    losses, _ = state["net"].train(case["steps"], batch=case["batch"], lr=LR, beta1=B1, beta2=B2, eps=EPS, seed=state["seed"])
    return {"losses": losses, "params": state["net"].get_params()}


# ---- what a pass cannot do without -----------------------------------------------------------------------

def work(case):
    kind = case["kind"]
    if kind in ("walk", "launch"):
        steps = STEPS[case["scene"]][1 if case.get("roulette") else 0] * case["photons"]
        dets = 7 if case["scene"] == "cover" else case["rings"]
        grid = 256 * 256 * 128 if case["scene"] == "ellipsoid" else 10 ** 6
        tris = {"heightfield": 4 * max(case["mesh"] - 1, 0) ** 2 + 4, "ellipsoid": 20 * 4 ** case["mesh"] + 8}.get(case["scene"], 10)
        out = 8 * grid + 32 * dets * (1 + case["bins"])
        if kind == "launch":
            out += 8 * grid * (1 + dets)
        return {"bytes": 48 * tris + out, "flops": STEP_OPS * steps}
    if kind == "batch":
        n = case["instances"]
        return {"bytes": n * (32 + 3 * 48) + 8 * n * (case["rings"] * (case["bins"] + 1) + 14),
                "flops": STEP_OPS * BATCH_STEPS * case["photons"]}
    dims = [15] + [case["hidden"]] * case["layers"] + [case["outputs"]]
    params = sum((a + 1) * b for a, b in zip(dims, dims[1:]))
    if kind == "forward":
        return {"bytes": 4 * (params + case["rows"] * (15 + case["outputs"])), "flops": 2 * params * case["rows"]}
    rows = case["steps"] * case["batch"]
    return {"bytes": 4 * rows * (15 + case["outputs"]) + 24 * params * case["steps"], "flops": 6 * params * rows}


# ---- the same in 64 bits ---------------------------------------------------------------------------------

def _layers(dims, flat, device):
    p, at, out = torch.from_numpy(flat).to(device, torch.float64), 0, []
    for a, b in zip(dims, dims[1:]):
        out.append([p[at:at + a * b].reshape(b, a).clone(), p[at + a * b:at + a * b + b].clone()])
        at += a * b + b
    return out


def _forward(layers, x):
    z, a = [], [x]
    for i, (w, b) in enumerate(layers):
        z.append(a[-1] @ w.T + b)
        a.append(z[-1] * torch.sigmoid(z[-1]) if i < len(layers) - 1 else z[-1])
    return z, a


def _philox(c0, c1, c2, c3, k0, k1):
    """First word of Philox4x32-10 (Salmon et al., SC'11) for arrays of counters."""
    m = np.uint64(0xFFFFFFFF)
    c = [np.asarray(v, dtype=np.uint64) for v in (c0, c1, c2, c3)]
    k0, k1 = np.uint64(k0), np.uint64(k1)
    for _ in range(10):
        p0, p1 = np.uint64(0xD2511F53) * c[0], np.uint64(0xCD9E8D57) * c[2]
        c = [(p1 >> np.uint64(32)) ^ c[1] ^ k0, p1 & m, (p0 >> np.uint64(32)) ^ c[3] ^ k1, p0 & m]
        k0, k1 = (k0 + np.uint64(0x9E3779B9)) & m, (k1 + np.uint64(0xBB67AE85)) & m
    return c[0]


def exact(case, seed):
    kind = case["kind"]
    if kind not in ("forward", "train"):
        return None  # integer tallies, and sums of them
    device = "cuda" if torch.cuda.is_available() else "cpu"
    rng = np.random.default_rng(seed)
    dims, flat = _net(case, rng)
    layers = _layers(dims, flat, device)
    if kind == "forward":
        x = rng.standard_normal((case["rows"], 15)).astype(np.float32)
        return _forward(layers, torch.from_numpy(x).to(device, torch.float64))[1][-1]
    x, t = (torch.from_numpy(v).to(device, torch.float64) for v in _data(case, rng, case["rows"]))
    w = _weights(case, rng)
    w = torch.ones(case["outputs"], device=device, dtype=torch.float64) if w is None else torch.from_numpy(w).to(device, torch.float64)
    moments = [[[torch.zeros_like(p), torch.zeros_like(p)] for p in layer] for layer in layers]
    rows, losses = np.arange(case["batch"]), []
    for step in range(1, case["steps"] + 1):
        u = _philox(rows, np.full_like(rows, step), np.full_like(rows, 0x6D6C70), 0 * rows, seed & 0xFFFFFFFF, seed >> 32)
        src = torch.from_numpy(((u * np.uint64(case["rows"])) >> np.uint64(32)).astype(np.int64)).to(device)
        z, a = _forward(layers, x[src])
        d = a[-1] - t[src]
        losses.append(float((w * d * d).sum()) / d.numel())
        dz = 2.0 / d.numel() * w * d
        alpha = LR * math.sqrt(1.0 - B2 ** step) / (1.0 - B1 ** step)
        for i in reversed(range(len(layers))):
            grads = (dz.T @ a[i], dz.sum(0))
            if i:
                s = torch.sigmoid(z[i - 1])
                dz = (dz @ layers[i][0]) * s * (1.0 + z[i - 1] * (1.0 - s))
            for p, g, (m, v) in zip(layers[i], grads, moments[i]):
                m.mul_(B1).add_(g, alpha=1.0 - B1)
                v.mul_(B2).addcmul_(g, g, value=1.0 - B2)
                p.sub_(alpha * m / (v.sqrt() + EPS))
    params = torch.cat([torch.cat([w_.reshape(-1), b_]) for w_, b_ in layers])
    return {"losses": np.array(losses), "params": params}

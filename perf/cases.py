"""The work that is timed: what a user of this framework has it do, through the Python package's public calls.

Kinds of case
  plain     a uniform-cooling realm (realm type cellular_automata): run to its end, or the first `steps` steps one call at a time
  batch     many uniform-cooling realms of uneven sizes in one launch
  track     an FE-coupled realm (cellular_automata_remelting): a laser track over a columnar baseplate, run to the end of its frames
  coupled   the same realm driven step by step by an FE solver of the caller's, which hands over node temperatures before each step
  raster    an FE-coupled realm whose frames come from the learned thermal model, back and forth over a block
  evaluate, gradients, train
            the learned thermal model by itself: temperatures of a list of points, gradients of one batch, a stretch of training

Sizes and physics are those of this repository's decks (amca3d_gb300/decks.py) and tests. Every realm is read from its deck once and
kept; a pass takes it back to its start, advances it and reads its fields into page-locked host arrays, as a parameter study does.
"""
import math

import numpy as np
import torch

import amca3d_gb300 as amca
from amca3d_gb300 import decks

HIDDEN, LAYERS, FREQ = 256, 4, 64
LIQUIDUS, BAND, THRESHOLD = 1700.0, 100.0, 5.0


def listed():
    return [
        # the smallest call: a host that advances a small realm step by step, where a step is one launch and its latency
        {"name": "plain_steps", "kind": "plain", "nx": 24, "ny": 24, "nz": 24, "bulk": 80, "surface": 60, "t_dot": -200.0, "steps": 24},
        # the physics of the reference's own nucleation example, 60^3 cells, to full solidification
        {"name": "plain_60", "kind": "plain", "nx": 60, "ny": 60, "nz": 60, "bulk": 270, "surface": 0, "t_dot": -20.0, "steps": 0},
        # an ordinary part of uneven edges with wall nucleation
        {"name": "plain_ragged", "kind": "plain", "nx": 149, "ny": 97, "nz": 61, "bulk": 700, "surface": 300, "t_dot": -50.0, "steps": 0},
        # the benchmark's domain: 33M cells, 20,000 bulk and 4,000 surface sites
        {"name": "plain_320", "kind": "plain", "nx": 320, "ny": 320, "nz": 320, "bulk": 20000, "surface": 4000, "t_dot": -50.0, "steps": 0},
        # a parameter sweep: 24 independent realms of 32 to 96 cells an edge in one launch, layout as the library picks it by itself
        {"name": "batch_24", "kind": "batch", "count": 24, "edge_lo": 32, "edge_hi": 96, "sizes": 3},
        # a short laser track over a small block, frames of the FE field resident on the device
        {"name": "track_small", "kind": "track", "nx": 75, "ny": 50, "nz": 30, "grains": 60, "frames": 420},
        # the laser powder-bed-fusion benchmark: 12.5M cells, 2,000 columnar grains, 1,550 frames
        {"name": "track_500", "kind": "track", "nx": 500, "ny": 250, "nz": 100, "grains": 2000, "frames": 1550},
        # an FE solver beside the realm: node temperatures from host memory before every step
        {"name": "coupled_steps", "kind": "coupled", "nx": 120, "ny": 60, "nz": 40, "grains": 60, "steps": 40},
        # two passes of a raster scan, every frame predicted by the learned model with the FE field near the liquidus
        {"name": "raster_model", "kind": "raster", "nx": 60, "ny": 60, "nz": 40, "grains": 60, "tracks": 2},
        # temperatures of a hundred thousand points of a part from the learned model
        {"name": "evaluate_100k", "kind": "evaluate", "points": 100003},
        # forward and backward pass of one batch of the model's own training schedule
        {"name": "gradients_32k", "kind": "gradients", "batch": 32768},
        # a stretch of that training schedule: Adam steps on batches gathered from a set on the device
        {"name": "train_32k", "kind": "train", "samples": 2000000, "steps": 24, "batch": 32768},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["plain", "plain", "plain", "batch", "track", "track", "coupled", "raster", "evaluate", "gradients", "train"])
    if kind == "plain":
        edge = math.exp(rng.uniform(math.log(12.0), math.log(300.0)))
        nx, ny, nz = (max(4, min(320, int(round(edge * math.exp(rng.uniform(-0.35, 0.35)))))) for _ in range(3))
        n = nx * ny * nz
        bulk = max(8, min(20000, _log_int(rng, 6e-4 * n, 6e-3 * n)))
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "bulk": bulk, "surface": rng.choice([0, max(1, bulk // 5)]),
                "t_dot": -float(rng.choice([20, 50, 100, 200])), "steps": rng.choice([0, 0, 0, rng.randint(1, 40)])}
    if kind == "batch":
        lo = rng.randint(16, 48)
        return {"kind": kind, "count": _log_int(rng, 4, 48), "edge_lo": lo, "edge_hi": lo + rng.randint(8, 64), "sizes": rng.randint(0, 9999)}
    if kind in ("track", "coupled", "raster"):
        most = {"track": 300, "coupled": 300, "raster": 90}[kind]
        nx = _log_int(rng, 40, most)
        ny, nz = max(24, int(nx * rng.uniform(0.45, 0.9))), max(16, int(nx * rng.uniform(0.2, 0.5)))
        c = {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "grains": _log_int(rng, 20, 1000)}
        if kind == "track":
            c["frames"] = rng.randint(250, 700)
        elif kind == "coupled":
            c["steps"] = rng.randint(4, 60)
        else:
            c["tracks"] = rng.randint(1, 2)
        return c
    if kind == "evaluate":
        return {"kind": kind, "points": _log_int(rng, 1, 1000000)}
    if kind == "gradients":
        return {"kind": kind, "batch": 128 * _log_int(rng, 1, 512)}
    return {"kind": kind, "samples": _log_int(rng, 200000, 4000000), "steps": rng.randint(4, 32), "batch": 128 * _log_int(rng, 16, 384)}


def _pinned(n, dtype):
    return torch.empty(n, dtype=dtype, pin_memory=True).numpy()  # the array keeps the page-locked tensor alive


def _cells(c):
    return c["nx"], c["ny"], c["nz"]


def _ghost_cells(c):
    return (c["nx"] + 2) * (c["ny"] + 2) * (c["nz"] + 2)


def _outputs_for(realm, names):
    kinds = {"int32": torch.int32, "float64": torch.float64, "uint8": torch.uint8}
    return {k: _pinned(realm.cells_with_ghosts, kinds[np.dtype(amca.FIELD_DTYPES[k]).name]) for k in names}


def _plain_deck(c, seed):
    h = 2e-6
    cells = _cells(c)
    return decks.PlainCase(name="part", cells=cells, cell_size=h, seed=seed, t_dot=c["t_dot"], time_step=0.001, termination_time=1.0e4,
                           bulk=(decks.bulk_density_for_sites(c["bulk"], cells, h), 3.0, 1.0),
                           surface=(decks.surface_density_for_sites(c["surface"], cells, h), 2.0, 0.5))


def _seed(seed):
    return 1 + seed % 1000003  # the realms' own seed is a small number


def _remelt_deck(c, seed):
    return decks.RemeltCase(name="block", cells=_cells(c), cell_size=2.0e-6, nucleation=True, seed=_seed(seed), bulk=(1.0e13, 8.0, 2.0),
                            surface=(0.0, 0.5, 0.1), melting_temperature=LIQUIDUS, solidus_temperature=1600.0, a=(0.0, 2.03e-4, 0.0),
                            microstructure="baseplate.txt", termination_time=1.0, time_step=1.0e-6, time_step_factor=0.4)


def _remelt_realm(c, seed):
    """The realm with its baseplate; frames are still to come."""
    case = _remelt_deck(c, seed)
    m = decks.columnar_microstructure(case.cells, case.cell_size, case.origin, c["grains"], seed)
    r = amca.CellularAutomataRealm(case.to_yaml(), seed=case.seed)
    r.set_microstructure(m["grain"], m["orient"], m["euler"], m["grain_cell"], m["grain_orient"], expected=m["expected"])
    return case, r


REMELT_FIELDS = ("orientation_id", "grain_id", "melted", "temperature")


# --- the learned thermal model -----------------------------------------------------------------------------------------------
def _uniform(seed, stream, i):
    """The model's counter-based uniform draws (splitmix64), of which its Fourier matrix is made."""
    full = (1 << 64) - 1

    def mix(z):
        z = (z + 0x9E3779B97F4A7C15) & full
        z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & full
        z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & full
        return z ^ (z >> 31)

    inner = mix((stream * 0x9E3779B97F4A7C15 + i) & full)
    return (mix(((seed * 0x100000001B3) & full) ^ inner) >> 11) * 2.0 ** -53


def _encoding(spec):
    """(Fourier matrix, input shift, input scale) of a model of this spec, as float32 values."""
    f = np.empty((FREQ, 5))
    for i in range(FREQ * 5):
        u1, u2 = max(_uniform(spec["seed"], 100, i), 1e-300), _uniform(spec["seed"], 101, i)
        sig = spec["fourier_sigma"] if i % 5 < 3 else spec["fourier_sigma_pv"]
        f.flat[i] = sig * math.sqrt(-2.0 * math.log(u1)) * math.cos(2.0 * math.pi * u2)
    lo = np.array(list(spec["window_lo"]) + [spec["power_lo"], spec["speed_lo"]])
    hi = np.array(list(spec["window_hi"]) + [spec["power_hi"], spec["speed_hi"]])
    return f.astype(np.float32), (0.5 * (lo + hi)).astype(np.float32), (2.0 / (hi - lo)).astype(np.float32)


def _field(spec, raw):
    """FE temperature (K) at raw inputs (offset along the track, across it, depth, power, speed), a tensor."""
    xi, dy, dz, power, speed = raw.unbind(1)
    r = torch.sqrt(xi * xi + dy * dy + dz * dz).clamp_min(1e-9)
    q = spec["absorptivity"] * power / (2.0 * math.pi * spec["conductivity"] * r)
    return (spec["t0"] + q * torch.exp(-(speed * (r + xi)) / (2.0 * spec["diffusivity"]))).clamp_max(spec["t_cap"])


def _points(spec, n, seed):
    """n raw inputs over the model's window, half of them around the melt pool where users look, as float32."""
    rng = np.random.default_rng(seed)
    raw = np.empty((n, 5), np.float32)
    near = rng.random(n) < 0.5
    for a in range(3):
        u = rng.random(n)
        lo, hi = spec["window_lo"][a], spec["window_hi"][a]
        nlo, nhi = spec["near_lo"][a], spec["near_hi"][a]
        raw[:, a] = np.where(near, nlo + (nhi - nlo) * u, lo + (hi - lo) * u)
    raw[:, 3] = rng.uniform(spec["power_lo"], spec["power_hi"], n)
    raw[:, 4] = rng.uniform(spec["speed_lo"], spec["speed_hi"], n)
    return raw


def _layers(p):
    """The parameter vector as [(W, b)] of the hidden layers and the head."""
    out, o = [], 0
    for rows, cols in [(HIDDEN, 2 * FREQ)] + [(HIDDEN, HIDDEN)] * (LAYERS - 1) + [(2, HIDDEN)]:
        out.append((p[o:o + rows * cols].reshape(rows, cols), p[o + rows * cols:o + rows * cols + rows]))
        o += rows * cols + rows
    return out


def _network(p, raw, enc):
    """(mu, log error) of the network in plain torch, in the type of p."""
    f, shift, scale = (torch.as_tensor(v, dtype=p.dtype, device=p.device) for v in enc)
    phase = 2.0 * math.pi * (((raw - shift) * scale) @ f.T)
    x = torch.cat([torch.sin(phase), torch.cos(phase)], 1)
    ls = _layers(p)
    for w, b in ls[:-1]:
        x = torch.nn.functional.silu(x @ w.T + b)
    y = x @ ls[-1][0].T + ls[-1][1]
    return y[:, 0], y[:, 1].clamp(-12.0, 4.0)


def _loss(p, raw, y, enc):
    """The model's training loss: squared error of mu, and the error head's likelihood with mu held."""
    mu, s = _network(p, raw, enc)
    r = (mu - y).detach()
    return (0.5 * (mu - y) ** 2 + 0.1 * (s + 0.5 * torch.exp(-2.0 * s) * r * r)).mean()


def _fitted(spec, seed, steps=240, batch=4096):
    """Parameters (float32) of a model fitted to the FE field in plain torch: what a saved model of a user holds."""
    enc = _encoding(spec)
    rng = np.random.default_rng(seed + 7)
    parts = []
    for rows, cols in [(HIDDEN, 2 * FREQ)] + [(HIDDEN, HIDDEN)] * (LAYERS - 1) + [(2, HIDDEN)]:
        k = math.sqrt(6.0 / (rows + cols)) * (0.1 if rows == 2 else 1.0)
        parts += [rng.uniform(-k, k, rows * cols), np.array([0.0, -2.0]) if rows == 2 else np.zeros(rows)]
    p = torch.tensor(np.concatenate(parts), dtype=torch.float32, device="cuda", requires_grad=True)
    raw = torch.tensor(_points(spec, batch * 32, seed + 8), device="cuda")
    y = (_field(spec, raw) - spec["t_shift"]) / spec["t_scale"]
    opt = torch.optim.Adam([p], lr=2e-3)
    for k in range(steps):
        for g in opt.param_groups:
            g["lr"] = 1e-5 + 2e-3 * 0.5 * (1.0 + math.cos(math.pi * k / steps))
        b = slice((k % 32) * batch, (k % 32 + 1) * batch)
        opt.zero_grad()
        _loss(p, raw[b], y[b], enc).backward()
        opt.step()
    return p.detach().cpu().numpy()


def _model(spec, params=None):
    m = amca.ThermalModel(**spec)
    if params is not None:
        m.set_params(params)
    return m


def _batch_of(c, seed):
    spec = decks.thermal_spec(seed=_seed(seed))
    raw = _points(spec, c["batch"], seed)
    y = (_field(spec, torch.tensor(raw, dtype=torch.float64)) - spec["t_shift"]) / spec["t_scale"]
    return spec, raw, y.numpy().astype(np.float32)


# --- the five functions ------------------------------------------------------------------------------------------------------
def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind == "plain":
        deck = _plain_deck(c, _seed(seed))
        realm = amca.CellularAutomataRealm(deck.to_yaml(), seed=deck.seed)
        realm.initialize()
        return {"case": c, "realm": realm, "out": _outputs_for(realm, ("orientation_id", "grain_id"))}
    if kind == "batch":
        realms = []  # edges, cooling rates and site densities are the study's own; the seeds place the sites
        for k, d in enumerate(decks.batched_instances(c["count"], c["sizes"], edges=(c["edge_lo"], c["edge_hi"]))):
            r = amca.CellularAutomataRealm(d.to_yaml(), seed=_seed(seed) + k)
            r.initialize()
            realms.append(r)
        return {"case": c, "realms": realms, "batch": amca.Batch(realms), "out": [_outputs_for(r, ("orientation_id",)) for r in realms]}
    if kind == "track":
        deck, realm = _remelt_realm(c, seed)
        realm.set_rosenthal_frames(**decks.pbf_frames(deck.cells, deck.cell_size, c["frames"]).rosenthal_kwargs())
        realm.initialize()
        return {"case": c, "realm": realm, "out": _outputs_for(realm, REMELT_FIELDS)}
    if kind == "coupled":
        deck, realm = _remelt_realm(c, seed)
        frames = decks.pbf_frames(deck.cells, deck.cell_size, 4)
        realm.set_rosenthal_frames(**frames.rosenthal_kwargs())  # the node grid; their values are replaced before each step
        realm.initialize()
        # the melt pool's tail, 0.45 mm behind the source, leaves the first part of the block; the source moves 0.5 um between two steps
        frames.source.x_start = 0.15 * c["nx"] * deck.cell_size + 4.5e-4
        frames.frame_dt = 5.0e-7
        return {"case": c, "realm": realm, "theta": [frames.frame_values(k) for k in range(c["steps"])],
                "out": _outputs_for(realm, REMELT_FIELDS)}
    spec = decks.thermal_spec(seed=_seed(seed))
    if kind == "raster":
        deck, realm = _remelt_realm(c, seed)
        scan = decks.scan_of(deck.cells, deck.cell_size, tracks=c["tracks"], hatch=4.0e-5, margin_end=2.0e-4)
        model = _model(spec, _fitted(spec, seed))
        realm.set_thermal_frames(model, LIQUIDUS, BAND, THRESHOLD, **scan)
        realm.initialize()
        return {"case": c, "realm": realm, "model": model, "out": _outputs_for(realm, REMELT_FIELDS)}
    if kind == "evaluate":
        return {"case": c, "model": _model(spec, _fitted(spec, seed)), "raw": _points(spec, c["points"], seed)}
    if kind == "gradients":
        spec, raw, y = _batch_of(c, seed)
        return {"case": c, "model": _model(spec, _fitted(spec, seed, steps=40)), "raw": raw, "target": y}
    return {"case": c, "model": _model(spec, _fitted(spec, seed, steps=40))}


def _fields(realm, out):
    for name, a in out.items():
        realm.field(name, out=a)
    return dict(out)


def run(state):
    c, kind = state["case"], state["case"]["kind"]
    if kind == "plain":
        realm = state["realm"]
        realm.reset()
        if c["steps"]:
            dt = [realm.single_integration_step() for _ in range(c["steps"])]
        else:
            realm.run()
            dt = []
        return {**_fields(realm, state["out"]), "dt": np.array(dt, np.float64), "liquid": realm.stats()["liquid_cells"]}
    if kind == "batch":
        state["batch"].run()
        out = [_fields(r, o)["orientation_id"] for r, o in zip(state["realms"], state["out"])]
        return {"orientation_id": out, "steps": np.array([r.stats()["step"] for r in state["realms"]], np.int64)}
    if kind in ("track", "raster"):
        realm = state["realm"]
        realm.reset()
        realm.run()
        s = realm.stats()
        return {**_fields(realm, state["out"]), "step": s["step"], "time": s["time"]}
    if kind == "coupled":
        realm = state["realm"]
        realm.reset()
        dt = []
        for theta in state["theta"]:
            realm.set_nodal_temperatures(theta)
            dt.append(realm.step_coupled(5.0e-7))
        return {**_fields(realm, state["out"]), "dt": np.array(dt, np.float64)}
    if kind == "evaluate":
        t, e = state["model"].eval(state["raw"])
        return {"temperature": t, "error": e}
    if kind == "gradients":
        g, pred = state["model"].gradients(state["raw"], state["target"])
        return {"gradient": g, "prediction": pred}
    st = state["model"].train(samples=c["samples"], steps=c["steps"], batch=c["batch"])
    return {"params": state["model"].params(), "loss": np.array([st["first_loss"], st["last_loss"]], np.float64)}


def _query_flops():
    return 2.0 * (HIDDEN * 2 * FREQ + (LAYERS - 1) * HIDDEN * HIDDEN + 2 * HIDDEN)


def _param_count():
    return HIDDEN * 2 * FREQ + (LAYERS - 1) * HIDDEN * HIDDEN + LAYERS * HIDDEN + 2 * HIDDEN + 2


def _window_nodes(c):
    """FE nodes inside the learned model's window, summed over the frames of a raster case."""
    spec = decks.thermal_spec()
    scan = decks.scan_of(_cells(c), 2.0e-6, tracks=c["tracks"], hatch=4.0e-5, margin_end=2.0e-4)
    axes = [scan["origin"][a] + scan["spacing"] * np.arange(scan["nodes"][a]) for a in range(3)]
    nz = np.sum((axes[2] >= scan["z_top"] - spec["window_hi"][2]) & (axes[2] <= scan["z_top"] - spec["window_lo"][2]))
    total = 0
    for f in range(scan["frames"]):
        t = f * scan["frame_dt"]
        k = min(int(t / scan["track_time"]), c["tracks"] - 1)
        along = scan["speed"] * (t - k * scan["track_time"])
        xi = (axes[0] - (scan["x_start"] + along)) if k % 2 == 0 else ((scan["x_turn"] - along) - axes[0])
        dy = axes[1] - (scan["y_line"] + k * scan["hatch"])
        total += int(np.sum((xi >= spec["window_lo"][0]) & (xi <= spec["window_hi"][0]))
                     * np.sum((dy >= spec["window_lo"][1]) & (dy <= spec["window_hi"][1])) * nz)
    return total


def work(case):
    c, kind = case, case["kind"]
    if kind == "plain":
        # sites (cell, threshold, orientation) in, two fields out
        return {"bytes": 8.0 * _ghost_cells(c) + 36.0 * (c["bulk"] + c["surface"]), "flops": 0.0}
    if kind == "batch":
        studied = decks.batched_instances(c["count"], c["sizes"], edges=(c["edge_lo"], c["edge_hi"]))
        sites = [d.bulk[0] * d.cell_size ** 3 * d.n_interior for d in studied]
        return {"bytes": sum(4.0 * d.n_ghost + 36.0 * s for d, s in zip(studied, sites)), "flops": 0.0}
    if kind in ("track", "coupled", "raster"):
        nodes = float(np.prod(decks.pbf_frames(_cells(c), 2.0e-6, 4).nodes))
        frames = {"track": c.get("frames", 0), "coupled": c.get("steps", 0), "raster": 0}[kind]
        flops = _query_flops() * _window_nodes(c) if kind == "raster" else 0.0
        # baseplate in (grain and orientation of each cell), frames in, four fields out
        return {"bytes": (8.0 + 17.0) * _ghost_cells(c) + 8.0 * nodes * frames, "flops": flops}
    if kind == "evaluate":
        return {"bytes": 28.0 * c["points"] + 2.0 * _param_count(), "flops": _query_flops() * c["points"]}
    if kind == "gradients":
        return {"bytes": 32.0 * c["batch"] + 8.0 * _param_count(), "flops": 3.0 * _query_flops() * c["batch"]}
    return {"bytes": c["steps"] * (24.0 * c["batch"] + 24.0 * _param_count()), "flops": c["steps"] * 3.0 * _query_flops() * c["batch"]}


def exact(case, seed):
    """The learned model's values in 64 bits. The realms' outputs are whole numbers, or temperatures and times that follow from a
    whole run of the reference's own order of operations, and have no such value."""
    c, kind = case, case["kind"]
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if kind == "evaluate":
        spec = decks.thermal_spec(seed=_seed(seed))
        p = torch.tensor(_fitted(spec, seed), dtype=torch.float64, device=dev)
        raw = torch.tensor(_points(spec, c["points"], seed), dtype=torch.float64, device=dev)
        t, e = [], []
        for part in raw.split(65536):
            mu, s = _network(p, part, _encoding(spec))
            t.append(spec["t_shift"] + spec["t_scale"] * mu)
            e.append(2.0 * spec["t_scale"] * torch.exp(s))
        return {"temperature": torch.cat(t), "error": torch.cat(e)}
    if kind == "gradients":
        spec, raw, y = _batch_of(c, seed)
        p = torch.tensor(_fitted(spec, seed, steps=40), dtype=torch.float64, device=dev, requires_grad=True)
        raw, y = (torch.tensor(v, dtype=torch.float64, device=dev) for v in (raw, y))
        pred = []
        for part, target in zip(raw.split(16384), y.split(16384)):
            (_loss(p, part, target, _encoding(spec)) * (len(part) / len(raw))).backward()
            with torch.no_grad():
                pred.append(torch.stack(_network(p, part, _encoding(spec)), 1))
        return {"gradient": p.grad, "prediction": torch.cat(pred)}
    return None

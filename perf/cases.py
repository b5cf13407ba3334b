"""What a user of the framework has it do, as measurable cases.

Five kinds of calls, all through the Python host mirror of the C ABI:

  run       a single simulation (jet or droplet) advances a number of time
            steps and its fields are read back into page-locked host arrays,
            as a driver does between two outputs; with an interval, the
            divergence watchdog checks the run while it advances
  ensemble  a batch of independent droplet boxes advances together, then the
            fields of every box are read back
  snapshot  a fine jet advances and becomes training data of the learned
            closure: samples, feature statistics, initial network, loss
  train     Adam on minibatches of a resident data set, then the mean loss
            over the whole set
  gradient  the summed training gradient over many samples

`exact` restates each of them in 64 bits with plain torch and numpy.
"""
import math

import numpy as np
import torch

import phasefieldlbm_gb300 as pf

# sizes of the closure network 8 -> 32 -> 32 -> 1 in its parameter blob
_IN, _H = 8, 32
_PARAMS = _H * _IN + _H + _H * _H + _H + _H + 1
_STORAGE = {"fp32": pf.STORAGE_FP32, "fp16": pf.STORAGE_FP16, "bf16": pf.STORAGE_BF16, "fp64": pf.STORAGE_FP64}
_BYTES = {"fp32": 4, "fp16": 2, "bf16": 2, "fp64": 8}
_AVERAGES = ("avg_phi", "avg_ux", "avg_uy", "avg_uz", "avg_uxux", "avg_uyuy", "avg_uzuz", "avg_uxuy", "avg_uxuz",
             "avg_uyuz")
# node updates of the largest listed case
_MOST_UPDATES = 256 * 256 * 1024 * 20


def listed():
    return [
        # the benchmark workload: the FP32 D3Q27 jet, 100 steps between outputs
        {"name": "jet_d3q27", "kind": "run", "flow": "jet", "vs": 27, "storage": "fp32", "nx": 128, "ny": 128,
         "nz": 512, "diam": 16, "noise": "uniform", "averages": False, "closure": False, "watchdog": 0, "steps": 100},
        # production-size jet in 16-bit storage (the precision study's grid)
        {"name": "jet_fp16_large", "kind": "run", "flow": "jet", "vs": 19, "storage": "fp16", "nx": 256, "ny": 256,
         "nz": 1024, "diam": 32, "noise": "uniform", "averages": False, "closure": False, "watchdog": 0, "steps": 20},
        # the reference's own jet: what the command line runs when nothing is changed
        {"name": "jet_default", "kind": "run", "flow": "jet", "vs": 19, "storage": "fp32", "nx": 64, "ny": 64,
         "nz": 128, "diam": 10, "noise": "gaussian", "averages": False, "closure": False, "watchdog": 0, "steps": 100},
        # a droplet box of the reference's size, watched for divergence every 10 steps
        {"name": "droplet_default", "kind": "run", "flow": "droplet", "vs": 19, "storage": "fp32", "nx": 128,
         "ny": 128, "nz": 128, "diam": 70, "noise": "none", "averages": False, "closure": False, "watchdog": 10,
         "steps": 100},
        # the smallest calls: a small box stepped a few steps at a time by a host loop
        {"name": "droplet64", "kind": "run", "flow": "droplet", "vs": 19, "storage": "fp32", "nx": 64, "ny": 64,
         "nz": 64, "diam": 32, "noise": "none", "averages": False, "closure": False, "watchdog": 0, "steps": 5},
        # a grid chosen by geometry, not by alignment: odd extents in every direction
        {"name": "jet_odd", "kind": "run", "flow": "jet", "vs": 27, "storage": "fp32", "nx": 101, "ny": 93, "nz": 251,
         "diam": 14, "noise": "uniform", "averages": False, "closure": False, "watchdog": 0, "steps": 50},
        # the double-precision run that other precisions are judged against
        {"name": "jet_fp64", "kind": "run", "flow": "jet", "vs": 19, "storage": "fp64", "nx": 96, "ny": 96, "nz": 256,
         "diam": 16, "noise": "uniform", "averages": False, "closure": False, "watchdog": 0, "steps": 40},
        # turbulence statistics with the learned closure attached (the closure study's coarse run)
        {"name": "jet_closure", "kind": "run", "flow": "jet", "vs": 19, "storage": "fp32", "nx": 128, "ny": 128,
         "nz": 512, "diam": 16, "noise": "uniform", "averages": True, "closure": True, "watchdog": 0, "steps": 50},
        # the seeded droplet ensemble, as created (not autotuned)
        {"name": "ensemble", "kind": "ensemble", "vs": 19, "boxes": 32, "steps": 50},
        # one training snapshot of a fine run
        {"name": "snapshot", "kind": "snapshot", "storage": "fp32", "nx": 128, "ny": 128, "nz": 512, "diam": 16,
         "stride": 2, "steps": 10},
        # a stretch of closure training
        {"name": "train", "kind": "train", "samples": 1 << 20, "batch": 16384, "iterations": 100},
        # full-data gradient (convergence checks, external optimisers)
        {"name": "gradient", "kind": "gradient", "samples": 1 << 20},
    ]


def _spread(rng, lo, hi):
    """An integer of [lo, hi], uniform in its logarithm; odd ones among them."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(("run", "run", "run", "run", "run", "ensemble", "snapshot", "train", "gradient"))
    if kind == "ensemble":
        return {"kind": kind, "vs": rng.choice((19, 27)), "boxes": _spread(rng, 2, 32), "steps": _spread(rng, 10, 40)}
    if kind == "snapshot":
        nx, ny = (2 * rng.randint(16, 64) for _ in range(2))
        return {"kind": kind, "storage": rng.choice(("fp32", "fp16")), "nx": nx, "ny": ny, "nz": 2 * _spread(rng, 24, 256),
                "diam": 2 * rng.randint(4, min(nx, ny) // 4 - 1), "stride": rng.choice((1, 2, 3)),
                "steps": _spread(rng, 1, 20)}
    if kind == "train":
        return {"kind": kind, "samples": _spread(rng, 20000, 1 << 20), "batch": _spread(rng, 256, 32768),
                "iterations": _spread(rng, 10, 100)}
    if kind == "gradient":
        return {"kind": kind, "samples": _spread(rng, 1000, 1 << 20)}
    flow = rng.choice(("jet", "jet", "droplet"))
    storage = rng.choice(("fp32", "fp32", "fp32", "fp16", "bf16", "fp64"))
    vs = rng.choice((19, 27))
    most = 128 if storage == "fp64" else 224
    nx, ny = _spread(rng, 24, most), _spread(rng, 24, most)
    if rng.random() < 0.5:
        nx = max(32, nx // 16 * 16)
    nz = _spread(rng, 24, most * 2 if flow == "jet" else most)
    if flow == "droplet":
        diam = 2 * max(3, int(min(nx, ny, nz) * rng.uniform(0.15, 0.3)))
    else:
        diam = 2 * rng.randint(3, max(3, min(nx, ny) // 4 - 2))
    wide = storage in ("fp32", "fp64")
    closure = wide and flow == "jet" and vs == 19 and rng.random() < 0.25
    most_steps = min(100, max(2, (_MOST_UPDATES // 12 if closure or storage == "fp64" else _MOST_UPDATES // 4) // (nx * ny * nz)))
    return {"kind": kind, "flow": flow, "vs": vs, "storage": storage, "nx": nx, "ny": ny, "nz": nz, "diam": diam,
            "noise": "none" if flow == "droplet" else rng.choice(("uniform", "gaussian")),
            "averages": rng.random() < (0.7 if closure else 0.15), "closure": closure,
            "watchdog": rng.choice((0, 0, 0, 10)), "steps": _spread(rng, 1, most_steps)}


# ------------------------------------------------------------------ inputs
def _config(case, seed):
    jet = case.get("flow", "jet") == "jet"
    c = pf.config_reference(pf.CASE_JET if jet else pf.CASE_DROPLET,
                            pf.VS_D3Q27 if case.get("vs", 19) == 27 else pf.VS_D3Q19)
    c.nx, c.ny, c.nz, c.diam = case["nx"], case["ny"], case["nz"], case["diam"]
    c.radius = c.diam // 2
    c.storage = _STORAGE[case["storage"]]
    c.device = torch.cuda.current_device()
    if jet:
        # the benchmark jet: u = 0.05, We = 500, Re = 5000 (10000 for the closure study)
        c.reynolds_water = c.reynolds_oil = 10000.0 if case.get("closure") else 5000.0
        c.sigma = float(np.float32(c.u_inf) * np.float32(c.u_inf) * np.float32(c.diam) / np.float32(500.0))
        if case.get("noise", "uniform") == "uniform":
            c.gamma = 0.05
            c.inflow_noise, c.noise_amp, c.seed = pf.NOISE_UNIFORM_UZ, 0.05, seed % (1 << 32)
    else:
        c.droplet_x_stretch = 1.0
        c.tau, c.sigma, c.gamma = 0.6, 0.01, 0.05
    if case.get("averages"):
        c.flags = pf.FLAG_TIME_AVERAGE | pf.FLAG_REYNOLDS_MOMENTS
    return c


def _waves(rng, shape, count=3):
    """A smooth random field of `shape` with values within +-1: a few separable waves."""
    f = torch.zeros(shape, dtype=torch.float32, device="cuda")
    for _ in range(count):
        axis = []
        for n in shape:
            k, ph = rng.randint(1, 5), rng.uniform(0.0, 2.0 * math.pi)
            axis.append(torch.sin(2.0 * math.pi * k * torch.arange(n, device="cuda") / n + ph).float())
        f += (1.0 / count) * axis[0][:, None, None] * axis[1][None, :, None] * axis[2][None, None, :]
    return f


def _initial_fields(case, cfg, seed):
    """rho, u and phi of a flow that is under way: a wavy jet over the whole length, or a drop off the centre in a stirred
    box. float32, with the reference's ghost shell."""
    rng = np.random.RandomState((seed * 2654435761 + 12345) % (1 << 32))
    nz, ny, nx = shape = (int(cfg.nz), int(cfg.ny), int(cfg.nx))
    z, y, x = (torch.arange(n, device="cuda", dtype=torch.float32) for n in shape)
    dx, dy = (x - (nx - 1) / 2)[None, None, :], (y - (ny - 1) / 2)[None, :, None]
    amp = 0.02
    if cfg.flow_case == pf.CASE_JET:
        k, ph = 2.0 * math.pi * rng.randint(2, 6) / nz, rng.uniform(0.0, 2.0 * math.pi)
        bend = 0.15 * cfg.radius * torch.sin(k * z + ph)[:, None, None]
        r = torch.sqrt((dx - bend) ** 2 + dy ** 2)
        phi = 0.5 + 0.5 * torch.tanh(2.0 * (cfg.radius - r) / 4.0)
        uz = cfg.u_inf * phi
        amp = cfg.u_inf
    else:
        off = rng.uniform(-2.0, 2.0, 3)
        dz = (z - (nz - 1) / 2 - off[0])[:, None, None]
        r = torch.sqrt((dx - off[2]) ** 2 + (dy - off[1]) ** 2 + dz ** 2)
        phi = 0.5 + 0.5 * torch.tanh(2.0 * (cfg.radius - r) / 4.0)
        uz = torch.zeros_like(phi)
    fields = {"rho": 1.0 + 1e-3 * _waves(rng, shape), "ux": 0.1 * amp * _waves(rng, shape),
              "uy": 0.1 * amp * _waves(rng, shape), "uz": uz + 0.1 * amp * _waves(rng, shape), "phi": phi}
    inside = torch.zeros(shape, dtype=torch.bool, device="cuda")
    inside[1:-1, 1:-1, 1:-1] = True
    for name, f in fields.items():
        f[~inside] = 1.0 if name == "rho" else 0.0
    if cfg.flow_case == pf.CASE_JET:
        fields["phi"][0] = (dx[0] ** 2 + dy[0] ** 2 <= float(cfg.radius) ** 2).float()
    return fields


def _network(seed):
    """A closure network in its parameter blob: Glorot weights, the feature statistics of a jet, nu_t of a few 1e-4."""
    rng = np.random.RandomState(seed % (1 << 32))
    b = np.zeros(pf.MLP_BLOB, np.float32)
    o = _offsets()
    b[o["w1"]:o["b1"]] = rng.uniform(-0.4, 0.4, _H * _IN)
    b[o["w2"]:o["b2"]] = rng.uniform(-0.3, 0.3, _H * _H)
    b[o["w3"]:o["b3"]] = rng.uniform(-0.4, 0.4, _H)
    b[o["b3"]] = -0.5
    b[o["mean"] + 6], b[o["mean"] + 7] = 0.1, 0.01
    b[o["inv"]:o["scale"]] = [2e4, 2e4, 2e4, 2e4, 2e4, 2e4, 4.0, 30.0]
    b[o["scale"]], b[o["scale"] + 1] = 5e-4, 1.0
    return b


def _offsets():
    o, at = {}, 0
    for name, n in (("w1", _H * _IN), ("b1", _H), ("w2", _H * _H), ("b2", _H), ("w3", _H), ("b3", 1), ("mean", _IN),
                    ("inv", _IN), ("scale", 2)):
        o[name] = at
        at += n
    return o


def _samples(case, seed):
    """Features and targets as snapshots give them: stresses of a few 1e-5, phi in [0, 1], targets many of which are 0."""
    rng = np.random.RandomState((seed * 40503 + 977) % (1 << 32))
    n = case["samples"]
    x = rng.standard_normal((n, _IN)).astype(np.float32)
    x[:, :6] *= np.float32(3e-5)
    x[:, 6] = 0.5 + 0.5 * np.tanh(2.0 * x[:, 6])
    x[:, 7] = 0.1 * np.abs(x[:, 7])
    s = np.sqrt((x[:, :6] * np.float32(3e4)) ** 2 @ np.ones(6, np.float32))
    y = np.clip(4e-4 * (s - 1.5) * (0.5 + x[:, 6]), 0.0, 2e-3)
    return x, y.astype(np.float32)


def _host(shape, dtype):
    return torch.empty(shape, dtype=dtype, pin_memory=True).numpy()


def _run_outputs(case):
    names = ["rho", "ux", "uy", "uz", "phi"]
    return names + list(_AVERAGES) if case["averages"] else names


def _ensemble_configs(case, seed):
    """The repository's seeded ensemble (boxes, radii, physics), each drop moved and each box stirred by the seed."""
    cfgs = pf.ensemble_configs(case["boxes"], 2026, pf.VS_D3Q27 if case["vs"] == 27 else pf.VS_D3Q19)
    rng = np.random.RandomState(seed % (1 << 32))
    for k, c in enumerate(cfgs):
        for i in range(3):
            c.center_offset[i] += float(rng.uniform(-1.0, 1.0))
        c.seed = (seed * 1000 + k) % (1 << 32)
        c.device = torch.cuda.current_device()
    return cfgs


def prepare(case, seed):
    kind = case["kind"]
    if kind == "run" or kind == "snapshot":
        cfg = _config(case, seed)
        sim = pf.Simulation(cfg)
        for name, f in _initial_fields(case, cfg, seed).items():
            sim.set_initial_field(name, f.cpu().numpy())
        if kind == "snapshot":
            stride, nxc, nyc, nzc = case["stride"], case["nx"] // 2, case["ny"] // 2, case["nz"] // 2
            count = len(range(-(-2 // stride) * stride, nxc - 2, stride)) * len(
                range(-(-2 // stride) * stride, nyc - 2, stride)) * (nzc - 4)
            return {"kind": kind, "sim": sim, "steps": case["steps"], "stride": stride, "seed": seed % (1 << 31),
                    "closure": pf.Closure(count, torch.cuda.current_device())}
        if case["closure"]:
            sim.set_closure(_network(seed), 1.0)
        if case["watchdog"]:
            sim.set_watchdog(case["watchdog"])
        wide = case["storage"] == "fp64"
        out = {n: _host(sim.shape, torch.float64 if wide else torch.float32) for n in _run_outputs(case)}
        return {"kind": kind, "sim": sim, "steps": case["steps"], "out": out,
                "dtype": np.float64 if wide else np.float32, "watched": case["watchdog"] > 0}
    if kind == "ensemble":
        cfgs = _ensemble_configs(case, seed)
        return {"kind": kind, "ens": pf.Ensemble(cfgs), "boxes": len(cfgs), "steps": case["steps"]}
    x, y = _samples(case, seed)
    closure = pf.Closure(case["samples"], torch.cuda.current_device())
    closure.set_samples(x, y)
    closure.init_params(seed % (1 << 31))
    return {"kind": kind, "closure": closure, "case": case, "seed": seed % (1 << 31)}


def run(state):
    kind = state["kind"]
    if kind == "run":
        sim = state["sim"]
        sim.step(state["steps"])
        out = {n: sim.get_field(n, out=a, dtype=state["dtype"]) for n, a in state["out"].items()}
        if state["watched"]:
            d = sim.reduce()
            out["diag"] = [d.phi_mass, d.rho_mass, d.max_speed, d.rho_in, d.rho_out, int(d.nonfinite)]
        return out
    if kind == "ensemble":
        ens = state["ens"]
        ens.step(state["steps"])
        return [[ens.get_field(k, "phi"), ens.get_field(k, "uz")] for k in range(state["boxes"])]
    closure = state["closure"]
    if kind == "snapshot":
        state["sim"].step(state["steps"])
        closure.set_samples(np.empty((0, _IN), np.float32), np.empty(0, np.float32))  # a new data set
        closure.add_snapshot(state["sim"], state["stride"])
        closure.init_params(state["seed"])
        x, y = closure.samples()
        return {"x": x, "y": y, "blob": closure.blob, "loss": closure.loss()}
    case = state["case"]
    if kind == "train":
        history = closure.train(case["iterations"], case["batch"], 2e-3, state["seed"])
        return {"history": history, "blob": closure.blob, "loss": closure.loss()}
    g, loss = closure.gradient(case["samples"])
    return {"gradient": g, "loss": loss}


# -------------------------------------------------------------------- work
def _step_work(vs, storage, averages, closure):
    """Bytes and operations per node and time step: populations read and written once, phi read and written once (and the
    ten running averages), the arithmetic of the stencils, moments and collision."""
    s = _BYTES[storage]
    t = 8 if storage == "fp64" else 4
    b = 2 * vs * s + 2 * t + (20 * t if averages else 0)
    f = (700 if vs == 27 else 480) + (60 if averages else 0) + (2 * _PARAMS + 8 * 64 if closure else 0)
    return b, f


def work(case):
    kind = case["kind"]
    if kind in ("run", "snapshot"):
        n = case["nx"] * case["ny"] * case["nz"]
        b, f = _step_work(case.get("vs", 19), case["storage"], case.get("averages"), case.get("closure"))
        nbytes, flops = n * b * case["steps"], n * f * case["steps"]
        if kind == "run":
            nbytes += n * len(_run_outputs(case)) * (8 if case["storage"] == "fp64" else 4)
        else:
            m = (n // 8) // case["stride"] ** 2
            nbytes += n * 5 * 4 + m * (_IN + 1) * 4 * 2
            flops += n * 20 + m * 2 * _PARAMS
        return {"bytes": nbytes, "flops": flops}
    if kind == "ensemble":
        n = sum(c.nodes for c in _ensemble_configs(case, 0))
        b, f = _step_work(case["vs"], "fp32", False, False)
        return {"bytes": n * (b * case["steps"] + 8), "flops": n * f * case["steps"]}
    per = (_IN + 1) * 4
    if kind == "train":
        seen = case["iterations"] * case["batch"]
        return {"bytes": (seen + case["samples"]) * per, "flops": 6 * _PARAMS * seen + 2 * _PARAMS * case["samples"]}
    return {"bytes": case["samples"] * per, "flops": 6 * _PARAMS * case["samples"]}


# ------------------------------------------------------------------- exact
_C = [(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (1, 1, 0), (-1, -1, 0), (1, 0, 1),
      (-1, 0, -1), (0, 1, 1), (0, -1, -1), (1, -1, 0), (-1, 1, 0), (1, 0, -1), (-1, 0, 1), (0, 1, -1), (0, -1, 1),
      (1, 1, 1), (-1, -1, -1), (1, 1, -1), (-1, -1, 1), (1, -1, 1), (-1, 1, -1), (-1, 1, 1), (1, -1, -1)]
_W = {19: (1 / 3, 1 / 18, 1 / 36, 0.0), 27: (8 / 27, 2 / 27, 1 / 54, 1 / 216)}
_M32 = 0xFFFFFFFF


def _hash32(x):
    x = (x ^ (x >> 16)) & _M32
    x = (x * 0x7FEB352D) & _M32
    x = (x ^ (x >> 15)) & _M32
    x = (x * 0x846CA68B) & _M32
    return x ^ (x >> 16)


def _uniform(h):
    return (h.double() + 0.5) / 4294967296.0


def _key(salt, x, y, t):
    return (0x9E3779B9 ^ salt) ^ x ^ ((y * 0x85EBCA6B) & _M32) ^ ((t * 0xC2B2AE35) & _M32)


def _dot(c, v):
    """c . v for a lattice direction c; None when c = 0."""
    s = None
    for a in range(3):
        if c[a]:
            t = v[a] if c[a] > 0 else -v[a]
            s = t if s is None else s + t
    return s


class _Exact:
    """The time step in 64 bits on arrays of (boxes, z, y, x). `f` holds for each direction what arrives at the interior
    nodes; what nothing sends there (the jet's inlet plane outside the inlet) keeps its first value."""

    def __init__(self, cfgs, fields, q, blob=None, averages=False):
        c = cfgs[0]
        self.cfg, self.q, self.jet, self.t = c, q, c.flow_case == pf.CASE_JET, 0
        d = {"dtype": torch.float64, "device": "cuda"}
        per = lambda get: torch.tensor([float(get(b)) for b in cfgs], **d)[:, None, None, None]  # noqa: E731
        self.sigma, self.gamma = per(lambda b: b.sigma), per(lambda b: b.gamma)
        self.omega = None if self.jet else per(lambda b: 1.0 / (0.5 + 3.0 * ((float(b.tau) - 0.5) / 3.0)))
        self.w = [_W[q][sum(map(abs, c_))] for c_ in _C[:q]]
        nz, ny, nx = (int(n) for n in (c.nz, c.ny, c.nx))
        self.inner = (slice(None), slice(1, nz - 1), slice(1, ny - 1), slice(1, nx - 1))
        self.shape = (len(cfgs), nz, ny, nx)
        self.phi = fields["phi"].clone()
        self.macro = {k: fields[k].clone() for k in ("rho", "ux", "uy", "uz", "phi")}
        u = [fields[k][self.inner] for k in ("ux", "uy", "uz")]
        rho = fields["rho"][self.inner]
        self.f = [self._feq(i, rho, u) for i in range(q)]
        self.avg = [torch.zeros(self.shape, **d) for _ in _AVERAGES] if averages else None
        self.ind = None
        self.net = None if blob is None else _Net(blob, rounded=True)
        if self.jet:
            yy, xx = torch.meshgrid(torch.arange(ny, device="cuda"), torch.arange(nx, device="cuda"), indexing="ij")
            self.xx, self.yy = xx, yy
            self.disc = (xx - (nx - 1) / 2) ** 2 + (yy - (ny - 1) / 2) ** 2 <= float(c.radius) ** 2
            nu = [float(c.u_inf) * float(c.diam) / float(r) for r in (c.reynolds_water, c.reynolds_oil)]
            self.nu, self.kg = nu, 1.0 + float(c.sponge_gain)
            cells = c.sponge_cells if c.sponge_cells >= 0 else nz // 12
            zn = torch.arange(1, nz - 1, **d) / (nz - 1)
            s = ((zn - (nz - 1 - cells) / (nz - 1)) * ((nz - 1) / max(cells, 1))).clamp(0.0, 1.0)
            self.ramp = (s * s * (3.0 - 2.0 * s))[None, :, None, None]

    def _feq(self, i, rho, u):
        w, uu = self.w[i], 1.5 * (u[0] * u[0] + u[1] * u[1] + u[2] * u[2])
        cu = _dot(_C[i], u)
        if cu is None:
            return w * rho * (1.0 - uu) - w
        cu = 3.0 * cu
        e = 1.0 - uu + cu + 0.5 * cu * cu
        if self.q == 27:
            e = e + cu * cu * cu / 6.0 - uu * cu
        return w * rho * e - w

    def _fneq(self, i, u, p):
        c, s = _C[i], 0.0
        for k, (a, b) in enumerate(((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))):
            if c[a] * c[b]:
                s = s + (1 if a == b else 2) * c[a] * c[b] * p[k]
        if self.q == 27:
            pxx, pyy, pzz, pxy, pxz, pyz = p
            ux, uy, uz = u
            third = ((c[1] * (3 * c[0] ** 2 - 1), lambda: pxx * uy + 2 * ux * pxy),
                     (c[2] * (3 * c[0] ** 2 - 1), lambda: pxx * uz + 2 * ux * pxz),
                     (c[0] * (3 * c[1] ** 2 - 1), lambda: pyy * ux + 2 * uy * pxy),
                     (c[2] * (3 * c[1] ** 2 - 1), lambda: pyy * uz + 2 * uy * pyz),
                     (c[0] * (3 * c[2] ** 2 - 1), lambda: pzz * ux + 2 * uz * pxz),
                     (c[1] * (3 * c[2] ** 2 - 1), lambda: pzz * uy + 2 * uz * pyz),
                     (c[0] * c[1] * c[2], lambda: 6 * (ux * pyz + uy * pxz + uz * pxy)))
            for a, h in third:
                if a:
                    s = s + a * h()
        return 4.5 * self.w[i] * s

    def _force(self, i, u, force):
        c = _C[i]
        uf = u[0] * force[0] + u[1] * force[1] + u[2] * force[2]
        cf = _dot(c, force)
        if cf is None:
            return -3.0 * self.w[i] * uf
        return 3.0 * self.w[i] * (cf - uf + 3.0 * _dot(c, u) * cf)

    def _shift(self, a, c):
        """`a` at the interior nodes' neighbours in direction c."""
        _, nz, ny, nx = self.shape
        return a[:, 1 + c[2]:nz - 1 + c[2], 1 + c[1]:ny - 1 + c[1], 1 + c[0]:nx - 1 + c[0]]

    def _gradient(self, a, axis):
        s = 0.0
        for i in range(1, self.q):
            if _C[i][axis]:
                s = s + self.w[i] * _C[i][axis] * self._shift(a, _C[i])
        return 3.0 * s

    def _inlet(self, t):
        """The inlet velocity at every ghost column."""
        c = self.cfg
        if c.inflow_noise == pf.NOISE_GAUSSIAN_UXY:
            sd, u = float(np.float32(c.noise_amp) * np.float32(c.u_inf)), []
            for salt in (0xA341316C, 0xC8013EA4):
                k = _key(salt, self.xx, self.yy, t)
                r = torch.sqrt(-2.0 * torch.log(_uniform(_hash32(k)).clamp(min=1e-12)))
                u.append(sd * r * torch.cos(2.0 * math.pi * _uniform(_hash32(k ^ 0x68BC21EB))))
            return [*u, torch.full_like(u[0], float(c.u_inf))]
        xi = 2.0 * _uniform(_hash32(_key(0x2545F491 ^ c.seed, self.xx, self.yy, t))) - 1.0
        return [torch.zeros_like(xi), torch.zeros_like(xi), float(c.u_inf) * (1.0 + float(c.noise_amp) * xi)]

    def step(self):
        I, q, t = self.inner, self.q, self.t
        # interface normals, curvature and force
        g = [self._gradient(self.phi, a) for a in range(3)]
        ind = torch.sqrt(g[0] * g[0] + g[1] * g[1] + g[2] * g[2])
        n = []
        for a in range(3):
            full = torch.zeros(self.shape, dtype=torch.float64, device="cuda")
            full[I] = g[a] / (ind + 1e-9)
            n.append(full)
        kappa = sum(self._gradient(n[a], a) for a in range(3))
        n = [a[I] for a in n]
        force = [-self.sigma * kappa * ind * a for a in n]
        # moments
        rho, j, m = 1.0, [0.0] * 3, [0.0] * 6
        pairs = ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))
        for i in range(q):
            c = _C[i]
            rho = rho + self.f[i]
            for a in range(3):
                if c[a]:
                    j[a] = j[a] + c[a] * self.f[i]
            for k, (a, b) in enumerate(pairs):
                if c[a] * c[b]:
                    m[k] = m[k] + c[a] * c[b] * self.f[i]
        u = [(j[a] + 0.5 * force[a]) / rho for a in range(3)]
        p = [m[k] - rho * u[a] * u[b] + 0.5 * (u[a] * force[b] + u[b] * force[a]) for k, (a, b) in enumerate(pairs)]
        trace = (p[0] + p[1] + p[2]) / 3.0
        p = [p[k] - trace if k < 3 else p[k] for k in range(6)]
        del j, m, g, kappa
        phi = self.phi[I]
        nu_t = self.net(torch.stack([*p, phi, ind], -1)) if self.net else 0.0
        if self.jet:
            tau = (1.0 - phi) * (0.5 + 3.0 * self.nu[0]) + phi * (0.5 + 3.0 * self.nu[1]) + 3.0 * nu_t
            tau_out = 0.5 + 3.0 * (((1.0 - phi) * self.nu[0] + phi * self.nu[1]) * self.kg)
            omega = 1.0 / (tau + self.ramp * (tau_out - tau))
        else:
            omega = 1.0 / (1.0 / self.omega + 3.0 * nu_t)
        if self.jet:
            inlet = self._inlet(t)
            mid, last = (slice(None), slice(0, 1)), (slice(None), slice(-1, None))
        # collision, then what arrives where
        for i in range(q):
            c = _C[i]
            v = self._feq(i, rho, u) + (1.0 - omega) * self._fneq(i, u, p) + 0.5 * self._force(i, u, force)
            v = torch.roll(v, (c[2], c[1], c[0]), (1, 2, 3))
            if self.jet and c[2] == 1:
                kept = self.f[i][mid].clone()
                # inflow: equilibrium of the inlet state, this node's non-equilibrium
                nz, ny, nx = self.shape[1:]
                src = (slice(1 - c[1], ny - 1 - c[1]), slice(1 - c[0], nx - 1 - c[0]))
                one = torch.ones((), dtype=torch.float64, device="cuda")
                eq = self._feq(i, one, [a[src] for a in inlet])
                om = 1.0 - 1.0 / (0.5 + 3.0 * self.nu[1])
                ne = self._fneq(i, [a[mid] for a in u], [a[mid] for a in p])
                v[mid] = torch.where(self.disc[src], eq + om * ne, kept)
            elif self.jet and c[2] == -1:
                # outflow: equilibrium of the column it comes from, this node's non-equilibrium and force
                back = lambda a: torch.roll(a[last], (c[1], c[0]), (2, 3))  # noqa: E731
                ub, pb = [back(a) for a in u], back(phi)
                om = 1.0 - 1.0 / (0.5 + 3.0 * (((1.0 - pb) * self.nu[0] + pb * self.nu[1]) * self.kg))
                v[last] = (self._feq(i, back(rho), ub) + om * self._fneq(i, [a[last] for a in u], [a[last] for a in p]) +
                           0.5 * self._force(i, ub, [a[last] for a in force]))
            self.f[i] = v
        # averages
        if self.avg is not None:
            now = [phi, *u] + [u[a] * u[b] for a, b in pairs]
            gate = [torch.ones_like(inlet[0]), *inlet] + [inlet[a] * inlet[b] for a, b in pairs] if self.jet else None
            for k, a in enumerate(self.avg):
                a[I] += (now[k] - a[I]) / (t + 1)
                if self.jet:
                    a[:, 0] = torch.where(self.disc, a[:, 0] + (gate[k] - a[:, 0]) / (t + 1), a[:, 0])
                    a[:, -1, 1:-1, 1:-1] = a[:, -2, 1:-1, 1:-1]
        # phase field
        sharp = self.gamma * phi * (1.0 - phi)
        flux = [4.0 * phi * u[a] + sharp * n[a] for a in range(3)]
        s = 0.25 * phi
        for a in range(3):
            for sign in (1, -1):
                v = torch.roll(0.125 * (phi + sign * flux[a]), sign, 3 - a)
                if self.jet and a == 2 and sign > 0:
                    uz = inlet[2] if self.cfg.inflow_noise == pf.NOISE_UNIFORM_UZ else torch.full_like(
                        inlet[2], float(self.cfg.u_inf))
                    v[:, 0] = torch.where(self.disc, 0.125 * (1.0 + 4.0 * uz), torch.zeros_like(uz))[1:-1, 1:-1]
                elif self.jet and a == 2:
                    v[:, -1] = 0.125 * phi[:, -1] * (1.0 - 4.0 * u[2][:, -1])
                s = s + v
        # the arrays as they stand after this step
        out = {"rho": torch.ones(self.shape, dtype=torch.float64, device="cuda")}
        for k in ("ux", "uy", "uz", "phi"):
            out[k] = torch.zeros(self.shape, dtype=torch.float64, device="cuda")
        for k, a in zip(("rho", "ux", "uy", "uz", "phi"), (rho, *u, phi)):
            out[k][I] = a
            if self.jet:
                out[k][:, -1, 1:-1, 1:-1] = out[k][:, -2, 1:-1, 1:-1]
        if self.jet:
            for k, a in zip(("ux", "uy", "uz", "phi"), (*inlet, torch.ones_like(inlet[0]))):
                out[k][:, 0] = torch.where(self.disc, a, torch.zeros_like(a))
        self.macro, self.ind = out, ind
        if self.jet:
            self.phi[:, -1, 1:-1, 1:-1] = phi[:, -1]
        self.phi[I] = s
        self.t += 1


class _Net:
    """The closure network, its forward pass in 64 bits; `rounded`: with the bfloat16 weights that a simulation runs."""

    def __init__(self, blob, rounded=False):
        b = np.array(blob, np.float32)
        if rounded:
            b[:_PARAMS] = pf.bf16_round(b[:_PARAMS])
        o, b = _offsets(), torch.tensor(b, dtype=torch.float64, device="cuda")
        self.p = [b[o["w1"]:o["b1"]].reshape(_H, _IN), b[o["b1"]:o["w2"]], b[o["w2"]:o["b2"]].reshape(_H, _H),
                  b[o["b2"]:o["w3"]], b[o["w3"]:o["b3"]], b[o["b3"]:o["b3"] + 1]]
        self.mean, self.inv, self.scale = b[o["mean"]:o["inv"]], b[o["inv"]:o["scale"]], b[o["scale"]]

    def relative(self, x):
        w1, b1, w2, b2, w3, b3 = self.p
        h = torch.nn.functional.silu((x - self.mean) * self.inv @ w1.T + b1)
        h = torch.nn.functional.silu(h @ w2.T + b2)
        z = h @ w3 + b3
        return torch.clamp(z, min=0.0) + torch.log1p(torch.exp(-z.abs()))

    def __call__(self, x):
        parts = [self.relative(c) for c in x.reshape(-1, _IN).split(1 << 21)]
        return self.scale * torch.cat(parts).reshape(x.shape[:-1])

    def loss_sum(self, x, y):
        return sum(((self.relative(a) - b / self.scale) ** 2).sum() for a, b in zip(x.split(1 << 21), y.split(1 << 21)))


def _mix64(x):
    with np.errstate(over="ignore"):
        x = (x ^ (x >> np.uint64(30))) * np.uint64(0xbf58476d1ce4e5b9)
        x = (x ^ (x >> np.uint64(27))) * np.uint64(0x94d049bb133111eb)
        return x ^ (x >> np.uint64(31))


def _first_network(x, y, seed):
    """The network that init_params makes from the data, as a blob in 64 bits."""
    o, b = _offsets(), np.zeros(pf.MLP_BLOB)
    x, y = x.double(), y.double()
    mean, var = x.mean(0), x.var(0, unbiased=False)
    b[o["mean"]:o["inv"]] = mean.cpu().numpy()
    b[o["inv"]:o["scale"]] = torch.where(var > 1e-30, var.rsqrt(), torch.ones_like(var)).cpu().numpy()
    rms = float(y.square().mean().sqrt())
    scale = rms if rms > 1e-30 else 1.0
    b[o["scale"]], b[o["scale"] + 1] = scale, 1.0

    def uniform(first, n):
        with np.errstate(over="ignore"):
            k = np.uint64(seed) * np.uint64(0x9E3779B97F4A7C15) + np.arange(first, first + n, dtype=np.uint64)
        return (_mix64(k) >> np.uint64(11)).astype(np.float64) * 2.0 ** -53

    b[o["w1"]:o["b1"]] = math.sqrt(6 / (_IN + _H)) * (2 * uniform(0, _H * _IN) - 1)
    b[o["w2"]:o["b2"]] = math.sqrt(6 / (2 * _H)) * (2 * uniform(10000, _H * _H) - 1)
    b[o["w3"]:o["b3"]] = math.sqrt(6 / (_H + 1)) * (2 * uniform(20000, _H) - 1)
    t0 = max(float(y.mean()) / scale, 1e-3)
    b[o["b3"]] = t0 if t0 > 20 else math.log(math.expm1(t0))
    return b


def _exact_training(case, seed):
    seed32 = seed % (1 << 31)
    x, y = (torch.from_numpy(a).cuda().double() for a in _samples(case, seed))
    blob = _first_network(x, y, seed32)
    net = _Net(blob)
    net.p = [p.clone().requires_grad_() for p in net.p]
    n = case["samples"]
    if case["kind"] == "gradient":
        total = 0.0
        for a, b in zip(x.split(1 << 19), y.split(1 << 19)):
            part = net.loss_sum(a, b)
            part.backward()
            total += float(part.detach())
        return {"gradient": torch.cat([p.grad.reshape(-1) for p in net.p]), "loss": total}
    m, v = [torch.zeros_like(p) for p in net.p], [torch.zeros_like(p) for p in net.p]
    history, batch = [], case["batch"]
    for t in range(1, case["iterations"] + 1):
        with np.errstate(over="ignore"):
            k = np.uint64(t) * np.uint64(0x100000001B3) + np.arange(batch, dtype=np.uint64)
            at = _mix64(np.uint64(seed32) * np.uint64(0x9E3779B97F4A7C15) + _mix64(k)) % np.uint64(n)
        at = torch.from_numpy(at.astype(np.int64)).cuda()
        loss = net.loss_sum(x[at], y[at]) / batch
        grads = torch.autograd.grad(loss, net.p)
        history.append(loss.detach())
        with torch.no_grad():
            for p, g, a, b in zip(net.p, grads, m, v):
                a.mul_(0.9).add_(g, alpha=0.1)
                b.mul_(0.999).add_(g * g, alpha=0.001)
                p -= 2e-3 * (a / (1 - 0.9 ** t)) / ((b / (1 - 0.999 ** t)).sqrt() + 1e-8)
    with torch.no_grad():
        loss = float(net.loss_sum(x, y)) / n
        o = _offsets()
        blob = torch.tensor(blob, device="cuda")
        blob[:o["mean"]] = torch.cat([p.reshape(-1) for p in net.p])
    return {"history": torch.stack(history), "blob": blob, "loss": loss}


def _exact_snapshot(case, cfg, sim, seed):
    """Training samples of the simulation's last step: box filter and restriction, sub-filter stress, targets."""
    nxc, nyc, nzc, stride = case["nx"] // 2, case["ny"] // 2, case["nz"] // 2, case["stride"]
    fine = {k: a[0] for k, a in sim.macro.items()}
    u = [fine[k] for k in ("ux", "uy", "uz")]
    pairs = ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))

    def filtered(a):
        for axis in range(3):
            n = a.shape[axis]
            at = torch.arange(0, n, 2, device="cuda")
            a = sum(a.index_select(axis, (at + d).clamp(0, n - 1)) for d in (-1, 0, 1)) / 3.0
        return a

    rho, phi, uc = filtered(fine["rho"]), filtered(fine["phi"]), [filtered(a) for a in u]
    tau = [filtered(u[a] * u[b]) - uc[a] * uc[b] for a, b in pairs]

    def inner(a, c=(0, 0, 0)):
        return a[2 + c[2]:nzc - 2 + c[2], 2 + c[1]:nyc - 2 + c[1], 2 + c[0]:nxc - 2 + c[0]]

    unit = ((1, 0, 0), (0, 1, 0), (0, 0, 1))
    g = [[0.5 * (inner(uc[b], unit[a]) - inner(uc[b], [-k for k in unit[a]])) for b in range(3)] for a in range(3)]
    s = [0.5 * (g[a][b] + g[b][a]) for a, b in pairs]
    tr = (s[0] + s[1] + s[2]) / 3.0
    nu = [float(cfg.u_inf) * float(cfg.diam) / float(r) for r in (cfg.reynolds_water, cfg.reynolds_oil)]
    ph = inner(phi)
    c = -2.0 * inner(rho) * ((1.0 - ph) * (0.5 + 3.0 * nu[0]) + ph * (0.5 + 3.0 * nu[1])) / 3.0
    w = _W[19]
    grad = [sum(w[sum(map(abs, d))] * d[a] * inner(phi, d) for d in _C[1:19] if d[a]) for a in range(3)]
    ind = 3.0 * torch.sqrt(grad[0] ** 2 + grad[1] ** 2 + grad[2] ** 2)
    t = [inner(a) for a in tau]
    ttr = (t[0] + t[1] + t[2]) / 3.0
    t = [a - ttr if k < 3 else a for k, a in enumerate(t)]
    two = (1, 1, 1, 2, 2, 2)
    num = -sum(k * a * b for k, a, b in zip(two, t, s))
    den = 2.0 * sum(k * b * b for k, b in zip(two, s))
    y = torch.where(den > 2e-10, (num / den).clamp(0.0, 2e-3), torch.zeros_like(den))
    feats = [c * (b - tr) if k < 3 else c * b for k, b in enumerate(s)] + [ph, ind]
    first = -(-2 // stride) * stride - 2
    pick = lambda a: a[:, first::stride, first::stride].reshape(-1)  # noqa: E731
    x, y = torch.stack([pick(a) for a in feats], -1), pick(y)
    blob = _first_network(x, y, seed % (1 << 31))
    loss = float(_Net(blob).loss_sum(x, y)) / len(y)
    return {"x": x, "y": y, "blob": torch.tensor(blob), "loss": loss}


def _diagnostics(m):
    inner = {k: a[0, 1:-1, 1:-1, 1:-1] for k, a in m.items()}
    rho, phi = inner["rho"], inner["phi"]
    speed = torch.sqrt(inner["ux"] ** 2 + inner["uy"] ** 2 + inner["uz"] ** 2).max()
    means = [float(rho[s].mean()) if bool(s.any()) else 0.0 for s in (phi > 0.9, phi < 0.1)]
    return [float(phi.sum()), float(rho.sum()), float(speed), *means, 0]


def _exact_ensemble(case, seed):
    cfgs = _ensemble_configs(case, seed)
    out = [None] * len(cfgs)
    for edge in sorted({int(c.nx) for c in cfgs}):
        at = [k for k, c in enumerate(cfgs) if int(c.nx) == edge]
        z, y, x = torch.meshgrid(*(torch.arange(edge, device="cuda"),) * 3, indexing="ij")
        inside = torch.zeros((edge,) * 3, dtype=torch.bool, device="cuda")
        inside[1:-1, 1:-1, 1:-1] = True
        fields = {k: [] for k in ("rho", "ux", "uy", "uz", "phi")}
        for c in (cfgs[k] for k in at):
            o = [(edge - 1) / 2 + float(v) for v in c.center_offset]
            r = torch.sqrt((x - o[0]) ** 2 + (y - o[1]) ** 2 + ((z - o[2]).double()) ** 2)
            fields["rho"].append(torch.ones_like(r))
            fields["phi"].append((0.5 + 0.5 * torch.tanh(2.0 * (c.radius - r) / float(c.interface_width))) * inside)
            for a, name in enumerate(("ux", "uy", "uz")):
                salt = 0x5851F42D ^ c.seed ^ ((a * 0x9E3779B9) & _M32)
                k = _key(salt, x, y, (z * 0x27D4EB2F) & _M32)
                fields[name].append(float(c.init_noise) * (2.0 * _uniform(_hash32(k)) - 1.0) * inside)
        sim = _Exact([cfgs[k] for k in at], {k: torch.stack(v) for k, v in fields.items()}, case["vs"])
        for _ in range(case["steps"]):
            sim.step()
        for i, k in enumerate(at):
            out[k] = [sim.macro["phi"][i], sim.macro["uz"][i]]
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind in ("train", "gradient"):
        return _exact_training(case, seed)
    if kind == "ensemble":
        return _exact_ensemble(case, seed)
    cfg = _config(case, seed)
    fields = {k: a.double()[None] for k, a in _initial_fields(case, cfg, seed).items()}
    blob = _network(seed) if case.get("closure") else None
    sim = _Exact([cfg], fields, case.get("vs", 19), blob, case.get("averages", False))
    for _ in range(case["steps"]):
        sim.step()
    if kind == "snapshot":
        return _exact_snapshot(case, cfg, sim, seed)
    out = {k: sim.macro[k][0] for k in ("rho", "ux", "uy", "uz", "phi")}
    if case["averages"]:
        out.update({k: a[0] for k, a in zip(_AVERAGES, sim.avg)})
    if case["watchdog"]:
        out["diag"] = _diagnostics(sim.macro)
    return out

"""Performance cases: what a user of this package has it do, through its public entry points.

* ``steps``: one engine advanced as the run loop does it: ``Gb300Engine.step`` for a chunk of time
  steps, the energy check, the running DFTs read back, and monitor planes of all six components
  (device to device) through the outer layers, the metal and the middle of the grid. The small
  box reads its whole fields back instead.
* ``sweep``: many instances with uneven grids stepped as one ``EngineBatch``, every instance's DFTs
  read back and one monitor plane each.
* ``epoch``: one epoch of the surrogate's training (``Mlp.run_epoch``, its captured steps), the
  weights after it.
* ``predict``: the surrogate's outputs for a set of parameter points (``Mlp.predict_device``).
* ``layer``: one hidden layer of every member, forward and backward (``oafdtd_mlp_gemm_tn``):
  activations, input gradients and weight gradients.

The engines start from seeded noise in every interior cell, so that each boundary layer, dispersive
edge and copper face is active from the first step.
"""

from __future__ import annotations

import functools
import math

import numpy as np
import torch

from open_analysis_gb300 import native
from open_analysis_gb300.batch import EngineBatch
from open_analysis_gb300.engine import Gb300Engine
from open_analysis_gb300.grid import Grid, uniform_lines
from open_analysis_gb300.model import LumpedPort, Model, Probe, Region, SoftSource, Waveform, compile_model
from open_analysis_gb300.pml import CpmlSpec
from open_analysis_gb300.structures import large_board, microstrip, sweep_instances, via_transition
from open_analysis_gb300.surrogate import HALF, Mlp, ViaGrid, via_instance, via_params

CHUNK = 64
EPS0 = 1.0 / (4e-7 * math.pi * 299792458.0**2)
MU0 = 4e-7 * math.pi


# ------------------------------------------------------------------------------------------ cases
def listed():
    return [
        # A small graded box with every kind of wall, a lossy slab and a lumped port: a unit check or
        # a resonance study, a few eager steps between field dumps. Launches and latency count.
        {"name": "box", "kind": "steps", "what": "box", "nx": 24, "ny": 20, "nz": 22, "steps": 16, "dtype": "float32"},
        # The plain 50-ohm microstrip as configured (both ports driven): a chunk between energy checks.
        {"name": "microstrip", "kind": "steps", "what": "microstrip", "nx": 120, "ny": 60, "nz": 40, "steps": CHUNK,
         "dtype": "float32"},
        # One via transition on the surrogate's own grid, one port driven, PEC walls in z.
        {"name": "via_single", "kind": "steps", "what": "via_single", "nx": 200, "ny": 200, "nz": 120, "steps": CHUNK,
         "dtype": "float32"},
        # The benchmark workload: two ports as a batch of two, Debye layers, copper faces, CPML.
        {"name": "via", "kind": "steps", "what": "via", "nx": 400, "ny": 400, "nz": 120, "steps": CHUNK,
         "dtype": "float32"},
        # A region of the large board at its full height: eight ports as a batch of eight, odd extents.
        {"name": "board", "kind": "steps", "what": "board", "nx": 397, "ny": 323, "nz": 160, "steps": CHUNK,
         "dtype": "float32"},
        # A convergence check of the via transition in float64, odd extents.
        {"name": "via_f64", "kind": "steps", "what": "via", "nx": 161, "ny": 143, "nz": 88, "steps": CHUNK,
         "dtype": "float64"},
        # A line on a causal broadband dielectric fitted with several Debye poles, with a PMC
        # symmetry wall.
        {"name": "broadband", "kind": "steps", "what": "broadband", "nx": 181, "ny": 90, "nz": 60, "steps": CHUNK,
         "dtype": "float32", "poles": 5},
        # A parameter sweep of microstrip and stripline instances with uneven grids, two ports each.
        {"name": "sweep", "kind": "sweep", "what": "lines", "n": 16, "first": 0, "steps": CHUNK, "dtype": "float32"},
        # A slice of the surrogate's training data: via transitions on its half grid, one port driven.
        {"name": "sweep_via", "kind": "sweep", "what": "vias", "n": 16, "first": 0, "steps": CHUNK, "dtype": "float32"},
        # One training epoch of the eight-member ensemble at the configured widths and batch.
        {"name": "epoch", "kind": "epoch", "members": 8, "width": 512, "depth": 6, "n_freq": 256, "batch": 256,
         "rows": 1100},
        # The ensemble answering the held-out tenth of a sweep.
        {"name": "predict", "kind": "predict", "members": 8, "width": 512, "depth": 6, "n_freq": 256, "rows": 412},
        # A hidden layer of the 32-member ensemble at the small sweep's batch, forward and backward.
        {"name": "layer", "kind": "layer", "members": 32, "width": 512, "batch": 64},
    ]


def _log(rng, lo, hi):
    """A whole number in lo..hi, spread evenly over its logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["box", "microstrip", "via_single", "via", "board", "via_f64", "broadband", "lines", "vias",
                       "epoch", "predict", "layer"])
    f32 = {"dtype": "float32"}
    if kind == "box":
        return {"kind": "steps", "what": "box", "nx": _log(rng, 18, 60), "ny": _log(rng, 14, 48),
                "nz": _log(rng, 14, 48), "steps": rng.randint(4, 40), **f32}
    if kind == "microstrip":
        return {"kind": "steps", "what": "microstrip", "nx": _log(rng, 60, 300), "ny": _log(rng, 40, 160),
                "nz": _log(rng, 28, 90), "steps": CHUNK, **f32}
    if kind == "via_single":
        return {"kind": "steps", "what": "via_single", "nx": _log(rng, 90, 220), "ny": _log(rng, 90, 220),
                "nz": rng.randint(118, 130), "steps": CHUNK, **f32}
    if kind == "via":
        return {"kind": "steps", "what": "via", "nx": _log(rng, 80, 400), "ny": _log(rng, 80, 400),
                "nz": _log(rng, 48, 120), "steps": CHUNK, **f32}
    if kind == "board":
        return {"kind": "steps", "what": "board", "nx": _log(rng, 140, 397), "ny": _log(rng, 140, 323),
                "nz": rng.randint(56, 160), "steps": CHUNK, **f32}
    if kind == "via_f64":
        return {"kind": "steps", "what": "via", "nx": _log(rng, 80, 200), "ny": _log(rng, 80, 200),
                "nz": _log(rng, 48, 100), "steps": CHUNK, "dtype": "float64"}
    if kind == "broadband":
        return {"kind": "steps", "what": "broadband", "nx": _log(rng, 80, 240), "ny": _log(rng, 50, 140),
                "nz": _log(rng, 40, 80), "steps": CHUNK, "poles": rng.randint(2, 8), **f32}
    if kind in ("lines", "vias"):
        return {"kind": "sweep", "what": kind, "n": _log(rng, 2, 20), "first": rng.randint(16, 40), "steps": CHUNK,
                **f32}
    net = {"members": rng.choice([1, 4, 8, 16, 32]), "width": rng.choice([256, 512])}
    if kind == "epoch":
        batch = rng.choice([64, 128, 256])
        return {"kind": "epoch", **net, "depth": rng.randint(3, 6), "n_freq": rng.choice([32, 64, 256]), "batch": batch,
                "rows": batch * rng.randint(1, 6) + rng.randint(0, batch - 1)}
    if kind == "predict":
        return {"kind": "predict", **net, "depth": rng.randint(3, 6), "n_freq": rng.choice([32, 64, 256]),
                "rows": _log(rng, 20, 4096)}
    return {"kind": "layer", **net, "batch": _log(rng, 32, 4096)}


# ------------------------------------------------------------------------------------- structures
def _graded(length, n, ratio):
    w = ratio ** np.arange(n)
    return np.concatenate([[0.0], np.cumsum(w) / w.sum() * length])


def _box(nx, ny, nz):
    """A graded box: CPML across x, PMC across y, PEC across z, a lossy slab with a PEC patch, a soft
    source, a lumped port, an E and an H probe; both sources driven."""
    d = 1e-3
    lx, ly, lz = nx * d, ny * d, nz * d
    g = Grid(_graded(lx, nx, 1.01), _graded(ly, ny, 1.0), _graded(lz, nz, 0.99))
    m = Model(g, Waveform("gauss_mod", 10e9, 20e9), np.array([2e9, 6e9, 10e9, 14e9]),
              walls=("cpml", "cpml", "pmc", "pmc", "pec", "pec"), cpml=CpmlSpec(cells=4))
    m.regions.append(Region((0, 0, 0.2 * lz), (lx, ly, 0.55 * lz), eps_r=4.4, sigma=0.02))
    m.regions.append(Region((0.35 * lx, 0.3 * ly, 0.55 * lz), (0.65 * lx, 0.7 * ly, 0.551 * lz), pec=True))
    m.sources.append(SoftSource("s", 2, (0.5 * lx, 0.5 * ly, 0.3 * lz), (0.5 * lx, 0.5 * ly, 0.3 * lz)))
    m.ports.append(LumpedPort("p", 2, (0.3 * lx, 0.5 * ly, 0.0), (0.3 * lx, 0.5 * ly, 0.2 * lz), 50.0))
    at = (0.65 * lx, 0.5 * ly, 0.1 * lz)
    m.probes.append(Probe("e", "E", 2, at, at))
    m.probes.append(Probe("h", "H", 1, at, at))
    m.drive = np.array([[1.0, 1.0], [0.0, -2.0]])
    return m


def _broadband(nx, ny, nz, poles):
    """A microstrip on a substrate with ``poles`` log-spaced Debye poles, a PMC wall at low y (half
    of a symmetric line), PEC ground, CPML elsewhere, both ports driven."""
    h = 50e-6
    g = Grid(uniform_lines(nx, h), uniform_lines(ny, h), uniform_lines(nz, h))
    m = Model(g, Waveform("gauss_mod", 10e9, 20e9), np.linspace(0.1e9, 20e9, 128),
              walls=("cpml", "cpml", "pmc", "cpml", "pec", "cpml"), cpml=CpmlSpec(cells=8, m=3.0, kappa_max=5.0))
    taus = 1.0 / (2 * math.pi * np.geomspace(1e7, 2e11, poles))
    sub = 8 * h
    m.regions.append(Region((-1, -1, 0.0), (1, 1, sub), 3.4, poles=tuple((0.5 / poles, float(t)) for t in taus)))
    x0, x1 = 12 * h, (nx - 12) * h
    m.regions.append(Region((x0, 0.0, sub), (x1, 4 * h, sub), pec=True))
    m.ports.append(LumpedPort("p1", 2, (x0, 2 * h, 0.0), (x0, 2 * h, sub), 50.0))
    m.ports.append(LumpedPort("p2", 2, (x1, 2 * h, 0.0), (x1, 2 * h, sub), 50.0))
    return m


def _models(case):
    what = case["what"]
    if what == "lines":
        return sweep_instances(case["first"] + case["n"])[case["first"]:]
    if what == "vias":
        return [via_instance(p, HALF) for p in via_params(case["first"] + case["n"])[case["first"]:]]
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    if what == "box":
        return [_box(nx, ny, nz)]
    if what == "microstrip":
        return [microstrip(nx, ny, nz)]
    if what == "via_single":
        return [via_instance(via_params(1)[0], ViaGrid(nx=nx, ny=ny, nz=nz))]
    if what == "via":
        return [via_transition(nx, ny, nz)]
    if what == "board":
        return [large_board(nx, ny, nz)]
    return [_broadband(nx, ny, nz, case["poles"])]


@functools.lru_cache(maxsize=1)
def _compiled_items(items):
    case = dict(items)
    return [compile_model(m, case["dtype"]) for m in _models(case)]


def _compiled(case):
    """The case's compiled problems (the structure does not depend on the seed)."""
    return _compiled_items(tuple(sorted((k, v) for k, v in case.items() if k != "name")))


def _noise(c, dtype, seed, device="cuda"):
    """Seeded noise in every interior cell, six fields ``(Z, B, Y, X)``: E of unit size, H as in a
    plane wave."""
    z, y, x = c.grid.shape
    nx, ny, nz = c.grid.n
    gen = torch.Generator(device=device)
    gen.manual_seed(int(seed))
    out = []
    for k in range(6):
        f = torch.zeros((z, c.batch, y, x), dtype=dtype, device=device)
        v = torch.randn((nz - 2, c.batch, ny - 2, nx - 2), generator=gen, dtype=torch.float32, device=device)
        f[2:nz, :, 2:ny, 2:nx] = (v if k < 3 else v / 376.73).to(dtype)
        out.append(f)
    return out


def _planes(c):
    """Monitor planes: inside the low and high outer layers, at the quarter points and the middle."""
    nz = c.grid.n[2]
    return sorted({3, nz // 4, nz // 2, (3 * nz) // 4, nz - 2})


def _engine(c, dtype, seed):
    eng = Gb300Engine(c, dtype)
    t = torch.float32 if dtype == "float32" else torch.float64
    for k, f in enumerate(_noise(c, t, seed)):
        torch.cuda.synchronize()
        for z in range(2, c.grid.n[2]):
            eng.plane_from_device(k, z, f[z].data_ptr())
    return eng


# ------------------------------------------------------------------------------------ surrogate data
def _net_arrays(case, seed):
    """Weights ``W[l] (members, fan_in, fan_out)`` and biases of every layer, FP32, and the rows."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    g = case["members"]
    sizes = [7] + [case["width"]] * case["depth"] + [4 * case["n_freq"]]
    w, b = [], []
    for a, n in zip(sizes[:-1], sizes[1:]):
        w.append(torch.randn((g, a, n), generator=gen, device="cuda") / math.sqrt(a))
        b.append(0.1 * torch.randn((g, n), generator=gen, device="cuda"))
    x = 2.0 * torch.rand((case["rows"], 7), generator=gen, device="cuda") - 1.0
    mix = torch.randn((7, sizes[-1]), generator=gen, device="cuda") / math.sqrt(7)
    t = torch.sin(2.0 * (x @ mix)) + 0.3 * torch.cos(x @ mix.flip(1))
    return sizes, w, b, x.cpu().numpy(), t.cpu().numpy()


def _net(case, seed, batch):
    sizes, w, b, x, t = _net_arrays(case, seed)
    net = Mlp(sizes, batch, seed=int(seed) % 100000, members=case["members"])
    flat = torch.zeros((case["members"], net.n_params), device="cuda")
    for (wo, a, n, bo), wl, bl in zip(net.layout, w, b):
        full = torch.zeros((case["members"], a, n), device="cuda")  # the first layer's padded inputs
        full[:, : wl.shape[1]] = wl
        flat[:, wo : wo + a * n] = full.reshape(case["members"], -1)
        flat[:, bo : bo + n] = bl
    net.load_flat(flat.reshape(-1))
    return net, x, t


def _layer_arrays(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    g, m, n = case["members"], case["batch"], case["width"]
    bf = torch.bfloat16
    x = torch.tanh(torch.randn((g, m, n), generator=gen, device="cuda")).to(bf)
    w = (torch.randn((g, n, n), generator=gen, device="cuda") / math.sqrt(n)).to(bf)
    bias = 0.1 * torch.randn((g, n), generator=gen, device="cuda")
    dy = (torch.randn((g, m, n), generator=gen, device="cuda") * 1e-3).to(bf)
    return x, w, bias, dy


# ------------------------------------------------------------------------------------ the interface
def prepare(case, seed):
    kind = case["kind"]
    if kind == "steps":
        c = _compiled(case)[0]
        eng = _engine(c, case["dtype"], seed)
        s = {"kind": kind, "eng": eng, "steps": case["steps"], "dump": case["what"] == "box", "at": _planes(c)}
        t = torch.float32 if case["dtype"] == "float32" else torch.float64
        z, y, x = c.grid.shape
        s["planes"] = torch.zeros((6, len(s["at"]), c.batch, y, x), dtype=t, device="cuda")
        return s
    if kind == "sweep":
        cs = _compiled(case)
        engines = [_engine(c, case["dtype"], seed + 1000 * i) for i, c in enumerate(cs)]
        t = torch.float32 if case["dtype"] == "float32" else torch.float64
        return {"kind": kind, "batch": EngineBatch(engines), "engines": engines, "steps": case["steps"],
                "at": [c.grid.n[2] // 2 for c in cs],
                "planes": [torch.zeros((c.batch, *c.grid.shape[1:]), dtype=t, device="cuda") for c in cs]}
    if kind == "epoch":
        net, x, t = _net(case, seed, case["batch"])
        net.prepare(x, t)
        return {"kind": kind, "net": net}
    if kind == "predict":
        net, x, _ = _net(case, seed, 256)
        return {"kind": kind, "net": net, "x": x}
    x, w, bias, dy = _layer_arrays(case, seed)
    g, m, n = case["members"], case["batch"], case["width"]

    def new(*shape, dtype=torch.bfloat16):
        return torch.zeros((g, *shape), dtype=dtype, device="cuda")

    return {"kind": kind, "lib": native.load(), "g": g, "m": m, "n": n, "x": x, "w": w, "bias": bias, "dy": dy,
            "xt": x.transpose(1, 2).contiguous(), "wt": w.transpose(1, 2).contiguous(),
            "dyt": dy.transpose(1, 2).contiguous(), "y": new(m, n), "yt": new(n, m),
            "dx": new(m, n, dtype=torch.float32), "dx16": new(m, n), "dxt": new(n, m),
            "dw": new(n, n, dtype=torch.float32), "status": torch.zeros(1, dtype=torch.int32, device="cuda")}


def run(s):
    kind = s["kind"]
    if kind == "steps":
        eng = s["eng"]
        eng.step(s["steps"])
        out = {"energy": eng.energy(), "dft": eng.results()}
        if s["dump"]:
            out["fields"] = eng.get_fields()
            return out
        planes = s["planes"]
        for k in range(6):
            for i, z in enumerate(s["at"]):
                eng.plane_to_device(k, z, planes[k, i].data_ptr())
        out["planes"] = planes
        return out
    if kind == "sweep":
        s["batch"].step(s["steps"])
        dft = np.stack([np.stack(list(e.results().values())) for e in s["engines"]])
        for e, z, p in zip(s["engines"], s["at"], s["planes"]):
            e.plane_to_device(2, z, p.data_ptr())
        return {"dft": dft, "planes": s["planes"]}
    if kind == "epoch":
        s["net"].run_epoch(1e-3)
        return s["net"].p32
    if kind == "predict":
        return s["net"].predict_device(s["x"])
    g, m, n, gemm = s["g"], s["m"], s["n"], s["lib"].oafdtd_mlp_gemm_tn
    st, stream = s["status"].data_ptr(), int(torch.cuda.current_stream().cuda_stream)
    # y = tanh(x W + b), also transposed for the next layer's weight gradient
    native.check(gemm(s["x"].data_ptr(), s["wt"].data_ptr(), None, s["y"].data_ptr(), s["yt"].data_ptr(),
                      s["bias"].data_ptr(), None, m, n, n, n, n, n, m, 3, 0.0, g, m * n, n * n, m * n, n * m, n, st,
                      stream), "forward")
    # dx = (dy W^T) (1 - x^2), in FP32 and BF16, also transposed
    native.check(gemm(s["dy"].data_ptr(), s["w"].data_ptr(), s["dx"].data_ptr(), s["dx16"].data_ptr(),
                      s["dxt"].data_ptr(), None, s["x"].data_ptr(), m, n, n, n, n, n, m, 4, 0.0, g, m * n, n * n,
                      m * n, n * m, 0, st, stream), "input gradient")
    # dW = x^T dy
    native.check(gemm(s["xt"].data_ptr(), s["dyt"].data_ptr(), s["dw"].data_ptr(), None, None, None, None, n, n, m, m,
                      m, n, n, 0, 0.0, g, n * m, n * m, n * n, 0, 0, st, stream), "weight gradient")
    return {k: s[k] for k in ("y", "yt", "dx", "dx16", "dxt", "dw")}


def work(case):
    """Per time step: every field value read and written once, the index of each edge read once, and
    the state of the boundary layers, Debye poles and copper faces read and written once. Networks:
    weights, inputs and outputs once, and the products."""
    if case["kind"] in ("steps", "sweep"):
        rb = 4 if case["dtype"] == "float32" else 8
        total = flops = 0.0
        for c in _compiled(case):
            nx, ny, nz = c.grid.n
            b, cells = c.batch, float(nx * ny * nz)
            per = cells * (12 * rb * b + 6)
            fl = cells * b * 36.0
            for k in c.pml.corrections:
                per += float(np.prod([k.box[a][1] - k.box[a][0] for a in range(3)])) * b * 2 * rb
            if c.ade is not None:
                edges = float(sum(np.asarray(f).size for f in c.ade.flat))
                per += edges * b * c.ade.tau.size * 2 * rb
                fl += edges * b * c.ade.tau.size * 5
            if c.sibc is not None:
                per += float(c.sibc.flat.size) * b * rb * (2 * (1 + c.sibc.cp.size) + 3)
                fl += float(c.sibc.flat.size) * b * c.sibc.cp.size * 4
            total += per * case["steps"]
            flops += fl * case["steps"]
        return {"bytes": total, "flops": flops}
    g, n = case["members"], case["width"]
    if case["kind"] == "layer":
        m = case["batch"]
        return {"bytes": g * (m * n * 2.0 * 8 + m * n * 4.0 + n * n * 8.0), "flops": 6.0 * g * m * n * n}
    sizes = [8] + [n] * case["depth"] + [4 * case["n_freq"]]
    mac = float(sum(a * b for a, b in zip(sizes[:-1], sizes[1:])))
    if case["kind"] == "predict":
        rows = case["rows"]
        return {"bytes": g * (2.0 * mac + rows * sizes[-1] * 4.0), "flops": 2.0 * g * rows * mac}
    nb = case["rows"] // case["batch"]
    # weights, both moments read and written, per step
    return {"bytes": nb * g * mac * 24.0, "flops": 6.0 * nb * g * case["batch"] * mac}


# ------------------------------------------------------------------------------------- in 64 bits
# (component, derivative axis, source component, sign) of E_c += cb d_a H_b; H_c the other way round
_CURL = ((0, 1, 2, 1.0), (0, 2, 1, -1.0), (1, 2, 0, 1.0), (1, 0, 2, -1.0), (2, 0, 1, 1.0), (2, 1, 0, -1.0))


def _win(f, box, axis=-1, shift=0):
    """View of a ``(B, z, y, x)`` tensor over a box of storage ranges (x, y, z)."""
    s = [slice(None)]
    for a in (2, 1, 0):
        d = shift if a == axis else 0
        s.append(slice(box[a][0] + d, box[a][1] + d))
    return f[tuple(s)]


def _line(v, axis, box):
    shape = [1, 1, 1, 1]
    shape[3 - axis] = box[axis][1] - box[axis][0]
    return v[box[axis][0] : box[axis][1]].reshape(shape)


def _march(c, fields, steps):
    """The leapfrog scheme in float64 torch from the compiled arrays: Yee updates, CPML, Debye
    currents, surface impedance, injection and running DFTs. Returns energy, DFTs and the fields."""
    dev = fields[0].device
    f64 = lambda a: torch.as_tensor(np.asarray(a, np.float64), device=dev)  # noqa: E731
    i64 = lambda a: torch.as_tensor(np.asarray(a, np.int64), device=dev)  # noqa: E731
    g, bsz, dt = c.grid, c.batch, c.dt
    n = g.n
    e, h = fields[:3], fields[3:]
    ip, idd = [f64(g.inv_primal(a)) for a in range(3)], [f64(g.inv_dual(a)) for a in range(3)]
    idx = [i64(m) for m in c.idx]
    ca, cb = f64(c.ca_tab), f64(c.cb_tab)
    full = tuple((1, n[a] + 2) for a in range(3))
    psi = [torch.zeros((bsz, *k.shape), dtype=torch.float64, device=dev) for k in c.pml.corrections]
    co = {a: {t: f64(getattr(v, t)) for t in ("eb", "ec", "ek", "hb", "hc", "hk")} for a, v in c.pml.coeffs.items()}
    ade = []
    if c.ade is not None:
        kp = f64(c.ade.kp)
        for comp, flat, beta, cbe in zip(c.ade.comp, c.ade.flat, c.ade.beta, c.ade.cbe):
            ade.append((comp, i64(flat), f64(beta), f64(cbe),
                        torch.zeros((c.ade.tau.size, bsz, len(flat)), dtype=torch.float64, device=dev)))
    sib = c.sibc
    if sib is not None:
        mat = i64(sib.mat)
        alpha = (f64(sib.rp)[mat] * f64(sib.cp)[None, :]).T[:, None, :]
        gp, r0 = f64(sib.gp)[:, None, None], f64(sib.r0)[mat][None]
        hs = [[(q, i64(np.flatnonzero((sib.hcomp[:, s] == q) & (sib.hsign[:, s] != 0)))) for q in range(3)]
              for s in range(2)]
        hflat, hsign = i64(sib.hflat), f64(sib.hsign)
        sel = [i64(np.flatnonzero(sib.comp == q)) for q in range(3)]
        sflat = i64(sib.flat)
        jprev = torch.zeros((bsz, sib.flat.size), dtype=torch.float64, device=dev)
        v = torch.zeros((sib.cp.size, *jprev.shape), dtype=torch.float64, device=dev)
    drive = f64(c.drive)
    chans = []
    for ch in c.channels:
        comps = np.broadcast_to(np.asarray(ch["comp"]), np.asarray(ch["flat"]).shape)
        chans.append([(int(q), i64(ch["flat"])[i64(np.flatnonzero(comps == q))],
                       f64(ch["amps"])[i64(np.flatnonzero(comps == q))]) for q in np.unique(comps)])
    omega = f64(2.0 * np.pi * c.frequencies)
    probes = [(q["name"], q["kind"], q["comp"], i64(q["flat"]), f64(q["weights"])) for q in c.probes]
    acc = {q[0]: torch.zeros((bsz, omega.numel()), dtype=torch.complex128, device=dev) for q in probes}

    def record(kind, t):
        ph = torch.exp(-1j * omega * t) * dt
        for name, kd, comp, flat, wt in probes:
            if kd == kind:
                val = ((e if kind == "E" else h)[comp].reshape(bsz, -1)[:, flat] * wt).sum(1)
                acc[name] += val[:, None] * ph[None]

    def layers(kind):
        for k, p in zip(c.pml.corrections, psi):
            if k.kind != kind:
                continue
            src, box, q, pre = (h if kind == "E" else e)[k.b], k.box, co[k.a], kind.lower()
            if kind == "E":
                d = (_win(src, box) - _win(src, box, k.a, -1)) * _line(idd[k.a], k.a, box)
                fac = cb[_win(idx[k.c][None], box)]
            else:
                d = (_win(src, box, k.a, 1) - _win(src, box)) * _line(ip[k.a], k.a, box)
                fac = dt / MU0
            p.mul_(_line(q[pre + "b"], k.a, box)).add_(_line(q[pre + "c"], k.a, box) * d)
            _win((e if kind == "E" else h)[k.c], box).add_(k.sign * fac * (_line(q[pre + "k"], k.a, box) * d + p))

    for step in range(steps):
        for comp in range(3):
            box = g.valid("H", comp)
            for q, a, b, sign in _CURL:
                if q == comp:
                    d = (_win(e[b], box, a, 1) - _win(e[b], box)) * _line(ip[a], a, box)
                    _win(h[comp], box).sub_(d, alpha=sign * dt / MU0)
        layers("H")
        for a in range(3):
            for side in range(2):
                if c.walls[2 * a + side] == "pmc":
                    dst, src = (0, 1) if side == 0 else (n[a] + 1, n[a])
                    for comp in range(3):
                        if comp != a:
                            h[comp].select(3 - a, dst).copy_(-h[comp].select(3 - a, src))
        record("H", (step + 0.5) * dt)
        old = [e[st[0]].reshape(bsz, -1)[:, st[1]] for st in ade]
        for comp in range(3):
            curl = None
            for q, a, b, sign in _CURL:
                if q == comp:
                    d = (_win(h[b], full) - _win(h[b], full, a, -1)) * _line(idd[a], a, full)
                    curl = sign * d if curl is None else curl.add_(d, alpha=sign)
            ix = _win(idx[comp][None], full)
            _win(e[comp], full).mul_(ca[ix]).add_(curl.mul_(cb[ix]))
        layers("E")
        if sib is not None:
            j = torch.zeros_like(jprev)
            for s in range(2):
                for q, ids in hs[s]:
                    j[:, ids] += hsign[ids, s] * h[q].reshape(bsz, -1)[:, hflat[ids, s]]
            v.mul_(gp).add_(alpha * (j - jprev)[None])
            out = r0 * j + v.sum(0)
            jprev = j
            for q in range(3):
                e[q].view(bsz, -1)[:, sflat[sel[q]]] = out[:, sel[q]]
        for ci, ch in enumerate(c.channels):
            wave = float(ch["waveform"](np.array([(step + 0.5) * dt]))[0])
            for q, flat, amp in chans[ci]:
                e[q].view(bsz, -1)[:, flat] += drive[:, ci : ci + 1] * wave * amp[None]
        for (comp, flat, beta, cbe, cur), eo in zip(ade, old):
            en = e[comp].view(bsz, -1)[:, flat]
            en = en - cbe * (0.5 * ((1.0 + kp)[:, None, None] * cur).sum(0))
            cur.mul_(kp[:, None, None]).add_(beta[:, None, :] * (en - eo)[None])
            e[comp].view(bsz, -1)[:, flat] = en
        record("E", (step + 1) * dt)
    energy = 0.0
    for k in range(6):
        comp, f = k % 3, (e + h)[k]
        w = torch.ones((1, 1, 1, 1), dtype=torch.float64, device=dev)
        for a in range(3):
            node = (a != comp) if k < 3 else (a == comp)
            wa = f64(g.node_weights(a) if node else g.cell_weights(a))
            shape = [1, 1, 1, 1]
            shape[3 - a] = wa.numel()
            w = w * wa.reshape(shape)
        w = w * (f64(c.eps_tab)[idx[comp]][None] * EPS0 if k < 3 else MU0)
        energy += 0.5 * float((f * f * w).sum())
    return energy, {k: a.cpu().numpy() for k, a in acc.items()}, e + h


def _exact_fields(c, dtype, seed):
    t = torch.float32 if dtype == "float32" else torch.float64
    return [f.to(torch.float64).transpose(0, 1).contiguous() for f in _noise(c, t, seed)]


def exact(case, seed):
    kind = case["kind"]
    if kind == "steps":
        c = _compiled(case)[0]
        energy, dft, fields = _march(c, _exact_fields(c, case["dtype"], seed), case["steps"])
        out = {"energy": energy, "dft": dft}
        if case["what"] == "box":
            out["fields"] = {k: f.cpu().numpy() for k, f in zip(("Ex", "Ey", "Ez", "Hx", "Hy", "Hz"), fields)}
        else:
            out["planes"] = torch.stack([torch.stack([f[:, z] for z in _planes(c)]) for f in fields])
        return out
    if kind == "sweep":
        dft, planes = [], []
        for i, c in enumerate(_compiled(case)):
            _, d, fields = _march(c, _exact_fields(c, case["dtype"], seed + 1000 * i), case["steps"])
            dft.append(np.stack(list(d.values())))
            planes.append(fields[2][:, c.grid.n[2] // 2].clone())
        return {"dft": np.stack(dft), "planes": planes}
    if kind == "layer":
        x, w, bias, dy = (a.double() for a in _layer_arrays(case, seed))
        y = torch.tanh(torch.bmm(x, w) + bias[:, None])
        dx = torch.bmm(dy, w.transpose(1, 2)) * (1.0 - x * x)
        return {"y": y, "yt": y.transpose(1, 2), "dx": dx, "dx16": dx, "dxt": dx.transpose(1, 2),
                "dw": torch.bmm(x.transpose(1, 2), dy)}
    sizes, w, b, x, t = _net_arrays(case, seed)
    w, b = [v.double() for v in w], [v.double() for v in b]
    x, t = torch.as_tensor(x, device="cuda").double(), torch.as_tensor(t, device="cuda").double()
    last = len(w) - 1

    def forward(inp):
        acts = [inp]
        for layer in range(len(w)):
            z = torch.bmm(acts[-1], w[layer]) + b[layer][:, None]
            acts.append(z if layer == last else torch.tanh(z))
        return acts

    g = case["members"]
    if kind == "predict":
        return forward(x.expand(g, -1, -1))[-1]
    m, rows = case["batch"], case["rows"]
    nb = rows // m
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed) % 100000 + 1)
    pick = torch.stack([torch.randperm(rows, generator=gen, device="cuda")[: nb * m].view(nb, m) for _ in range(g)], 1)
    mom = [[torch.zeros_like(v), torch.zeros_like(v)] for v in w + b]
    for step in range(nb):
        acts = forward(x[pick[step]])
        dz = (acts[-1] - t[pick[step]]) * (2.0 / (m * sizes[-1]))
        grads_w, grads_b = [None] * len(w), [None] * len(w)
        for layer in range(last, -1, -1):
            grads_w[layer], grads_b[layer] = torch.bmm(acts[layer].transpose(1, 2), dz), dz.sum(1)
            if layer:
                dz = torch.bmm(dz, w[layer].transpose(1, 2)) * (1.0 - acts[layer] ** 2)
        for p, gr, mv in zip(w + b, grads_w + grads_b, mom):
            mv[0].mul_(0.9).add_(0.1 * gr)
            mv[1].mul_(0.999).add_(0.001 * gr * gr)
            p.sub_(1e-3 * (mv[0] / (1 - 0.9 ** (step + 1))) / ((mv[1] / (1 - 0.999 ** (step + 1))).sqrt() + 1e-8))
    # every member's parameters in one flat block, each array on a multiple of 64 values
    up = lambda k: (k + 63) // 64 * 64  # noqa: E731
    blocks = []
    for wl, bl in zip(w, b):
        a = (wl.shape[1] + 7) // 8 * 8
        full = torch.zeros((g, a, wl.shape[2]), dtype=torch.float64, device="cuda")
        full[:, : wl.shape[1]] = wl
        for v in (full.reshape(g, -1), bl):
            blocks.append(torch.nn.functional.pad(v, (0, up(v.shape[1]) - v.shape[1])))
    return torch.cat(blocks, 1).reshape(-1)

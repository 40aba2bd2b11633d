"""Workloads of this package as its users run them, for timing and for checking outputs.

A case is one plain dict. Its ``kind`` says which public entry points it goes through:

* ``room`` -- one ``CudaAcousticFDTD`` put at rest, run for a block of steps, recordings and the
  final pressure read back (``scheme`` absent: the constructor's own default);
* ``response`` -- ``simulate_impulse_response``, from the room's description to its impulse
  responses, a new solver each time;
* ``batch`` -- a ``RoomBatch`` of uneven rooms run together, every recording read back;
* ``gradient`` -- a ``DifferentiableRoom``: recorded forward run and adjoint of a least-squares
  misfit (walls, source signal, initial pressure, optionally the air's processes);
* ``gradient_batch`` -- the same over a ``DifferentiableBatch`` of rooms with patched walls;
* ``metrics`` -- deconvolution, Schroeder decay, T20, T30, EDT, C50 and C80 of a set of
  receiver signals that are already on the GPU.

Sizes are those of the package's own workloads (``ac_fdtd_b200/workloads.py``: 64^3 and 384^3
rooms, uneven rooms of 60-200 cells per axis, a 128^3 inversion, patched rooms of 96-160 cells)
and of its tests (20 x 17 x 15), with odd ones between them. Runs are blocks of the full length:
enough steps that a pass is the step loop and not its setup.
"""

from __future__ import annotations

import math

import numpy as np
import torch

from ac_fdtd_b200 import (
    AbsorbingLayer,
    AirAbsorption,
    CudaAcousticFDTD,
    Grid,
    Room,
    RoomBatch,
    WallAdmittances,
    pinned_array,
    simulate_impulse_response,
)
from ac_fdtd_b200 import postprocess
from ac_fdtd_b200.adjoint import DifferentiableBatch, DifferentiableRoom
from ac_fdtd_b200.boundaries import WallPatches

C = 331.3 * ((20.0 + 273.15) / 273.15) ** 0.5      # the default medium: air at 20 C
RHO = 101325.0 / (287.058 * (20.0 + 273.15))
FACES = ((0, 0), (0, 1), (1, 0), (1, 1), (2, 0), (2, 1))
ON_CHIP_BYTES = 126 << 20                          # L2: a smaller state need not leave the chip


def listed():
    return [
        # The smallest call: the parity tests' grid with every term active, 100 steps. Launch
        # and synchronisation latency is all of it.
        {"name": "tiny_everything_fp32", "kind": "room", "nx": 20, "ny": 17, "nz": 15, "steps": 100,
         "dtype": "float32", "walls": True, "layer": 3, "layer_faces": 6, "air": True, "receivers": 1},
        # The plain small room in the constructor's defaults (float64, default scheme): a first
        # simulation, and the room the reference's own numbers are quoted on.
        {"name": "small_room_fp64", "kind": "room", "nx": 64, "ny": 64, "nz": 64, "steps": 500,
         "dtype": "float64", "walls": True, "layer": 0, "layer_faces": 0, "air": False, "receivers": 1},
        # The whole room-acoustics workflow in its defaults: a 3.4 x 2.7 x 2.4 m room to 700 Hz,
        # ISO air, one new solver per call, deconvolved responses out.
        {"name": "impulse_response_fp64", "kind": "response", "lx": 3.4, "ly": 2.7, "lz": 2.4,
         "max_frequency": 700.0, "steps": 600, "dtype": "float64", "receivers": 2},
        # A medium room with ragged counts in single precision and the default scheme: walls and
        # ISO air, as a parameter study runs it.
        {"name": "ragged_room_fp32", "kind": "room", "nx": 97, "ny": 131, "nz": 77, "steps": 300,
         "dtype": "float32", "walls": True, "layer": 0, "layer_faces": 0, "air": True, "receivers": 2},
        # The headline room: 384^3, walls, two-face sponge, ISO air, four receivers, one sweep
        # per step.
        {"name": "large_room_fp32", "kind": "room", "nx": 384, "ny": 384, "nz": 384, "steps": 150,
         "dtype": "float32", "scheme": "fused", "walls": True, "layer": 16, "layer_faces": 2, "air": True,
         "receivers": 4},
        # A large room in double precision with the default scheme, ragged, everything on: the
        # accurate run a study is checked against.
        {"name": "large_room_fp64", "kind": "room", "nx": 203, "ny": 187, "nz": 211, "steps": 80,
         "dtype": "float64", "walls": True, "layer": 12, "layer_faces": 2, "air": True, "receivers": 4},
        # Walls only, pressure-only scheme: the cheap scheme at a large size.
        {"name": "pressure_only_fp32", "kind": "room", "nx": 320, "ny": 300, "nz": 340, "steps": 200,
         "dtype": "float32", "scheme": "pressure_only", "walls": True, "layer": 0, "layer_faces": 0,
         "air": False, "receivers": 2},
        # Uneven rooms in one batch, one launch per step for all of them.
        {"name": "uneven_batch_fp32", "kind": "batch", "rooms": 8, "low": 60, "high": 200, "shape_seed": 3,
         "steps": 150, "dtype": "float32", "scheme": "fused"},
        # The 128^3 wall inversion: one gradient of six admittances and a source signal.
        {"name": "wall_gradient_fp32", "kind": "gradient", "nx": 128, "ny": 128, "nz": 128, "steps": 200,
         "dtype": "float32", "air": False, "receivers": 4},
        # Fitting the air's relaxation strengths and times as well: history of every cell.
        {"name": "air_gradient_fp32", "kind": "gradient", "nx": 101, "ny": 86, "nz": 92, "steps": 120,
         "dtype": "float32", "air": True, "receivers": 4},
        # Patched walls (4 x 4 per wall), sponge on one face, ISO air, several rooms at once.
        {"name": "patch_gradients_fp32", "kind": "gradient_batch", "rooms": 3, "low": 96, "high": 160,
         "shape_seed": 5, "steps": 100, "dtype": "float32"},
        # Room-acoustics figures of a receiver grid: 48 signals of two seconds at 48 kHz.
        {"name": "decay_metrics_fp64", "kind": "metrics", "channels": 48, "samples": 96000},
    ]


def _between(rng, low, high):
    """A whole number of [low, high], spread over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(("room", "room", "room", "room", "response", "batch", "gradient", "gradient",
                       "gradient_batch", "metrics"))
    if kind == "room":
        scheme = rng.choice(("", "", "fused", "pressure_only"))
        side = _between(rng, 16, 300)
        shape = [max(8, int(side * rng.uniform(0.75, 1.25))) for _ in range(3)]
        cells = math.prod(shape)
        case = {"kind": kind, "nx": shape[0], "ny": shape[1], "nz": shape[2],
                "steps": max(60, min(500, int(4e8 / cells))), "dtype": rng.choice(("float32", "float64")),
                "walls": rng.random() < 0.85, "layer": 0, "layer_faces": 0, "air": False,
                "receivers": rng.randint(1, 4)}
        if scheme:
            case["scheme"] = scheme
        if scheme != "pressure_only":
            case["air"] = rng.random() < 0.6
            if rng.random() < 0.4 and min(shape) >= 12:
                case["layer"], case["layer_faces"] = rng.randint(2, min(16, min(shape) // 4)), rng.choice((1, 2, 6))
        return case
    if kind == "response":
        return {"kind": kind, "lx": round(rng.uniform(1.5, 4.5), 2), "ly": round(rng.uniform(1.5, 4.0), 2),
                "lz": round(rng.uniform(1.5, 3.0), 2), "max_frequency": float(_between(rng, 300, 800)),
                "steps": rng.randint(300, 800), "dtype": rng.choice(("float64", "float64", "float32")),
                "receivers": rng.randint(1, 4)}
    if kind == "batch":
        high = _between(rng, 40, 200)
        return {"kind": kind, "rooms": rng.randint(3, 8), "low": max(16, high // 3), "high": high,
                "shape_seed": rng.randint(0, 1 << 20), "steps": max(60, min(400, int(1.2e8 / high**3))),
                "dtype": rng.choice(("float32", "float32", "float64")), "scheme": rng.choice(("fused", "two_sweeps"))}
    if kind == "gradient":
        side, air = _between(rng, 24, 140), rng.random() < 0.4
        shape = [max(8, int(side * rng.uniform(0.8, 1.2))) for _ in range(3)]
        return {"kind": kind, "nx": shape[0], "ny": shape[1], "nz": shape[2],
                "steps": max(60, min(300, int(3e8 / math.prod(shape)))),
                "dtype": rng.choice(("float32", "float32", "float64")), "air": air, "receivers": rng.randint(1, 4)}
    if kind == "gradient_batch":
        high = _between(rng, 32, 160)
        return {"kind": kind, "rooms": rng.randint(2, 4), "low": max(24, high * 3 // 5), "high": high,
                "shape_seed": rng.randint(0, 1 << 20), "steps": rng.randint(60, 100), "dtype": "float32"}
    return {"kind": kind, "channels": rng.randint(1, 48), "samples": _between(rng, 4000, 96000)}


# ---------------------------------------------------------------------------------- inputs


def _xi(alpha):
    r = math.sqrt(1.0 - alpha)
    return (1.0 - r) / (1.0 + r)


def _signal(steps, dt, frequency):
    """A Gaussian pulse 40 dB down at ``frequency``."""
    width = math.sqrt(math.log(100.0)) / (math.pi * frequency)
    t = (np.arange(steps) + 0.5) * dt
    return np.exp(-(((t - 3.0 * width) / width) ** 2))


def _margins(shape):
    return [min(4, (n - 1) // 2) for n in shape]


def _point(rng, shape):
    return tuple(int(rng.integers(m, n - m)) for m, n in zip(_margins(shape), shape))


def _description(rng, shape, steps, *, walls, layer, layer_faces, air, receivers, dx, patches=0):
    """One room's inputs as plain numbers, drawn from ``rng``."""
    dt = dx / (C * math.sqrt(3.0))
    alphas = rng.uniform(0.05, 0.5, (6, patches, patches) if patches else 6)
    xi = np.vectorize(_xi)(alphas)
    source = _point(rng, shape)
    reach = max(1, steps // 6)      # cells: the pulse gets to the receivers well within the run

    def near():
        low = [max(m, s - reach) for m, s in zip(_margins(shape), source)]
        high = [min(n - m, s + reach + 1) for n, m, s in zip(shape, _margins(shape), source)]
        return tuple(int(rng.integers(a, b)) for a, b in zip(low, high))

    return {
        "shape": shape, "steps": steps, "dx": dx, "dt": dt, "xi": xi if walls else None,
        "layer": (layer, [tuple(f) for f in FACES[:layer_faces]]) if layer else None,
        "air": (float(rng.uniform(15.0, 25.0)), float(rng.uniform(30.0, 70.0))) if air else None,
        "source": source, "signal": _signal(steps, dt, C / (10.0 * dx)) * float(rng.uniform(0.5, 2.0)),
        "receivers": [near() for _ in range(receivers)],
    }


def _objects(d):
    """The package's value objects for a description."""
    out = {"grid": Grid(dx=d["dx"], nx=d["shape"][0], ny=d["shape"][1], nz=d["shape"][2])}
    if d["xi"] is not None:
        out["walls"] = WallAdmittances(*d["xi"]) if d["xi"].ndim == 1 else WallPatches(d["xi"])
    if d["layer"]:
        out["absorbing_layer"] = AbsorbingLayer(thickness=d["layer"][0], faces=tuple(d["layer"][1]))
    if d["air"]:
        out["air_absorption"] = AirAbsorption(temperature=d["air"][0], relative_humidity=d["air"][1])
    return out


def _metres(d, cell):
    return tuple((i + 0.5) * d["dx"] for i in cell)


def _batch_shapes(case):
    rng = np.random.default_rng(case["shape_seed"])
    return [tuple(int(v) for v in rng.integers(case["low"], case["high"] + 1, 3)) for _ in range(case["rooms"])]


def _descriptions(case, seed):
    """Every room of a case as plain numbers."""
    rng = np.random.default_rng([seed, 7])
    kind = case["kind"]
    if kind == "room":
        return [_description(rng, (case["nx"], case["ny"], case["nz"]), case["steps"], walls=case["walls"],
                             layer=case["layer"], layer_faces=case["layer_faces"], air=case["air"],
                             receivers=case["receivers"], dx=0.02)]
    if kind == "gradient":
        return [_description(rng, (case["nx"], case["ny"], case["nz"]), case["steps"], walls=True, layer=0,
                             layer_faces=0, air=case["air"], receivers=case["receivers"], dx=0.02)]
    if kind == "batch":
        return [_description(rng, s, case["steps"], walls=True, layer=0, layer_faces=0, air=True, receivers=2,
                             dx=0.05) for s in _batch_shapes(case)]
    return [_description(rng, s, case["steps"], walls=True, layer=8 if min(s) >= 32 else 4, layer_faces=1, air=True,
                         receivers=4, dx=0.017, patches=4) for s in _batch_shapes(case)]


def _targets(case, seed, rooms):
    """Measured signals the misfit compares with: decaying noise of the recordings' size."""
    rng = np.random.default_rng([seed, 11])
    out = []
    for d in rooms:
        decay = np.exp(-3.0 * np.arange(d["steps"]) / d["steps"])
        out.append(rng.standard_normal((len(d["receivers"]), d["steps"])) * decay)
    return out


def _response(case, seed):
    rng = np.random.default_rng([seed, 13])
    size = (case["lx"], case["ly"], case["lz"])
    points = [tuple(float(rng.uniform(0.25, 0.75)) * v for v in size) for _ in range(1 + case["receivers"])]
    dx = C / (10.0 * case["max_frequency"])
    return {"size": size, "absorption": float(rng.uniform(0.05, 0.4)), "source": points[0], "receivers": points[1:],
            "air": (20.0, float(rng.uniform(30.0, 70.0))), "dx": dx, "dt": dx / (C * math.sqrt(3.0))}


def _decays(case, seed):
    """What receivers record of decaying responses excited by a short pulse, and that pulse."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    n, channels = case["samples"], case["channels"]
    t = torch.arange(n, device="cuda", dtype=torch.float64) / n
    rate = 5.0 + 4.0 * torch.rand(channels, 1, generator=g, device="cuda", dtype=torch.float64)
    x = torch.randn(channels, n, generator=g, device="cuda", dtype=torch.float64) * torch.exp(-rate * t)
    excitation = torch.zeros(n, device="cuda", dtype=torch.float64)
    excitation[:17] = torch.hann_window(17, periodic=False, dtype=torch.float64, device="cuda")
    recorded = torch.fft.irfft(torch.fft.rfft(x) * torch.fft.rfft(excitation), n=n)
    return recorded, excitation


# ------------------------------------------------------------------------------ the passes


def prepare(case, seed):
    kind = case["kind"]
    if kind == "metrics":
        x, excitation = _decays(case, seed)
        return {"case": case, "x": x, "excitation": excitation, "rate": 48000.0}
    if kind == "response":
        r = _response(case, seed)
        room = Room(dimensions=r["size"], absorption=r["absorption"],
                    air=AirAbsorption(temperature=r["air"][0], relative_humidity=r["air"][1]))
        return {"case": case, "room": room, "r": r, "duration": case["steps"] * r["dt"]}
    rooms = _descriptions(case, seed)
    dtype = np.dtype(case["dtype"])
    state = {"case": case}
    options = {"scheme": case["scheme"]} if "scheme" in case else {}
    if kind == "room":
        d = rooms[0]
        objects = _objects(d)
        solver = CudaAcousticFDTD(objects.pop("grid"), dtype=dtype, **objects, **options)
        solver.add_volume_source(_metres(d, d["source"]), d["signal"])
        for cell in d["receivers"]:
            solver.add_pressure_receiver(_metres(d, cell))
        state.update(solver=solver, p=pinned_array(d["shape"], dtype))
    elif kind == "batch":
        batch = RoomBatch([_objects(d) for d in rooms], dtype=dtype, **options)
        for r, d in enumerate(rooms):
            batch.add_volume_source(r, _metres(d, d["source"]), d["signal"])
            for cell in d["receivers"]:
                batch.add_pressure_receiver(r, _metres(d, cell))
        state.update(batch=batch)
    elif kind == "gradient":
        d = rooms[0]
        objects = _objects(d)
        room = DifferentiableRoom(objects.pop("grid"), dtype=dtype, **objects, max_steps=case["steps"],
                                  wrt=("signal", "walls", "air") if case["air"] else ("signal", "walls"))
        room.solver.add_volume_source(_metres(d, d["source"]), d["signal"])
        for cell in d["receivers"]:
            room.solver.add_pressure_receiver(_metres(d, cell))
        state.update(room=room, target=_targets(case, seed, rooms)[0])
    else:
        batch = DifferentiableBatch([_objects(d) for d in rooms], dtype=dtype, max_steps=case["steps"])
        for r, d in enumerate(rooms):
            batch.batch.add_volume_source(r, _metres(d, d["source"]), d["signal"])
            for cell in d["receivers"]:
                batch.batch.add_pressure_receiver(r, _metres(d, cell))
        state.update(batch=batch, targets=_targets(case, seed, rooms))
    return state


def run(state):
    case = state["case"]
    kind, steps = case["kind"], case.get("steps")
    if kind == "room":
        solver = state["solver"]
        solver.reset_state()
        solver.step_index = 0
        solver.run(steps)
        recorded = solver.recorded_pressure
        solver.get_state(p=state["p"])
        return {"recorded": recorded, "p": state["p"]}
    if kind == "response":
        r = state["r"]
        out = simulate_impulse_response(state["room"], r["source"], r["receivers"], case["max_frequency"],
                                        duration=state["duration"], dtype=np.dtype(case["dtype"]))
        return {"signals": out.signals, "recorded": out.recorded}
    if kind == "batch":
        batch = state["batch"]
        batch.reset_state()
        batch.step_index = 0
        batch.run(steps)
        return {"recorded": [batch.recorded_pressure(r) for r in range(len(batch))]}
    if kind == "gradient":
        room = state["room"]
        recorded = room.forward(steps)
        g = room.backward(recorded - state["target"])
        out = {"recorded": recorded, "signal": g.signal, "walls": g.walls, "initial_p": g.initial_p,
               "wall_cells": g.wall_cells}
        if case["air"]:
            out.update(strength=g.strength, relaxation_time=g.relaxation_time)
        return out
    if kind == "gradient_batch":
        batch = state["batch"]
        recorded = batch.forward(steps)
        gradients = batch.backward([x - t for x, t in zip(recorded, state["targets"])])
        return {"recorded": recorded, "signal": [g.signal for g in gradients], "walls": [g.walls for g in gradients],
                "wall_cells": [g.wall_cells for g in gradients]}
    rate = state["rate"]
    response = postprocess.deconvolve(state["x"], state["excitation"], 1.0 / rate, 0.45 * rate, as_numpy=False)
    return {"response": response, "decay": postprocess.schroeder_decay(response, as_numpy=False),
            "t20": postprocess.reverberation_time(response, rate, 20.0),
            "t30": postprocess.reverberation_time(response, rate, 30.0),
            "edt": postprocess.early_decay_time(response, rate), "c50": postprocess.clarity(response, rate, 0.05),
            "c80": postprocess.clarity(response, rate, 0.08)}


# ------------------------------------------------------------- what a pass cannot do without


def _cells(case):
    kind = case["kind"]
    if kind == "response":
        r = _response(case, 0)
        return math.prod(max(1, round(v / r["dx"])) for v in r["size"])
    if kind in ("batch", "gradient_batch"):
        return sum(math.prod(s) for s in _batch_shapes(case))
    return case["nx"] * case["ny"] * case["nz"]


def work(case):
    """Bytes and operations of one pass. A state that fits the chip's caches has to cross HBM once
    per run; a larger one is read and written every step: p, v, the relaxation states (p twice for
    the pressure-only scheme, which has no v). An adjoint step moves the adjoint state the same way
    and reads what the forward run recorded."""
    if case["kind"] == "metrics":
        n = case["channels"] * case["samples"]
        return {"bytes": 8 * n * 3, "flops": n * (10 * math.log2(case["samples"]) + 40)}
    cells, steps = _cells(case), case["steps"]
    size = 4 if case["dtype"] == "float32" else 8
    air = case.get("air", case["kind"] in ("response", "batch", "gradient_batch"))
    relax = 3 if air else 0
    fields = 4 + relax
    flops = 22 + 8 * relax + (9 if case.get("layer") or case["kind"] == "gradient_batch" else 0)
    per_step = 2 * fields
    if case.get("scheme") == "pressure_only":
        fields, per_step, flops = 2, 3, 9
    state = cells * size * fields
    one_way = state * 2 if state <= ON_CHIP_BYTES else cells * size * per_step * steps
    total_bytes, total_flops = one_way, flops * cells * steps
    if case["kind"] in ("gradient", "gradient_batch"):
        total_bytes += one_way
        total_flops += (flops + 6 + 6 * relax) * cells * steps
        if case["kind"] == "gradient" and air:
            total_bytes += 2 * (1 + relax) * cells * size * steps     # D and psi, written and read
    return {"bytes": total_bytes, "flops": total_flops}


# ---------------------------------------------------------------- the same in plain 64 bits


def _processes(temperature, humidity, dt):
    """ISO 9613-1 oxygen and nitrogen relaxation and the classical term at Nyquist."""
    kelvin = temperature + 273.15
    tr = kelvin / 293.15
    h = humidity * 10.0 ** (-6.8346 * (273.16 / kelvin) ** 1.261 + 4.6151)
    f_o = 24.0 + 4.04e4 * h * (0.02 + h) / (0.391 + h)
    f_n = tr**-0.5 * (9.0 + 280.0 * h * math.exp(-4.170 * (tr ** (-1.0 / 3.0) - 1.0)))
    oxygen = tr**-2.5 * 0.01275 * math.exp(-2239.1 / kelvin)
    nitrogen = tr**-2.5 * 0.1068 * math.exp(-3352.0 / kelvin)
    nyquist = 0.5 / dt
    terms = ((oxygen, f_o), (nitrogen, f_n), (1.84e-11 * tr**0.5 * nyquist, nyquist))
    return [k * C / math.pi for k, _ in terms], [1.0 / (2.0 * math.pi * f) for _, f in terms]


def _maps(d, xi):
    """Wall admittance of every boundary cell of each face, six 2D tensors."""
    out = []
    for f, (axis, _) in enumerate(FACES):
        nb, nc = [d["shape"][a] for a in range(3) if a != axis]
        if xi.ndim == 1:
            out.append(xi[f].expand(nb, nc).clone())
        else:
            p = xi.shape[-1]
            ib, ic = (torch.arange(n, device=xi.device) * p // n for n in (nb, nc))
            out.append(xi[f][ib][:, ic])
    return out


def _on_face(shape, f, values):
    """``values`` (one per cell of face ``f``) on the room's grid, zero elsewhere."""
    axis, side = FACES[f]
    values = values.unsqueeze(axis)
    rest = shape[axis] - 1
    if rest == 0:
        return values
    pad = [0] * 6
    pad[2 * (2 - axis) + (1 if side == 0 else 0)] = rest
    return torch.nn.functional.pad(values, pad)


def _profiles(d):
    """The sponge's factors at cell centres and faces of each axis."""
    thickness, faces = d["layer"]
    depth = thickness * d["dx"]
    sigma = -4.0 * C * math.log(1e-5) / (2.0 * depth)

    def profile(x, extent, axis):
        distance = torch.full_like(x, math.inf)
        if (axis, 0) in faces:
            distance = torch.minimum(distance, x)
        if (axis, 1) in faces:
            distance = torch.minimum(distance, extent - x)
        inside = torch.clamp(1.0 - distance / depth, 0.0, 1.0)
        view = [1, 1, 1]
        view[axis] = -1
        return torch.exp(-sigma * inside**3 * d["dt"]).reshape(view)

    cell, face = [], []
    for axis, n in enumerate(d["shape"]):
        k = torch.arange(n + 1, device="cuda", dtype=torch.float64)
        cell.append(profile((k[:-1] + 0.5) * d["dx"], n * d["dx"], axis))
        face.append(profile(k * d["dx"], n * d["dx"], axis))
    return cell, face


def _damping(factors):
    """The factors that damp anything, in axis order."""
    return [f for f in factors if bool((f < 1.0).any())]


def _leapfrog(d, maps=None, signal=None, p0=None, strength=None, tau=None, grad=False):
    """The staggered leapfrog in float64 torch: (recordings, final pressure)."""
    shape, dx, dt = d["shape"], d["dx"], d["dt"]
    f64 = {"dtype": torch.float64, "device": "cuda"}
    if maps is None and d["xi"] is not None:
        maps = _maps(d, torch.as_tensor(d["xi"], **f64))
    if signal is None:
        signal = torch.as_tensor(d["signal"], **f64)
    cv, cp, cs = dt / (RHO * dx), RHO * C * C * dt / dx, RHO * C * C * dt
    p = torch.zeros(shape, **f64) if p0 is None else p0
    v = [torch.zeros([n - 1 if a == axis else n for a, n in enumerate(shape)], **f64) for axis in range(3)]
    if d["air"] and strength is None:
        strength, tau = (torch.as_tensor(x, **f64) for x in _processes(*d["air"], dt))
    psi = []
    if strength is not None:
        relaxed = C * C / (1.0 + strength.sum())
        gain = RHO * relaxed * strength / dx
        decay = torch.exp(-dt / tau)
        mean = dt * (tau / dt) * (1.0 - decay)
        scale = dt * gain.sum()
        psi = [torch.zeros(shape, **f64) for _ in range(len(strength))]
    fu = fp = None
    if maps is not None:
        a = sum(_on_face(shape, f, (C * dt / (2.0 * dx)) * m) for f, m in enumerate(maps))
        fu, fp = 1.0 / (1.0 + a), a / (1.0 + a)
    damp_p, damp_v = [], [[], [], []]
    if d["layer"]:
        cell, face = _profiles(d)
        damp_p = _damping(cell)
        for axis in range(3):
            n = shape[axis]
            inner = face[axis].narrow(axis, 1, n - 1)
            damp_v[axis] = _damping([inner if b == axis else cell[b] for b in range(3)])
    at = tuple(torch.tensor([i], device="cuda") for i in d["source"])
    heard = tuple(torch.tensor([c[a] for c in d["receivers"]], device="cuda") for a in range(3))
    recorded = []
    for n in range(d["steps"]):
        for axis in range(3):
            if shape[axis] > 1:
                difference = torch.diff(p, dim=axis)
                v[axis] = v[axis] - cv * difference if grad else v[axis].sub_(difference, alpha=cv)
                for f in damp_v[axis]:
                    v[axis] = v[axis] * f if grad else v[axis].mul_(f)
        div = 0.0
        for axis in range(3):
            pad = [0] * 6
            pad[2 * (2 - axis)] = pad[2 * (2 - axis) + 1] = 1
            div = div + torch.diff(torch.nn.functional.pad(v[axis], pad), dim=axis)
        q = p
        for r in range(len(psi)):
            target = div * gain[r]
            offset = psi[r] - target
            psi[r] = offset * decay[r] + target
            q = q + offset * mean[r]
        q = q - div * (cp - scale) if psi else q - div * cp
        if fu is not None:
            q = q * fu - p * fp
        for f in damp_p:
            q = q * f
        p = q.index_put(at, cs * signal[n : n + 1], accumulate=True)
        recorded.append(p[heard])
    return torch.stack(recorded, 1), p


def _gradients(d, target):
    f64 = {"dtype": torch.float64, "device": "cuda"}
    maps = [m.requires_grad_() for m in _maps(d, torch.as_tensor(d["xi"], **f64))]
    signal = torch.as_tensor(d["signal"], **f64).requires_grad_()
    p0 = torch.zeros(d["shape"], **f64, requires_grad=True)
    leaves = [signal, p0, *maps]
    strength = tau = None
    if d["air"]:
        strength, tau = (torch.as_tensor(x, **f64).requires_grad_() for x in _processes(*d["air"], d["dt"]))
        leaves += [strength, tau]
    recorded, _ = _leapfrog(d, maps, signal, p0, strength, tau, grad=True)
    loss = 0.5 * (recorded - torch.as_tensor(target, **f64)).square().sum()
    g = torch.autograd.grad(loss, leaves)
    cells = list(g[2:8])
    if d["xi"].ndim == 1:
        walls = torch.stack([m.sum() for m in cells])
    else:
        n = d["xi"].shape[-1]
        walls = torch.zeros((6, n, n), **f64)
        for f, m in enumerate(cells):
            ib, ic = (torch.arange(k, device="cuda") * n // k for k in m.shape)
            walls[f].index_put_((ib[:, None].expand(m.shape), ic[None].expand(m.shape)), m, accumulate=True)
    return recorded.detach(), g, walls, cells


def _decay_seconds(decay, rate, upper, lower):
    """Seconds per 60 dB of a least-squares line between two levels of each decay curve."""
    out = []
    for curve in decay:
        start, end = (int((curve <= level).to(torch.int8).argmax()) for level in (upper, lower))
        y = curve[start:end]
        x = torch.arange(start, end, device="cuda", dtype=torch.float64) / rate
        x = x - x.mean()
        out.append(-60.0 / float((x * (y - y.mean())).sum() / x.square().sum()))
    return np.array(out)


def _deconvolve(x, excitation, dt, frequency):
    spectrum, source = torch.fft.rfft(x), torch.fft.rfft(excitation)
    power = source.abs().square()
    out = spectrum * source.conj() / (power + 1e-6 * power.max())
    k = torch.arange(out.shape[-1], device=out.device, dtype=torch.float64)
    out[..., k / (x.shape[-1] * dt) > frequency] = 0.0
    return torch.fft.irfft(out, n=x.shape[-1])


def exact(case, seed):
    kind = case["kind"]
    if kind == "metrics":
        x, excitation = _decays(case, seed)
        rate = 48000.0
        h = _deconvolve(x, excitation, 1.0 / rate, 0.45 * rate)
        energy = h.square()
        tail = energy.flip(-1).cumsum(-1).flip(-1)
        decay = (10.0 * torch.log10((tail / tail[:, :1]).clamp(min=1e-300))).clamp(min=-120.0)
        out = {"response": h, "decay": decay}
        for name, upper, lower in (("t20", -5.0, -25.0), ("t30", -5.0, -35.0), ("edt", 0.0, -10.0)):
            out[name] = _decay_seconds(decay, rate, upper, lower)
        for name, split in (("c50", 0.05), ("c80", 0.08)):
            k = int(round(split * rate))
            out[name] = 10.0 * torch.log10(energy[:, :k].sum(-1) / energy[:, k:].sum(-1))
        return out
    if kind == "response":
        r = _response(case, seed)
        shape = tuple(max(1, round(v / r["dx"])) for v in r["size"])

        def cell(point):
            return tuple(min(max(math.floor(x / r["dx"] + 1e-6), 0), n - 1) for x, n in zip(point, shape))

        steps, dt = case["steps"], r["dt"]
        half = int(np.ceil(4.0 / (case["max_frequency"] * dt)))
        offsets = np.arange(-half, half + 1)
        kernel = 2.0 * case["max_frequency"] * dt * np.sinc(2.0 * case["max_frequency"] * dt * offsets)
        excitation = np.zeros(steps)
        excitation[: kernel.size] = kernel * np.hanning(kernel.size)
        d = {"shape": shape, "steps": steps, "dx": r["dx"], "dt": dt, "xi": np.full(6, _xi(r["absorption"])),
             "layer": None, "air": r["air"], "source": cell(r["source"]), "signal": excitation,
             "receivers": [cell(x) for x in r["receivers"]]}
        recorded, _ = _leapfrog(d)
        signals = _deconvolve(recorded, torch.as_tensor(excitation, device="cuda"), dt, case["max_frequency"])
        return {"signals": signals, "recorded": recorded}
    rooms = _descriptions(case, seed)
    if kind == "room":
        recorded, p = _leapfrog(rooms[0])
        return {"recorded": recorded, "p": p}
    if kind == "batch":
        return {"recorded": [_leapfrog(d)[0] for d in rooms]}
    targets = _targets(case, seed, rooms)
    if kind == "gradient":
        recorded, g, walls, cells = _gradients(rooms[0], targets[0])
        out = {"recorded": recorded, "signal": g[0][None], "walls": walls, "initial_p": g[1], "wall_cells": cells}
        if case["air"]:
            out.update(strength=g[8], relaxation_time=g[9])
        return out
    out = {"recorded": [], "signal": [], "walls": [], "wall_cells": []}
    for d, target in zip(rooms, targets):
        recorded, g, walls, cells = _gradients(d, target)
        out["recorded"].append(recorded)
        out["signal"].append(g[0][None].detach())
        out["walls"].append(walls)
        out["wall_cells"].append(cells)
        del g
    return out

"""The workloads this project's speed is measured on, each one a pass through
the public entry points (engine, batch, studies, closure, C ABI).

Every case is a dict of plain values; its `kind` says what a pass is:

  sim      a whole small simulation: a new grid, its scene voxelized, CPML,
           engine.run (sources and probes included), the FieldBlock snapshot
  wave     a validation study's plane-wave run (nx x 8 x 8, periodic y and z,
           hard sheet source, probe trace)
  step     `steps` more steps of a resident grid; FP32 grids hand back their
           device fields, 16-bit grids the FP32 view in pinned host memory,
           grids with probes the probe sums too
  pool     wf_step_fields_noalloc on the caller's own device fields
  batch    `steps` steps of a DeviceBatch of uneven cubes
  closure  steps of a thin-CPML grid with the learned boundary closure
  train    one training step of the closure network

Sizes, CPML depths, materials and sources follow configs.py, studies.py,
closure.py, bench.py and the tests.  The inputs of a case are made from its
seed on the GPU: fields start as noise (E of order 1, H of order 1/eta0), so
that every cell and every psi carries values from the first step on.
`exact` is an independent float64 restatement in plain torch.
"""
from __future__ import annotations

import ctypes as C
import math
import random

import numpy as np
import torch

import wavefront_b200 as wb
from wavefront_b200 import closure as wc
from wavefront_b200 import studies

DEV = "cuda"
C0 = 299792458.0
EPS0, MU0 = np.float32(8.854188e-12), np.float32(1.2566371e-6)
DX = 1.0e-3
DT = float(np.float32(0.99 / math.sqrt(3.0) * DX / C0))
OMEGA_DT = 2.0 * math.pi * (C0 / (20.0 * DX)) * DT  # 20 cells per wavelength
F0 = float(np.float32(C0 / (20.0 * DX)))


def listed():
    return [
        # the plain 64^3 run end to end (configs.plain_cube_64 with a scene): what
        # a caller with many small jobs pays per job, set-up and results included
        {"name": "sim_64", "kind": "sim", "n": 64, "steps": 500, "cells": 10},
        # one run of the dispersion and reflection studies: a long, tiny domain,
        # periodic y and z, 1000 steps, launches and latency only
        {"name": "wave_560", "kind": "wave", "nx": 560, "steps": 1000, "cells": 16},
        # the smallest call: one step of a 32^3 grid per call, as in a loop that
        # looks at the fields after every step
        {"name": "step1_32", "kind": "step", "nx": 32, "ny": 32, "nz": 32, "steps": 1, "cells": 8,
         "exact_pml": False, "arith": "exact", "precision": "f32", "periodic": "", "probes": 0},
        # ten steps of an application's own 64^3 fields, nothing allocated
        {"name": "pool_64", "kind": "pool", "nx": 64, "ny": 64, "nz": 64, "steps": 10,
         "arith": "exact", "periodic": ""},
        # the reference's benchmark shape: 256^3, 8-cell CPML (fields larger than L2)
        {"name": "demo_256", "kind": "step", "nx": 256, "ny": 256, "nz": 256, "steps": 50,
         "cells": 8, "exact_pml": False, "arith": "exact", "precision": "f32", "periodic": "",
         "probes": 0},
        # the headline throughput run: 512^3, 16-cell CPML, source and 8 probes read
        {"name": "spheres_512", "kind": "step", "nx": 512, "ny": 512, "nz": 512, "steps": 32,
         "cells": 16, "exact_pml": False, "arith": "exact", "precision": "f32", "periodic": "",
         "probes": 8},
        # ragged extents, a per-cell 10-cell CPML and the FMA arithmetic
        {"name": "ragged_fma", "kind": "step", "nx": 264, "ny": 136, "nz": 200, "steps": 24,
         "cells": 10, "exact_pml": True, "arith": "fma", "precision": "f32", "periodic": "",
         "probes": 2},
        # binary16 storage: a hundred steps, then the FP32 view of the state read
        {"name": "half_320", "kind": "step", "nx": 320, "ny": 320, "nz": 320, "steps": 100,
         "cells": 16, "exact_pml": False, "arith": "exact", "precision": "f16", "periodic": "",
         "probes": 4},
        # a photonic-crystal cell: periodic in x and y, CPML in z
        {"name": "periodic_xy", "kind": "step", "nx": 192, "ny": 160, "nz": 256, "steps": 20,
         "cells": 16, "exact_pml": True, "arith": "exact", "precision": "f32", "periodic": "xy",
         "probes": 2},
        # the parameter sweep: 48 cubes of 32-128 cells stepped together
        {"name": "batch_48", "kind": "batch", "scenes": 48, "lo": 32, "hi": 128, "steps": 32,
         "cells": 10},
        # the thin 4-cell layer with the learned closure after every step
        {"name": "closure_232", "kind": "closure", "n": 232, "steps": 4},
        # one training step of the closure network on a batch of crops
        {"name": "train_128", "kind": "train", "batch": 128, "crop": 16},
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _m8(v, lo=8):
    return max(lo, int(round(v / 8.0)) * 8)


def draw(rng: random.Random):
    kind = rng.choices(["step", "half", "periodic", "sim", "wave", "pool", "batch", "closure",
                        "train"], [6, 2, 2, 2, 1, 1, 2, 1, 1])[0]
    if kind == "sim":
        return {"kind": "sim", "n": _m8(_log_uniform(rng, 32, 128)), "steps": rng.randint(100, 500),
                "cells": rng.choice([0, 4, 8, 10, 16])}
    if kind == "wave":
        return {"kind": "wave", "nx": _m8(_log_uniform(rng, 300, 1680)),
                "steps": rng.randint(400, 1500), "cells": rng.choice([0, 8, 16, 32])}
    if kind == "pool":
        d = [_m8(_log_uniform(rng, 8, 64)) for _ in range(3)]
        return {"kind": "pool", "nx": d[0], "ny": d[1], "nz": d[2], "steps": rng.randint(1, 40),
                "arith": rng.choice(["exact", "exact", "fma"]),
                "periodic": rng.choice(["", "yz", "xyz"])}
    if kind == "batch":
        lo = _m8(_log_uniform(rng, 24, 64))
        return {"kind": "batch", "scenes": int(_log_uniform(rng, 3, 60)), "lo": lo,
                "hi": lo + 8 * rng.randint(1, 9), "steps": rng.randint(8, 64),
                "cells": rng.choice([4, 8, 10])}
    if kind == "closure":
        return {"kind": "closure", "n": _m8(_log_uniform(rng, 40, 240)), "steps": rng.randint(2, 8)}
    if kind == "train":
        return {"kind": "train", "batch": int(_log_uniform(rng, 16, 256)),
                "crop": rng.choice([8, 12, 16, 20, 24])}
    if kind == "periodic":
        d = [_m8(_log_uniform(rng, 16, 256)) for _ in range(3)]
        axes = rng.choice(["x", "xy", "yz", "xyz"])
        prec, arith, top = "f32", rng.choice(["exact", "exact", "fma"]), 256 ** 3
        cells = rng.choice([0, 4, 10, 16])
    elif kind == "half":
        d = [_m8(_log_uniform(rng, 64, 384)) for _ in range(3)]
        axes, prec, arith, top = "", rng.choice(["f16", "bf16"]), "exact", 320 ** 3
        cells = rng.choice([4, 8, 10, 16, 24])
    else:
        m = _log_uniform(rng, 32, 440)
        d = [_m8(m * rng.uniform(0.6, 1.5)) for _ in range(3)]
        axes, prec, arith, top = "", "f32", rng.choice(["exact", "exact", "exact", "fma"]), 480 ** 3
        cells = rng.choice([0, 4, 8, 8, 10, 16, 16, 24, 32])
    while d[0] * d[1] * d[2] > top:
        k = d.index(max(d))
        d[k] = _m8(0.8 * d[k])
    most = max(1, min(64, (1 << 31) // (d[0] * d[1] * d[2])))
    return {"kind": "step", "nx": d[0], "ny": d[1], "nz": d[2],
            "steps": max(1, int(_log_uniform(rng, 1, most))), "cells": cells,
            "exact_pml": rng.random() < 0.5, "arith": arith, "precision": prec, "periodic": axes,
            "probes": rng.choice([0, 1, 4, 8])}


# ---- inputs shared by prepare and exact ---------------------------------------


def _q16(eps_r, sigma):
    """{ca, cb, da, db} of a material as Q16.16 integers (f32 arithmetic)."""
    f = np.float32
    eps, mu, dt, dx = f(eps_r) * EPS0, f(1.0) * MU0, f(DT), f(DX)
    loss = f(sigma) * dt / (f(2.0) * eps)
    vals = [(f(1) - loss) / (f(1) + loss), (dt / (eps * dx)) / (f(1) + loss), f(1), dt / (mu * dx)]
    return [int(math.floor(float(v * f(65536.0)) + 0.5)) for v in vals]


def _profile(n, t, dt=DT, dx=DX):
    """b, a, 1/kappa along an axis of n cells with a t-cell graded layer (f32)."""
    f = np.float32
    b, a, ik = np.ones(n, f), np.zeros(n, f), np.ones(n, f)
    if t > 0:
        depth = f(t) * f(dx)
        smax = -(f(4.0)) * np.log(f(1e-6)) / (f(2.0) * np.sqrt(MU0 / EPS0) * depth)
        for g in range(t):
            rho = f(t - g) / f(t)
            sig, kap = smax * rho ** f(3.0), f(1.0) + f(6.0) * rho ** f(3.0)
            alpha = f(0.05) * (f(1.0) - rho)
            bb = np.exp(-(sig / kap + alpha) * f(dt) / EPS0)
            den = kap * (sig + kap * alpha)
            for i in (g, n - 1 - g):
                b[i], ik[i] = bb, f(1.0) / kap
                a[i] = sig * (bb - f(1.0)) / den if abs(den) > 1e-30 else f(0.0)
    return b, a, ik


def _spheres(rng, dims, count):
    """`count` spheres (eps_r, sigma, centre, radius), coordinates in quarters."""
    out = []
    for _ in range(count):
        c = [rng.randrange(0, 4 * d) / 4.0 for d in dims]
        r = max(2.0, rng.randrange(int(min(dims) / 4), int(min(dims)) + 1) / 4.0)
        out.append((rng.randrange(8, 64) / 8.0, rng.choice([0.0, rng.randrange(1, 64) / 6400.0]), c, r))
    return out


def _text(spheres):
    return "".join(f"sphere {e:.9g} 1.0 {s:.9g} {c[0]:.9g} {c[1]:.9g} {c[2]:.9g} {r:.9g}\n"
                   for e, s, c, r in spheres)


def _graded(dims, cells, exact_pml, periodic):
    """Graded thickness per axis: rounded to whole blocks as the engine does, or per cell."""
    if not exact_pml:
        t = 8 * min(-(-cells // 8), max(1, (min(dims) // 8) // 2)) if cells else 0
        ts = [t, t, t]
    else:
        ts = [min(cells, d // 2) for d in dims]
    return [0 if "xyz"[i] in periodic else ts[i] for i in range(3)]


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _noise(out, seed):
    """Fills a [6][nz][ny][nx] float32 device tensor with E ~ 1, H ~ 1/eta0."""
    out.normal_(generator=_gen(seed))
    out[3:].mul_(1.0 / 377.0)
    return out


def _wave_table(n):
    return np.sin(OMEGA_DT * (np.arange(n) + 1.0)).astype(np.float32)


def _source_at(rng, dims):
    return tuple(rng.randrange(d // 4, max(d // 4 + 1, 3 * d // 4)) for d in dims)


def _probe_at(dims, k):
    return (dims[0] // 16 + (dims[0] * k) // 9, dims[1] // 2, (7 * dims[2]) // 8)


class _Device:
    """A device array of the library as torch sees it; `owner` lives as long as
    the tensor does (torch holds this object, which holds the owner)."""

    def __init__(self, ptr, shape, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": tuple(shape), "typestr": "<f4",
                                         "data": (int(ptr), False), "version": 2}


def _view(ptr, dims, owner):
    return torch.as_tensor(_Device(ptr, (6, dims[2], dims[1], dims[0]), owner), device=DEV)


def _weights(seed):
    g = torch.Generator().manual_seed(int(seed))
    out = []
    for layer, (ci, co) in enumerate(((10, 16), (16, 16), (16, 6))):
        scale = math.sqrt(2.0 / (ci * 27)) * (0.05 if layer == 2 else 1.0)
        out.append(torch.randn(6, co, ci, 27, generator=g) * scale)
    return out


# ---- prepare / run --------------------------------------------------------------


def _case_dims(case):
    return (case["nx"], case["ny"], case["nz"])


def _fill_state(grid, dims, seed, s):
    """Noise into the grid's current FP32 fields, where they are."""
    grid.sync()
    _noise(_view(grid.device_field_ptrs()[0], dims, grid), seed)
    torch.cuda.synchronize()
    s["views"] = {}


def _fields(s):
    p = s["grid"].device_field_ptrs()[0]
    v = s["views"].get(p)
    if v is None:
        v = s["views"][p] = _view(p, s["dims"], s["grid"])
    return v


def _prepare_step(case, seed):
    dims, rng = _case_dims(case), random.Random(seed)
    g = wb.DeviceFieldGrid(wb.GridDims(*dims), arith=case["arith"], precision=case["precision"],
                           boundary=tuple("periodic" if a in case["periodic"] else "zero" for a in "xyz"))
    g.set_scene(_text(_spheres(rng, dims, 3)), wb.MaterialTable.vacuum_filled(DT, DX), DT, DX)
    for ax, t in enumerate(_graded(dims, case["cells"], case["exact_pml"], case["periodic"])):
        if t:
            g.set_pml_axis(ax, t, *_profile(dims[ax], t))
    # tables for a long-running program: at least 65 536 steps
    n = 1 << (20 if dims[0] * dims[1] * dims[2] <= 1 << 21 else 16)
    x, y, z = _source_at(rng, dims)
    g.add_source_values(x, y, z, 2, _wave_table(n))
    for k in range(case["probes"]):
        ph = OMEGA_DT * (np.arange(n) + 1.0)
        g.add_probe_tables(*_probe_at(dims, k), 2, np.cos(ph)[:, None], np.sin(ph)[:, None])
    s = {"grid": g, "dims": dims}
    if case["precision"] == "f32":
        _fill_state(g, dims, seed, s)
    else:
        # the FP32 view crosses the host link through a pinned buffer
        s["host"] = torch.empty((6, dims[2], dims[1], dims[0]), pin_memory=True)
        s["host"].copy_(_noise(torch.empty(s["host"].shape, device=DEV), seed))
        g.set_fields(s["host"].numpy())
    return s


def _run_step(case, s):
    g = s["grid"]
    g.step(case["steps"])
    out = {}
    if case["probes"]:
        sums = [g.probe_sums(k, 1) for k in range(case["probes"])]
        out["cos"] = np.array([c[0] for c, _, _ in sums])
        out["sin"] = np.array([c[0] for _, c, _ in sums])
    if case["precision"] == "f32":
        out["fields"] = _fields(s)
    else:
        L = wb.lib()
        st = L.wf_get_fields(g._h, C.cast(s["host"].data_ptr(), C.POINTER(C.c_float)))
        if st:
            raise wb.WfError(st, "wf_get_fields")
        out["fields"] = s["host"]
    return out


def _prepare_sim(case, seed):
    n, rng = case["n"], random.Random(seed)
    dims = wb.GridDims(n, n, n)
    x, y, z = _source_at(rng, (n, n, n))
    return {"dims": dims, "text": _text(_spheres(random.Random(seed), (n, n, n), 3)),
            "pml": wb.PmlContext.build(dims, wb.PmlConfig(thickness=case["cells"]), DT, DX),
            "source": wb.Source(x, y, z, wb.FieldComponent.Ez, 1.0, wb.default_waveform("ricker", F0))}


def _run_sim(case, s):
    n = case["n"]
    with wb.DeviceFieldGrid(s["dims"]) as g:
        g.set_scene(s["text"], wb.MaterialTable.vacuum_filled(DT, DX), DT, DX)
        if case["cells"]:
            g.set_pml(s["pml"])
        p = wb.Probe(n // 2, n // 2, n // 4, wb.ProbeComponent.Ez, [F0], record_trace=True)
        wb.run(g, [s["source"]], [p], wb.EngineConfig(case["steps"], DT))
        return {"blocks": g.download_blocks(), "trace": p.trace, "cos": p.sum_cos, "sin": p.sum_sin}


def _wave_case(case, seed):
    """nx, dx, dt, freq, source and probe columns, steps, layer of a study's run."""
    f = np.float32
    freq = f(3.0e10 * (0.9 + 0.2 * random.Random(seed).random()))
    dx = f(f(f(C0) / f(3.0e10)) / f(20.0))
    dt = f(f(f(0.4) * dx) / f(C0))
    xs = case["nx"] // 3
    return case["nx"], dx, dt, freq, xs, xs + min(120, case["nx"] // 4), case["steps"], case["cells"]


def _prepare_pool(case, seed):
    dims, rng = _case_dims(case), random.Random(seed)
    ids, table = _ids_and_table(_spheres(rng, dims, 3), dims)
    q = np.ascontiguousarray(table, np.int32)
    f = _noise(torch.empty((6, dims[2], dims[1], dims[0]), device=DEV), seed)
    bnd = (C.c_int32 * 3)(*[int(a in case["periodic"]) for a in "xyz"])
    return {"fields": f, "ids": ids.contiguous(), "q": q, "bnd": bnd}


def _run_pool(case, s):
    st = wb.lib().wf_step_fields_noalloc(
        s["fields"].data_ptr(), s["ids"].data_ptr(), s["q"].ctypes.data_as(C.POINTER(C.c_int32)),
        case["nx"], case["ny"], case["nz"], s["bnd"], int(case["arith"] == "fma"), case["steps"],
        torch.cuda.current_stream().cuda_stream)
    if st:
        raise wb.WfError(st, wb.lib().wf_noalloc_last_error().decode())
    return {"fields": s["fields"]}


def _batch_sizes(case, seed):
    rng = random.Random(seed)
    ns = [_m8(rng.uniform(case["lo"], case["hi"])) for _ in range(case["scenes"])]
    return ns, [rng.randrange(1 << 30) for _ in ns]


def _prepare_batch(case, seed):
    # the sizes are the case's own (the same sweep for every seed); contents are the seed's
    ns, _ = _batch_sizes(case, case["scenes"] * 1000 + case["lo"])
    _, seeds = _batch_sizes(case, seed)
    b = wb.DeviceBatch([wb.GridDims(n, n, n) for n in ns])
    steps = 1 << 16
    wave = _wave_table(steps)
    ph = OMEGA_DT * (np.arange(steps) + 1.0)
    cos, sin = np.cos(ph)[:, None], np.sin(ph)[:, None]
    for g, n, sd in zip(b.grids, ns, seeds):
        rng = random.Random(sd)
        g.set_scene(_text(_spheres(rng, (n, n, n), 2)), wb.MaterialTable.vacuum_filled(DT, DX), DT, DX)
        t = min(case["cells"], n // 2)
        prof = _profile(n, t)
        for ax in range(3):
            g.set_pml_axis(ax, t, *prof)
        g.add_source_values(*_source_at(rng, (n, n, n)), 2, wave)
        g.add_probe_tables(n // 2, n // 2, n // 4, 2, cos, sin)
    b.sync()
    for g, n, sd in zip(b.grids, ns, seeds):
        _noise(_view(g.device_field_ptrs()[0], (n, n, n), b), sd)
    torch.cuda.synchronize()
    return {"batch": b, "ns": ns, "views": {}}


def _run_batch(case, s):
    b = s["batch"]
    b.step(case["steps"])
    b.sync()
    out = []
    for g, n in zip(b.grids, s["ns"]):
        p = g.device_field_ptrs()[0]
        if p not in s["views"]:
            s["views"][p] = _view(p, (n, n, n), b)
        out.append(s["views"][p])
    return out


def _thin_profile(n):
    """The innermost 4 cells of a 16-cell grading (closure.truncated_profiles)."""
    b, a, ik = _profile(n + 24, 16)
    return tuple(np.ascontiguousarray(v[12:12 + n]) for v in (b, a, ik))


def _prepare_closure(case, seed):
    n, rng = case["n"], random.Random(seed)
    dims = (n, n, n)
    g = wb.DeviceFieldGrid(wb.GridDims(n, n, n))
    g.set_scene(_text(_spheres(rng, dims, 3)), wb.MaterialTable.vacuum_filled(DT, DX), DT, DX)
    for ax in range(3):
        g.set_pml_axis(ax, 4, *_thin_profile(n))
    g.add_source_values(*_source_at(rng, dims), 2, _wave_table(1 << 16))
    net = wc.ClosureNet(seed=0)
    net.load_state({"w": [w.numpy() for w in _weights(seed)], "gain_e": 1.0, "gain_h": wc.ETA0, "t": 0})
    torch.cuda.synchronize()
    net.attach(g)
    s = {"grid": g, "dims": dims, "net": net}
    _fill_state(g, dims, seed, s)
    return s


def _run_closure(case, s):
    s["grid"].step(case["steps"])
    return {"fields": _fields(s)}


def _train_data(case, seed):
    m, c = case["batch"], case["crop"]
    g = _gen(seed)
    x = torch.randn(m, 10, 8, c, c, device=DEV, generator=g)
    t = torch.randn(m, 6, 8, c, c, device=DEV, generator=g)
    face = torch.randint(0, 6, (m,), device=DEV, generator=g).to(torch.int32)
    return x, t, face


def _prepare_train(case, seed):
    net = wc.ClosureNet(seed=0)
    net.load_state({"w": [w.numpy() for w in _weights(seed)], "gain_e": 1.0, "gain_h": wc.ETA0, "t": 0})
    return {"net": net, "data": _train_data(case, seed)}


def _run_train(case, s):
    net = s["net"]
    loss = net.train_step(*s["data"], lr=3e-4)
    return {"loss": loss, "grad": list(net.dw), "w": list(net.w)}


def prepare(case, seed):
    kind = case["kind"]
    if kind == "wave":
        s = {"args": _wave_case(case, seed)}
    else:
        s = {"step": _prepare_step, "sim": _prepare_sim, "pool": _prepare_pool,
             "batch": _prepare_batch, "closure": _prepare_closure, "train": _prepare_train}[kind](case, seed)
    s["case"] = case
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "wave":
        return {"trace": studies.plane_wave_trace(*s["args"])}
    return {"step": _run_step, "sim": _run_sim, "pool": _run_pool, "batch": _run_batch,
            "closure": _run_closure, "train": _run_train}[kind](case, s)


# ---- the work of a pass ---------------------------------------------------------


def _slab_cells(dims, ts):
    n = dims[0] * dims[1] * dims[2]
    return sum(n // dims[i] * min(2 * ts[i], dims[i]) for i in range(3))


def _step_work(dims, ts, elem=4):
    """One step: every field read and written once, the id read, every psi read and written."""
    n = dims[0] * dims[1] * dims[2]
    p = _slab_cells(dims, ts)
    return n * (12 * elem + 1) + 32 * p, 36 * n + 16 * p


def work(case):
    kind, steps = case["kind"], case.get("steps", 1)
    if kind == "train":
        m, p = case["batch"], 8 * case["crop"] ** 2
        macs = 27 * (10 * 16 + 16 * 16 + 16 * 6) * m * p
        w = 27 * 6 * (160 + 256 + 96)
        return {"bytes": 4 * m * p * (10 + 6) + 30 * w, "flops": 2 * (3 * macs - 27 * 160 * m * p)}
    if kind == "batch":
        ns, _ = _batch_sizes(case, case["scenes"] * 1000 + case["lo"])
        each = [_step_work((n, n, n), [min(case["cells"], n // 2)] * 3) for n in ns]
        return {"bytes": steps * sum(b for b, _ in each), "flops": steps * sum(f for _, f in each)}
    if kind == "wave":
        dims, ts = (case["nx"], 8, 8), [case["cells"], 0, 0]
    elif kind in ("sim", "closure"):
        dims = (case["n"],) * 3
        ts = [4] * 3 if kind == "closure" else _graded(dims, case["cells"], False, "")
    elif kind == "pool":
        dims, ts = _case_dims(case), [0, 0, 0]
    else:
        dims = _case_dims(case)
        ts = _graded(dims, case["cells"], case["exact_pml"], case["periodic"])
    b, f = _step_work(dims, ts, 2 if case.get("precision", "f32") != "f32" else 4)
    b, f = b * steps, f * steps
    n = dims[0] * dims[1] * dims[2]
    if kind == "closure":  # the bands read (6 fields, 4 psi) and corrected (6 fields), the network
        p = 6 * 8 * dims[0] ** 2
        b += steps * 4 * p * (6 + 4 + 12)
        f += steps * 2 * 27 * (10 * 16 + 16 * 16 + 16 * 6) * p
    if kind == "sim" or case.get("precision", "f32") != "f32":
        b += 24 * n  # the state handed to the host
    return {"bytes": b, "flops": f}


# ---- float64 restatement ----------------------------------------------------------


def _ids_and_table(spheres, dims):
    """Cell ids [nz][ny][nx] (later spheres overwrite, equal materials share an
    id) and the 256-entry Q16.16 table."""
    x, y, z = (torch.arange(d, device=DEV, dtype=torch.float64) + 0.5 for d in dims)
    ids = torch.zeros((dims[2], dims[1], dims[0]), dtype=torch.uint8, device=DEV)
    table = np.tile(np.array(_q16(1.0, 0.0)), (256, 1))
    known = []
    for e, sg, c, r in spheres:
        if (e, sg) not in known:
            known.append((e, sg))
            table[len(known)] = _q16(np.float32(float(f"{e:.9g}")), np.float32(float(f"{sg:.9g}")))
        d2 = ((x - c[0]) ** 2)[None, None, :] + ((y - c[1]) ** 2)[None, :, None]
        for k in range(dims[2]):  # plane by plane: no grid-sized temporaries
            ids[k][(d2[0] + (z[k] - c[2]) ** 2) <= r * r] = known.index((e, sg)) + 1
    return ids, table


class _Yee:
    """H, E, CPML, sources and probes in float64."""

    def __init__(self, dims, ids, table, fields, profiles, periodic=""):
        coef = torch.tensor(np.asarray(table, np.float64) / 65536.0, device=DEV)
        i = ids.long()
        self.ca, self.cb, self.da, self.db = (coef[:, k][i] for k in range(4))
        self.f = list(fields.double().unbind(0)) if fields is not None else [
            torch.zeros(ids.shape, dtype=torch.float64, device=DEV) for _ in range(6)]
        self.prof, self.periodic = [], periodic
        for ax, p in enumerate(profiles):
            shape = [1, 1, 1]
            shape[2 - ax] = -1
            self.prof.append(None if p is None else tuple(
                torch.tensor(v, dtype=torch.float64, device=DEV).reshape(shape) for v in p))
        self.psi = [None if p is None else [torch.zeros(ids.shape, dtype=torch.float64, device=DEV)
                                            for _ in range(4)] for p in profiles]

    def _diff(self, v, ax, up, k):
        """Forward (up) or backward difference along axis ax, corrected; k is its psi slot."""
        dim = 2 - ax
        n = v.shape[dim]
        r = torch.roll(v, -1 if up else 1, dim)
        if "xyz"[ax] not in self.periodic:
            r.select(dim, n - 1 if up else 0).zero_()
        d = r.sub_(v) if up else v - r
        if self.prof[ax] is not None:
            b, a, ik = self.prof[ax]
            psi = self.psi[ax][k]
            psi.mul_(b).add_(a * d)
            d = d.mul_(ik).add_(psi)
        return d

    def step(self):
        f, d = self.f, self._diff
        cx = d(f[2], 1, True, 0) - d(f[1], 2, True, 0)
        cy = d(f[0], 2, True, 1) - d(f[2], 0, True, 0)
        cz = d(f[1], 0, True, 1) - d(f[0], 1, True, 1)
        for k, c in ((3, cx), (4, cy), (5, cz)):
            f[k] = self.da * f[k] - self.db * c
        cx = d(f[5], 1, False, 2) - d(f[4], 2, False, 2)
        cy = d(f[3], 2, False, 3) - d(f[5], 0, False, 2)
        cz = d(f[4], 0, False, 3) - d(f[3], 1, False, 3)
        for k, c in ((0, cx), (1, cy), (2, cz)):
            f[k] = self.ca * f[k] + self.cb * c


def _conv(x, w, faces):
    """3x3x3 convolutions, each sample with its face's weights [6][co][ci][27]."""
    out = x.new_empty((x.shape[0], w.shape[1]) + x.shape[2:])
    parts = []
    for f in range(6):
        sel = torch.nonzero(faces == f).flatten()
        if sel.numel():
            k = w[f].reshape(w.shape[1], w.shape[2], 3, 3, 3)
            parts.append((sel, torch.nn.functional.conv3d(x[sel], k, padding=1)))
    order = torch.cat([s for s, _ in parts])
    out = torch.cat([p for _, p in parts])
    return out[torch.argsort(order)]


def _gelu(z):
    return 0.5 * z * (1.0 + torch.erf(z / math.sqrt(2.0)))


def _close(sim, ws, ge, gh):
    """The closure on the six 8-cell bands of a cubic grid."""
    def bands(v, ax):  # [n along the axis][u][v] view
        v = v.permute(2, 1, 0)
        return v if ax == 0 else v.permute(1, 0, 2) if ax == 1 else v.permute(2, 0, 1)

    xs = []
    for face in range(6):
        ax = face // 2
        rows = []
        for k, v in enumerate(sim.f + sim.psi[ax]):
            b = bands(v, ax)
            b = b[:8] if face % 2 == 0 else b[-8:].flip(0)
            gain = ge if k < 3 or 6 <= k < 8 else gh
            rows.append(b * gain)
        xs.append(torch.stack(rows))
    x = torch.stack(xs)
    rms = x[:, :3].square().mean(dim=(1, 2, 3, 4)).sqrt().reshape(6, 1, 1, 1, 1)
    faces = torch.arange(6, device=DEV)
    a = _gelu(_conv(x / rms, ws[0], faces))
    a = _gelu(_conv(a, ws[1], faces))
    y = _conv(a, ws[2], faces) * rms
    for face in range(6):
        ax = face // 2
        for k in range(6):
            b = bands(sim.f[k], ax)
            yk = y[face, k] / (ge if k < 3 else gh)
            if face % 2 == 0:
                b[:8] += yk
            else:
                b[-8:] += yk.flip(0)


def _march(sim, steps, at=None, values=None, sheet=None, probes=(), after=None):
    """`steps` steps with one Ez source; returns the probes' Ez samples [steps][probe]."""
    rows = []
    for s in range(steps):
        sim.step()
        if after is not None:
            after(sim)
        if sheet is not None:
            sim.f[2][:, :, sheet] = float(values[s])
        elif at is not None:
            sim.f[2][at[2], at[1], at[0]] += float(values[s])
        if probes:
            rows.append(torch.stack([sim.f[2][z, y, x] for x, y, z in probes]))
    return torch.stack(rows).cpu().numpy() if rows else None


def _dft(rows, omega_dt=None, phase=None):
    ph = omega_dt * (np.arange(len(rows)) + 1.0) if phase is None else phase
    return (rows * np.cos(ph)[:, None]).sum(0), (rows * np.sin(ph)[:, None]).sum(0)


def _exact_step(case, seed):
    dims, rng = _case_dims(case), random.Random(seed)
    ids, table = _ids_and_table(_spheres(rng, dims, 3), dims)
    ts = _graded(dims, case["cells"], case["exact_pml"], case["periodic"])
    f = _noise(torch.empty((6, dims[2], dims[1], dims[0]), device=DEV), seed)
    sim = _Yee(dims, ids, table, f, [_profile(dims[i], ts[i]) if ts[i] else None for i in range(3)],
               case["periodic"])
    del f
    at = _source_at(rng, dims)
    rows = _march(sim, case["steps"], at, _wave_table(case["steps"]),
                  probes=[_probe_at(dims, k) for k in range(case["probes"])])
    out = {"fields": torch.stack(sim.f)}
    if case["probes"]:
        out["cos"], out["sin"] = _dft(rows, OMEGA_DT)
    return out


def _exact_sim(case, seed):
    n = case["n"]
    dims, rng = (n, n, n), random.Random(seed)
    at = _source_at(rng, dims)
    ids, table = _ids_and_table(_spheres(random.Random(seed), dims, 3), dims)
    t = _graded(dims, case["cells"], False, "")[0]
    sim = _Yee(dims, ids, table, None, [_profile(n, t) if t else None] * 3)
    f = np.float32
    time = (np.arange(case["steps"], dtype=f) + f(1.0)) * f(DT)
    arg = f(np.pi) * f(F0) * (time - f(1.0) / f(F0))
    values = (f(1.0) - f(2.0) * arg * arg) * np.exp(-(arg * arg))
    rows = _march(sim, case["steps"], at, values, probes=[(n // 2, n // 2, n // 4)])
    blocks = torch.stack(sim.f).reshape(6, n // 8, 8, n // 8, 8, n // 8, 8).permute(1, 3, 5, 0, 2, 4, 6)
    cos, sin = _dft(rows, phase=2.0 * math.pi * float(f(F0)) * time.astype(np.float64))
    return {"blocks": blocks.reshape(-1), "trace": rows[:, 0], "cos": cos, "sin": sin}


def _exact_wave(case, seed):
    nx, dx, dt, freq, xs, xp, steps, cells = _wave_case(case, seed)
    f = np.float32
    t = 8 * min(-(-cells // 8), (nx // 8) // 2)
    dims = (nx, 8, 8)
    q = [int(math.floor(float(v * f(65536.0)) + 0.5)) for v in
         (f(1), dt / (EPS0 * dx), f(1), dt / (MU0 * dx))]
    sim = _Yee(dims, torch.zeros((8, 8, nx), dtype=torch.uint8, device=DEV), np.tile(np.array(q), (256, 1)),
               None, [_profile(nx, t, dt, dx) if t else None, None, None], "yz")
    time = (np.arange(steps, dtype=f) + f(1.0)) * dt
    values = np.sin(f(2.0) * f(np.pi) * freq * time)
    rows = _march(sim, steps, values=values, sheet=xs, probes=[(xp, 0, 0)])
    return {"trace": rows[:, 0]}


def _exact_pool(case, seed):
    dims, rng = _case_dims(case), random.Random(seed)
    ids, table = _ids_and_table(_spheres(rng, dims, 3), dims)
    f = _noise(torch.empty((6, dims[2], dims[1], dims[0]), device=DEV), seed)
    sim = _Yee(dims, ids, table, f, [None] * 3, case["periodic"])
    _march(sim, case["steps"])
    return {"fields": torch.stack(sim.f)}


def _exact_batch(case, seed):
    ns, _ = _batch_sizes(case, case["scenes"] * 1000 + case["lo"])
    _, seeds = _batch_sizes(case, seed)
    out = []
    for k, (n, sd) in enumerate(zip(ns, seeds)):
        if k % 6:  # every sixth grid: all of them would take minutes
            out.append(None)
            continue
        dims, rng = (n, n, n), random.Random(sd)
        ids, table = _ids_and_table(_spheres(rng, dims, 2), dims)
        t = min(case["cells"], n // 2)
        sim = _Yee(dims, ids, table, _noise(torch.empty((6, n, n, n), device=DEV), sd),
                   [_profile(n, t)] * 3)
        _march(sim, case["steps"], _source_at(rng, dims), _wave_table(case["steps"]))
        out.append(torch.stack(sim.f))
    return out


def _exact_closure(case, seed):
    n, rng = case["n"], random.Random(seed)
    dims = (n, n, n)
    ids, table = _ids_and_table(_spheres(rng, dims, 3), dims)
    sim = _Yee(dims, ids, table, _noise(torch.empty((6, n, n, n), device=DEV), seed),
               [_thin_profile(n)] * 3)
    ws = [w.to(DEV).to(torch.bfloat16).double() for w in _weights(seed)]
    gh = float(np.float32(wc.ETA0))
    _march(sim, case["steps"], _source_at(rng, dims), _wave_table(case["steps"]),
           after=lambda s: _close(s, ws, 1.0, gh))
    return {"fields": torch.stack(sim.f)}


def _exact_train(case, seed):
    x, t, face = _train_data(case, seed)
    w32 = [w.to(DEV) for w in _weights(seed)]
    ws = [w.to(torch.bfloat16).double().requires_grad_(True) for w in w32]
    a = _gelu(_conv(x.double(), ws[0], face))
    a = _gelu(_conv(a, ws[1], face))
    loss = (_conv(a, ws[2], face) - t.double()).square().mean()
    loss.backward()
    w_new = []
    for w, p in zip(w32, ws):  # the first Adam step: both moments start at zero
        g = p.grad
        w_new.append(w.double() - 3e-4 * g / (g.abs() + 1e-8))
    return {"loss": loss.detach().reshape(1), "grad": [p.grad for p in ws], "w": w_new}


def exact(case, seed):
    with torch.backends.cudnn.flags(enabled=False):
        return {"step": _exact_step, "sim": _exact_sim, "wave": _exact_wave, "pool": _exact_pool,
                "batch": _exact_batch, "closure": _exact_closure, "train": _exact_train}[case["kind"]](case, seed)

"""GPU: the bounds-checked device build (libwavefront_gpu_checked.so).

compute-sanitizer is not available on the GPU pool, so the library has a
debugging variant compiled with -DWF_BOUNDS_CHECK: every global access of
the step kernels (fused and split: field and psi loads and stores) and of
the step tail (source and probe cells) tests its index against its buffer
and, when it is out of range, latches a device error flag (reported by
wf_sync) and skips the access.  Here the small-grid parity cases run under
that build in a fresh process (the library is chosen when it is loaded):
results must equal the oracle's bit for bit with no flag raised.
"""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SCRIPT = r'''
import os, sys
import numpy as np
sys.path.insert(0, os.environ["WF_ROOT"])
import wavefront_b200 as wf
from wavefront_b200 import _lib as L, configs
from oracle import oracle as O
assert L.LIB_PATH.endswith("libwavefront_gpu_checked.so")

def run(sc, steps, prec="f32", arith="exact", **kw):
    g = configs.device_grid(sc, precision=prec, arith=arith, **{k: v for k, v in kw.items() if k == "kernel"})
    if "columns" in kw:
        g.set_column_tiles(kw["columns"])
    for s in sc.sources:
        g.add_source_values(s.x, s.y, s.z, s.component, s.values(sc.dt, steps), s.mode)
    for p in sc.probes:
        c, si = p.tables(sc.dt, steps)
        g.add_probe_tables(p.x, p.y, p.z, p.component, c, si, p.first_step(sc.dt))
    g.step(steps)
    g.sync()  # raises on a latched device flag
    f, sums = g.fields(), [g.probe_sums(i, len(p.frequencies_hz)) for i, p in enumerate(sc.probes)]
    psi = [g.psi(w) for w in range(12)] if sc.pml is not None else []
    g.close()
    return f, sums, psi

def check(sc, steps, storage="f32", arith="exact", **kw):
    sim = O.sim_from_scenario(sc, steps=steps, storage=storage, arith=arith)
    sim.step(steps, os.cpu_count() or 1)
    f, sums, psi = run(sc, steps, prec=storage, arith=arith, **kw)
    assert np.array_equal(f, sim.fields()), (sc.name, kw, int(np.count_nonzero(f != sim.fields())))
    for i, p in enumerate(sc.probes):
        oc, os_, on = sim.probe_sums(i, len(p.frequencies_hz))
        assert np.array_equal(sums[i][0], oc) and sums[i][2] == on, (sc.name, i)
    for w, a in enumerate(psi):
        assert np.array_equal(a, sim.psi(w)), (sc.name, kw, w)
    sim.close()

cube = configs.plain_cube_64(steps=120)
check(cube, 120, kernel="fused", columns=True)
check(cube, 120, kernel="fused", columns=False)
check(cube, 120, kernel="split")
check(cube, 60, arith="fma", kernel="fused")
check(configs.plain_cube_64(steps=80, exact_pml=True), 80, kernel="fused")
check(configs.two_spheres(n=64, steps=80), 80, storage="f16", kernel="fused")
check(configs.two_spheres(n=96, steps=60), 60, kernel="fused")
print("BOUNDS_OK")
'''


def test_bounds_checked_build_matches_oracle_without_flags():
    lib = os.path.join(ROOT, "wavefront_b200", "lib", "libwavefront_gpu_checked.so")
    assert os.path.exists(lib), "build the bounds-checked variant (wavefront_b200/build.py)"
    env = dict(os.environ, WF_BOUNDS_CHECK="1", WF_ROOT=ROOT)
    r = subprocess.run([sys.executable, "-c", SCRIPT], cwd=ROOT, env=env, capture_output=True,
                       text=True, timeout=900)
    assert r.returncode == 0 and "BOUNDS_OK" in r.stdout, (r.stdout[-2000:], r.stderr[-3000:])


# The same checks form by form: bricks, marching tiles with and without column
# tiles, the mixed step and batches, each in the arithmetic and storage it runs.
FORMS = SCRIPT.split("cube = configs")[0].replace('if "columns" in kw:', '''if "tiling" in kw:
        g.set_tiling(*kw["tiling"])
    if "columns" in kw:''') + r'''
cube, ten = configs.plain_cube_64(steps=40), configs.plain_cube_64(steps=40, exact_pml=True)
two = configs.two_spheres(n=96, steps=24)
for form in (dict(tiling=(8, 4, 1)), dict(tiling=(4, 12, 3)), dict(tiling=(8, 16, 3), columns=False)):
    check(cube, 40, kernel="fused", **form)
    check(cube, 40, arith="fma", kernel="fused", **form)
    check(ten, 40, kernel="fused", **form)
    check(ten, 40, arith="fma", kernel="fused", **form)
    check(two, 24, kernel="fused", **form)
for form in (dict(tiling=(8, 4, 1)), dict(tiling=(4, 12, 3)), dict(tiling=(4, 12, 3), columns=False)):
    check(two, 24, storage="f16", kernel="fused", **form)
    check(ten, 24, storage="bf16", kernel="fused", **form)

# thin slabs on every axis, and an interior of marching tiles with bricks around
# it, against the split pair of the same build
def same(dims, depth, steps, tiling=None, precision="f32", ref=None):
    out = []
    for k in (0, 1):
        g = wf.DeviceFieldGrid(wf.GridDims(*dims), kernel="split" if k and not ref else "auto", precision=precision)
        dt = configs.courant_dt(1e-3)
        g.set_materials(wf.MaterialGrid(wf.GridDims(*dims)), wf.MaterialTable.vacuum_filled(dt, 1e-3))
        for ax, n in enumerate(dims):
            p = wf.PmlProfile1D.build(n, wf.PmlConfig(thickness=depth[ax]), dt, 1e-3, depth[ax])
            g.set_pml_axis(ax, depth[ax], p.b, p.a, p.inv_kappa)
        t = ref if k else tiling
        if t:
            g.set_tiling(*t)
        g.set_fields(np.random.default_rng(3).standard_normal((6, *dims[::-1])).astype(np.float32))
        g.step(steps)
        g.sync()
        out.append([g.fields()] + [g.psi(w) for w in range(12)])
        g.close()
    assert all(np.array_equal(a, b) for a, b in zip(*out)), (dims, depth, tiling, precision)

for depth in ((1, 1, 1), (2, 3, 1), (5, 1, 2), (4, 0, 0)):
    for tiling in ((8, 4, 1), (4, 12, 3)):
        same((72, 24, 16), depth, 6, tiling)
    same((72, 24, 16), depth, 6, (8, 4, 1), "f16", ref=(4, 5, 3))
for depth in ((7, 5, 9), (1, 16, 4)):
    same((520, 200, 264), depth, 3)  # the mixed step
    same((520, 200, 264), depth, 2, None, "f16", ref=(4, 32, 3))

for tiling in (None, (8, 4, 1), (4, 16, 3), (32, 16, 3)):
    scenes = configs.batched_sweep(3, steps=20, seed=19, sizes=(32, 40, 64))
    b = configs.device_batch(scenes)
    if tiling:
        b.set_tiling(*tiling)
    b.step(20)
    b.sync()
    for i, sc in enumerate(scenes):
        sim = O.sim_from_scenario(sc, steps=20)
        sim.step(20, os.cpu_count() or 1)
        assert np.array_equal(b.grid(i).fields(), sim.fields()), (tiling, i)
        sim.close()
    b.close()
print("BOUNDS_OK")
'''


def test_every_form_of_the_step_stays_in_bounds():
    env = dict(os.environ, WF_BOUNDS_CHECK="1", WF_ROOT=ROOT)
    r = subprocess.run([sys.executable, "-c", FORMS], cwd=ROOT, env=env, capture_output=True, text=True, timeout=900)
    assert r.returncode == 0 and "BOUNDS_OK" in r.stdout, (r.stdout[-2000:], r.stderr[-3000:])

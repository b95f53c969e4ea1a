"""GPU: the brick step against the split and marching kernels, bit for bit, at
the sizes where it can go wrong: x extents that leave a brick 8, 16 or 24
cells wide, single bricks, CPML depths that are not multiples of 4 (groups
that straddle the slab), that meet in the middle or exceed 64 positions,
periodic axes with and without CPML, more than 32 sources, sheet sources."""
import numpy as np
import pytest

import wavefront_b200 as wf
from wavefront_b200 import configs

pytestmark = pytest.mark.gpu

BRICK = (8, 4, 1)


def _grid(dims, kernel, seed, pml=(0, 0, 0), periodic="", arith="exact", precision="f32",
          tiling=None, nsrc=2, sheet=False, steps=9):
    nx, ny, nz = dims
    rng = np.random.default_rng(seed)
    d = wf.GridDims(nx, ny, nz)
    dx = 1e-3
    dt = configs.courant_dt(dx)
    g = wf.DeviceFieldGrid(d, kernel=kernel, arith=arith, precision=precision,
                           boundary=tuple("periodic" if a in periodic else "zero" for a in "xyz"))
    ids = rng.integers(0, 3, nx * ny * nz).astype(np.uint8)
    table = wf.MaterialTable.vacuum_filled(dt, dx)
    table.set_material(1, 4.0, 1.0, 0.01, dt, dx)
    table.set_material(2, 2.25, 1.5, 0.0, dt, dx)
    g.set_materials(wf.MaterialGrid(d, ids), table)
    for ax, t in enumerate(pml):
        if t:
            p = wf.PmlProfile1D.build(dims[ax], wf.PmlConfig(thickness=t), dt, dx, t)
            g.set_pml_axis(ax, t, p.b, p.a, p.inv_kappa)
    if tiling:
        g.set_tiling(*tiling)
    f = rng.standard_normal((6, nz, ny, nx)).astype(np.float32)
    f[3:] /= 377.0
    g.set_fields(f)
    if sheet:
        g.add_source_values(nx - 1, 0, 0, 2, np.linspace(0.5, 1.0, steps), mode=1)
    for k in range(nsrc):
        # two share a cell: list order matters
        x, y, z = (int(v) for v in (rng.integers(0, nx), rng.integers(0, ny), rng.integers(0, nz)))
        for c in ([0, 0] if k == 0 else [k % 3]):
            g.add_source_values(x, y, z, c, rng.standard_normal(steps).astype(np.float32))
    for c in range(6):
        tab = rng.standard_normal((steps, 2))
        g.add_probe_tables(int(rng.integers(0, nx)), int(rng.integers(0, ny)), int(rng.integers(0, nz)), c,
                           tab, tab + 1.0, 2, True)
    g.step(steps)
    g.sync()
    out = [g.fields()] + [g.psi(w) for w in range(12)]
    for c in range(6):
        s = g.probe_sums(c, 2)
        out += [s[0], s[1], np.array(s[2]), g.probe_trace(c, steps)]
    g.close()
    return out


def _same(a, b):
    for i, (u, v) in enumerate(zip(a, b)):
        assert np.array_equal(u, v), f"output {i}: {int((u != v).sum())} values differ"  # +0 == -0


@pytest.mark.parametrize("dims,pml,periodic,kw", [
    ((8, 8, 8), (0, 0, 0), "", {}),
    ((8, 8, 8), (4, 3, 4), "", {}),
    ((40, 16, 8), (10, 5, 2), "", {}),
    ((48, 8, 24), (24, 4, 1), "", {"nsrc": 33}),
    ((56, 72, 16), (7, 16, 8), "", {"arith": "fma"}),
    ((72, 16, 16), (36, 8, 8), "", {}),
    ((160, 16, 16), (40, 0, 0), "", {}),
    ((32, 24, 24), (0, 0, 10), "xy", {"sheet": True}),
    ((24, 8, 40), (0, 0, 0), "xyz", {"arith": "fma"}),
    ((64, 88, 16), (9, 0, 0), "yz", {"sheet": True}),
    ((96, 8, 8), (16, 0, 0), "x", {}),
])
def test_brick_equals_split(dims, pml, periodic, kw):
    want = _grid(dims, "split", 3, pml, periodic, **kw)
    got = _grid(dims, "auto", 3, pml, periodic, tiling=BRICK, **kw)
    assert np.abs(want[0]).max() > 0
    _same(got, want)


@pytest.mark.parametrize("precision", ["f16", "bf16"])
@pytest.mark.parametrize("dims,pml", [((8, 8, 8), (0, 0, 0)), ((40, 16, 24), (10, 5, 9)),
                                      ((72, 8, 32), (16, 4, 8))])
def test_brick_equals_marching_16bit(precision, dims, pml):
    want = _grid(dims, "fused", 5, pml, precision=precision, tiling=(4, 5, 3))
    got = _grid(dims, "fused", 5, pml, precision=precision, tiling=BRICK)
    _same(got, want)


# Large grids whose x axis has CPML: an interior of marching tiles with bricks
# around it, for interiors cut by a ragged x extent, by slabs of several depths
# and open on the axes without CPML.
@pytest.mark.parametrize("dims,pml,kw", [
    ((680, 200, 200), (7, 5, 9), {}),
    ((520, 264, 200), (16, 16, 16), {"arith": "fma", "nsrc": 33}),
    ((1032, 136, 104), (10, 0, 0), {"sheet": True}),
    ((360, 200, 264), (7, 5, 9), {"precision": "f16"}),
    ((328, 264, 200), (4, 0, 12), {"precision": "bf16"}),
])
def test_bricks_around_marching_interior(dims, pml, kw):
    g = wf.DeviceFieldGrid(wf.GridDims(*dims), precision=kw.get("precision", "f32"))
    for ax, t in enumerate(pml):
        if t:
            g.set_pml_axis(ax, t, *(np.ones(2 * t, np.float32),) * 3)
    assert g.tiling()[0] == 4 and not g.column_tiles  # both kernels
    g.close()
    other = dict(kernel="fused", tiling=(4, 24, 3)) if "precision" in kw else dict(kernel="split")
    want = _grid(dims, seed=7, pml=pml, **other, **kw)
    got = _grid(dims, "auto", 7, pml, **kw)
    assert np.abs(want[0]).max() > 0
    _same(got, want)


def test_default_tiling_round_trips_and_marching_stays_selectable():
    g = wf.DeviceFieldGrid(wf.GridDims(64, 64, 64))
    try:
        assert g.tiling() == BRICK and not g.column_tiles
        g.set_tiling(*g.tiling())
        g.step(2)
        g.set_tiling(4, 12, 3)
        assert g.tiling() == (4, 12, 3)
        g.step(2)
        g.sync()
    finally:
        g.close()


# CPML depths on x that leave every group straddling the slab: at depth 1 the
# group that meets the high slab begins two positions before the slab array's row.
@pytest.mark.parametrize("dims,pml,kw", [
    ((8, 8, 8), (1, 0, 0), {}),
    ((40, 16, 8), (1, 1, 1), {}),
    ((40, 16, 8), (2, 1, 3), {"arith": "fma"}),
    ((72, 8, 16), (3, 2, 0), {"nsrc": 33}),
    ((64, 24, 8), (5, 0, 1), {}),
])
def test_thin_x_slabs_equal_split(dims, pml, kw):
    _same(_grid(dims, "auto", 11, pml, tiling=BRICK, **kw), _grid(dims, "split", 11, pml, **kw))


@pytest.mark.parametrize("precision", ["f16", "bf16"])
@pytest.mark.parametrize("depth", [1, 2, 3, 5])
def test_thin_x_slabs_equal_marching_16bit(precision, depth):
    dims, pml = (40, 16, 24), (depth, 1, 2)
    _same(_grid(dims, "auto", 13, pml, precision=precision, tiling=BRICK),
          _grid(dims, "fused", 13, pml, precision=precision, tiling=(4, 5, 3)))


@pytest.mark.parametrize("depth", [1, 2, 3, 5])
def test_thin_x_slabs_around_a_marching_interior(depth):
    dims, pml = (520, 200, 264), (depth, 9, 4)
    _same(_grid(dims, "auto", 17, pml), _grid(dims, "split", 17, pml))


def test_thin_x_slabs_in_a_batch():
    sizes, depths = ((40, 16, 8), (32, 8, 8), (72, 24, 16), (8, 8, 8)), (1, 2, 3, 1)
    dt = configs.courant_dt(1e-3)

    def load(g, k):
        nx, ny, nz = sizes[k]
        rng = np.random.default_rng(100 + k)
        g.set_materials(wf.MaterialGrid(wf.GridDims(nx, ny, nz)), wf.MaterialTable.vacuum_filled(dt, 1e-3))
        for ax, n in enumerate(sizes[k]):
            p = wf.PmlProfile1D.build(n, wf.PmlConfig(thickness=depths[k]), dt, 1e-3, depths[k])
            g.set_pml_axis(ax, depths[k], p.b, p.a, p.inv_kappa)
        g.set_fields(rng.standard_normal((6, nz, ny, nx)).astype(np.float32))
        return g

    b = wf.DeviceBatch([wf.GridDims(*s) for s in sizes])
    try:
        for k in range(len(sizes)):
            load(b.grid(k), k)
        b.step(6)
        b.sync()
        for k, s in enumerate(sizes):
            with wf.DeviceFieldGrid(wf.GridDims(*s), kernel="split") as g:
                load(g, k)
                g.step(6)
                g.sync()
                _same([b.grid(k).fields()] + [b.grid(k).psi(w) for w in range(12)],
                      [g.fields()] + [g.psi(w) for w in range(12)])
    finally:
        b.close()


# The automatic step, whichever form its price picks: the split pair on short
# rows, bricks, marching tiles.
@pytest.mark.parametrize("dims,pml,periodic,kw", [
    ((16, 128, 256), (4, 4, 4), "", {}),
    ((8, 128, 256), (0, 0, 0), "xyz", {"sheet": True, "nsrc": 33}),
    ((16, 128, 128), (4, 0, 0), "yz", {"arith": "fma"}),
    ((24, 128, 256), (0, 0, 0), "yz", {}),
    ((104, 264, 200), (0, 0, 0), "", {"nsrc": 33}),
    ((136, 40, 200), (40, 3, 9), "", {}),
])
def test_automatic_step_equals_split(dims, pml, periodic, kw):
    _same(_grid(dims, "auto", 19, pml, periodic, **kw), _grid(dims, "split", 19, pml, periodic, **kw))


def test_the_form_follows_the_cpml_between_steps():
    """A grid whose cheapest form is bricks, then the split pair, then bricks
    again as its CPML is set: sources and probes run once a step in each."""
    dims, steps = (16, 128, 256), 4
    dt = configs.courant_dt(1e-3)
    f = np.random.default_rng(23).standard_normal((6, *dims[::-1])).astype(np.float32)

    def run(kernel):
        g = wf.DeviceFieldGrid(wf.GridDims(*dims), kernel=kernel)
        g.set_materials(wf.MaterialGrid(wf.GridDims(*dims)), wf.MaterialTable.vacuum_filled(dt, 1e-3))
        g.set_fields(f)
        g.add_source_values(9, 60, 100, 2, np.linspace(1.0, 2.0, 3 * steps).astype(np.float32))
        g.add_probe_tables(8, 64, 128, 1, np.ones((3 * steps, 1)), np.full((3 * steps, 1), 2.0), 0, True)
        out, launches = [], []
        for t in (0, 4, 8):
            for ax, n in enumerate(dims):
                p = wf.PmlProfile1D.build(n, wf.PmlConfig(thickness=t), dt, 1e-3, t)
                g.set_pml_axis(ax, t, p.b, p.a, p.inv_kappa)
            before = g.kernel_launches
            g.step(steps)
            g.sync()
            launches.append((g.kernel_launches - before) // steps)
            out += [g.fields()] + ([g.psi(w) for w in range(12)] if t else [])
        s = g.probe_sums(0, 1)
        out += [s[0], s[1], np.array(s[2]), g.probe_trace(0, 3 * steps)]
        g.close()
        return out, launches

    got, launches = run("auto")
    want, split_launches = run("split")
    assert launches == [1, split_launches[1], 1] and split_launches[1] > 1
    _same(got, want)


def test_grids_beyond_a_brick_launch_run_other_forms():
    """More than 65535 bands of 64 rows do not fit a launch of bricks: the tiling
    is refused, a step and a batch of such a grid (13 GB) run other forms."""
    dims, steps = wf.GridDims(8, 4194312, 8), 3

    def load(g):
        for y in (0, 2000003, dims.ny - 1):
            g.add_source_values(4, y, 3, 2, np.linspace(1.0, 2.0, steps).astype(np.float32))
            g.add_probe_tables(5, y, 4, 0, np.zeros((steps, 0)), np.zeros((steps, 0)), 0, True)
            g.add_probe_tables(4, y, 3, 2, np.zeros((steps, 0)), np.zeros((steps, 0)), 0, True)

    def traces(g):
        return [g.probe_trace(k, steps) for k in range(6)]

    try:
        out = {}
        for kernel in ("auto", "fused", "split"):
            with wf.DeviceFieldGrid(dims, kernel=kernel) as g:
                t = wf.MaterialTable.vacuum_filled(configs.courant_dt(1e-3), 1e-3)
                g.set_scene("", t, configs.courant_dt(1e-3), 1e-3)
                with pytest.raises(wf.WfError):
                    g.set_tiling(*BRICK)
                load(g)
                g.step(steps)
                g.sync()
                out[kernel] = traces(g)
        with wf.DeviceBatch([dims]) as b:
            assert b.tiling() == (4, 16, 3)
            b.grid(0).set_scene("", wf.MaterialTable.vacuum_filled(configs.courant_dt(1e-3), 1e-3),
                                configs.courant_dt(1e-3), 1e-3)
            load(b.grid(0))
            b.step(steps)
            b.sync()
            out["batch"] = traces(b.grid(0))
        assert all(np.abs(t).max() > 0 for t in out["split"])
        for form in ("auto", "fused", "batch"):
            _same(out[form], out["split"])
    finally:
        wf.lib().wf_release_cached_memory(-1)


def test_asking_for_the_default_column_tiles_leaves_a_grid_automatic():
    dims = wf.GridDims(64, 64, 64)
    for kernel, enable, tiling, columns in (("auto", True, BRICK, False), ("auto", False, (4, 12, 3), False),
                                            ("fused", True, (4, 12, 3), True), ("fused", False, (4, 12, 3), False)):
        with wf.DeviceFieldGrid(dims, kernel=kernel) as g:
            p = wf.PmlProfile1D.build(64, wf.PmlConfig(thickness=8), 1e-12, 1e-3, 8)
            for ax in range(3):
                g.set_pml_axis(ax, 8, p.b, p.a, p.inv_kappa)
            g.set_column_tiles(enable)
            assert (g.tiling(), g.column_tiles) == (tiling, columns), (kernel, enable)
            if kernel == "auto":  # off and on again: automatic
                g.set_column_tiles(False)
                g.set_column_tiles(True)
                assert g.tiling() == BRICK
            g.step(2)
            g.sync()


# The marching tiles, which a grid of these sizes runs only when asked: FMA and
# exact, every CPML class, column tiles on (the default) and off.
@pytest.mark.parametrize("tiling", [(4, 12, 3), (8, 16, 3), (16, 5, 3), (4, 24, 4)])
@pytest.mark.parametrize("dims,pml,kw", [
    ((136, 72, 40), (10, 10, 10), {"arith": "fma"}),
    ((136, 72, 40), (16, 0, 12), {"arith": "fma", "nsrc": 33}),
    ((264, 40, 56), (7, 5, 0), {"arith": "fma", "sheet": True}),
    ((72, 72, 48), (20, 9, 16), {"arith": "fma"}),
    ((136, 72, 40), (10, 10, 10), {}),
])
def test_marching_equals_split(tiling, dims, pml, kw):
    _same(_grid(dims, "fused", 43, pml, tiling=tiling, **kw), _grid(dims, "split", 43, pml, **kw))

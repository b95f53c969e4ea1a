"""GPU: batched stepping (wf_batch_*) of many independent grids of uneven
size by one persistent kernel per step.  Every grid must equal the oracle
bit for bit (fields, every psi array, probe sums), through runs long enough
to replay the captured 32-step graphs; the autotuner must leave the state
as it found it; lockstep violations are reported, not run."""
import os

import numpy as np
import pytest

import wavefront_b200 as wf
from wavefront_b200 import configs

pytestmark = pytest.mark.gpu
NT = min(os.cpu_count() or 1, 32)


def _eq(got, want, what):
    bad = got != want  # +0 == -0
    if bad.any():
        raise AssertionError(f"{what}: {bad.sum()} values differ, first {np.argwhere(bad)[:3].tolist()}")


def _check_against_oracle(oracle, b, scenes, steps):
    for i, sc in enumerate(scenes):
        sim = oracle.sim_from_scenario(sc, steps=steps)
        sim.step(steps, NT)
        g = b.grid(i)
        _eq(g.fields(), sim.fields(), f"scene {i} ({sc.dims.nx}^3) fields")
        for w in range(12):
            _eq(g.psi(w), sim.psi(w), f"scene {i} {wf.PSI_NAMES[w]}")
        gc, gs, gn = g.probe_sums(0, 1)
        oc, os_, on = sim.probe_sums(0, 1)
        assert gn == on and np.array_equal(gc, oc) and np.array_equal(gs, os_), i
        assert g.steps_done == steps
        sim.close()


def test_batch_matches_oracle_through_graph_replays(oracle):
    """9 scenes of 32..96 cells, 70 steps: two 32-step graph replays plus 6
    directly launched steps."""
    scenes = configs.batched_sweep(9, steps=70, seed=7, sizes=(32, 48, 64, 96))
    b = configs.device_batch(scenes)
    try:
        b.step(70)
        b.sync()
        # per step: one persistent launch per non-empty CPML class, then the tail
        per_step, rest = divmod(b.kernel_launches, 70)
        assert rest == 0 and 2 <= per_step <= 9, b.kernel_launches
        _check_against_oracle(oracle, b, scenes, 70)
    finally:
        b.close()


def test_narrow_batch_is_one_launch_per_step_and_matches_oracle(oracle):
    """The narrow tiling (tile_rows 32: every grid in 16-wide, 32-row tiles,
    all items in one persistent launch of the all-axes body): one step
    kernel plus the tail per step, bit for bit against the oracle, on grids
    whose x extent is not a multiple of the 16-cell tile (40, 56, 120)."""
    scenes = configs.batched_sweep(7, steps=70, seed=13, sizes=(32, 40, 56, 120))
    b = configs.device_batch(scenes)
    try:
        b.set_tiling(32, 16, 3)
        b.step(70)
        b.sync()
        assert b.kernel_launches == 2 * 70, b.kernel_launches
        _check_against_oracle(oracle, b, scenes, 70)
    finally:
        b.close()


@pytest.mark.parametrize("tiling", [(8, 16, 4), (4, 1000, 3), (16, 8, 3), (32, 1000, 3), (32, 7, 3)])
def test_batch_tilings_match_oracle(oracle, tiling):
    scenes = configs.batched_sweep(5, steps=40, seed=11, sizes=(32, 48, 64))
    b = configs.device_batch(scenes)
    try:
        b.set_tiling(*tiling)
        b.step(40)
        b.sync()
        _check_against_oracle(oracle, b, scenes, 40)
    finally:
        b.close()


def test_batch_autotune_restores_state(oracle):
    scenes = configs.batched_sweep(4, steps=35, seed=3, sizes=(32, 64))
    b = configs.device_batch(scenes)
    try:
        best, ms = b.autotune(2)
        assert best in [(ty, zc, s) for ty in (4, 8, 16) for s in (3, 4)
                        for zc in (8, 12, 16, 24, 32, 64, 128)] + [
                            (32, zc, 3) for zc in (8, 12, 16, 24, 32, 64, 128)]
        assert ms > 0
        b.step(35)
        b.sync()
        _check_against_oracle(oracle, b, scenes, 35)
    finally:
        b.close()


def test_batch_requires_lockstep():
    scenes = configs.batched_sweep(2, steps=10, seed=5, sizes=(32,))
    b = configs.device_batch(scenes)
    try:
        b.grid(0).step(1)  # one grid alone: the batch is out of lockstep
        with pytest.raises(wf.WfError, match="same steps"):
            b.step(1)
    finally:
        b.close()


@pytest.mark.parametrize("tiling", [(4, 16, 3), (32, 16, 3), (8, 4, 1)])
def test_grids_stepped_alone_around_batched_steps(tiling):
    """Each grid alone for 40 steps (a captured graph of 32 among them), the
    batch for 33, each alone again: building the batch replaces a grid's
    descriptors and work lists, so the graph captured before must not be
    replayed after."""
    sizes = (64, 48)
    scenes = configs.batched_sweep(2, steps=113, seed=29, sizes=(64,))[:1] + configs.batched_sweep(
        1, steps=113, seed=31, sizes=(48,))
    b = configs.device_batch(scenes)
    try:
        b.set_tiling(*tiling)
        for g in b.grids:
            g.set_tiling(4, 12, 3)
        for g in b.grids:
            g.step(40)
        b.step(33)
        for g in b.grids:
            g.step(40)
        b.sync()
        for i, sc in enumerate(scenes):
            assert sc.dims.nx == sizes[i]
            h = configs.device_grid(sc, kernel="split")
            for s_ in sc.sources:
                h.add_source_values(s_.x, s_.y, s_.z, s_.component, s_.values(sc.dt, 113), s_.mode)
            for p_ in sc.probes:
                c, si = p_.tables(sc.dt, 113)
                h.add_probe_tables(p_.x, p_.y, p_.z, p_.component, c, si, p_.first_step(sc.dt))
            h.step(113)
            h.sync()
            _eq(b.grid(i).fields(), h.fields(), f"grid {i} fields")
            for w in range(12):
                _eq(b.grid(i).psi(w), h.psi(w), f"grid {i} {wf.PSI_NAMES[w]}")
            a, z = b.grid(i).probe_sums(0, 1), h.probe_sums(0, 1)
            assert np.array_equal(a[0], z[0]) and np.array_equal(a[1], z[1]) and a[2] == z[2]
            h.close()
    finally:
        b.close()


@pytest.mark.parametrize("sizes,depth,tiling", [
    ((96, 96, 96, 96, 96, 96, 96, 96), 0, (4, 16, 3)),
    ((96, 96, 96, 96, 96, 96, 96, 96), 10, (8, 4, 1)),
    ((32, 64), 0, (8, 4, 1)),
])
def test_default_batch_takes_the_cheaper_form(sizes, depth, tiling):
    """Without CPML the marching items are the cheaper form of all but small
    batches (16 cubes of 128 cells: 302 us a step against 460 as bricks); a set
    tiling stays set; both forms give the same bits."""
    dt = configs.courant_dt(1e-3)

    def run(set_to=None):
        b = wf.DeviceBatch([wf.GridDims(n, n, n) for n in sizes])
        try:
            for k, (g, n) in enumerate(zip(b.grids, sizes)):
                g.set_materials(wf.MaterialGrid(wf.GridDims(n, n, n)), wf.MaterialTable.vacuum_filled(dt, 1e-3))
                if depth:
                    p = wf.PmlProfile1D.build(n, wf.PmlConfig(thickness=depth), dt, 1e-3, depth)
                    for ax in range(3):
                        g.set_pml_axis(ax, depth, p.b, p.a, p.inv_kappa)
                f = np.random.default_rng(k).standard_normal((6, n, n, n)).astype(np.float32)
                g.set_fields(f)
            if set_to:
                b.set_tiling(*set_to)
            used = b.tiling()
            b.step(5)
            b.sync()
            assert b.tiling() == used
            return used, [g.fields() for g in b.grids]
        finally:
            b.close()

    used, got = run()
    assert used == tiling
    other = (8, 4, 1) if tiling == (4, 16, 3) else (4, 16, 3)
    set_used, want = run(other)
    assert set_used == other
    for i, (x, y) in enumerate(zip(got, want)):
        _eq(x, y, f"grid {i}")


def test_default_batch_of_bricks_is_one_launch_and_the_tail():
    scenes = configs.batched_sweep(3, steps=40, seed=37, sizes=(32, 48))
    b = configs.device_batch(scenes)
    try:
        assert b.tiling() == (8, 4, 1)
        b.step(40)
        b.sync()
        assert b.kernel_launches == 2 * 40
    finally:
        b.close()

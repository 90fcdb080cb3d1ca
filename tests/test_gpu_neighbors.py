"""Neighbour lists and the 10M-particle configuration against the oracle, on a B200.

The neighbour lists the density pass records (and the force pass and boundary reactions
read) are exported through vxl_sph_export_neighbors and compared, entry for entry and in
order, with the oracle's UniformGrid::for_neighbors_in walk
(crates/vxl-phys-fluid/src/grid.rs:115-155) over the same positions: all neighbours of a
fluid particle, the fluid ones of a boundary particle (fluid_density.rs:59-69). Cases: the
16k dam break at h-sized bins, a doubled-bin tank (2h cells), lists
longer than the 64 recorded entries (walked again), and a flowing state after a few ticks.

The 10M configuration (9,938,375 fluid particles in the 2.5 x 1.2 x 1.2 m tank, Akinci
walls, 64 boxes, c0 = 20, alpha = 0.05, eps = 0.5, bins doubled to 2h by the cell budget)
is stepped one substep from identical state on the GPU and on the oracle, and compared bit
for bit: cell table, density, pressure, acceleration, XSPH, per-boundary-particle
reaction, and the integrated positions and velocities
(crates/vxl-phys-fluid/src/fluid_step.rs:91-127).
"""
import os

import numpy as np
import pytest

from test_gpu_parity import F32, _custom, assert_bits, compare_grid, compare_state, f32_dt

pytestmark = pytest.mark.gpu


def _threads():
    return max(1, len(os.sched_getaffinity(0)))


def _compare_lists(g, o, label):
    go, ge = g.export_neighbors()
    oo, oe = o.neighbors()
    assert go.shape == oo.shape, label
    if not np.array_equal(go, oo):
        i = int(np.nonzero(go != oo)[0][0])
        raise AssertionError(f"{label}: list lengths differ first at particle {max(i - 1, 0)}")
    if not np.array_equal(ge, oe):
        k = int(np.nonzero(ge != oe)[0][0])
        i = int(np.searchsorted(oo, k, side="right") - 1)
        raise AssertionError(f"{label}: entry {k} (particle {i}) differs: {ge[k]} vs {oe[k]}")
    return go, ge


DENSITY = [0, 1]  # the tuning's density: both accepted values run the one density pass


def _lists_after(vxl, oracle_mod, spec, warm_ticks=0, substeps_before=0, density=0):
    """GPU and oracle from identical state; optionally advanced together; then the oracle's
    lists from its current positions and the GPU's lists of its next substep."""
    g = vxl.Scene(spec.params, spec.pos, spec.vel, spec.pmass, spec.n_fluid)
    g.set_tuning(256, 256, 0, density)
    o = oracle_mod.OracleSystem.from_scene(spec, threads=_threads())
    dt_tick = float(F32(1) / F32(60))
    for _ in range(warm_ticks):
        g.step_tick(dt_tick, spec.spans)
        o.step(dt_tick)
    dt = f32_dt(spec.params.substeps)
    for _ in range(substeps_before):
        g.substep(dt)
        o.substep(dt)
    compare_state(g, o, "before the listed substep")
    g.substep(dt)
    return g, o


@pytest.mark.parametrize("density", DENSITY)
def test_neighbor_lists_dam0_bit_exact(vxl, oracle_mod, density):
    from vxl_sph import scenes
    spec = scenes.dam0()
    g, o = _lists_after(vxl, oracle_mod, spec, density=density)
    offs, ent = _compare_lists(g, o, "dam0")
    counts = np.diff(offs.astype(np.int64))
    assert counts[:spec.n_fluid].mean() > 20 and ent.size > 0


@pytest.mark.parametrize("density", DENSITY)
def test_neighbor_lists_flowing_state(vxl, oracle_mod, density):
    """After two ticks of the dam break (particles moved, cells reordered)."""
    from vxl_sph import scenes
    spec = scenes.dam0()
    g, o = _lists_after(vxl, oracle_mod, spec, warm_ticks=2, substeps_before=3, density=density)
    _compare_lists(g, o, "dam0 after 2 ticks + 3 substeps")


@pytest.mark.parametrize("density", DENSITY)
def test_neighbor_lists_doubled_bins(vxl, oracle_mod, density):
    """The 10M tank's grid rule with a 40^3 block: the budget doubles the bins to 2h, so the
    density pass takes a cell's particles by octant."""
    from vxl_sph import scenes
    spec = scenes.dam10m_block(40)
    g, o = _lists_after(vxl, oracle_mod, spec, density=density)
    _, _, _, info = g.export_grid()
    assert info.bin >= 2 * spec.params.smoothing_radius * 0.999
    _compare_lists(g, o, "dam10m tank, 40^3 block")


@pytest.mark.parametrize("density", DENSITY)
def test_neighbor_lists_longer_than_the_recorded_cap(vxl, oracle_mod, density):
    """h = 3 s: about 110 neighbours per particle, past the 64 recorded entries, so every
    interior list is walked again; boundary particles keep only their fluid neighbours."""
    from vxl_sph import scenes
    s = 0.02
    params = scenes.baseline_params(s, substeps=4, smoothing_radius=3 * s)
    fluid = scenes.jitter(scenes.fluid_block((0.0, 0.0, 0.0), (14, 12, 14), s), s, 5)
    spec = scenes.assemble("wide", params, fluid, scenes.tank_bodies((0.4, 0.4, 0.4), 2 * s), s, 2)
    g, o = _lists_after(vxl, oracle_mod, spec, density=density)
    offs, _ = _compare_lists(g, o, "h = 3 s")
    assert np.diff(offs.astype(np.int64)).max() > 64


def _channel(vxl, max_bins, plate=0.0):
    """A channel of fluid 1,200 particles long in x (more than 36,000: one lane per particle), over a plate."""
    from vxl_sph import scenes
    s = 0.005
    pos = scenes.jitter(scenes.fluid_block((0.0, 0.0, 0.0), (1200, 6, 6), s), s, 8, 0.2)
    b = None
    if plate:
        b = scenes.body_particles([scenes.Body(0, (plate / 2, s, 0.03), (3.0, -1.5 * s, 0.015))], s, 2 * s, 1, 1000.0)
    return _custom(vxl, pos, h=2 * s, spacing=s, max_bins=max_bins, boundary=b)


@pytest.mark.parametrize("max_bins,plate,walls", [(3000, 0.0, False), (3000, 2.0, False), (3000, 5.5, False), (3000, 0.0, True),
                                                  (200, 0.0, False), (20, 0.0, False)])
def test_lists_of_a_scene_long_in_x(vxl, oracle_mod, max_bins, plate, walls):
    """List entries by rows: at bins of 2h, with boundary reactions of few and of many boundary particles, with
    provider walls, and at 8h and 32h, where three cells hold up to 1,728 and 6,912 particles (past the
    12 bits, walked again)."""
    from vxl_sph import scenes
    spec = _channel(vxl, max_bins, plate)
    assert plate < 5 or spec.n_boundary > 20000
    g = vxl.Scene(spec.params, spec.pos, spec.vel, spec.pmass, spec.n_fluid)
    o = oracle_mod.OracleSystem.from_scene(spec, threads=_threads())
    if walls:
        for x in (g, o):
            x.set_providers([scenes.floor_provider(), scenes.box_obstacle((3.0, 0.0, 0.0), (0.5, 0.01, 0.01))])
    dt = f32_dt(40)
    g.set_record(True)
    for _ in range(2):
        g.substep(dt)
        o.substep(dt)
    bf = g.read_fields()[4]
    if plate:
        assert np.any(bf != 0)
        assert_bits(bf, o.read_f32()["bforce"][spec.n_fluid:], "bforce")
    compare_grid(g, o, "channel")
    compare_state(g, o, "channel")
    g.substep(dt)
    _compare_lists(g, o, "channel")  # the oracle's from its positions, the next substep's


def test_long_scene_beside_a_short_one(vxl):
    """Entries by rows and by planes in one handle, each scene bitwise as alone."""
    from vxl_sph import scenes
    specs = [scenes.small_dam(n=(9, 8, 7), spacing=0.05, tank=(0.7, 0.6, 0.5), seed=8), _channel(vxl, 3000, 1.0),
             _custom(vxl, scenes.jitter(scenes.fluid_block((0, 0, 0), (12, 10, 8), 0.05), 0.05, 11), max_bins=64)]
    both = vxl.Batch(specs)
    alone = [vxl.Batch([x]) for x in specs]
    for t in range(2):
        rb = both.step_tick(1.0 / 600.0)
        ra = [r for g in alone for r in g.step_tick(1.0 / 600.0)]
        for (b1, f1, t1), (b2, f2, t2) in zip(ra, rb):
            assert b1 == b2 and f1.tobytes() == f2.tobytes() and t1.tobytes() == t2.tobytes(), (t, b1)
        for q, g in enumerate(alone):
            for x, y in zip(both.read_state(q), g.read_state(0)):
                assert x.tobytes() == y.tobytes(), (t, q)


@pytest.mark.parametrize("dims,max_bins,tile", [((900, 30, 30), 60000, 256), ((700, 12, 6), 1500, 16384)])
def test_force_pass_of_a_long_scene_is_no_slower_along_x(vxl, dims, max_bins, tile):
    """The lists hold whichever way a scene is long and however few tiles it has: the force pass of a block 900 long in
    x takes at most twice that of the same block along z (walked again for want of lists it took six times as long)."""
    from vxl_sph import scenes
    ms = []
    for dims in (dims, dims[::-1]):
        s = 0.005
        pos = scenes.jitter(scenes.fluid_block((0.0, 0.0, 0.0), dims, s), s, 1)
        spec = _custom(vxl, pos, h=2 * s, spacing=s, max_bins=max_bins)
        g = vxl.Batch([spec])
        g.set_tuning(256, tile, 0)
        g.substep(1e-5)
        g.set_profile(True)
        for _ in range(5):
            g.substep(1e-5)
        total, n = g.profile()["k_force"]
        ms.append(total / n)
        g.close()
    assert ms[0] < 2 * ms[1], ms


def test_neighbor_lists_before_any_substep_is_not_ready(vxl):
    from vxl_sph import scenes
    spec = scenes.small_dam()
    g = vxl.Scene(spec.params, spec.pos, spec.vel, spec.pmass, spec.n_fluid)
    with pytest.raises(vxl.VxlError) as e:
        g.export_neighbors()
    assert e.value.status == vxl.NOT_READY


def test_dam10m_substep_bit_exact(vxl, oracle_mod):
    """The 10M configuration, one substep from identical state (doubled bins, walls, 64
    boxes, the configuration's constants): every per-particle quantity bit for bit, with
    either value of the tuning's density."""
    from vxl_sph import scenes
    spec = scenes.dam10m()
    assert spec.n_fluid == 9938375 and len(spec.spans) == 69
    o = oracle_mod.OracleSystem.from_scene(spec, threads=_threads())
    dt = f32_dt(spec.params.substeps)
    o.substep(dt)
    r = o.read_f32()
    nf = spec.n_fluid
    for density in DENSITY:
        g = vxl.Scene(spec.params, spec.pos, spec.vel, spec.pmass, spec.n_fluid)
        g.set_tuning(256, 256, 0, density)
        g.set_record(True)
        g.substep(dt)
        _, _, _, info = g.export_grid()
        assert info.bin >= 2 * spec.params.smoothing_radius * 0.999, "the cell budget doubles the bins"
        compare_grid(g, o, f"dam10m density {density}")
        dens, press, acc, xsph, bf = g.read_fields()
        assert_bits(dens, r["dens"], "density")
        assert_bits(press, r["press"], "pressure")
        assert_bits(acc[:nf], r["acc"][:nf], "acceleration")
        assert_bits(xsph[:nf], r["xsph"][:nf], "xsph")
        assert_bits(bf, r["bforce"][nf:], "boundary reaction per particle")
        compare_state(g, o, f"dam10m after one substep, density {density}")
        g.close()
    o.close()

"""The density walk's candidate filter: never drops a neighbour.

On the CPU the words and the byte dot product of csrc/sph_device.cuh are restated in numpy
and held to the exact test r2 <= h2 over grids of h-sized and doubled bins, far origins, the
16,384-cell axis cap and particles clamped into the last cell. On a B200 the density kernel's
fields, table and state are compared bitwise with the oracle over the same kinds of scenes.
"""
import numpy as np
import pytest

F32 = np.float32


def _axis(o, v, inv, n):
    with np.errstate(all="ignore"):
        f = ((v - F32(o)).astype(F32) * F32(inv)).astype(F32)
        c = np.minimum(np.maximum(np.floor(f), 0).astype(np.int64), n - 1)
        sub = (f * F32(64)).astype(F32) - (c.astype(F32) * F32(64)).astype(F32)
    return c, np.clip(sub, 0, 63).astype(np.int64)


def _kept(pos, i, j, h, lo, bin_, dims):
    """Whether the filter keeps slot j as a candidate of particle i (cells within one of each other)."""
    inv = F32(1.0) / F32(bin_)
    c, q = zip(*(_axis(lo[a], pos[:, a], inv, dims[a]) for a in range(3)))
    d = [c[a][j] - c[a][i] for a in range(3)]
    near = (np.abs(d[0]) <= 1) & (np.abs(d[1]) <= 1) & (np.abs(d[2]) <= 1)
    b = [64 * ((c[0][j] - c[0][i] % 3 + 1) % 3) + q[0][j] - 96, q[1][j] - 32, q[2][j] - 32]
    norm = (b[0] ** 2 + b[1] ** 2 + b[2] ** 2) // 90
    assert norm.max() <= 127 and max(np.abs(x).max() for x in b) <= 128
    A = [q[0][i] - 32, q[1][i] - 64 * d[1] - 32, q[2][i] - 64 * d[2] - 32]
    assert all(np.abs(a[near]).max(initial=0) <= 127 for a in A)
    reach = F32(64) * (F32(h) / F32(bin_)) + (F32(1.75) + F32(4.2e-5) * F32(max(dims)))
    T = int(np.ceil(reach * reach))
    AA = A[0] ** 2 + A[1] ** 2 + A[2] ** 2
    over = -((T - AA) >> 1) - 1
    dot = -(A[0] * b[0] + A[1] * b[1] + A[2] * b[2]) + 45 * norm
    return near, dot + over < 0


@pytest.mark.parametrize("bins,shift,span", [(1, 0.0, 6), (2, 0.0, 9), (4, -3.0, 9), (8, 1e3, 9), (1, 1e4, 5),
                                             (1, 0.0, 16400), (2, -7.0, 33000)])
def test_filter_keeps_every_neighbour(bins, shift, span):
    h = F32(0.1)
    bin_ = F32(h * F32(bins))
    rng = np.random.default_rng(bins * 7 + span)
    n = 30000
    base = rng.uniform(0, 1, (n, 3)) * np.array([span, 4 * bins, 4 * bins]) * float(h)
    base[: n // 4, 0] = (span - rng.uniform(0, 4, n // 4)) * float(h)  # at the far end of the axis
    # partners on and around the sphere of radius h
    u = rng.normal(size=(n, 3))
    u /= np.linalg.norm(u, axis=1)[:, None]
    off = u * (float(h) * rng.choice([1.0, 1.0 - 1e-6, 0.999, 0.97, 0.5], n))[:, None]
    pos = (np.concatenate([base, base + off]) + shift).astype(F32)
    lo, hi = pos.min(0), pos.max(0)
    dims = [int(min(max(np.floor((hi[a] - lo[a]) / bin_) + 1, 1), 16384)) for a in range(3)]
    i, j = np.arange(n), np.arange(n, 2 * n)
    near, kept = _kept(pos, i, j, h, lo, bin_, dims)
    dx = (pos[i] - pos[j]).astype(F32)
    r2 = ((dx[:, 0] * dx[:, 0] + dx[:, 1] * dx[:, 1]) + dx[:, 2] * dx[:, 2]).astype(F32)
    accepted = r2 <= F32(h * h)
    assert accepted.sum() > n // 3
    assert np.all(near[accepted]) and np.all(kept[accepted])
    if bins <= 2:
        far = near & (r2 > F32(h * h) * F32(1.6 if bins == 1 else 2.2))
        assert not np.any(kept[far])  # and it does drop what is well outside


@pytest.mark.gpu
@pytest.mark.parametrize("max_bins,shift", [(0, 0.0), (0, 300.0), (900, -2.0), (120, 0.0), (20, 50.0), (1, 0.0)])
def test_density_walk_bit_exact_over_bin_sizes(vxl, oracle_mod, max_bins, shift):
    """A ragged cloud (dense core, sparse rim, walls through it) at bins of h, 2h, 4h, ... one cell,
    near and far from the origin: windows cut at every word offset, with eight lanes per particle."""
    from vxl_sph import scenes
    from test_gpu_parity import _custom, _run_both
    rng = np.random.default_rng(max_bins + 5)
    core = rng.uniform(0.0, 0.5, (1500, 3))
    rim = rng.uniform(-0.4, 0.9, (700, 3))
    pos = (np.concatenate([core, rim]) + shift).astype(F32)
    b = scenes.body_particles([scenes.Body(0, (0.3, 0.05, 0.3), (0.25 + shift, -0.1 + shift, 0.25 + shift))], 0.05, 0.1, 1,
                              1000.0)
    _run_both(vxl, oracle_mod, _custom(vxl, pos, max_bins=max_bins, boundary=b), substeps=2)


@pytest.mark.gpu
def test_density_walk_batch_of_bin_sizes(vxl):
    """Scenes of h-sized, doubled and single-cell bins side by side in one batch, each bitwise the same alone:
    windows run up to and past a neighbouring scene's slots."""
    from test_gpu_parity import _custom
    rng = np.random.default_rng(3)
    specs = [_custom(vxl, rng.uniform(0.0, w, (n, 3)).astype(F32), max_bins=mb)
             for n, w, mb in ((37, 0.3, 0), (501, 0.6, 64), (5, 0.2, 0), (260, 0.3, 1), (1, 0.1, 0), (333, 0.9, 300))]
    bat = vxl.Batch(specs)
    alone = [vxl.Scene(s.params, s.pos, s.vel, s.pmass, s.n_fluid) for s in specs]
    for _ in range(3):
        bat.substep(1.0 / 240.0)
        for g in alone:
            g.substep(1.0 / 240.0)
    for q, g in enumerate(alone):
        for a, b in zip(bat.read_state(q), g.read_state()):
            assert a.tobytes() == b.tobytes(), q
        for a, b in zip(bat.export_grid(q)[:3], g.export_grid()[:3]):
            assert np.array_equal(a, b), q


def _cloud(vxl, name):
    """Small scenes for the one-lane walk: name, rows with more windows than its queue of 18."""
    from vxl_sph import scenes
    from test_gpu_parity import _custom
    rng = np.random.default_rng(12)
    if name.startswith("lattice"):  # in random order in one cell or eight: some 38 windows of a row hold a few kept slots each
        pos = scenes.jitter(scenes.fluid_block((0.0, 0.0, 0.0), (16, 16, 16), 0.05), 0.05, 3, 0.2)
        return _custom(vxl, pos[rng.permutation(len(pos))], max_bins=int(name.split()[1]))
    pos = np.concatenate([rng.uniform(0.26, 0.34, (2000, 3)), rng.uniform(0.0, 0.6, (700, 3))]).astype(F32)  # a crowded bin
    b = scenes.body_particles([scenes.Body(0, (0.3, 0.05, 0.3), (0.25, -0.1, 0.25))], 0.05, 0.1, 1, 1000.0)
    return _custom(vxl, pos, max_bins=int(name.split()[1]), boundary=b)


@pytest.mark.gpu
@pytest.mark.parametrize("walls", [False, True])
@pytest.mark.parametrize("cloud", ["lattice 1", "lattice 8", "crowd 0", "crowd 60", "crowd 1"])
def test_one_lane_walk_past_its_queue(vxl, oracle_mod, cloud, walls):
    """Rows of well over 18 windows of 32 slots (the queue is emptied in mid-row) at bins of h, 2h and more, beside a
    block that brings the density pass to one lane per particle: table, state, density and lists bit for bit."""
    import ctypes
    from vxl_sph import scenes
    from test_gpu_parity import _custom, assert_bits, f32_dt
    spec = _cloud(vxl, cloud)
    n = spec.n_total
    g = vxl.Batch([spec, _custom(vxl, scenes.fluid_block((0.0, 0.0, 0.0), (34, 34, 34), 0.05))])
    o = oracle_mod.OracleSystem.from_scene(spec, threads=8)
    if walls:
        for x in (g, o):
            x.set_providers([scenes.floor_provider(), scenes.box_obstacle((0.1, 0.0, 0.1), (0.08, 0.05, 0.08))])
    dt = f32_dt(400)
    g.substep(dt)
    o.substep(dt)
    r, og = o.read_f32(), o.grid()
    dens = np.empty(n, F32)
    assert g.lib.vxl_sph_read_fields_scene(g._h, 0, vxl._fptr(dens), None, None, None, None) == vxl.OK
    assert_bits(dens, r["dens"], "density")
    items, start, _, info = g.export_grid(0)
    assert list(info.dims) == list(og["dims"]) and np.array_equal(start, og["start"]) and np.array_equal(items, og["items"])
    row = np.diff(start.astype(np.int64)).reshape(tuple(info.dims)).sum(0).max()
    assert row > 18 * 32 * 1.5, row
    p, v = g.read_state(0)
    assert_bits(p, r["pos"], "pos")
    assert_bits(v, r["vel"], "vel")
    g.substep(dt)
    off, tot = np.empty(n + 1, np.uint64), ctypes.c_uint64()
    op = off.ctypes.data_as(ctypes.POINTER(ctypes.c_uint64))
    assert g.lib.vxl_sph_export_neighbors(g._h, op, n + 1, None, 0, ctypes.byref(tot)) == vxl.OK
    ent = np.empty(tot.value, np.uint32)
    assert g.lib.vxl_sph_export_neighbors(g._h, op, n + 1, vxl._u32ptr(ent), tot.value, ctypes.byref(tot)) == vxl.OK
    oo, oe = o.neighbors()
    assert np.array_equal(off, oo) and np.array_equal(ent, oe)
    if cloud.startswith("lattice"):
        assert np.median(np.diff(oo.astype(np.int64))) <= 64  # lists that are recorded, not walked again

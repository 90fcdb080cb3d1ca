"""Span reactions, wall separation and pair quotients where their kernels can go wrong (B200).

The compacted span sums against the sequential float32 loop over the recorded reactions; the
tiled separation check and the force pass's shared-reciprocal quotients against the oracle.
"""
import numpy as np
import pytest

from test_gpu_parity import F32, _custom, _run_both, assert_bits, compare_state, pair

pytestmark = pytest.mark.gpu


def _sequential(bf, bpos, origin, start, end):
    f = np.zeros(6, F32)
    with np.errstate(all="ignore"):
        for k in range(start, end):
            r = (bpos[k] - origin).astype(F32)
            v = bf[k]
            t = (r[1] * v[2] - r[2] * v[1], r[2] * v[0] - r[0] * v[2], r[0] * v[1] - r[1] * v[0])
            f = (f + np.array([v[0], v[1], v[2], *t], F32)).astype(F32)
    return f


@pytest.mark.parametrize("origin", [(0.1, 0.2, -0.3), (3e18, 0.0, 0.0), (np.inf, 1.0, 0.0)])
def test_span_sums_equal_the_sequential_loop(vxl, origin):
    """Spans of every alignment to the mask's words, empty, one, a warp, a chunk, past the length that takes a
    block, wet in places only; and torque origins with which a dry particle's term is not zero."""
    from vxl_sph import scenes
    s = 0.02
    b = scenes.body_particles([scenes.Body(0, (0.75, 0.03, 0.75), (0.75, -0.05, 0.75))], s, 2 * s, 1, 1000.0)
    nb = b[0].shape[0]
    assert nb > 11000
    rng = np.random.default_rng(2)
    fluid = scenes.jitter(scenes.fluid_block((0.3, -0.02, 0.4), (30, 4, 9), s), s, 4, 0.2)
    fluid = np.concatenate([fluid, rng.uniform((0.0, -0.02, 0.0), (1.5, 0.0, 1.5), (60, 3))]).astype(F32)
    cuts = [(0, 0), (5, 5), (0, 1), (31, 32), (31, 33), (7, 39), (64, 96), (1, 1025), (100, 8292), (3, 8196), (0, nb),
            (17, nb - 5), (nb - 1, nb)]
    spec = _custom(vxl, fluid, h=2 * s, spacing=s, boundary=(b[0], b[1], b[2], [(k, origin, i, j) for k, (i, j) in enumerate(cuts)]),
                   substeps=1)
    g = vxl.Scene(spec.params, spec.pos, spec.vel, spec.pmass, spec.n_fluid)
    g.set_record(True)
    got = g.step_tick(1.0 / 600.0, spec.spans)
    bf = g.read_fields()[4]
    assert 0 < np.count_nonzero(np.any(bf != 0, axis=1)) < nb // 2
    for (i, j), (_, force, torque) in zip(cuts, got):
        want, have = _sequential(bf, b[0], np.array(origin, F32), i, j), np.concatenate([force, torque])
        nan = np.isnan(want)  # the NaN's payload is the machine's own
        assert np.array_equal(nan, np.isnan(have)), (i, j, want, have)
        assert_bits(have[~nan], want[~nan], f"span {i}:{j}")


@pytest.mark.parametrize("n,close", [(2, (0, 1)), (130, (3, 129)), (128, (126, 127)), (300, (5, 290)), (300, None)])
def test_separation_check_over_tiles(vxl, oracle_mod, n, close):
    """n pushed particles on a line under the floor, one pair (or none) closer than 0.2 h, within and across
    the check's tiles."""
    from vxl_sph import scenes
    x = 0.05 * np.arange(n)
    pos = np.stack([x, np.full(n, -0.001), np.zeros(n)], 1).astype(F32)
    if close:
        pos[close[1]] = pos[close[0]] + np.array([0.0001, 0.0, 0.0], F32)
    pos = np.concatenate([pos, [[-1.0, 0.5, 0.5]]]).astype(F32)
    spec = _custom(vxl, pos, h=0.1, spacing=0.05)
    g, o = pair(vxl, oracle_mod, spec, threads=1)
    g.set_providers([scenes.floor_provider()])
    o.set_providers([scenes.floor_provider()])
    for _ in range(3):
        g.substep(1.0 / 240.0)
        o.substep(1.0 / 240.0)
        compare_state(g, o, f"{n} pushed, close {close}")


def _pushed_line(vxl, n, close=()):
    """n particles on a line under the floor, two of them 1e-4 apart."""
    pos = np.stack([0.05 * np.arange(n), np.full(n, -0.001), np.zeros(n)], 1).astype(F32)
    if close:
        pos[close[1]] = pos[close[0]] + np.array([0.0001, 0.0, 0.0], F32)
    return _custom(vxl, pos, h=0.1, spacing=0.05)


def _floored(vxl, specs):
    from vxl_sph import scenes
    b = vxl.Batch(specs)
    for q in range(len(specs)):
        b.set_providers([scenes.floor_provider()], q)
    return b


def test_separation_check_over_scenes(vxl):
    """Scenes shorter and longer than the check's tiles side by side, at the same places, some with a close pair:
    each as alone."""
    specs = [_pushed_line(vxl, n, c) for n, c in ((1, ()), (130, (3, 129)), (5, ()), (127, ()), (300, (5, 290)), (2, (0, 1)),
                                                  (256, ()), (700, (0, 699)), (1, ()))]
    both = _floored(vxl, specs)
    alone = [_floored(vxl, [s]) for s in specs]
    for t in range(2):
        both.substep(1.0 / 240.0)
        for q, g in enumerate(alone):
            g.substep(1.0 / 240.0)
            for x, y in zip(both.read_state(q), g.read_state(0)):
                assert x.tobytes() == y.tobytes(), (t, q)


def test_separation_check_grows_with_the_scenes_not_their_square(vxl):
    """Eight times the scenes (2,048 pushed particles each) take at most eight times the wall kernels' time; with
    the pairs of all scenes tested it was 64 times the pairs."""
    ms = []
    for n in (8, 64):
        line = _pushed_line(vxl, 2048)
        b = _floored(vxl, [line] * n)
        b.set_profile(True)
        for _ in range(5):
            for q in range(n):
                b.write_state(q, line.pos, line.vel)
            b.substep(1e-4)
        total, launches = b.profile()["k_walls"]
        assert launches > 0
        ms.append(total / launches)
        b.close()
    assert ms[1] < 8 * ms[0], ms


@pytest.mark.parametrize("h,over", [(0.1, {}), (0.1, dict(tensile_instability_suppression=False)), (3e-4, {}), (2e-3, {}),
                                    (900.0, {}), (3000.0, {}), (0.1, dict(artificial_viscosity=0.0)),
                                    (0.1, dict(artificial_viscosity=3e3)), (0.1, dict(rest_density=1e-15)),
                                    (0.1, dict(rest_density=1e12))])
def test_pair_quotients_over_scales(vxl, oracle_mod, h, over):
    """Smoothing lengths, viscosities and densities inside and outside the shared-reciprocal range, pressures of
    both signs, pairs at rest, slow (1e-20) and fast, coincident pairs: forces and reactions bit for bit."""
    from vxl_sph import scenes
    s = 0.5 * h
    rng = np.random.default_rng(9)
    pos = scenes.jitter(scenes.fluid_block((0.0, 0.0, 0.0), (6, 5, 6), s), s, 3, 0.3)
    pos[7] = pos[6]
    vel = np.zeros_like(pos)
    vel[:60] = rng.normal(size=(60, 3))
    vel[60:120] = rng.normal(size=(60, 3)) * 1e-20
    b = scenes.body_particles([scenes.Body(0, (3 * s, s, 3 * s), (3 * s, -1.2 * s, 3 * s))], s, h, 1, over.get("rest_density", 1000.0))
    _run_both(vxl, oracle_mod, _custom(vxl, pos, vel=vel, h=h, spacing=s, boundary=b, **over), substeps=2)


def test_reciprocals_and_quotients_on_the_device(tmp_path):
    """recip_rn against 1 / b for every significand (it rests on rcp.approx being within 1 ulp), quot_rn against a / b
    for every divisor's numerators nearest a rounding midpoint: every pair that the step could round wrongly."""
    import subprocess
    from pathlib import Path
    from vxl_sph import build
    exe = tmp_path / "quotients"
    flags = [f for f in build.NVCC_FLAGS if f != "-shared"]
    src = Path(__file__).resolve().parent / "c" / "quotients.cu"
    subprocess.run([build.nvcc(), *flags, "-I", str(build.CSRC), "-o", str(exe), str(src)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    assert int(r.stdout.split()[3]) > 5e7, r.stdout


def _edge_scenes(vxl):
    from vxl_sph import scenes
    rng = np.random.default_rng(17)
    s = 0.025
    plate = scenes.body_particles([scenes.Body(0, (0.2, 0.05, 0.2), (0.125, -0.05, 0.125))], s, 4 * s, 1, 1000.0)
    walled = scenes.small_dam(n=(9, 8, 7), spacing=0.05, tank=(0.7, 0.6, 0.5), seed=8)
    return [_custom(vxl, rng.uniform(0.0, 0.08, (230, 3)).astype(F32), h=0.1),  # one crowded cell
            _custom(vxl, scenes.jitter(scenes.fluid_block((0, 0, 0), (9, 8, 9), s), s, 5), h=3 * s, spacing=s),  # > 64 neighbours
            _custom(vxl, scenes.fluid_block((0.0, 0.0, 0.0), (10, 8, 10), s), h=4 * s, spacing=s, boundary=plate),  # reactions too
            _custom(vxl, rng.uniform(0.0, 0.9, (701, 3)).astype(F32), h=0.1, max_bins=100),  # doubled bins
            walled]


@pytest.mark.parametrize("filler", [19000, 30000, 50000])
def test_scenes_step_the_same_beside_a_filler(vxl, filler):
    """The lanes per particle follow the whole batch's size: edge scenes alone (eight lanes) and beside a block that
    brings the passes to four lanes and to one, bitwise, with their reactions."""
    from vxl_sph import scenes
    specs = _edge_scenes(vxl)
    alone = vxl.Batch(specs)
    n = int(round(filler ** (1 / 3)))
    big = _custom(vxl, scenes.jitter(scenes.fluid_block((0, 0, 0), (n, n, n), 0.05), 0.05, 6))
    both = vxl.Batch(specs + [big])
    for t in range(2):
        ra, rb = alone.step_tick(1.0 / 60.0), both.step_tick(1.0 / 60.0)
        assert len(ra) == len(rb) >= 6
        for (b1, f1, t1), (b2, f2, t2) in zip(ra, rb):
            assert b1 == b2 and f1.tobytes() == f2.tobytes() and t1.tobytes() == t2.tobytes(), (t, b1)
        for q in range(len(specs)):
            for x, y in zip(alone.read_state(q), both.read_state(q)):
                assert x.tobytes() == y.tobytes(), (t, q)


@pytest.mark.parametrize("walls", [2600, 14000, 23000])
def test_boundary_forces_over_lane_counts(vxl, walls):
    """Boundary forces with eight, four and one lane per particle: the edge scenes' reactions beside a dry plate
    of `walls` boundary particles."""
    from vxl_sph import scenes
    specs = [_edge_scenes(vxl)[k] for k in (2, 0)]  # (a handle of one scene takes its spans per call)
    half = 0.02 * (walls / 2) ** 0.5 / 2
    plate = scenes.body_particles([scenes.Body(0, (half, 0.02, half), (0.0, -0.5, 0.0))], 0.02, 0.04, 1, 1000.0)
    assert 0.7 * walls < plate[0].shape[0] < 1.4 * walls
    far = _custom(vxl, [[0.0, 0.5, 0.0]], h=0.04, spacing=0.02, boundary=plate)
    alone, both = vxl.Batch(specs), vxl.Batch(specs + [far])
    for t in range(2):
        a, b = alone.step_tick(1.0 / 60.0)[0], both.step_tick(1.0 / 60.0)[0]
        assert np.any(a[1] != 0)
        assert a[1].tobytes() == b[1].tobytes() and a[2].tobytes() == b[2].tobytes(), t

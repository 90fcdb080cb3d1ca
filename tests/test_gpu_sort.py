"""The table's per-cell order and the gathered state, over cell sizes around the ranking loop's steps (B200)."""
import numpy as np
import pytest

from test_gpu_parity import F32, _custom, _run_both, compare_grid, pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(1, 2, 3, 4, 5), (7, 8, 9, 31, 32, 33), (63, 64, 65, 255, 256, 257), (700, 1, 2)])
def test_cells_of_every_size_sort(vxl, oracle_mod, sizes):
    """Cells two bins apart holding `sizes` particles each, the indices dealt out across them, over three substeps
    (the second and third start from the order the first left)."""
    rng = np.random.default_rng(sum(sizes))
    pos = np.concatenate([rng.uniform(0.01, 0.09, (n, 3)) + (0.2 * k, 0.0, 0.1 * (k % 2)) for k, n in enumerate(sizes)])
    pos = pos[rng.permutation(len(pos))].astype(F32)
    _run_both(vxl, oracle_mod, _custom(vxl, pos, h=0.1), substeps=3)


def _static(vxl, pos, h, max_bins):
    import ctypes as C
    import torch
    n = pos.shape[0]
    d_pos = torch.from_numpy(np.ascontiguousarray(pos, F32)).cuda()
    items = torch.full((n,), -1, dtype=torch.int32, device="cuda")
    start = torch.full((max_bins + 1,), -1, dtype=torch.int32, device="cuda")
    info = vxl.GridInfo()
    info.hdr = vxl.header(vxl.GridInfo)
    st = vxl.load().vxl_sph_build_grid_static(C.c_void_p(d_pos.data_ptr()), n, h, max_bins, C.c_void_p(items.data_ptr()),
                                              C.c_void_p(start.data_ptr()), max_bins + 1, C.byref(info),
                                              C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert st == vxl.OK
    return items.cpu().numpy().view(np.uint32), start[: int(info.total) + 1].cpu().numpy().view(np.uint32), info


@pytest.mark.parametrize("n,cells", [(1, 1), (31, 3), (257, 2), (2048, 1), (2049, 1), (4100, 2), (70000, 30), (100000, 20)])
def test_static_grid_over_cell_sizes(vxl, oracle_mod, n, cells):
    """The allocation-free table around the ranking limit (2,048 entries a cell; larger ones by bitmap), called
    twice so that the second starts from the first's leftovers, against the oracle's table."""
    rng = np.random.default_rng(n)
    pos = rng.uniform(0.0, 0.09, (n, 3))
    pos[:, 0] += 0.1 * rng.integers(0, cells, n)
    pos[0] = 0.0
    if n > 2:
        pos[1] = np.nan  # never in the box; binned into the first cell
    pos = pos.astype(F32)
    ref_start, ref_items, _ = oracle_mod.rebuild_grid(pos, 0.1, 4096)
    for _ in range(2):
        items, start, info = _static(vxl, pos, 0.1, 4096)
        assert np.array_equal(start, ref_start) and np.array_equal(items, ref_items), (n, cells)


@pytest.mark.parametrize("cells", [1, 2, 511, 512, 513, 1024, 1300])
def test_grid_export_over_tile_edges(vxl, oracle_mod, cells):
    """The exported table of grids that end within, at and past the export's tiles, full and empty cells mixed."""
    rng = np.random.default_rng(cells)
    x = np.concatenate([[0.05, 0.1 * cells - 0.05], 0.1 * rng.integers(0, cells, 700) + 0.05])
    pos = np.stack([x, rng.uniform(0.0, 0.09, 702), np.zeros(702)], 1).astype(F32)
    spec = _custom(vxl, pos)
    g, o = pair(vxl, oracle_mod, spec)
    g.substep(1e-4)
    o.substep(1e-4)
    assert abs(int(g.export_grid()[3].total) - cells) <= 1
    compare_grid(g, o, f"{cells} cells")


def test_grid_export_takes_about_a_state_read(vxl):
    """A sparse tank's table of a million cells (8 MB out) takes less than twice the time of its 10 MB of state (0.7 ms
    each): the scan of the cells goes over the whole GPU, one block took 1.2 ms for it."""
    import time
    from vxl_sph import scenes
    spec = scenes.dam_break("sparse", (20, 20, 20), 0.01, (2.0, 2.0, 2.0), 1, 3)
    g = vxl.Scene(spec.params, spec.pos, spec.vel, spec.pmass, spec.n_fluid)
    g.substep(1e-4)
    out = (np.empty_like(spec.pos), np.empty_like(spec.vel))
    best = [1e9, 1e9]
    for _ in range(7):
        for k, call in enumerate((lambda: g.export_grid(), lambda: g.read_state(out=out))):
            t = time.perf_counter()
            call()
            best[k] = min(best[k], time.perf_counter() - t)
    assert g.export_grid()[3].total > 1000000
    assert best[0] < 2 * best[1], best

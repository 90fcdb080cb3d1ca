"""The table's per-cell order and the gathered state, over cell sizes around the ranking loop's steps (B200)."""
import numpy as np
import pytest

from test_gpu_parity import F32, _custom, _run_both

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(1, 2, 3, 4, 5), (7, 8, 9, 31, 32, 33), (63, 64, 65, 255, 256, 257), (700, 1, 2)])
def test_cells_of_every_size_sort(vxl, oracle_mod, sizes):
    """Cells two bins apart holding `sizes` particles each, the indices dealt out across them, over three substeps
    (the second and third start from the order the first left)."""
    rng = np.random.default_rng(sum(sizes))
    pos = np.concatenate([rng.uniform(0.01, 0.09, (n, 3)) + (0.2 * k, 0.0, 0.1 * (k % 2)) for k, n in enumerate(sizes)])
    pos = pos[rng.permutation(len(pos))].astype(F32)
    _run_both(vxl, oracle_mod, _custom(vxl, pos, h=0.1), substeps=3)

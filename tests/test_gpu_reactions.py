"""Wall separation where its check's tiles can go wrong (B200), against the oracle."""
import numpy as np
import pytest

from test_gpu_parity import F32, _custom, compare_state, pair

pytestmark = pytest.mark.gpu


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

"""The binning at its line between worlds whose blocks scan the tiles' counts
themselves (up to 4,096 tiles of 16x8x8 cells) and worlds whose occupied tiles
are listed by kernels, bit for bit against the oracle."""
import numpy as np
import pytest

import scenarios
from mls_mpm_b200 import scenes
from runner import GpuScene, cpu_run, diff_report

pytestmark = pytest.mark.gpu


def _scene(grid, n, seed):
    """n particles in the first and the last tile, in a block in the middle and all over."""
    rng = np.random.default_rng(seed)
    low, high = np.array([2.0, 2.0, 2.0]), np.array(grid) - 2.0
    mid = np.array(grid) / 2.0
    k = n // 4
    pos = np.concatenate([rng.uniform(low, low + 6, (k, 3)), rng.uniform(high - 6, high, (k, 3)),
                          rng.uniform(mid - 9, mid + 9, (k, 3)), rng.uniform(low, high, (n - 3 * k, 3))])
    return scenes.Scene(grid, pos.astype(np.float32), rng.uniform(-2, 2, (n, 3)).astype(np.float32), name="tile_lines")


# 16 x 16 x 16 = 4,096 tiles, a layer of tiles one cell deep more, and 5,250 tiles
@pytest.mark.parametrize("grid", [(256, 128, 128), (256, 128, 129), (657, 40, 200)])
@pytest.mark.parametrize("n", [4, 3001])
def test_tiles_on_both_sides_of_the_line(gpu, grid, n):
    sc = scenarios.Scenario("tile_lines", _scene(grid, n, n), 3)
    g = GpuScene(gpu, sc.scene)
    try:
        for k, ((P, W, H, dims, gen, adv), o) in enumerate(zip(sc.frames(), cpu_run(sc, "oracle", threads=16))):
            g.frame(P, W, H, dims)
            bad = diff_report(g.state(), o)
            assert not bad, f"substep {k}: {bad}"
    finally:
        g.close()

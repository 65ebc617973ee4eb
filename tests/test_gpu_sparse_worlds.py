"""Few particles in a large grid: a substep follows the particles and not the tiles."""
import time

import numpy as np
import pytest

import scenarios
from mls_mpm_b200 import scenes
from mls_mpm_b200.abi import check
from runner import GpuScene

pytestmark = pytest.mark.gpu


def test_few_particles_in_a_large_grid(gpu):
    def substep_us(grid):
        sc = scenes.small_box(grid=(24, 24, 24), n=1000, seed=1, name="few")
        g = GpuScene(gpu, scenes.Scene(grid, sc.pos[:, :3].copy(), sc.vel[:, :3].copy(), name="few"))
        try:
            (P, W, H, dims, _, _), = scenarios.Scenario("few", g.scene, 1).frames()
            g.frame(P, W, H, dims, substeps=40)
            best = np.inf
            for _ in range(5):
                check(gpu.mpm_sync(g.h), "sync")
                t = time.perf_counter()
                check(gpu.mpm_step(g.h, 200), "step")
                check(gpu.mpm_sync(g.h), "sync")
                best = min(best, (time.perf_counter() - t) / 200 * 1e6)
            return best
        finally:
            g.close()

    small, large = substep_us((128, 128, 128)), substep_us((512, 512, 512))   # 2,048 and 131,072 tiles
    assert large < 1.6 * small, (small, large)   # (1.1; one block's loop over all tiles made it 2.2)

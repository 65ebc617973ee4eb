"""The binning's two ways to place the tiles: worlds of up to 16,384 tiles of
16x8x8 cells, whose binning blocks scan the tiles' particle counts themselves,
and larger ones, where a kernel lists the occupied tiles first.  Particles sit
in the first and the last tiles and in blocks that cross the 1,024-tile groups
of the scans; every array bit-exact against the oracle after each substep, and
again after a second upload of other particles."""
import numpy as np
import pytest

import scenarios
from mls_mpm_b200 import abi, scenes
from mls_mpm_b200.abi import check
from runner import GpuScene, cpu_run, diff_report

pytestmark = pytest.mark.gpu


def _scene(grid, seed):
    rng = np.random.default_rng(seed)
    X, Y, Z = grid
    low, high = np.array([2.0, 2.0, 2.0]), np.array([X, Y, Z]) - 2.0
    parts = [rng.uniform(low, low + 6, (700, 3)),            # the first tile
             rng.uniform(high - 6, high, (513, 3)),          # the last one
             rng.uniform([X / 2 - 20, 2, Z / 2 - 3], [X / 2 + 20, 12, Z / 2 + 3], (1500, 3)),
             rng.uniform(low, high, (300, 3))]               # one to a tile, all over
    pos = np.concatenate(parts).astype(np.float32)
    vel = rng.uniform(-2, 2, pos.shape).astype(np.float32)
    return scenes.Scene(grid, pos, vel, name="many_tiles")


# 32 x 32 x 16 = 16,384 tiles, and 32 x 32 x 17 (the last row of tiles one cell deep)
@pytest.mark.parametrize("grid", [(512, 256, 128), (509, 256, 129)])
def test_tile_placement_bit_exact(gpu, grid):
    sc = scenarios.Scenario("many_tiles", _scene(grid, 1), 3)
    g = GpuScene(gpu, sc.scene)
    try:
        for again in range(2):
            if again:
                sc = scenarios.Scenario("many_tiles", _scene(grid, 2), 2)
                s = sc.scene
                check(gpu.mpm_upload_particles(g.h, abi.ptr(s.pos), abi.ptr(s.vel), abi.ptr(s.affine), abi.ptr(s.mass),
                                               s.n), "upload")
            for k, ((P, W, H, dims, gen, adv), o) in enumerate(zip(sc.frames(), cpu_run(sc, "oracle", threads=16))):
                g.frame(P, W, H, dims)
                bad = diff_report(g.state(), o)
                assert not bad, f"upload {again} substep {k}: {bad}"
    finally:
        g.close()

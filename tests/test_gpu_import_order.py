"""Loading particles in any order: a load counts the particles of each tile in a
table per block, with a slot per tile modulo 1,024.  Many shuffled particles, in
tiles that share slots and in few tiles, bit for bit against the oracle; and a
load in shuffled order costs about what one in the order of the cells does."""
import ctypes
import time

import numpy as np
import pytest

import oracle as O
from mls_mpm_b200 import abi, scenes
from mls_mpm_b200.abi import check
from mls_mpm_b200.batch import default_params
from runner import GpuScene, diff_report

pytestmark = pytest.mark.gpu


def _scene(grid, lo, hi, n, seed, ordered=False):
    rng = np.random.default_rng(seed)
    pos = rng.uniform(lo, hi, (n, 3)).astype(np.float32)
    if ordered:
        cell = np.floor(pos).astype(np.int64)
        pos = pos[np.argsort((cell[:, 2] * grid[1] + cell[:, 1]) * grid[0] + cell[:, 0])]
    return scenes.Scene(grid, pos, rng.uniform(-0.5, 0.5, (n, 3)).astype(np.float32), name="import_order")


# more particles than blocks of 256 at twelve an SM; 2,304 tiles (three to a slot) and one tile; one particle
@pytest.mark.parametrize("grid,lo,hi,n", [((128, 144, 128), 2.5, (125.5, 141.5, 125.5), 500_003),
                                          ((128, 144, 128), (35.0, 33.0, 33.0), (46.0, 38.0, 38.0), 20_001),
                                          ((128, 144, 128), 60.0, 61.0, 1)])
def test_shuffled_loads_bit_exact(gpu, grid, lo, hi, n):
    sc = _scene(grid, lo, hi, n, 5)
    P, W, st = default_params(grid, n), abi.WallParams(), O.new_state(sc)
    g = GpuScene(gpu, sc)
    try:
        for k in range(2):
            g.frame(P, W, None, None)
            O.substep(st, P, W, threads=16)
            bad = diff_report(g.state(), st)
            assert not bad, f"substep {k}: {bad}"
    finally:
        g.close()


def test_order_costs_little(gpu):
    n, grid = 2_000_000, (64, 64, 64)   # 256 tiles

    def load_us(ordered):
        g = GpuScene(gpu, _scene(grid, 2.5, 61.5, n, 6, ordered))
        try:
            Ps = [default_params(grid, n - 1), default_params(grid, n)]
            g.frame(Ps[1], abi.WallParams(), None, None, substeps=2)
            best = np.inf
            for _ in range(6):
                check(gpu.mpm_sync(g.h), "sync")
                t = time.perf_counter()
                for k in range(20):   # a changed count loads the scene again, here without a substep
                    check(gpu.mpm_set_params(g.h, ctypes.byref(Ps[k % 2])), "params")
                    check(gpu.mpm_step(g.h, 0), "step")
                check(gpu.mpm_sync(g.h), "sync")
                best = min(best, (time.perf_counter() - t) / 20 * 1e6)
            return best
        finally:
            g.close()

    ordered, shuffled = load_us(True), load_us(False)
    print(f"load: in order {ordered:.0f} us, shuffled {shuffled:.0f} us")
    assert shuffled < 1.5 * ordered, (ordered, shuffled)

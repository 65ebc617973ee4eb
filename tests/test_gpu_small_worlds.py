"""Worlds on both sides of the line up to which P2G_MOM decodes the cell masses itself (one 256-particle chunk for each of
four blocks on every SM) instead of a pass of its own: every array bit-exact against the oracle, the decoded grid included,
and a batch that falls below the line when a scene leaves it."""
import numpy as np
import pytest

import oracle as O
import scenarios
from mls_mpm_b200 import abi, scenes
from runner import GpuScene, diff_report

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("over", [None, -1, 0, 1, 40000])
def test_worlds_around_the_line(gpu, over):
    import torch
    line = torch.cuda.get_device_properties(0).multi_processor_count * 4 * 256
    n = 1 if over is None else line + over
    sc = scenarios.Scenario("line", scenes.small_box(grid=(72, 60, 70), n=n, seed=11, name="line"), 3,
                            walls=scenarios._walls_moving)
    st = O.new_state(sc.scene)
    g = GpuScene(gpu, sc.scene)
    try:
        for P, W, H, dims, gen, adv in sc.frames():
            O.substep(st, P, W, H, dims, gen, adv, threads=8)
            g.frame(P, W, H, dims)
            bad = diff_report(g.state(), st)
            assert not bad, bad
    finally:
        g.close()


def test_batch_shrinks_below_the_line(gpu):
    """A batch above the line loses a scene and falls below it; the scene that stays is bit-exact throughout."""
    from mls_mpm_b200.batch import Batch, default_params
    big = scenes.small_box(grid=(72, 60, 70), n=150000, seed=3, name="big")
    keep = scenes.small_box(grid=(24, 20, 22), n=3000, seed=4, name="keep")
    P = default_params(keep.grid, keep.n)
    b = Batch(big.n + keep.n, big.cells + keep.cells, 2)
    try:
        ib = b.add(default_params(big.grid, big.n), big.pos, big.mass, big.vel, big.affine)
        ik = b.add(P, keep.pos, keep.mass, keep.vel, keep.affine)
        st = O.new_state(keep)
        for step in range(6):
            if step == 3:
                b.remove(ib)
            b.step(1)
            O.substep(st, P, abi.WallParams())
            for k in ("pos", "vel", "density", "cell_mass_f32", "cell_mv_f32"):
                got = b.read(ik, k)
                assert np.array_equal(got.reshape(-1).view(np.uint32), np.ascontiguousarray(st[k]).reshape(-1).view(np.uint32)), (step, k)
    finally:
        b.close()

"""The density of a scene added to a batch that has already stepped reads 0
until its first substep, as it does in a new batch, also where it takes
positions that an earlier, longer layout used; every scene's density follows
the oracle from then on."""
import numpy as np
import pytest

import oracle as O
from mls_mpm_b200 import abi, scenes
from mls_mpm_b200.batch import Batch, default_params

pytestmark = pytest.mark.gpu

GRID = (28, 24, 26)


@pytest.mark.parametrize("late", [1, 700, 2000, 4500])   # fewer and more particles than the positions left behind
@pytest.mark.parametrize("stepped_without", [False, True])   # the removed scene's holes still there, or compacted away
def test_density_of_a_scene_added_late(gpu, late, stepped_without):
    b = Batch(12000, 3 * 28 * 24 * 26, 3)
    W = abi.WallParams()

    def add(n, seed):
        sc = scenes.small_box(grid=GRID, n=n, seed=seed, name=f"late{seed}")
        return b.add_scene(sc), O.new_state(sc), default_params(GRID, n)

    def step(live, k=1):
        b.step(k)
        for _, st, P in live:
            for _ in range(k):
                O.substep(st, P, W)

    def compare(live):
        for sid, st, _ in live:
            assert np.array_equal(b.read(sid, "density").view(np.uint32), st["density"].view(np.uint32)), sid

    try:
        live = [add(3000, 1), add(2500, 2)]
        compare(live)                     # before the first substep
        step(live, 2)
        compare(live)
        b.remove(live.pop()[0])
        if stepped_without:
            step(live)
        live.append(add(late, 3))
        compare(live)                     # zeros for the new scene, the others' untouched
        step(live)
        compare(live)
    finally:
        b.close()

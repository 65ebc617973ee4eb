"""Diffuse free-list passes at the edges of their segments (64 groups of 256 ids, 512 segments before a segment holds
more groups): pools whose last group or segment is ragged, one of more than 512 segments, and pools that fill up, so that
only the spawners of the lowest ids find a slot.  Pool, stack and top are bit-exact against the oracle."""
import numpy as np
import pytest

import oracle as O
import scenarios
from mls_mpm_b200 import scenes
from runner import ENGINES, GpuScene

pytestmark = pytest.mark.gpu

# (slots, particles): a pool of one slot; one group and one slot more; a segment less, exactly and more than its
# 16,384 ids, with as many particles; a pool of 513 segments
SIZES = [(1, 3000), (257, 3000), (16383, 9000), (16384, 16385), (16500, 33000), (8388609, 4000)]
SUBSTEPS = 12   # the first slots are freed after about nine


@pytest.mark.parametrize("engine", list(ENGINES))
@pytest.mark.parametrize("slots,n", SIZES)
def test_free_list_at_segment_edges(gpu, engine, slots, n):
    sc = scenarios.Scenario("pool", scenes.small_box(grid=(36, 30, 34), n=n, seed=5, name="pool"), SUBSTEPS,
                            diffuse_max=slots, hand=scenarios._hand_sweep)
    # falling fast, so that many particles spawn at once; a short life, so that many slots are freed
    sc.scene.vel[:, 1] = -2.0
    st = O.new_state(sc.scene, slots)
    g = GpuScene(gpu, sc.scene, slots, flags=ENGINES[engine])
    spawned = 0
    try:
        for s, (P, W, H, dims, gen, adv) in enumerate(sc.frames()):
            O.substep(st, P, W, H, dims, gen, adv)
            g.frame(P, W, H, dims)
            spawned = max(spawned, slots - int(st["top"][0]))
            if s + 3 < SUBSTEPS:
                continue
            for k in ("top", "free_list", "diffuse"):
                a = g.read(k)
                assert np.array_equal(a.view(np.uint8), np.ascontiguousarray(st[k]).view(np.uint8)), k
        assert spawned >= min(slots, 200), spawned
    finally:
        g.close()

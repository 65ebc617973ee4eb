"""The serving loop's host blocks: jobs of one server, run after run, in blocks
that earlier jobs used (larger ones, smaller ones, with and without initial
velocities), whose states leave the blocks in one piece or several.  Every final
state is bit-exact against the oracle running that scene alone."""
import numpy as np
import pytest

import oracle as O
from mls_mpm_b200 import abi, scenes
from mls_mpm_b200.batch import default_params
from mls_mpm_b200.server import Server

pytestmark = pytest.mark.gpu

# particle counts of successive runs: the smallest block (64 KB, 1820 particles) and one more; a state of just over one
# and over three pieces of 256 KB; then each in a block left by another
RUNS = [(1, 1820, 1821, 7300), (22000, 900, 7281, 1), (7282, 15000, 1821)]


@pytest.mark.parametrize("keep", [True, False])
def test_blocks_serve_one_run_after_another(gpu, keep):
    srv = Server(1 << 28, scene_capacity=3, cells_per_particle=4.0, flags=abi.SERVER_KEEP_STATE if keep else 0)
    try:
        for r, counts in enumerate(RUNS):
            jobs = []
            for i, n in enumerate(counts):
                sc = scenes.small_box(grid=(24, 20, 28), n=n, seed=10 * r + i, name=f"run{r}job{i}")
                vel = sc.vel if (r + i) % 2 else None
                steps = 2 + 3 * ((i + r) % 3)
                P = default_params(sc.grid, sc.n)
                jobs.append((sc, vel, steps, P, srv.submit(P, sc.pos, sc.mass, steps, 0.0, vel4=vel)))
            assert srv.run().jobs == len(jobs)
            for sc, vel, steps, P, j in jobs:
                res = srv.job(j)
                assert res.done
                if not keep:
                    with pytest.raises(abi.MpmError):
                        srv.download(j, "pos")
                    continue
                want = O.new_state(sc)
                if vel is None:
                    want["vel"][:] = 0.0
                for _ in range(steps):
                    O.substep(want, P, abi.WallParams())
                for k in ("pos", "vel", "density"):
                    got = srv.download(j, k)
                    assert np.array_equal(got.view(np.uint32), np.ascontiguousarray(want[k]).view(np.uint32)), (sc.name, k)
    finally:
        srv.close()

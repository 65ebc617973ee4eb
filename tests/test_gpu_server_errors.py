"""A serving run that ends with an error keeps what it finished: jobs that
retired before it are done, their final states can be downloaded and equal the
oracle's, their host blocks serve later submissions, and the job that could not
be admitted stays queued."""
import numpy as np
import pytest

import oracle as O
from mls_mpm_b200 import abi, scenes
from mls_mpm_b200.batch import default_params
from mls_mpm_b200.server import Server

pytestmark = pytest.mark.gpu


BUDGET = 1 << 28   # 610,000 particles, 2.4M cells and 7,400 tiles of 16x8x8 cells at four cells a particle
# submit accepts it (its 2M cells fit) and no batch admits it: 5 x 5 cells pad to a whole tile, 10,000 of them
MISFIT = (5, 5, 80000)


# particle counts of the jobs before it: states of less than one, of several and of many pieces of 256 KB
@pytest.mark.parametrize("counts", [(900,), (22000,), (3000, 22000, 1, 60000)])
@pytest.mark.parametrize("keep", [True, False])
def test_finished_jobs_survive_a_later_failure(gpu, counts, keep):
    srv = Server(BUDGET, scene_capacity=3, cells_per_particle=4.0, flags=abi.SERVER_KEEP_STATE if keep else 0)
    try:
        for again in range(2):   # the misfit, submitted once, is the last in order of arrival both times
            jobs = []
            for i, n in enumerate(counts):
                sc = scenes.small_box(grid=(44, 30, 48), n=n, seed=7 * again + i, name=f"job{i}")
                P = default_params(sc.grid, sc.n)
                jobs.append((sc, P, 2 + i, srv.submit(P, sc.pos, sc.mass, 2 + i, 0.0, vel4=sc.vel)))
            if not again:
                bad = scenes.small_box(grid=(24, 20, 28), n=10, seed=1, name="misfit")
                thin = srv.submit(default_params(MISFIT, 10), bad.pos, bad.mass, 3, 1e-6)
            with pytest.raises(abi.MpmError) as err:
                srv.run()
            assert abi.status_name(err.value.status) == "MPM_ERR_CAPACITY"
            assert not srv.job(thin).done
            for sc, P, steps, j in jobs:
                res = srv.job(j)
                assert res.done and res.finish_s > 0.0
                if not keep:
                    continue
                want = O.new_state(sc)
                for _ in range(steps):
                    O.substep(want, P, abi.WallParams(), threads=4)
                for k in ("pos", "vel", "density"):
                    got = srv.download(j, k)
                    assert np.array_equal(got.view(np.uint32), np.ascontiguousarray(want[k]).view(np.uint32)), (sc.n, k)
    finally:
        srv.close()

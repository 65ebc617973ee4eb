"""Which scenes get their render buffers from the pass after G2P: those of
1,500,000 active particles or more, 65 substeps after a load.  The pass is one
launch more a substep, so the launch count tells; the bound buffers equal what a
scene without bound buffers downloads."""
import ctypes

import numpy as np
import pytest

from mls_mpm_b200 import abi
from mls_mpm_b200.abi import BUF, check
from mls_mpm_b200.batch import default_params
from mls_mpm_b200.fluid_gpu import Desc

pytestmark = pytest.mark.gpu

GRID = (100, 96, 104)
LINE = 1_500_000


class _Scene:
    def __init__(self, lib, n, capacity, bound):
        self.lib, self.n = lib, n
        rng = np.random.default_rng(n)
        pos = np.zeros((n, 4), np.float32)
        pos[:, :3] = rng.uniform(2.5, np.array(GRID) - 2.5, (n, 3))
        vel = np.zeros((n, 4), np.float32)
        vel[:, :3] = rng.uniform(-0.5, 0.5, (n, 3))
        mass = np.ones(n, np.float32)
        self.h = ctypes.c_void_p()
        check(lib.mpm_create(ctypes.byref(Desc(*GRID, capacity, 0, 0)), ctypes.byref(self.h)), "create")
        check(lib.mpm_upload_particles(self.h, abi.ptr(pos), abi.ptr(vel), None, abi.ptr(mass), n), "upload")
        P = default_params(GRID, n)
        check(lib.mpm_set_params(self.h, ctypes.byref(P)), "params")
        self.ptrs = {}
        for name in ("pos", "vel", "density") if bound else ():
            p, sz = ctypes.c_void_p(), ctypes.c_size_t()
            check(lib.mpm_get_buffer(self.h, BUF[name], ctypes.byref(p), ctypes.byref(sz)), "get_buffer")
            self.ptrs[name] = p.value

    def step(self, k):
        """Launches of k substeps."""
        a, b = ctypes.c_uint64(), ctypes.c_uint64()
        check(self.lib.mpm_launch_count(self.h, ctypes.byref(a)), "launches")
        check(self.lib.mpm_step(self.h, k), "step")
        check(self.lib.mpm_launch_count(self.h, ctypes.byref(b)), "launches")
        return b.value - a.value

    def read(self, name):
        from cuda.bindings import driver
        out = np.empty((self.n, 4) if name != "density" else (self.n,), np.float32)
        if name in self.ptrs:
            check(self.lib.mpm_sync(self.h), "sync")
            err, = driver.cuMemcpyDtoH(out.ctypes.data, self.ptrs[name], out.nbytes)
            assert err == driver.CUresult.CUDA_SUCCESS, err
        else:
            check(self.lib.mpm_download(self.h, BUF[name], abi.ptr(out), out.nbytes), "download")
        return out.view(np.uint32)

    def delete(self):
        """Removes the particles around an axis; returns how many are left."""
        m = ctypes.c_uint32()
        o, d = (ctypes.c_double * 3)(50.0, 0.0, 50.0), (ctypes.c_double * 3)(0.0, 1.0, 0.0)
        check(self.lib.mpm_delete_near(self.h, o, d, 6.0, ctypes.byref(m)), "delete")
        self.n = m.value
        return m.value

    def close(self):
        self.lib.mpm_destroy(self.h)


@pytest.mark.parametrize("n", [40_000, LINE - 1, LINE, LINE + 1025])
def test_pass_follows_the_active_particles(gpu, n):
    a, b = _Scene(gpu, n, LINE + 100_000, True), _Scene(gpu, n, LINE + 100_000, False)
    try:
        extra = int(n >= LINE)
        assert a.step(64) == b.step(64)
        assert a.step(4) == b.step(4) + 4 * extra
        a.step(20), b.step(20)              # past the eagerly launched substeps
        assert a.step(2) == b.step(2) + 2 * extra
        for name in ("pos", "vel", "density"):
            assert np.array_equal(a.read(name), b.read(name)), name
        # an edit that takes the scene below the line ends the pass
        assert a.delete() == b.delete() < LINE
        assert a.step(3) == b.step(3)
        a.step(20), b.step(20)
        assert a.step(2) == b.step(2)
        for name in ("pos", "vel", "density"):
            assert np.array_equal(a.read(name), b.read(name)), name
    finally:
        a.close()
        b.close()

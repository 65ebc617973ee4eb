"""Render buffers of large scenes: written by G2P in the first 64 substeps after
the load, by the pass that reads them from the layout's records afterwards.
The smallest capacities on both sides of the rule, few active particles in them
(counts on both sides of the pass's 1,024 a block): the bytes at the bound
pointers equal the oracle's state in the substeps around the change, after
edits and after a new load."""
import ctypes

import numpy as np
import pytest

import oracle as O
from mls_mpm_b200 import abi, scenes
from mls_mpm_b200.abi import BUF, check
from mls_mpm_b200.batch import default_params
from mls_mpm_b200.fluid_gpu import Desc
from runner import diff_report

pytestmark = pytest.mark.gpu


def _read(ptr, shape):
    from cuda.bindings import driver
    out = np.empty(shape, np.float32)
    err, = driver.cuMemcpyDtoH(out.ctypes.data, ptr, out.nbytes)
    assert err == driver.CUresult.CUDA_SUCCESS, err
    return out


def _scene(seed, n):
    rng = np.random.default_rng(seed)
    pos = rng.uniform(2.2, 21.8, (n, 3)).astype(np.float32)
    return scenes.Scene((24, 24, 24), pos, rng.uniform(-1, 1, (n, 3)).astype(np.float32), name="gather")


@pytest.mark.parametrize("capacity", [1_499_999, 1_500_000])
@pytest.mark.parametrize("n", [1, 1024, 3001])
def test_bound_buffers_follow_every_step(gpu, capacity, n):
    h = ctypes.c_void_p()
    check(gpu.mpm_create(ctypes.byref(Desc(24, 24, 24, capacity, 0, 0)), ctypes.byref(h)), "create")

    def load(sc):
        check(gpu.mpm_upload_particles(h, abi.ptr(sc.pos), abi.ptr(sc.vel), abi.ptr(sc.affine), abi.ptr(sc.mass), sc.n),
              "upload")
        return O.new_state(sc)

    def step(st, k, compare_from):
        count = len(st["mass"])
        P, W = default_params((24, 24, 24), count), abi.WallParams()
        check(gpu.mpm_set_params(h, ctypes.byref(P)), "params")
        for i in range(k):
            check(gpu.mpm_step(h, 1), "step")
            O.substep(st, P, W)
            if i < compare_from:
                continue
            check(gpu.mpm_sync(h), "sync")
            got = {"pos": _read(ptrs["pos"], (count, 4)), "vel": _read(ptrs["vel"], (count, 4)),
                   "density": _read(ptrs["density"], (count,))}
            bad = diff_report(got, st)
            assert not bad, f"step {i}: {bad}"

    try:
        st = load(_scene(3, n))
        ptrs = {}
        for name in ("pos", "vel", "density"):
            p, sz = ctypes.c_void_p(), ctypes.c_size_t()
            check(gpu.mpm_get_buffer(h, BUF[name], ctypes.byref(p), ctypes.byref(sz)), "get_buffer")
            ptrs[name] = p.value
        step(st, 68, 62)
        if n > 100:   # an edit keeps the substep count: the pass goes on with fewer particles
            m = ctypes.c_uint32()
            o, d = (ctypes.c_double * 3)(12.0, 0.0, 12.0), (ctypes.c_double * 3)(0.0, 1.0, 0.0)
            check(gpu.mpm_delete_near(h, o, d, 3.0, ctypes.byref(m)), "delete")
            P = default_params((24, 24, 24), n)
            c, po, vo, mo = O.compact(P, abi.RayParams(12.0, 0.0, 12.0, 3.0, 0.0, 1.0, 0.0, 0.0), st["pos"], st["vel"],
                                      st["mass"])
            assert c == m.value
            sc = scenes.Scene((24, 24, 24), po[:c, :3], vo[:c, :3], name="kept")
            sc.affine[:], sc.mass[:] = st["affine"][:c], mo[:c]
            st = O.new_state(sc)
            st["pos"][:, 3], st["vel"][:, 3] = po[:c, 3], vo[:c, 3]
            step(st, 20, 0)
        st = load(_scene(4, n))   # a new load: G2P writes them again
        step(st, 3, 0)
    finally:
        gpu.mpm_destroy(h)

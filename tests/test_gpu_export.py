"""Reading single particle buffers back: each read exports only the buffer asked
for (and, in a batch right after a step, only the scene's own range of the
layout).  Every buffer of every scene against the oracle, in changing orders,
right after scenes are added and removed and after steps, long enough that both
the eagerly launched and the captured substeps are read from."""
import ctypes

import numpy as np
import pytest

import oracle as O
from mls_mpm_b200 import abi, scenes
from mls_mpm_b200.abi import BUF, check
from mls_mpm_b200.batch import Batch, default_params
from runner import GpuScene, diff_report

pytestmark = pytest.mark.gpu

BUFFERS = ("pos", "vel", "affine", "mass", "density")


def _scene(seed, n, grid):
    rng = np.random.default_rng(seed)
    pos = rng.uniform(2.2, np.array(grid) - 2.2, (n, 3)).astype(np.float32)
    sc = scenes.Scene(grid, pos, rng.uniform(-1, 1, (n, 3)).astype(np.float32), name=f"export_{seed}")
    sc.mass[:] = rng.uniform(0.5, 2.0, n).astype(np.float32)
    return sc


@pytest.mark.parametrize("steps", [1, 3, 20])   # 20: past the eagerly launched substeps of an unchanged batch
def test_batch_reads_every_scene_and_buffer(gpu, steps):
    b = Batch(20_000, 120_000, 6)
    live = {}
    W = abi.WallParams()

    def add(seed, n, grid):
        sc = _scene(seed, n, grid)
        sid = b.add_scene(sc)
        live[sid] = (O.new_state(sc), default_params(grid, n))

    def check_all(order):
        for sid, (st, _) in live.items():
            for name in order:
                bad = diff_report({name: b.read(sid, name)}, {name: st[name]})
                assert not bad, f"scene {sid}: {bad}"

    def step(k):
        b.step(k)
        for st, P in live.values():
            for _ in range(k):
                O.substep(st, P, W)

    try:
        add(1, 3001, (40, 24, 33))
        add(2, 2500, (33, 30, 20))
        add(3, 1, (16, 16, 16))
        check_all(BUFFERS)
        step(steps)
        check_all(BUFFERS[::-1])
        # a scene goes; one that takes its tiles and slot comes, and one behind the rest
        first = next(iter(live))
        b.remove(first)
        del live[first]
        check_all(("density", "pos"))
        add(4, 700, (20, 18, 17))
        add(5, 5000, (48, 20, 24))
        check_all(("vel", "affine", "mass"))
        step(steps)
        check_all(("affine", "density", "vel", "pos", "mass"))
    finally:
        b.close()


@pytest.mark.parametrize("bind", [False, True])   # without and with the render buffers kept by the substeps
def test_scene_reads_after_steps_and_raycasts(gpu, bind):
    sc = _scene(7, 4000, (36, 28, 30))
    g = GpuScene(gpu, sc)
    st = O.new_state(sc)
    P, W = default_params(sc.grid, sc.n), abi.WallParams()
    o, d = (ctypes.c_double * 3)(18.0, 60.0, 15.0), (ctypes.c_double * 3)(0.0, -1.0, 0.0)
    ray = abi.RayParams(18.0, 60.0, 15.0, 2.0, 0.0, -1.0, 0.0, 0.0)
    orders = [("affine",), ("pos", "density"), (), ("mass", "vel", "affine"), ("density", "pos", "vel", "mass", "affine")]
    try:
        if bind:
            p, sz = ctypes.c_void_p(), ctypes.c_size_t()
            check(gpu.mpm_get_buffer(g.h, BUF["vel"], ctypes.byref(p), ctypes.byref(sz)), "mpm_get_buffer")
        for k in range(25):
            g.frame(P, W, None, None)
            O.substep(st, P, W)
            if k % 2:
                hit, t, hp = ctypes.c_int(), ctypes.c_float(), (ctypes.c_double * 3)()
                check(gpu.mpm_raycast_fluid(g.h, o, d, 2.0, ctypes.byref(hit), ctypes.byref(t), hp), "raycast")
                bits = int(np.float32(t.value).view(np.uint32)) if hit.value else 0xFFFFFFFF
                assert bits == O.raycast(P, ray, st["pos"]), k
            names = orders[k % len(orders)]
            bad = diff_report({n: g.read(n) for n in names}, {n: st[n] for n in names})
            assert not bad, f"substep {k}: {bad}"
    finally:
        g.close()

"""Particles and foam far outside the grid, where the cell of a coordinate
saturates at the ends of the 32-bit range: no index test may take such a stencil
for one inside.  Every array bit-exact against the oracle."""
import numpy as np
import pytest

import oracle as O
import scenarios
from mls_mpm_b200 import abi, scenes
from mls_mpm_b200.abi import BUF, check
from runner import GpuScene, diff_report

pytestmark = pytest.mark.gpu

# the first saturated coordinate, the last exact one, beyond, and as far below
INT_MAX = (1 << 31) - 1
FAR = np.array([2147483648.0, 2147483520.0, 3e9, -2147483648.0, -2147483904.0, -3e9], np.float32)


def _far_rows():
    """(axes, coordinate): each axis alone, pairs, and all three."""
    return [(ax, x) for ax in ((0,), (1,), (2,), (0, 1), (1, 2), (0, 2), (0, 1, 2)) for x in FAR]


def _records(grid, lo, hi, infinite):
    """Live foam and bubble records, one far coordinate or more each, among ordinary ones."""
    rng = np.random.default_rng(4)
    rows = _far_rows() + ([((ax,), x) for ax in range(3) for x in (np.float32(np.inf), np.float32(-np.inf))] if infinite else [])
    rec = np.zeros(2 * len(rows) + 64, abi.DIFFUSE_DTYPE)
    rec["pos"][:, :3] = rng.uniform(lo, np.array(grid) - lo, (len(rec), 3))
    rec["vel"][:, :3] = rng.uniform(-1, 1, (len(rec), 3))
    rec["ptype"] = np.arange(len(rec)) % 2 + 1            # foam, bubble
    rec["alive"], rec["lifetime"] = 1, 5.0
    for i, (axes, x) in enumerate(rows):
        for ax in axes:
            rec["pos"][2 * i:2 * i + 2, ax] = x
    return rec


def test_far_foam_is_sampled_nowhere(gpu):
    sc = scenes.small_box(grid=(24, 20, 22), n=3000, seed=8, name="far_foam")
    rec = _records(sc.grid, 2.5, 2.5, True)
    M = len(rec) + 40
    s = scenarios.Scenario("far_foam", sc, 3, diffuse_max=M)
    st = O.new_state(sc, M)
    st["diffuse"][:len(rec)] = rec
    st["free_list"][:40] = np.arange(len(rec), M)
    st["top"][0] = 40
    g = GpuScene(gpu, sc, M)
    try:
        for name, buf in (("diffuse", "diffuse"), ("free_list", "free_list"), ("top", "free_top")):
            a = np.ascontiguousarray(st[name])
            check(gpu.mpm_upload(g.h, BUF[buf], abi.ptr(a), a.nbytes), "mpm_upload")
        for k, (P, W, H, dims, gen, adv) in enumerate(s.frames()):
            g.frame(P, W, H, dims)
            O.substep(st, P, W, H, dims, gen, adv)
            bad = diff_report(g.state(), st)
            assert not bad, f"substep {k}: {bad}"
    finally:
        g.close()


def _misses_grid(cell, grid):
    """True when the reference's linear index (shaders.js:303-304), which wraps, puts no stencil cell into the grid."""
    X, Y, Z = grid
    base = ((cell[2] - 1) * Y + cell[1] - 1) * X + cell[0] - 1
    return all((base + (k * Y + j) * X + i) % (1 << 32) >= X * Y * Z for k in range(3) for j in range(3) for i in range(3))


def test_far_particles_take_the_guarded_path(gpu):
    # odd dims: few saturated cells wrap back into the grid
    sc = scenes.small_box(grid=(25, 21, 23), n=3000, seed=9, name="far_fluid")
    far = []
    for i, (axes, x) in enumerate(_far_rows()):
        pos = sc.pos[40 * i].copy()
        pos[list(axes)] = x
        cell = [int(min(max(np.floor(float(c)), -(1 << 31)), (1 << 31) - 1)) for c in pos[:3]]
        # (three saturated axes: the weights' product overflows, and infinity times a zero mass is NaN)
        if _misses_grid(cell, sc.grid) and max(map(abs, cell)) * len(axes) < 3 * (INT_MAX - 200):
            sc.pos[40 * i] = pos
            far.append(40 * i)
    assert len(far) > 20
    near = np.setdiff1d(np.arange(sc.n), far)
    # the oracle (which, as the reference, indexes unchecked) runs the other particles alone: far ones weigh nothing
    alone = scenes.Scene(sc.grid, sc.pos[near, :3].copy(), sc.vel[near, :3].copy(), name="near")
    alone.affine[:], alone.mass[:] = sc.affine[near], sc.mass[near]
    st = O.new_state(alone)
    (P, W, H, dims, gen, adv), = scenarios.Scenario("near", alone, 1).frames()
    O.substep(st, P, W, H, dims, gen, adv)
    g = GpuScene(gpu, sc)
    try:
        (P, W, H, dims, gen, adv), = scenarios.Scenario("far_fluid", sc, 1).frames()
        g.frame(P, W, H, dims)
        got = g.state()
        want = {k: st[k] for k in got}
        bad = diff_report({k: v[near] if len(v) == sc.n else v for k, v in got.items()}, want)
        assert not bad, bad
        assert not got["density"][far].any() and not got["affine"][far].any()
        hi = np.array([P.hard_max_x, P.hard_max_y, P.hard_max_z], np.float32)
        assert np.array_equal(got["pos"][far, :3], np.clip(sc.pos[far, :3], np.float32(P.hard_min), hi))
    finally:
        g.close()

"""COMPACT at the sizes where its passes change: one tile of 2,048 particles and
its neighbours, and 4,096 tiles, up to which a block adds up the counts before
its own (8,388,608 particles) and beyond which a scan runs.  Survivors, order
and count against a plain mask of the pass's own test in 32 bits, everything
kept, nothing kept and some."""
import ctypes

import pytest

from mls_mpm_b200 import abi
from mls_mpm_b200.abi import check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 256, 2047, 2048, 2049, 65_537, 8_388_608, 8_388_609])
@pytest.mark.parametrize("radius", [0.0, 9.5, 1000.0])
@pytest.mark.parametrize("fn", ["mpm_compact", "mpm_compact_noalloc"])
def test_compact_matches_mask(gpu, n, radius, fn):
    import torch
    dev = torch.device("cuda:0")
    g = torch.Generator(dev)
    g.manual_seed(n)
    pos = torch.rand((n, 4), generator=g, device=dev) * 32
    vel = torch.rand((n, 4), generator=g, device=dev) - 0.5
    mass = torch.rand((n,), generator=g, device=dev)
    d = [0.43643578, 0.87287156, 0.21821789]
    ray = abi.RayParams(16.0, 16.0, 16.0, radius, *d, 0.0)
    d = [ray.dx, ray.dy, ray.dz]
    # shaders.js:80-84 and 536-540, operation by operation
    to = [pos[:, a] - 16.0 for a in range(3)]
    t = to[0] * d[0] + to[1] * d[1] + to[2] * d[2]
    perp = [to[a] - t * d[a] for a in range(3)]
    keep = ~((perp[0] * perp[0] + perp[1] * perp[1] + perp[2] * perp[2]).sqrt() < radius)
    m = int(keep.sum())
    out = [torch.full_like(a, -7.0) for a in (pos, vel, mass)]
    count = torch.full((1,), 99, dtype=torch.int32, device=dev)
    check(getattr(gpu, fn)(ctypes.byref(ray), n, pos.data_ptr(), vel.data_ptr(), mass.data_ptr(), out[0].data_ptr(),
                           out[1].data_ptr(), out[2].data_ptr(), count.data_ptr(),
                           torch.cuda.current_stream().cuda_stream), fn)
    torch.cuda.synchronize()
    assert int(count.item()) == m
    for got, src in zip(out, (pos, vel, mass)):
        assert torch.equal(got[:m], src[keep])
        assert bool((got[m:] == -7.0).all())   # nothing past the survivors is written

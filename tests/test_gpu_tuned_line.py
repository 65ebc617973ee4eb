"""The line between worlds with and without a DECODE_MASS launch (one small chunk
for each of four blocks an SM) does not depend on the launch shape: every shape
the autotuner tries, and the one it keeps, launches the same kernels."""
import pytest

from mls_mpm_b200 import abi, scenes
from mls_mpm_b200.batch import Batch

pytestmark = pytest.mark.gpu


def _sms():
    from cuda.bindings import runtime
    err, v = runtime.cudaDeviceGetAttribute(runtime.cudaDeviceAttr.cudaDevAttrMultiProcessorCount, 0)
    assert err == runtime.cudaError_t.cudaSuccess, err
    return v


@pytest.mark.parametrize("beyond", [1, 50_000])
def test_launches_do_not_depend_on_the_shape(gpu, beyond):
    n = 4 * _sms() * 256 + beyond
    b = Batch(n, 2 * 80 ** 3, 2, flags=abi.BATCH_AUTOTUNE)
    try:
        for i, m in enumerate((n // 2, n - n // 2)):
            b.add_scene(scenes.small_box(grid=(80, 80, 80), n=m, seed=i, name="tuned"))
        counts, shapes = [], set()
        b.step(1)                       # the first substep counts every particle
        for _ in range(40):
            before = b.info().launches
            b.step(1)
            counts.append(b.info().launches - before)
            shapes.add(b.info().item_blocks)
        assert len(shapes) >= 4         # the trials' shapes
        assert set(counts) == {7}, counts
    finally:
        b.close()

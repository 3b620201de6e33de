"""Short calls of engines of many systems go kernel by kernel (a cluster that
rebuilds its lists would keep each such call waiting), longer ones inside
clusters: the same bits whatever the calls' lengths, events on either side of the
line included."""
import numpy as np
import pytest

from test_gpu_cluster_run import _engine, _same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes,min_steps", [
    ([1000] * 7, 1), ([4000], 1), ([2000] * 8, 1), ([4000] * 8, 2), ([1000] * 33, 1), ([2000] * 16, 2), ([500] * 34, 1),
    ([1000] * 34, 2), ([2000] * 34, 3), ([4000] * 34, 4), ([500] * 75, 2), ([1000] * 75, 3), ([4000] * 75, 7)])
@pytest.mark.parametrize("precision", [0, 1])
def test_line(cuda_lib, sizes, min_steps, precision):
    from activechi4_b200 import Engine, default_params
    e = Engine([default_params(n, precision=precision, list_mode=1, rebuild_factor=4.0) for n in sizes])
    assert e.run_plan()["min_steps"] == min_steps
    e.close()


@pytest.mark.parametrize("prepare", [False, True])
@pytest.mark.parametrize("sizes", [[700] * 34, [600] * 74 + [1900]])
def test_bits_do_not_depend_on_the_calls(cuda_lib, sizes, prepare):
    a, b, c = (_engine(sizes, 1) for _ in range(3))
    k = a.run_plan()["min_steps"]
    assert k > 1
    for e in (a, b, c):
        for r in (0, len(sizes) - 1):
            e.start_ramp(r, 0.3, 0.304, 0.1)
            e.obs_configure(r, 200, 8, 1.4, 0, 0.3, np.array([[1, 0, 0], [2, 1, 0]]), 4)
    if prepare:
        a.prepare()
    for m in (k - 1, k, 1, 2 * k, 30 - 4 * k):  # the calls of one step shuffle and remove drift too
        a.step(m)
    a.bench_steps(k - 1, 0)
    a.bench_steps(k, 0)
    n = a.thermo(1)["step"]
    for _ in range(n):
        b.step(1)
    c.step(n)
    for e in (b, c):
        _same(a, e)
        for r in (0, len(sizes) - 1):
            assert np.array_equal(a.obs_sums(r)[1], e.obs_sums(r)[1])

"""Which engines step inside clusters, and how: the plan behind the equality tests
of test_gpu_cluster_run.py (an engine that fell back to kernel by kernel would pass
those whatever the cluster kernel does)."""
import pytest

pytestmark = pytest.mark.gpu


def _plan(sizes, precision=0, **kw):
    from activechi4_b200 import Engine, default_params
    e = Engine([default_params(n, precision=precision, list_mode=1, rebuild_factor=4.0, **kw) for n in sizes])
    p = e.run_plan()
    e.close()
    return p


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("count,cluster", [(1, 16), (7, 16), (8, 8), (15, 8), (16, 4), (33, 4), (34, 2), (74, 2),
                                           (75, 1), (300, 1)])
def test_cluster_by_count(cuda_lib, count, cluster, precision):
    p = _plan([600] * count, precision)
    assert (p["cluster"], p["threads"], p["resident"]) == (cluster, 512, 1)


@pytest.mark.parametrize("n", [460, 513, 870, 1000, 2961, 4031])
@pytest.mark.parametrize("precision", [0, 1])
def test_one_system(cuda_lib, n, precision):
    p = _plan([n], precision)
    assert (p["cluster"], p["threads"], p["resident"]) == (16, 512, 1)


@pytest.mark.parametrize("precision,threads", [(0, 512), (1, 1024)])
@pytest.mark.parametrize("count,cluster", [(34, 2), (75, 1)])
def test_state_in_memory(cuda_lib, count, cluster, precision, threads):
    p = _plan([700] * (count - 1) + [3500], precision)
    assert (p["cluster"], p["threads"], p["resident"]) == (cluster, threads, 0)


@pytest.mark.parametrize("sizes,kw", [
    ([300], {}), ([4505], {}), ([1000, 6000], {}), ([1000, 300], {}), ([1000], dict(thermostat=3)),
    ([1000], dict(thermostat=5)), ([1000], dict(shuffle=2))])
def test_kernel_by_kernel(cuda_lib, sizes, kw):
    assert _plan(sizes, **kw) == dict(cluster=0, threads=0, resident=0, min_steps=0, max_steps=0)
    assert _plan([1000], thermostat=2)["cluster"] == 16

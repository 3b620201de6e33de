"""Launches of clusters that occupy the whole chip are bounded in time, so other
streams' work is not held off for the length of a call; the bits do not depend on
where a call is cut."""
import numpy as np
import pytest

from test_gpu_cluster_run import _engine, _same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes,precision,full", [
    ([4000], 1, False), ([4000] * 7, 0, False), ([1000] * 33, 1, False), ([2000] * 75, 1, False),
    ([3000] * 74, 0, True), ([4000] * 140, 1, True), ([500, 1500, 2500, 3500] * 64, 1, True), ([1000] * 600, 0, True)])
def test_bound(cuda_lib, sizes, precision, full):
    e = _engine(sizes, precision)
    k = e.run_plan()["max_steps"]
    if not full:
        assert k == 2048
        return
    e.step(300)  # off the lattice
    k = min(k, 256)  # (acg_bench_steps times up to 256 steps in one launch)
    ms = min(e.bench_steps(k, 0)[0] for _ in range(3))
    # a launch of k steps (cut where a drift removal is due); the bound is an estimate: within a factor of two
    assert k >= 40 and (ms < 40.0 or k == 40)


@pytest.mark.parametrize("precision", [0, 1])
def test_cut_calls(cuda_lib, precision):
    sizes = [460 + (37 * r) % 900 for r in range(150)]
    a, b = (_engine(sizes, precision) for _ in range(2))
    k = a.run_plan()["max_steps"]
    assert 40 <= k < 700
    a.step(2 * k + 1)  # three launches
    b.step(k + 1)
    b.step(k)
    _same(a, b)
    if precision == 0:
        c = _engine(sizes, precision)
        c.step_eager(2 * k + 1)
        _same(a, c)
    assert a.thermo(3)["step"] == 2 * k + 1 and np.isfinite(a.thermo(3)["pe"])

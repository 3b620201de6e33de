"""Engines of many systems whose mean momentum is removed every few steps: each
piece between two removals is a launch of its own, so such calls step kernel by
kernel however long they are; the bits are those of single steps."""
import numpy as np
import pytest

from test_gpu_cluster_run import _engine, _same

pytestmark = pytest.mark.gpu


def _with_cadence(sizes, every):
    from activechi4_b200 import Engine, default_params, lattice_state
    e = Engine([default_params(n, T=0.6, f0=1.0, tau_p_steps=7, precision=1, seed=40 + r, list_mode=1,
                               rebuild_factor=4.0, drift_every=every) for r, n in enumerate(sizes)])
    for r, n in enumerate(sizes):
        e.set_state(r, lattice_state(n, 0.6, seed=3 + r))
        e.set_nhc(r, np.zeros(3), np.array([0.2, -0.1, 0.05]))
    return e


@pytest.mark.parametrize("every,inside", [(1, False), (2, False), (3, False), (12, True), (50, True)])
def test_route_and_bits(cuda_lib, every, inside):
    sizes = [700] * 33 + [1800]  # clusters from three steps on
    a, b = (_with_cadence(sizes, every) for _ in range(2))
    k = a.run_plan()["min_steps"]
    assert 2 < k < 12
    a.step(60)
    for _ in range(60):
        b.step(1)
    _same(a, b)
    # launches of 60 steps inside clusters: a run per piece and two kernels a removal
    launches = a.bench_steps(60, 0)[1]
    assert (launches < 60) == inside
    b.step(60)
    _same(a, b)


@pytest.mark.parametrize("count", [1, 8])
def test_single_cadence(cuda_lib, count):
    """(clusters whatever the call: few particles a block)"""
    a, b = (_engine([900] * count, 0) for _ in range(2))
    assert a.run_plan()["min_steps"] == 1
    a.step(110)
    b.step_eager(110)
    _same(a, b)

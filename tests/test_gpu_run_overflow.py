"""List overflow inside a cluster: rows that hold the box's mean neighbour count but
not that of a droplet in it (rows below the mean send an engine kernel by kernel)."""
import dataclasses

import numpy as np
import pytest

from test_gpu_cluster_run import _same

pytestmark = pytest.mark.gpu


def _droplets(count, precision):
    from activechi4_b200 import Engine, default_params, lattice_state
    e = Engine([default_params(900, density=0.8, T=0.6, f0=1.0, tau_p_steps=7, precision=precision, seed=40 + r,
                               list_mode=1, rebuild_factor=4.0, nb_capacity=96) for r in range(count)])
    for r in range(count):
        st = lattice_state(900, 0.6, seed=3 + r)  # density 1.2
        L = (900 / 0.8) ** 0.33333333
        x = st.x * st.L / L
        e.set_state(r, dataclasses.replace(st, L=L, x=x, xu=x.copy()))
        e.set_nhc(r, np.zeros(3), np.array([0.2, -0.1, 0.05]))
    return e


@pytest.mark.parametrize("count,cluster", [(1, 16), (34, 2), (75, 1)])
@pytest.mark.parametrize("precision", [0, 1])
def test_droplets(cuda_lib, count, cluster, precision):
    a, b = (_droplets(count, precision) for _ in range(2))
    assert a.run_plan()["cluster"] == cluster
    some = 0
    for k in (4, 8, 20):
        a.step(k)
        b.step_eager(k)
        some += a.thermo(0)["overflow"]
        _same(a, b)
    assert some > 0


def test_rows_below_the_mean(cuda_lib):
    from activechi4_b200 import Engine, default_params
    for cap, run in ((64, False), (96, False), (128, True), (0, True)):
        e = Engine(default_params(1000, nb_capacity=cap))
        assert (e.run_plan()["cluster"] > 0) == run
        e.close()

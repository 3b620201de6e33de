"""Whole-box lists of the kernel-by-kernel step, one particle a warp (engines of up
to 16384 such particles) and by bricks (more): the same lists, so the same bits for
a system in engines on either side of the line."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [460, 870, 1000, 3000, 4031])
@pytest.mark.parametrize("precision", [0, 1])
def test_either_side(cuda_lib, n, precision):
    from activechi4_b200 import Engine, default_params, lattice_state
    sizes = [n, 4000, 4000, 4000, 16384 - 12000 - n], [n, 4000, 4000, 4000, 16385 - 12000 - n]
    sizes = [[s for s in z if s >= 300] for z in sizes]
    if sizes[0] == sizes[1]:
        sizes[1] = sizes[1] + [1000]
    out = []
    for z in [[n]] + sizes:
        e = Engine([default_params(s, T=0.6, thermostat=3, precision=precision, seed=7 + r, list_mode=1, rebuild_factor=4.0)
                    for r, s in enumerate(z)])
        assert e.run_plan()["cluster"] == 0
        for r, s in enumerate(z):
            e.set_state(r, lattice_state(s, 0.6, seed=2 + r))
        e.step(40)
        out.append(e.get_state(0))
        assert e.thermo(0)["rebuilds"] > 2
    for o in out[1:]:
        for u, w in zip(out[0], o):
            assert np.array_equal(u, w)

"""acg_compute_forces and acg_rebuild leave the systems without a state alone (all
their particles lie at the origin: listing and summing them costs a system's
square and gives no number), and evaluate the others as an engine of their own."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(700, 900), (300, 700), (1000, 9000), (700, 21000)])
def test_forces_of_the_loaded(cuda_lib, sizes):
    from activechi4_b200 import Engine, default_params, lattice_state
    ps = [default_params(n, T=0.6, f0=1.0, seed=9 + r) for r, n in enumerate(sizes)]
    st = lattice_state(sizes[0], 0.6, seed=5)
    e, a = Engine(ps), Engine([ps[0]])
    for x in (e, a):
        x.set_state(0, st)
        x.compute_forces()
        x.rebuild()
        x.compute_forces()
    assert np.array_equal(a.get_state(0)[3], e.get_state(0)[3])
    t = e.thermo(1)
    assert (t["rebuilds"], t["overflow"], t["pe"], t["virial"]) == (0, 0, 0.0, 0.0)
    assert not e.get_state(1)[3].any()
    _, counts, members = e.cells(1)
    assert not counts.any() and np.array_equal(members, np.arange(sizes[1]))

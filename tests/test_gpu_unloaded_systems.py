"""Systems of an engine that hold no state yet are left alone when others are
primed: the loaded systems' results are those of an engine of their own, and a
system loaded after the others have stepped starts as if it were alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(700, 900), (1000, 9000)])
def test_loaded_later(cuda_lib, sizes):
    from activechi4_b200 import Engine, default_params, lattice_state
    ps = [default_params(n, T=0.6, seed=9 + r) for r, n in enumerate(sizes)]
    st = [lattice_state(n, 0.6, seed=r) for r, n in enumerate(sizes)]
    e = Engine(ps)
    e.set_state(0, st[0])
    a = Engine([ps[0]])
    a.set_state(0, st[0])
    for x in (e, a):
        x.set_nhc(0, np.zeros(3), np.array([0.1, 0.05, -0.1]))
        x.step(20)
    for u, w in zip(a.get_state(0), e.get_state(0)):
        assert np.array_equal(u, w)
    e.set_state(1, st[1])
    b = Engine([ps[1]])
    b.set_state(0, st[1])
    b.compute_forces()
    e.compute_forces()
    assert np.array_equal(b.get_state(0)[3], e.get_state(1)[3])
    assert e.thermo(1)["pe"] == b.thermo(0)["pe"] and np.isfinite(e.thermo(1)["pe"])

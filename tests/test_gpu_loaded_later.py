"""A system loaded after the others have stepped starts with the chain and box it
was created with (the thermostat does not run on a system that holds no state):
its trajectory is that of an engine of its own, bit for bit, without set_nhc.
Its step counter has gone on with the engine's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(700, 900), (1000, 10200)])
@pytest.mark.parametrize("thermostat", [1, 2, 3, 4, 5])
def test_starts_as_alone(cuda_lib, sizes, thermostat):
    from activechi4_b200 import Engine, default_params, lattice_state
    ps = [default_params(n, T=0.6, f0=1.0, P=5.0, shuffle=0, drift_every=0, thermostat=thermostat, seed=9 + r)
          for r, n in enumerate(sizes)]
    st = [lattice_state(n, 0.6, seed=r) for r, n in enumerate(sizes)]
    e = Engine(ps)
    e.set_state(0, st[0])
    e.step(25)
    e.set_state(1, st[1])
    a = Engine([ps[1]])
    a.set_state(0, st[1])
    for x in (e, a):
        x.step(20)
    for u, w in zip(a.get_state(0), e.get_state(1)):
        assert np.isfinite(u).all() and np.array_equal(u, w)
    ta, te = a.thermo(0), e.thermo(1)
    for f in ("pe", "ke", "virial", "L"):
        assert ta[f] == te[f], f
    assert np.array_equal(ta["p_eta"], te["p_eta"]) and np.array_equal(ta["eta"], te["eta"])
    assert (ta["step"], te["step"]) == (20, 45)


def test_drift_removal_leaves_unloaded_alone(cuda_lib):
    from activechi4_b200 import Engine, default_params, lattice_state
    ps = [default_params(700 + 200 * r, T=0.6, P=5.0, thermostat=5, shuffle=0, drift_every=4) for r in range(2)]
    e = Engine(ps)
    e.set_state(0, lattice_state(700, 0.6, seed=0))
    L = e.thermo(1)["L"]
    e.step(10)
    t = e.thermo(1)
    assert t["L"] == L and not t["p_eta"].any() and t["step"] == 10

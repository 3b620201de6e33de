"""Directions set before a system's state: the system steps along with the
loaded ones without moving, however long, and every system's result is that of an
engine of its own, bit for bit.

An unloaded system's slots once held particle 0 each, active along the first
direction, so directions set first made it drift past its skin and sort a
particle list that was no permutation."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(700, 900), (900, 600, 500), (1000, 9000), (700, 21000)])
def test_directions_before_state(cuda_lib, sizes):
    from activechi4_b200 import Engine, default_params, lattice_state
    ps = [default_params(n, T=0.6, f0=2.0, shuffle=0, drift_every=0, seed=9 + r) for r, n in enumerate(sizes)]
    st = [lattice_state(n, 0.6, seed=r) for r, n in enumerate(sizes)]
    chain = np.zeros(3), np.array([0.1, 0.05, -0.1])
    alone = []
    for p, s in zip(ps, st):
        a = Engine([p])
        a.set_state(0, s)
        a.set_nhc(0, *chain)
        alone.append(a)
    e = Engine(ps)
    for r, s in enumerate(st):
        e.set_directions(r, np.ones_like(s.k))
    e.set_state(0, st[0])
    e.set_nhc(0, *chain)
    for x in (e, alone[0]):
        x.step(300)  # with f0 k on every particle, 100 steps pass the skin
    for r in range(1, len(sizes)):
        for a in e.get_state(r)[:3]:
            assert not a.any()
    for r in range(1, len(sizes)):
        e.set_state(r, st[r])
        e.set_nhc(r, *chain)
    e.step(40)
    for r, a in enumerate(alone):
        a.step(40)
        for u, w in zip(a.get_state(0), e.get_state(r)):
            assert np.array_equal(u, w)
        assert a.thermo(0)["pe"] == e.thermo(r)["pe"]

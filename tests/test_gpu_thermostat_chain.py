"""The thermostat chain's link factors on both sides of the series' range.

A link moves x = dt/4 p_eta/q: up to |x| = 1/16 the factors come from a Taylor
series (truncation below 1e-19), beyond from exp().  The chain momenta here put
the links well inside, at both sides of and well beyond the edge; the states
after five steps are compared with the oracle's, whose links all use exp().
Tolerance: the oracle's (1 - exp(-x)) / x carries a rounding of 1e-16 / x,
about 1e-13 at the smallest x of a chain in use, on terms of order one; five
steps of two halves leave it below 1e-11 of the momenta."""
import numpy as np
import pytest

from conftest import golden_state

pytestmark = pytest.mark.gpu

T = 0.45
EDGE = 0.0625 * (T * 0.04) / (0.25 * 0.005)  # chain momentum of a link at |x| = 1/16


@pytest.mark.parametrize("p1,p2", [(0.1, -0.1), (0.999 * EDGE, -0.999 * EDGE), (1.001 * EDGE, -1.001 * EDGE),
                                   (-1.001 * EDGE, 0.1), (3.0, -2.5)])
def test_chain_links(cuda_lib, g1000, p1, p2):
    from activechi4_b200 import Engine, default_params
    from oracle import Oracle
    st = golden_state(g1000)
    p_eta = np.array([1.0, p1, p2])
    e = Engine(default_params(st.n, T=T, f0=1.0, shuffle=0, drift_every=0))
    e.set_state(0, st)
    e.set_nhc(0, np.zeros(3), p_eta)
    e.step(5)
    o = Oracle.from_state(st, T, 1.0, p_eta=p_eta)
    o.run(5, shuffle=False, drift=False)
    _, _, p, _ = e.get_state(0)
    _, _, po, _ = o.get_state()
    assert np.abs(p - po).max() <= 1e-11 * np.sqrt((po ** 2).mean())
    e.close()

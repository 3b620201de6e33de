"""The direction shuffle applied in windows of swaps against the sequential
swaps (MDcode/active.c:58-75 on numpy's MT19937), bit for bit, at the edges of a
window (640 swaps, 624 draws of the stream) and with every place active."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sequential(k, seed):
    n = k.shape[1]
    words = np.random.RandomState(seed).randint(0, 1 << 32, size=3 * n, dtype=np.uint32)
    k = k.copy()
    for c in range(3):
        for i in range(n):
            j = int(n * (int(words[c * n + i]) / 4294967296.0))
            k[c, i], k[c, j] = k[c, j], k[c, i]
    return k


@pytest.mark.parametrize("n,nact", [(1000, 1), (1000, 2), (1000, 207), (1000, 208), (1000, 209), (1000, 1000),
                                    (2000, 623), (2000, 625), (6000, 640), (6000, 1281), (40000, 25600),
                                    (40000, 32768), (40000, 32769)])
def test_windows(cuda_lib, n, nact):
    from activechi4_b200 import Engine, default_params, lattice_state
    st = lattice_state(n, 0.5, seed=2, nact=nact)
    e = Engine(default_params(n, nact=nact, seed=4242))
    e.set_state(0, st)
    assert np.array_equal(e.get_directions(), st.k)
    e.shuffle()
    k = _sequential(np.asarray(st.k), 4242)
    assert np.array_equal(e.get_directions(), k)
    if n <= 4000:  # the same inside a step's cluster run (step 0 shuffles)
        b = Engine(default_params(n, nact=nact, seed=4242))
        b.set_state(0, st)
        b.set_nhc(0, np.zeros(3), np.array([0.1, 0.05, -0.1]))
        b.step(1)
        assert np.array_equal(b.get_directions(), k)

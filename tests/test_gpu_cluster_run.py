"""Whole runs inside a thread-block cluster (acg_step on whole-box systems)
against the same steps kernel by kernel (acg_step_eager): the same bits.

Both sum in an order that depends on the system's slots alone, so no tolerance
is needed.  Sizes: the smallest with list sub-cells, one past a multiple of 32
slots, the cell-count edges of the whole-box range; the engines' cluster sizes
16, 8, 4, 2 and 1 (by the number of systems); state in shared memory and in
global memory; lists that overflow; ramps, observables, direction shuffles."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _engine(sizes, precision, tpp=2, thermostat=1, **kw):
    from activechi4_b200 import Engine, default_params, lattice_state
    ps = [default_params(n, T=0.6, f0=1.0, tau_p_steps=7, precision=precision, seed=40 + r, list_mode=1,
                         rebuild_factor=4.0, thermostat=thermostat, drift_every=50, **kw) for r, n in enumerate(sizes)]
    e = Engine(ps)
    e.set_group_tpp(tpp)
    for r, n in enumerate(sizes):
        e.set_state(r, lattice_state(n, 0.6, seed=3 + r))
        e.set_nhc(r, np.zeros(3), np.array([0.2, -0.1, 0.05]))
    return e


def _same(a, b):
    for r in range(a.nsys):
        for u, w in zip(a.get_state(r), b.get_state(r)):
            assert np.array_equal(u, w)
        assert np.array_equal(a.get_directions(r), b.get_directions(r))
        ta, tb = a.thermo(r), b.thermo(r)
        for f in ("pe", "ke", "virial", "vir_act", "maxD", "step", "rebuilds", "overflow"):
            assert ta[f] == tb[f], f
        assert np.array_equal(ta["p_eta"], tb["p_eta"])


@pytest.mark.parametrize("n", [460, 513, 870, 1000, 2961, 4031])
@pytest.mark.parametrize("precision,tpp", [(0, 1), (0, 2), (1, 2), (1, 4)])
def test_run_equals_eager(cuda_lib, n, precision, tpp):
    a, b = (_engine([n], precision, tpp) for _ in range(2))
    for k in (1, 2, 60):
        a.step(k)
        b.step_eager(k)
        _same(a, b)


@pytest.mark.parametrize("count", [7, 8, 16, 34, 75])
@pytest.mark.parametrize("precision", [0, 1])
def test_cluster_sizes(cuda_lib, count, precision):
    rng = np.random.default_rng(count)
    sizes = [int(s) for s in rng.integers(460, 1300, count - 1)] + [3500]
    a, b = (_engine(sizes, precision) for _ in range(2))
    a.step(45)
    b.step_eager(45)
    _same(a, b)


@pytest.mark.parametrize("thermostat", [0, 2])
def test_other_integrators(cuda_lib, thermostat):
    a, b = (_engine([1200], 0, thermostat=thermostat) for _ in range(2))
    a.step(50)
    b.step_eager(50)
    _same(a, b)


@pytest.mark.parametrize("count", [1, 75])
def test_overflowing_lists(cuda_lib, count):
    """Rows of 64 entries: most particles are served by the all-pairs scan."""
    a, b = (_engine([900] * count, 1, nb_capacity=64) for _ in range(2))
    a.step(20)
    b.step_eager(20)
    assert a.thermo(0)["overflow"] > 0
    _same(a, b)


@pytest.mark.parametrize("count", [1, 8])
def test_ramp_and_observables(cuda_lib, count):
    a, b = (_engine([1000 + 33 * r for r in range(count)], 0) for _ in range(2))
    for e in (a, b):
        for r in range(count):
            e.start_ramp(r, 0.3, 0.304, 0.1)
            e.obs_configure(r, 200, 8, 1.4, 0, 0.3, np.array([[1, 0, 0], [2, 1, 0]]), 4)
    a.step(60)
    b.step_eager(60)
    _same(a, b)
    for r in range(count):
        assert np.array_equal(a.obs_sums(r)[1], b.obs_sums(r)[1])

"""The allocation-free forces where their split of the work changes: pieces of a
neighbourhood above the staged capacity with the cell itself in the first, a
later or two pieces, cells shared by several blocks, grids of few particles a
cell (by particles from 14 cells per side on, fewer than four a cell), the most
cells (32 per side, where the FP32 test's margin is tightest, with pairs on both
sides of each cut and across the faces), droplets in an empty box; coordinates
outside [0, 1); particles whose position is no number.  Forces, energy, virial
and active virial against a plain FP64 sum in torch; tolerance: the entry point's
documented 1e-12 of the rms force (the scalars: of the sum of the magnitudes of
the terms that a pair's energy and virial are made of; at the cut these cancel)."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

IS2, E4 = (1.0, 1.5625, 1.0 / 0.88 ** 2), (4.0, 6.0, 2.0)


def _plain(x, typ, L):
    """F, pe, virial and the sums of the terms' magnitudes, by rows of all pairs."""
    import torch
    n, dev = x.shape[0], x.device
    is2 = torch.tensor(IS2, dtype=torch.float64, device=dev)
    e4 = torch.tensor(E4, dtype=torch.float64, device=dev)
    F, pe, vir, mag = torch.zeros_like(x), 0.0, 0.0, [0.0, 0.0]
    for r in torch.arange(n, device=dev).split(max(1, 20_000_000 // n)):
        d = x[r][:, None, :] - x[None]
        d -= d.round()
        tp = typ[r][:, None] + typ[None]
        dr2 = (d * d).sum(-1) * L * L
        ok = (dr2 * is2[tp] < 6.25) & (r[:, None] != torch.arange(n, device=dev)[None])
        i, j = ok.nonzero(as_tuple=True)
        t, dr2, d = tp[i, j], dr2[i, j], d[i, j]
        rs2 = dr2 * is2[t]
        s2 = 1.0 / rs2
        s6 = s2 ** 3
        g = 2 * e4[t] * is2[t] * (6 * s6 * (s6 - 0.5) * s2 + 0.001949973872640)
        F.index_add_(0, r[i], g[:, None] * d * L)
        u = e4[t] * (s6 * (s6 - 1) + 0.0162665594880 - 0.001949973872640 * rs2)
        pe, vir = pe + 0.5 * float(u.sum()), vir + float((g * dr2).sum()) / 6
        mag[0] += 0.5 * float((e4[t] * (s6 * s6 + s6 + 0.0162665594880 + 0.001949973872640 * rs2)).sum())
        mag[1] += float((2 * e4[t] * rs2 * ((6 * s6 + 3) * s6 * s2 + 0.001949973872640)).sum()) / 6
    return F, pe, vir, mag


def _call(lib, x, typ, act, k, L, f0):
    import torch
    n, dev = x.shape[0], x.device
    F = torch.full((n, 3), float("nan"), dtype=torch.float64, device=dev)
    out = torch.full((3,), float("nan"), dtype=torch.float64, device=dev)
    p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    rc = lib.acg_forces_noalloc(p(x), None, p(typ), p(act), p(k), n, k.shape[1], L, f0, p(F), p(out),
                                C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0, lib.acg_last_error().decode()
    return F, out


def _check(lib, x, typ, L, seed, skip=None):
    """`skip`: particles that take part in nothing (position no number)."""
    import torch
    dev = torch.device("cuda:0")
    rng = np.random.default_rng(seed)
    n, nact = len(x), max(1, len(x) // 7)
    act = np.full(n, -1, dtype=np.int32)
    act[rng.permutation(n)[:nact]] = np.arange(nact)
    k = rng.integers(-1, 2, (3, nact)).astype(np.int32)
    up = lambda a, t: torch.tensor(np.ascontiguousarray(a), dtype=t, device=dev)  # noqa: E731
    X, T, A, K = up(x, torch.float64), up(typ, torch.int32), up(act, torch.int32), up(k, torch.int32)
    F, out = _call(lib, X, T, A, K, L, 1.5)
    if skip is not None:
        act[skip] = -1
        X = X.clone()
        X[up(skip, torch.int64)] = float("nan")
    want, pe, vir, mag = _plain(X, T.long(), L)
    a = torch.where(up(act, torch.int64)[:, None] >= 0, 1.5 * K.double().T[up(np.maximum(act, 0), torch.int64)], 0.0)
    keep = torch.ones(n, dtype=torch.bool, device=dev)
    if skip is not None:
        keep[up(skip, torch.int64)] = False
    rms = float((want + a)[keep].square().sum(1).mean().sqrt())
    assert float((F - want - a)[keep].abs().max()) <= 1e-12 * rms
    assert abs(float(out[0]) - pe) <= 1e-12 * mag[0] and abs(float(out[1]) - vir) <= 1e-12 * mag[1]
    if skip is None:
        va = (a * X).sum(1)
        assert abs(float(out[2]) - float(va.sum())) <= 1e-12 * float((a * X).abs().sum())


def _grid(n, L, rng, jitter=0.05):
    m = int(np.ceil(n ** (1.0 / 3.0)))
    g = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)[rng.permutation(m ** 3)[:n]]
    return (g + 0.5 + rng.uniform(-jitter, jitter, g.shape)) / m


@pytest.mark.parametrize("n,density", [
    (1280, 1.2), (1281, 1.2), (1500, 1.2), (2561, 2.2), (3000, 6.0), (3041, 1.2), (6500, 1.2),  # pieces
    (277, 1.2), (700, 1.2), (1000, 1.2), (4100, 1.2), (9000, 1.2), (15000, 2.5),                  # shared cells
    (10975, 0.175), (10976, 0.175), (10977, 0.175), (8788, 0.175), (3000, 0.03), (64, 0.004)])    # few a cell
def test_split(cuda_lib, n, density):
    rng = np.random.default_rng(n)
    L = (n / density) ** (1.0 / 3.0)
    _check(cuda_lib, _grid(n, L, rng), (rng.random(n) < 0.2).astype(np.int32), L, n)


def _pairs_at_cuts(L, rng):
    """Pairs of each type a relative 1e-9 to 3e-4 of the cut squared inside and
    outside it, in the box's middle and across its faces and corners."""
    x, typ = [], []
    spots = [np.array(s) / 8.0 for s in np.ndindex(8, 8, 8)]
    rng.shuffle(spots)
    at = iter(spots)
    for t in ((0, 0), (0, 1), (1, 1)):
        for off in (1e-9, 1e-6, 1e-5, 5e-5, 1.5e-4, 3e-4):
            for s in (-1, 1):
                for _ in range(4):
                    r = np.sqrt(6.25 * (1 + s * off) / IS2[sum(t)]) / L
                    u = rng.standard_normal(3)
                    a = next(at) + rng.uniform(-0.4, 0.4, 3) * r
                    x += [a % 1.0, (a + r * u / np.linalg.norm(u)) % 1.0]
                    typ += list(t)
    return np.array(x), np.array(typ, dtype=np.int32)


@pytest.mark.parametrize("fill", [0, 140000])
def test_most_cells(cuda_lib, fill):
    """32 cells per side; without and with other particles (by particles, by cells)."""
    rng = np.random.default_rng(fill)
    L = 93.9
    x, typ = _pairs_at_cuts(L, rng)
    if fill:
        # the others on a grid, none within two of a pair's particles
        g = _grid(fill, L, rng)
        cells = {tuple(c) for p in x for c in
                 ((np.floor(p * 30).astype(int) + o) % 30 for o in np.ndindex(3, 3, 3))}
        cells = {tuple((np.array(c) - 1) % 30) for c in cells}
        keep = np.array([tuple(c) not in cells for c in np.floor(g * 30).astype(int)])
        x, typ = np.concatenate([x, g[keep]]), np.concatenate([typ, (rng.random(keep.sum()) < 0.2).astype(np.int32)])
    _check(cuda_lib, x, typ, L, 7)


def test_droplet(cuda_lib):
    """All particles of an otherwise empty large box in one corner, across its faces."""
    rng = np.random.default_rng(3)
    L, n = 60.0, 2500
    l = (n / 1.3) ** (1.0 / 3.0)
    x = (_grid(n, l, rng) - 0.5) * l / L
    _check(cuda_lib, x % 1.0, (rng.random(n) < 0.2).astype(np.int32), L, 5)


@pytest.mark.parametrize("n", [700, 1000, 1500])
@pytest.mark.parametrize("most", [1, 5, 100000])
def test_unfolded(cuda_lib, n, most):
    """Up to three cells per side every cell neighbours every other, so the sums
    never depended on the coordinates being folded into the box."""
    rng = np.random.default_rng(n + most)
    L = (n / 1.2) ** (1.0 / 3.0)
    # whole boxes away: the folded coordinates are exact multiples of 2^-32
    x = np.floor(_grid(n, L, rng) * 2.0 ** 32) / 2.0 ** 32
    some = rng.random(n) < 0.3
    x[some] += rng.integers(-most, most + 1, (some.sum(), 3))
    _check(cuda_lib, x, (rng.random(n) < 0.2).astype(np.int32), L, 11)


@pytest.mark.parametrize("n,density", [(700, 1.2), (1500, 1.2), (1500, 6.0), (3500, 1.2), (8000, 0.02)])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_no_number(cuda_lib, n, density, bad):
    """A particle whose position is no number takes part in no pair."""
    rng = np.random.default_rng(n)
    L = (n / density) ** (1.0 / 3.0)
    x = _grid(n, L, rng)
    skip = rng.permutation(n)[:3]
    x[skip, rng.integers(0, 3, 3)] = bad
    _check(cuda_lib, x, (rng.random(n) < 0.2).astype(np.int32), L, 13, skip)

"""The allocation-free forces at the edges of their staging: two cells per side
(8 neighbour cells), three, neighbourhoods above the staged capacity (a dense
box, evaluated from memory), an empty cell, and the most cells; against a plain
FP64 all-pairs or cell sum in torch.  Tolerance: the entry point's documented
1e-12 of the rms force."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _plain(x, typ, L, rows):
    import torch
    is2 = torch.tensor([1.0, 1.5625, 1.0 / 0.88 ** 2], dtype=torch.float64, device=x.device)
    e4 = torch.tensor([4.0, 6.0, 2.0], dtype=torch.float64, device=x.device)
    out, pe = [], 0.0
    for r in rows:
        d = x[r][:, None, :] - x[None]
        d -= d.round()
        tp = typ[r][:, None] + typ[None]
        rs2 = (d * d).sum(-1) * L * L * is2[tp]
        ok = (rs2 < 6.25) & (r[:, None] != torch.arange(x.shape[0], device=x.device)[None])
        s2 = 1.0 / torch.where(ok, rs2, torch.ones_like(rs2))
        s6 = s2 ** 3
        g = torch.where(ok, 2 * e4[tp] * is2[tp] * (6 * s6 * (s6 - 0.5) * s2 + 0.001949973872640), 0 * s6)
        out.append((g[..., None] * d).sum(1) * L)
        pe += float(torch.where(ok, e4[tp] * (s6 * (s6 - 1) + 0.0162665594880 - 0.001949973872640 * rs2), 0 * s6).sum())
    return torch.cat(out), 0.5 * pe


@pytest.mark.parametrize("n,density", [(300, 1.2), (870, 1.2), (900, 1.2), (1500, 6.0), (3000, 2.5), (700, 0.05),
                                       (4000, 1.2), (20000, 0.03)])
def test_edges(cuda_lib, n, density):
    import torch
    dev = torch.device("cuda:0")
    L = (n / density) ** (1.0 / 3.0)
    rng = np.random.default_rng(n)
    m = int(np.ceil(n ** (1.0 / 3.0)))
    g = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)[rng.permutation(m ** 3)[:n]]
    x = torch.tensor(((g + 0.5 + rng.uniform(-0.05, 0.05, g.shape)) / m), dtype=torch.float64, device=dev)
    typ = torch.tensor((rng.random(n) < 0.2).astype(np.int32), device=dev)
    act = torch.full((n,), -1, dtype=torch.int32, device=dev)
    F = torch.full((n, 3), float("nan"), dtype=torch.float64, device=dev)
    out = torch.full((3,), float("nan"), dtype=torch.float64, device=dev)
    p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    rc = cuda_lib.acg_forces_noalloc(p(x), None, p(typ), p(act), None, n, 0, L, 0.0, p(F), p(out),
                                     C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0, cuda_lib.acg_last_error().decode()
    want, pe = _plain(x, typ.long(), L, torch.arange(n, device=dev).split(512))
    rms = float(want.square().sum(1).mean().sqrt())
    assert float((F - want).abs().max()) <= 1e-12 * max(rms, 1e-300)
    assert abs(float(out[0]) - pe) <= 1e-12 * abs(pe)

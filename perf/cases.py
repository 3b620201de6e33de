"""Performance cases of the timestep: what programs that use this library have it do.

Each case is one call pattern of the public entry points (the C ABI of
include/activechi4.h and its Python mirror), on the active Kob-Andersen glass
at density 1.2:

* ``run``: one system per engine, advanced a chunk of steps, its scalars and
  state read back into the caller's pinned buffers (the drop-in run loop and
  every plain run);
* ``served``: the same on an engine set up by the run server (FP32 pair forces,
  observables accumulated in place);
* ``batch``: many replicas of uneven size in one engine, every replica's state
  read back after the chunk;
* ``forces``: calculate_forces at the current positions (cells, neighbour lists
  and forces) and the forces read back;
* ``device_forces``: the allocation-free force evaluation on device arrays.

All inputs are the library's seeded lattice states, where every run of the
reference and of the server begins.  States of FP32 pair forces are returned in
single precision (their own), all others in double; their chunks are 48 steps,
short enough that the rounding of single precision has not grown (by the
divergence of neighbouring trajectories) past single precision.
"""
import ctypes as C
import math

import numpy as np
import torch

from activechi4_b200 import Engine, _abi, default_params, lattice_state
from activechi4_b200.batch import make_engine, replica_set
from activechi4_b200.serve import RunRequest, request_params, start_run

DT = 0.005
TAU_T = 0.20
PAIRS = 32.6  # interacting pairs per particle within the cut at this density, each counted once
F0_SET = (0.0, 0.5, 1.0, 2.0)
T_SET = (0.45, 0.5, 0.6)
TAU_SET = (20, 200, 2000)


def listed():
    return [
        # a host program that drives the run loop itself, one step per call, and
        # reads the step's energies and state (the reference's size, FP64)
        dict(name="n1000_one_step", kind="run", n=1000, steps=1, precision=0, T=0.45, f0=1.0, tau_p=200, thermostat=1),
        # the reference's default system in chunks of steps
        dict(name="n1000_chunk", kind="run", n=1000, steps=64, precision=0, T=0.45, f0=1.0, tau_p=200, thermostat=1),
        # NVE at the size of the energy-drift checks
        dict(name="n4000_nve", kind="run", n=4000, steps=64, precision=0, T=0.45, f0=0.0, tau_p=200, thermostat=0),
        # the large plain run (FP64)
        dict(name="n100000_chunk", kind="run", n=100000, steps=64, precision=0, T=0.45, f0=1.0, tau_p=200,
             thermostat=1),
        # the largest size served, FP64, directions renewed every 0.1 time units
        dict(name="n256000_tau20", kind="run", n=256000, steps=64, precision=0, T=0.6, f0=2.0, tau_p=20, thermostat=1),
        # runs of the server: small ones are bound by step latency, large ones by arithmetic
        dict(name="served_n4505", kind="served", n=4505, steps=48, T=0.5, f0=1.0, tau_p=20),
        dict(name="served_n11154", kind="served", n=11154, steps=48, T=0.45, f0=0.5, tau_p=200),
        dict(name="served_n88250", kind="served", n=88250, steps=48, T=0.45, f0=1.0, tau_p=2000),
        # the batched workload: 256 replicas of 500 to 4000 particles
        dict(name="batch256", kind="batch", count=256, n_min=500, n_max=4000, replicas=11, steps=48, precision=1),
        # calculate_forces of a program that moves the particles itself
        dict(name="forces_n100000", kind="forces", n=100000, precision=0, f0=1.0),
        # force evaluation inside a framework that owns all device memory
        dict(name="device_forces_n20000", kind="device_forces", n=20000, f0=1.0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("run", "run", "served", "served", "batch", "forces", "device_forces"))
    f0 = rng.choice(F0_SET)
    if kind == "run":
        n = _log_int(rng, 500, 256000)
        precision = rng.choice((0, 0, 1))
        steps = rng.randint(1, 48 if precision else 64)
        return dict(kind=kind, n=n, steps=steps, precision=precision, T=rng.choice(T_SET), f0=f0,
                    tau_p=rng.choice(TAU_SET), thermostat=rng.choice((1, 1, 1, 0, 2)))
    if kind == "served":
        return dict(kind=kind, n=_log_int(rng, 1000, 256000), steps=rng.randint(24, 48), T=rng.choice(T_SET), f0=f0,
                    tau_p=rng.choice(TAU_SET))
    if kind == "batch":
        lo = _log_int(rng, 500, 2000)
        return dict(kind=kind, count=_log_int(rng, 4, 256), n_min=lo, n_max=rng.randint(lo, 4000),
                    replicas=rng.randint(0, 9999), steps=rng.randint(16, 48), precision=rng.choice((0, 1, 1)))
    if kind == "forces":
        return dict(kind=kind, n=_log_int(rng, 500, 256000), precision=rng.choice((0, 0, 1)), f0=f0)
    return dict(kind=kind, n=_log_int(rng, 500, 100000), f0=f0)


def _params(case, seed):
    return default_params(case["n"], T=case["T"], f0=case["f0"], tau_p_steps=case["tau_p"],
                          thermostat=case["thermostat"], precision=case["precision"], seed=seed % 1000003 + 1,
                          list_mode=1, rebuild_factor=4.0)


def _request(case, seed):
    return RunRequest(0, case["n"], 100000, case["T"], case["f0"], case["tau_p"], seed=seed % 100003)


def _pinned(n, width):
    return torch.empty((n, width), dtype=torch.float64).pin_memory()


def _replicas(case, seed):
    """The batch's sizes and parameters are the case's (its own draw); the states are the seed's."""
    reps = replica_set(case["count"], case["n_min"], case["n_max"], seed=case["replicas"], precision=case["precision"])
    return [(p, lattice_state(p.n, p.T, seed=(seed % 100003) * 1000 + r)) for r, (p, _) in enumerate(reps)]


def prepare(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng(seed)
    s = {"kind": kind, "steps": case.get("steps", 0), "single": case.get("precision", 1 if kind == "served" else 0) == 1}
    if kind == "device_forces":
        st = lattice_state(case["n"], 0.45, seed=seed)
        # a configuration off the lattice: every coordinate moved by up to 0.05
        x = st.x + rng.uniform(-0.05, 0.05, st.x.shape) / st.L
        x -= np.floor(x)
        x[x >= 1.0] = 0.0
        dev = torch.device("cuda")
        as_i = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.int32)).to(dev)  # noqa: E731
        s.update(n=st.n, nact=st.nact, L=st.L, f0=case["f0"], x=torch.from_numpy(x).to(dev), type=as_i(st.type),
                 act=as_i(st.act_tag), k=as_i(st.k.reshape(-1)),
                 F=torch.empty((st.n, 3), dtype=torch.float64, device=dev),
                 out=torch.empty(3, dtype=torch.float64, device=dev))
        return s
    if kind == "batch":
        e = make_engine(_replicas(case, seed))
    elif kind == "served":
        e = start_run(_request(case, seed))
    else:
        c = case if kind == "run" else dict(case, T=0.45, tau_p=200, thermostat=1)
        e = Engine(_params(c, seed))
        st = lattice_state(case["n"], c["T"], seed=seed)
        if kind == "forces":
            st.x = st.x + rng.uniform(-0.05, 0.05, st.x.shape) / st.L
            st.xu = st.x.copy()
            st.x -= np.floor(st.x)
            st.x[st.x >= 1.0] = 0.0
        e.set_state(0, st)
        if c["thermostat"] == 1:
            e.set_nhc(0, np.zeros(3), _p_eta(case["n"], c["T"], rng.standard_normal(3)))
    # the graphs of the chunk are built before the run starts
    if kind != "forces":
        e.prepare()
    e.sync()
    total = sum(n for n, _ in e.sizes)
    s.update(engine=e, offset=np.cumsum([0] + [n for n, _ in e.sizes]).tolist(), xu=_pinned(total, 3),
             p=_pinned(total, 3), F=_pinned(total, 3))
    return s


def _read(s, want):
    """Every system's state into the caller's pinned buffers, one system after another."""
    e, lib = s["engine"], _abi.lib()
    at = lambda name, k: C.c_void_p(s[name].data_ptr() + 24 * s["offset"][k]) if name in want else None  # noqa: E731
    for k in range(e.nsys):
        _abi.check(lib.acg_get_state(e.h, k, None, at("xu", k), at("p", k), at("F", k)))
    return {name: s[name].to(torch.float32) if s["single"] else s[name] for name in want}


def run(s):
    if s["kind"] == "device_forces":
        p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
        _abi.check(_abi.lib().acg_forces_noalloc(
            p(s["x"]), None, p(s["type"]), p(s["act"]), p(s["k"]), s["n"], s["nact"], s["L"], s["f0"], p(s["F"]),
            p(s["out"]), C.c_void_p(torch.cuda.current_stream().cuda_stream)))
        return {"F": s["F"], "scalars": s["out"]}
    e = s["engine"]
    if s["kind"] == "forces":
        e.compute_forces()
        out = _read(s, ("F",))
    else:
        e.step(s["steps"])
        out = _read(s, ("xu", "p") if s["kind"] == "batch" else ("xu", "p", "F"))
    if s["kind"] != "batch":
        t = e.thermo(0)
        scalars = torch.tensor([t["pe"], t["ke"], t["virial"]], dtype=torch.float64)
        out["scalars"] = scalars.to(torch.float32) if s["single"] else scalars
    return out


def work(case):
    """Bytes: a step reads each particle's wrapped and unfolded position, momentum and type and writes
    the three back; a force evaluation reads positions and types and writes forces.  Operations: 30 a pair."""
    kind = case["kind"]
    if kind in ("forces", "device_forces"):
        return {"bytes": case["n"] * (24 + 4 + 24), "flops": case["n"] * PAIRS * 30}
    n = case["n"] if kind != "batch" else case["count"] * 0.5 * (case["n_min"] + case["n_max"])
    return {"bytes": case["steps"] * n * 148.0, "flops": case["steps"] * n * (PAIRS * 30 + 60)}


# ---- the same in plain torch, FP64 -------------------------------------------
_IS2 = (1.0, 1.5625, 1.0 / (0.88 * 0.88))
_E4 = (4.0, 6.0, 2.0)


class _Plain:
    """One system: every pair with its minimum image (small N) or from a padded table of the
    particles within the cut and a margin, renewed when one has moved half the margin."""

    CUT, MARGIN, DENSE = 2.5, 1.4, 5000

    def __init__(self, st, f0):
        dev = torch.device("cuda")
        self.n, self.L, self.f0 = st.n, st.L, f0
        as_t = lambda a: torch.tensor(np.asarray(a, dtype=np.float64), device=dev)  # noqa: E731
        self.x, self.xu, self.p = as_t(st.x), as_t(st.xu), as_t(st.p)
        self.type = torch.tensor(np.asarray(st.type, dtype=np.int64), device=dev)
        self.act = torch.tensor(np.asarray(st.act_tag, dtype=np.int64), device=dev)
        self.k = np.array(st.k, dtype=np.int64)
        self.table, self.at = None, None
        self.is2 = torch.tensor(_IS2, dtype=torch.float64, device=dev)
        self.e4 = torch.tensor(_E4, dtype=torch.float64, device=dev)

    def _renew(self):
        n, dev = self.n, self.x.device
        cut2 = ((self.CUT + self.MARGIN) / self.L) ** 2
        nc = int(self.L / (self.CUT + self.MARGIN))
        rows = []
        ids = torch.arange(n, device=dev)
        if nc >= 3:
            c = (self.x * nc).long().clamp_(0, nc - 1)
            cell = c[:, 0] + nc * (c[:, 1] + nc * c[:, 2])
            order = torch.argsort(cell, stable=True)
            count = torch.bincount(cell, minlength=nc ** 3)
            start = torch.cumsum(count, 0) - count
            cap = int(count.max())
            slot = torch.full((nc ** 3, cap), -1, dtype=torch.long, device=dev)
            sc = cell[order]
            slot[sc, torch.arange(n, device=dev) - start[sc]] = order
            shift = torch.tensor([(a, b, d) for a in (-1, 0, 1) for b in (-1, 0, 1) for d in (-1, 0, 1)], device=dev)
        for i0 in range(0, n, 8192):
            i = ids[i0:i0 + 8192]
            if nc >= 3:
                q = (c[i][:, None, :] + shift[None]) % nc
                cand = slot[q[..., 0] + nc * (q[..., 1] + nc * q[..., 2])].reshape(len(i), -1)
            else:
                cand = ids[None].expand(len(i), n)
            d = self.x[i][:, None, :] - self.x[cand.clamp(min=0)]
            d -= d.round()
            ok = (cand >= 0) & (cand != i[:, None]) & ((d * d).sum(-1) < cut2)
            width = int(ok.sum(1).max())
            key = torch.where(ok, cand, torch.full_like(cand, n))
            rows.append(torch.sort(key, dim=1)[0][:, :width])
        width = max(r.shape[1] for r in rows)
        self.table = torch.cat([torch.nn.functional.pad(r, (0, width - r.shape[1]), value=n) for r in rows])
        self.at = self.xu.clone()

    def forces(self):
        n, L = self.n, self.L
        F = torch.empty_like(self.x)
        pe = torch.zeros((), dtype=torch.float64, device=self.x.device)
        vir = torch.zeros_like(pe)
        dense = n <= self.DENSE
        if not dense and (self.at is None or float((self.xu - self.at).square().sum(1).max()) * L * L
                          > (0.5 * self.MARGIN) ** 2):
            self._renew()
        step = 4096 if dense else 65536
        ids = torch.arange(n, device=self.x.device)
        for i0 in range(0, n, step):
            i = ids[i0:i0 + step]
            if dense:
                d = self.x[i][:, None, :] - self.x[None]
                tp = self.type[i][:, None] + self.type[None]
                ok = i[:, None] != ids[None]
            else:
                j = self.table[i]
                ok = j < n
                j = j.clamp(max=n - 1)
                d = self.x[i][:, None, :] - self.x[j]
                tp = self.type[i][:, None] + self.type[j]
            d -= d.round()
            is2, e4 = self.is2[tp], self.e4[tp]
            r2 = (d * d).sum(-1) * (L * L)
            rs2 = r2 * is2
            ok &= rs2 < 6.25
            rs2 = torch.where(ok, rs2, torch.ones_like(rs2))
            s2 = 1.0 / rs2
            s6 = s2 * s2 * s2
            zero = torch.zeros((), dtype=torch.float64, device=d.device)
            pe += torch.where(ok, e4 * (s6 * (s6 - 1.0) + 0.0162665594880 - 0.001949973872640 * rs2), zero).sum()
            g = torch.where(ok, 2.0 * e4 * is2 * (6.0 * s6 * (s6 - 0.5) * s2 + 0.001949973872640), zero)
            F[i] = (g[..., None] * d).sum(1) * L
            vir += (g * r2).sum()
        on = self.act >= 0
        kk = torch.tensor(self.k.astype(np.float64), device=d.device)
        if self.k.shape[1]:
            F[on] += self.f0 * kk[:, self.act[on]].T
        self.F, self.pe, self.vir = F, 0.5 * float(pe), 0.5 * float(vir) / 3.0
        return F

    def ke2(self):
        return float((self.p * self.p).sum())


def _half(chain, T, dof, k2):
    """U4 U3 U4 of the three-link chain for half a step; returns the velocity scale."""
    eta, pe = chain
    q = [dof * T * TAU_T ** 2, T * TAU_T ** 2, T * TAU_T ** 2]
    t4, t3 = 0.25 * DT, 0.5 * DT

    def link(j, k2):
        g = k2 - dof * T if j == 0 else pe[j - 1] ** 2 / q[j - 1] - T
        if j == 2:
            pe[j] += t4 * g
        else:
            x = t4 * pe[j + 1] / q[j + 1]
            pe[j] = pe[j] * math.exp(-x) + t4 * g * ((1.0 - math.exp(-x)) / x if x else 1.0)

    for j in (2, 1, 0):
        link(j, k2)
    s = math.exp(-t3 * pe[0] / q[0])
    for j in range(3):
        eta[j] += t3 * pe[j] / q[j]
    for j in (0, 1, 2):
        link(j, s * s * k2)
    return s


def _shuffle(k, words):
    n = k.shape[1]
    for c in range(3):
        row = k[c].tolist()
        for i in range(n):
            j = int(n * (int(words[c * n + i]) / 4294967296.0))
            row[i], row[j] = row[j], row[i]
        k[c] = row


def _trajectory(st, steps, T, f0, tau_p, thermostat, seed, p_eta):
    s = _Plain(st, f0)
    dof = 3.0 * s.n - 3.0
    chain = ([0.0] * 3, list(p_eta))
    words = np.random.RandomState(seed & 0xffffffff)
    s.forces()
    k2 = s.ke2()
    for step in range(steps):
        if step % tau_p == 0 and s.k.shape[1]:
            _shuffle(s.k, words.randint(0, 1 << 32, size=3 * s.k.shape[1], dtype=np.uint32))
        if thermostat == 1:
            s.p *= _half(chain, T, dof, k2)
        s.p += s.F * (0.5 * DT)
        dx = s.p * (DT / s.L)
        s.xu += dx
        s.x = s.x + dx
        s.x -= s.x.floor()
        s.forces()
        s.p += s.F * (0.5 * DT)
        k2 = s.ke2()
        if thermostat == 1:
            f = _half(chain, T, dof, k2)
            s.p *= f
            k2 *= f * f
        elif thermostat == 2:
            s.p *= math.sqrt(1.0 + (T / (k2 / dof) - 1.0) * DT / 0.20)
        if step == 0:  # the mean momentum is removed after every 100000th step, the first among them
            s.p -= s.p.mean(0)
            k2 = s.ke2()
    return s, k2


def _p_eta(n, T, normals):
    q = np.array([(3.0 * n - 3.0) * T * TAU_T ** 2, T * TAU_T ** 2, T * TAU_T ** 2])
    return np.sqrt(T * q) * normals


def exact(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng(seed)
    if kind in ("forces", "device_forces"):
        st = lattice_state(case["n"], 0.45, seed=seed)
        st.x = st.x + rng.uniform(-0.05, 0.05, st.x.shape) / st.L
        st.xu = st.x.copy()
        st.x = st.x - np.floor(st.x)
        st.x[st.x >= 1.0] = 0.0
        s = _Plain(st, case["f0"])
        s.forces()
        if kind == "forces":
            return {"F": s.F, "scalars": torch.tensor([s.pe, 0.5 * s.ke2(), s.vir], dtype=torch.float64)}
        # the active virial takes the unfolded positions, here the wrapped ones
        on = st.act_tag >= 0
        va = case["f0"] * float((st.k[:, st.act_tag[on]].T * st.x[on]).sum())
        return {"F": s.F, "scalars": torch.tensor([s.pe, s.vir, va], dtype=torch.float64)}
    if kind == "batch":
        if case["count"] * case["steps"] > 8192 and case["n_max"] > 2500:
            return None
        normals = np.random.default_rng(7)
        got = []
        for p, st in _replicas(case, seed):
            s, _ = _trajectory(st, case["steps"], p.T, p.f0, p.tau_p_steps, 1, p.seed,
                               _p_eta(st.n, p.T, normals.standard_normal(3)))
            got.append((s.xu, s.p))
        return {"xu": torch.cat([a for a, _ in got]), "p": torch.cat([b for _, b in got])}
    if kind == "served":
        r = _request(case, seed)
        st = lattice_state(case["n"], case["T"], seed=r.seed)
        p_eta = _p_eta(case["n"], case["T"], np.random.default_rng(r.seed).standard_normal(3))
        s, k2 = _trajectory(st, case["steps"], case["T"], case["f0"], case["tau_p"], 1, request_params(r).seed, p_eta)
    else:
        st = lattice_state(case["n"], case["T"], seed=seed)
        p_eta = _p_eta(case["n"], case["T"], rng.standard_normal(3)) if case["thermostat"] == 1 else np.zeros(3)
        s, k2 = _trajectory(st, case["steps"], case["T"], case["f0"], case["tau_p"], case["thermostat"],
                            seed % 1000003 + 1, p_eta)
    if kind == "run" and case["thermostat"] == 2:
        k2 = None  # the Berendsen step reports its kinetic energy from before the scaling
    scalars = None if k2 is None else torch.tensor([s.pe, 0.5 * k2, s.vir], dtype=torch.float64)
    return {"xu": s.xu, "p": s.p, "F": s.F, "scalars": scalars}

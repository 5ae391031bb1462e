"""The work that a user of vring_b200 has it do, as cases that can be timed and
compared: RK3 time steps of single rings and of ensembles, the reference's
per-routine call sequence, particles, the axisymmetric pressure solves (Krylov,
learned and direct), a training step of the learned preconditioner and the
batched tridiagonal solver.

Grids, Reynolds numbers, time steps and particle counts are those of the
workloads the tests and the benchmark run: r in [0, 4], z in [0, 12] (16 for
the head-on pair), a Gaussian-core ring with seeded noise of 1e-4; the
512 x 1024 axisymmetric grid clustered toward r = 1.

A pass of a time-stepping case is what a program does between two outputs: a
few steps, then the velocity (and the particles) to pinned host memory through
the library's asynchronous copies.
"""
from __future__ import annotations

import ctypes
import functools
import math

import numpy as np
import torch

import vring_b200 as V
from vring_b200 import api, learned, synthetic

DEV = "cuda"


# ---- the cases ------------------------------------------------------------------
def _ring(name, nth, nr, nz, steps, precision="fp64", wth="modified", inflow="off", re=3000.0, dt=5e-4, tracers=0,
          inertial=0, pair=False):
    return dict(name=name, kind="ring", nth=nth, nr=nr, nz=nz, steps=steps, precision=precision, wth=wth,
                inflow=inflow, re=re, dt=dt, tracers=tracers, inertial=inertial, pair=pair)


def listed():
    return [
        # the smallest run in use (the one the CPU build of the reference can do): launches and latency
        _ring("ring_64x32x128", 32, 64, 128, 10, wth="exact", re=1000.0, dt=2e-3, tracers=16384),
        # the benchmark grid in double precision
        _ring("ring_256x128x512", 128, 256, 512, 4),
        # the head-on pair's long theta and z lines, mixed precision, at a quarter of its radial cells
        _ring("pair_mixed_128x256x1024", 256, 128, 1024, 2, precision="mixed", re=5000.0, dt=2.5e-4, pair=True),
        # a grid that is no power of two in any direction, with the piston inflow of the reference's deck
        _ring("ring_inflow_100x48x180", 48, 100, 180, 10, wth="exact", inflow="reference", re=1500.0, dt=1e-3),
        # particles: tracers and inertial particles of one run, whole state read back
        _ring("particles_128x64x256", 64, 128, 256, 10, re=2000.0, dt=1e-3, tracers=262144, inertial=65536),
        # a Fortran host that keeps its own loop and calls the routines one by one
        dict(name="routines_128x64x256", kind="routines", nth=64, nr=128, nz=256, steps=4, re=2000.0, dt=1e-3,
             wth="exact"),
        # a parameter study: independent rings of uneven grids, mixed precision, tracers
        dict(name="ensemble_8_rings", kind="ensemble", rings=8, draw=1, steps=5, tracers=16384),
        # the axisymmetric pressure solve, fastest plain method, on the deck's grid
        dict(name="krylov_pcg_512x1024", kind="krylov", nr=512, nz=1024, method="pcg"),
        # the same with the trained network, from the previous step's pressure
        dict(name="krylov_learned_512x1024", kind="krylov", nr=512, nz=1024, method="learned"),
        # the direct solve that makes the training pairs
        dict(name="direct_512x1024", kind="direct", nr=512, nz=1024),
        # one Adam step of the network's training
        dict(name="train_512x1024", kind="train", nr=512, nz=1024, pool=4, c0=16, c1=32, c2=48, c3=64, batch=8),
        # solve_lap_thom on device arrays, a radial system per (theta mode, z mode) pair
        dict(name="thomas_257x1024", kind="thomas", n=257, nbatch=1024),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["ring", "ring", "ring", "routines", "ensemble", "krylov", "krylov", "direct", "train", "thomas"])
    if kind in ("ring", "routines"):
        if rng.random() < 0.5:  # power-of-two lines, any radial extent
            nth, nz = rng.choice([16, 32, 64, 128, 256]), rng.choice([64, 128, 256, 512, 1024])
        else:
            nth, nz = rng.randint(12, 100), rng.randint(48, 320)
        nr = max(24, min(_logint(rng, 24, 256), (1 << 24) // (nth * nz)))
        cells = nth * nr * nz
        steps = max(1, min(10, (1 << 23) // cells))
        c = dict(kind=kind, nth=nth, nr=nr, nz=nz, steps=steps, re=rng.uniform(500.0, 4000.0), dt=5e-4,
                 wth=rng.choice(["exact", "modified"]))
        if kind == "ring":
            c.update(precision=rng.choice(["fp64", "mixed"]), inflow=rng.choice(["off", "off", "reference"]),
                     tracers=rng.choice([0, _logint(rng, 500, 131072)]),
                     inertial=rng.choice([0, 0, _logint(rng, 500, 32768)]), pair=False)
        return c
    if kind == "ensemble":
        return dict(kind=kind, rings=rng.randint(2, 8), draw=rng.randint(2, 1000), steps=rng.randint(2, 5),
                    tracers=_logint(rng, 1000, 16384))
    if kind == "krylov":
        return dict(kind=kind, nr=_logint(rng, 32, 512), nz=_logint(rng, 64, 1024),
                    method=rng.choice(["cg", "pcg", "bicgstab", "fcg_jacobi"]))
    if kind == "direct":
        return dict(kind=kind, nr=_logint(rng, 32, 512), nz=_logint(rng, 64, 1024))
    if kind == "train":
        pool = rng.choice([2, 4])
        f = pool ** 3
        return dict(kind=kind, nr=f * max(1, round(_logint(rng, 64, 512) / f)),
                    nz=f * max(1, round(_logint(rng, 128, 1024) / f)), pool=pool, c0=8 * rng.randint(1, 3),
                    c1=8 * rng.randint(2, 4), c2=8 * rng.randint(3, 6), c3=8 * rng.randint(4, 8),
                    batch=rng.randint(1, 4))
    n = _logint(rng, 16, 1024)
    return dict(kind="thomas", n=n, nbatch=max(1, min(_logint(rng, 64, 4096), (1 << 19) // n)))


# ---- inputs ---------------------------------------------------------------------
@functools.lru_cache(maxsize=32)
def _base(nr, nz, zmax, rings):
    """q2 and q3 of the unperturbed ring(s) on one (r, z) plane."""
    _, q2, q3 = synthetic.ring_fields(1, nr, nz, 4.0, zmax, noise=0.0, rings=list(rings))
    return tuple(np.ascontiguousarray(q[0].T) for q in (q2, q3))  # (nz + 3, nr + 3)


def _set_velocity(run, nth, nr, nz, zmax, rings, seed):
    """The ring plus noise of 1e-4 on the interior, made on the GPU."""
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    q2, q3 = (torch.from_numpy(a).to(DEV) for a in _base(nr, nz, zmax, rings))
    for name, b, (j0, k0) in (("q1", torch.zeros_like(q2), (1, 1)), ("q2", q2, (2, 1)), ("q3", q3, (1, 2))):
        q = b[:, :, None].repeat(1, 1, nth)
        part = q[k0:nz + 1, j0:nr + 1]
        part += 1e-4 * torch.randn(part.shape, dtype=torch.float64, device=DEV, generator=g)
        host = q.cpu()
        run.set_ptr(name, host.data_ptr())


def _host(shape, dtype=torch.float64):
    return torch.empty(shape, dtype=dtype, pin_memory=True)


class _Stepped:
    """A run, where its velocity goes on the host, and its particle classes."""

    def __init__(self, run, nth, nr, nz):
        self.run = run
        self.q = {n: _host((nz + 3, nr + 3, nth)) for n in ("q1", "q2", "q3")}
        self.parts = []

    def add(self, pid, mode, n, r0, r1, z0, z1, seed):
        if not n:
            return
        p = V.Part(self.run, pid, n, mode)
        u = np.zeros((n, 117), order="F")
        u[:, 0], u[:, 1], u[:, 2] = synthetic.annulus_particles(n, r0, r1, z0, z1, seed=seed)
        v = np.zeros((n, 3), order="F")
        v[:, 2] = np.arange(1, n + 1)
        p.set_state(u, v, None, n)
        p.attach(True)
        self.parts.append((p, _host((117, n)), _host((3, n)), _host((n,), torch.int32)))

    def read(self, stream):
        for n, t in self.q.items():
            self.run.get_async(n, t.data_ptr(), stream)
        out = dict(self.q)
        for i, (p, u, v, f) in enumerate(self.parts):
            cnt = (ctypes.c_int32 * 4)()
            p._chk(api.lib().vr_part_get_state(p._h, ctypes.c_void_p(u.data_ptr()), ctypes.c_void_p(v.data_ptr()),
                                               ctypes.c_void_p(f.data_ptr()), cnt))
            out["part%d" % i] = (u, v, f)
        return out


def _single(c, seed):
    pair, nth, nr, nz = c.get("pair", False), c["nth"], c["nr"], c["nz"]
    zmax = 16.0 if pair else 12.0
    rings = ((1.0, 0.15, 1.0, 5.0), (1.0, 0.15, -1.0, 11.0)) if pair else ((1.0, 0.2, 1.0, 3.0),)
    run = V.Run(nth, nr, nz, 4.0, zmax, c["dt"], c["re"], 1.0, 1.0, precision=c.get("precision", "fp64"),
                theta_wavenumber=c["wth"], inflow=c.get("inflow", "off"))
    _set_velocity(run, nth, nr, nz, zmax, rings, seed)
    s = _Stepped(run, nth, nr, nz)
    s.add(8, 1, c.get("tracers", 0), 0.5, 1.5, 2.0, 4.0, seed)
    s.add(1, 0, c.get("inertial", 0), 0.5, 1.5, 2.0, 4.0, seed + 1)
    return s


def _ensemble_specs(c):
    from vring_b200.ensemble import ensemble_specs
    return ensemble_specs(c["rings"], c["draw"])


def _rhs(faces, nr, nz, zmax, seed):
    """(f_t, p_{t-1}) of a seeded pressure sequence; K in plain numpy."""
    seq = learned.RingSequence(2 + seed % 20, faces, nz, zmax)
    t = 1 + seed % 900
    return _apply_k(faces, nz, zmax, seq.pressure(t)), seq.pressure(t - 1)


def _coef(faces, nz, zmax):
    dz = zmax / nz
    rm, dr = 0.5 * (faces[:-1] + faces[1:]), np.diff(faces)
    c = faces[1:-1] * dz / np.diff(rm)
    aw, ae = np.concatenate([[0.0], c]), np.concatenate([c, [0.0]])
    return aw, ae, rm * dr / dz, rm * dr * dz, 2.0 * faces[-1] * dz / dr[-1]


def _apply_s(faces, nz, zmax, x):
    """The symmetric operator of the axisymmetric pressure problem, x (nr, nz)."""
    aw, ae, az, _, gam = _coef(faces, nz, zmax)
    y = np.zeros_like(x)
    y[1:] += aw[1:, None] * (x[1:] - x[:-1])
    y[:-1] += ae[:-1, None] * (x[:-1] - x[1:])
    y[-1] += gam * x[-1].mean()
    y[:, 1:] += az[:, None] * (x[:, 1:] - x[:, :-1])
    y[:, :-1] += az[:, None] * (x[:, :-1] - x[:, 1:])
    return y


def _apply_k(faces, nz, zmax, x):
    return _apply_s(faces, nz, zmax, x) / _coef(faces, nz, zmax)[3][:, None]


def _solve_k(faces, nz, zmax, f):
    """K x = f by a z cosine transform and a radial elimination per z mode."""
    nr = faces.size - 1
    aw, ae, _, vol, gam = _coef(faces, nz, zmax)
    dz, q = zmax / nz, np.arange(nz)
    c = np.cos(np.pi * np.outer(q, 2 * q + 1) / (2 * nz))
    fh = f @ c.T / nz
    lo, up = -aw / vol, -ae / vol
    wz = 2.0 / dz ** 2 * (1.0 - np.cos(q * np.pi / nz))
    d = ((aw + ae) / vol)[:, None] + wz
    d[-1, 0] += gam / vol[-1]
    for j in range(1, nr):
        w = lo[j] / d[j - 1]
        d[j] -= w * up[j - 1]
        fh[j] -= w * fh[j - 1]
    fh[-1] /= d[-1]
    for j in range(nr - 2, -1, -1):
        fh[j] = (fh[j] - up[j] * fh[j + 1]) / d[j]
    c[1:] *= 2.0
    return fh @ c


def _dev(a):
    """A (nr, nz) array as the library lays vectors out (r fastest)."""
    return torch.from_numpy(np.ascontiguousarray(a.T)).to(DEV)


def _layers(c):
    """(cin, cout) of the 14 3x3 layers, then the head."""
    a, b, d, e = c["c0"], c["c1"], c["c2"], c["c3"]
    return [(1, a), (a, a), (a, b), (b, b), (b, d), (d, d), (d, e), (e, e), (e + d, d), (d, d), (d + b, b), (b, b),
            (b + a, a), (a, a)]


def _weights(c, rng):
    w = [rng.standard_normal((co, 3, 3, ci)) / math.sqrt(9 * ci) for ci, co in _layers(c)]
    w.append(rng.standard_normal(c["c0"]) / math.sqrt(c["c0"]))
    return np.concatenate([x.ravel() for x in w]).astype(np.float32)


def _errors(c, rng, faces):
    """A training batch: increments of pressure sequences, smooth fields and scaled noise."""
    nr, nz, zmax, out = c["nr"], c["nz"], learned.ZMAX, []
    rm, zm = learned.cell_centres(faces, nz, zmax)
    aw, ae, az, _, gam = _coef(faces, nz, zmax)
    diag = (aw + ae)[:, None] + az[:, None] * (2.0 - (np.arange(nz) == 0) - (np.arange(nz) == nz - 1))
    diag[-1] += gam / nz
    for b in range(c["batch"]):
        if b % 4 < 2:
            seq, t = learned.RingSequence(int(rng.integers(2, 22)), faces, nz, zmax), int(rng.integers(1, 1000))
            e = seq.pressure(t) - seq.pressure(t - 1)
        elif b % 4 == 2:
            e = sum(rng.normal() / (1.0 + kr + kz) * np.outer(np.cos(np.pi * kr * rm / faces[-1]), np.cos(np.pi * kz * zm / zmax))
                    for kr, kz in rng.integers(0, min(nr, nz) // 2, (8, 2)))
        else:
            e = rng.standard_normal((nr, nz)) / np.sqrt(diag)
        out.append(e)
    return np.stack(out)


LR_FIRST, LR = 1e-8, 1e-3  # the first step of a run warms the moments up


def _training_inputs(c, seed):
    rng = np.random.default_rng(seed)
    faces = learned.tanh_faces(c["nr"])
    return faces, _weights(c, rng), _errors(c, rng, faces), _errors(c, rng, faces)


def _systems(c, seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    u = [torch.rand((c["nbatch"], c["n"]), dtype=torch.float64, device=DEV, generator=g) for _ in range(4)]
    return u[0] * 2 - 1, u[1] * 2 - 1, u[2] + 2.5, u[3] * 2 - 1  # rhs, aa, bb, cc: diagonally dominant


def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind in ("ring", "routines"):
        return dict(case=c, s=[_single(c, seed)], stream=torch.cuda.Stream())
    if kind == "ensemble":
        from vring_b200 import ensemble as E
        made = []
        for i, sp in enumerate(_ensemble_specs(c)):
            nth, nr, nz = sp["nth"], sp["nr"], sp["nz"]
            run = V.Run(nth, nr, nz, E.RMAX, E.ZMAX, E.DT, sp["re"], 1.0, 1.0, precision="mixed",
                        theta_wavenumber="modified")
            _set_velocity(run, nth, nr, nz, E.ZMAX, ((sp["R"], sp["sr"] * sp["R"], 1.0, E.Z0),), seed + i)
            s = _Stepped(run, nth, nr, nz)
            s.add(8, 1, c["tracers"], 0.5 * sp["R"], 1.5 * sp["R"], E.Z0 - 1.0, E.Z0 + 1.0, seed + i)
            made.append(s)
        return dict(case=c, s=made, ens=V.Ensemble([s.run for s in made]), stream=torch.cuda.Stream())
    if kind in ("krylov", "direct"):
        k = learned.make_solver(nr=c["nr"], nz=c["nz"])
        f, p = _rhs(k.faces, c["nr"], c["nz"], learned.ZMAX, seed)
        st = dict(case=c, k=k, f=_dev(f), x0=_dev(p))
        st["x"] = torch.zeros_like(st["x0"])
        if c.get("method") == "learned":
            st["net"] = learned.make_net()
            learned.load_weights(st["net"])
            k.set_preconditioner(st["net"])
        return st
    if kind == "train":
        faces, w, e0, e1 = _training_inputs(c, seed)
        k = learned.make_solver(nr=c["nr"], nz=c["nz"])
        net = learned.make_net(nr=c["nr"], nz=c["nz"], ch=(c["c0"], c["c1"], c["c2"], c["c3"]), pool=c["pool"])
        net.set_params(w)
        e0, e1 = (torch.from_numpy(np.ascontiguousarray(e.transpose(0, 2, 1))).to(DEV) for e in (e0, e1))
        torch.cuda.synchronize()  # the library's streams do not wait for torch's
        net.train_step(k, e0.data_ptr(), c["batch"], LR_FIRST)
        return dict(case=c, k=k, net=net, e=e1)
    t = _systems(c, seed)
    return dict(case=c, t=t, sol=torch.empty_like(t[0]))


def run(state):
    c = state["case"]
    kind = c["kind"]
    if kind == "ring":
        s = state["s"][0]
        s.run.iterate(c["steps"])
        return s.read(state["stream"].cuda_stream)
    if kind == "ensemble":
        state["ens"].iterate(c["steps"])
        return [s.read(state["stream"].cuda_stream) for s in state["s"]]
    if kind == "routines":
        s = state["s"][0]
        r = s.run
        _, t, n = r.clock
        for i in range(1, c["steps"] + 1):
            for irk in (1, 2, 3):
                r.set_clock(irk, t + i * c["dt"], n + i)
                r.ucoeff()
                r.coesys()
                r.hdnbc()
                r.hdnl1()
                r.hdnl2()
                r.hdnl3()
                r.step()
                r.divq()
                r.laplace_solve()
                r.upsol()
                r.uppres()
        return s.read(state["stream"].cuda_stream)
    if kind == "krylov":
        state["x"].copy_(state["x0"])
        torch.cuda.current_stream().synchronize()  # the library's stream does not wait for torch's
        state["k"].solve_dev(state["f"].data_ptr(), state["x"].data_ptr(), c["method"], tol=1e-12, maxit=40000)
        return state["x"]
    if kind == "direct":
        state["k"].direct_dev(state["f"].data_ptr(), state["x"].data_ptr())
        return state["x"]
    if kind == "train":
        loss = state["net"].train_step(state["k"], state["e"].data_ptr(), c["batch"], LR)
        return loss, state["net"].get_params()
    r, a, b, d = state["t"]
    api.solve_lap_thom_noalloc(r.data_ptr(), state["sol"].data_ptr(), a.data_ptr(), b.data_ptr(), d.data_ptr(),
                               c["n"], c["nbatch"], torch.cuda.current_stream().cuda_stream)
    return state["sol"]


# ---- the same in 64 bits ----------------------------------------------------------
def _net(c, w, x):
    """N(x) in float64 on weights rounded to bfloat16 (what the network's weights are); x (nr, nz)."""
    import torch.nn.functional as F
    parts, off = [], 0
    for ci, co in _layers(c):
        n = 9 * ci * co
        parts.append(w[off:off + n].reshape(co, 3, 3, ci).permute(0, 3, 1, 2))
        off += n
    head, pool = w[off:], c["pool"]

    def two(t, i):
        return F.conv2d(F.conv2d(t, parts[i], padding=1), parts[i + 1], padding=1)

    e0 = two(x[None, None], 0)
    e1 = two(F.avg_pool2d(e0, pool), 2)
    e2 = two(F.avg_pool2d(e1, pool), 4)
    t = two(F.avg_pool2d(e2, pool), 6)
    for skip, i in ((e2, 8), (e1, 10), (e0, 12)):
        t = two(torch.cat([F.interpolate(t, scale_factor=pool, mode="nearest"), skip], 1), i)
    return (t[0] * head[:, None, None]).sum(0)


def _train_exact(c, seed):
    faces, w, e0, e1 = _training_inputs(c, seed)
    nz, zmax = c["nz"], learned.ZMAX
    aw, ae, az, _, gam = (torch.as_tensor(v, dtype=torch.float64, device=DEV) for v in _coef(faces, nz, zmax))

    def S(x):
        y = gam * torch.zeros_like(x)
        y[1:] += aw[1:, None] * (x[1:] - x[:-1])
        y[:-1] += ae[:-1, None] * (x[:-1] - x[1:])
        y[-1] += gam * x[-1].mean()
        y[:, 1:] += az[:, None] * (x[:, 1:] - x[:, :-1])
        y[:, :-1] += az[:, None] * (x[:, :-1] - x[:, 1:])
        return y

    k = torch.arange(nz, device=DEV)
    diag = (aw + ae)[:, None] + az[:, None] * (2.0 - (k == 0).double() - (k == nz - 1).double())
    diag[-1] += gam / nz
    d = diag.rsqrt()
    w = torch.from_numpy(w).to(DEV).double()
    m, v = torch.zeros_like(w), torch.zeros_like(w)
    for t, (batch, lr) in enumerate(((e0, LR_FIRST), (e1, LR)), 1):
        w16 = w.float().bfloat16().double().requires_grad_(True)
        total = 0.0
        for b in range(c["batch"]):
            e = torch.from_numpy(batch[b]).to(DEV)
            r = S(e)
            s = (d * r).square().mean().sqrt()
            y = s * d * _net(c, w16, d * r / s)
            loss = ((y - e) * S(y - e)).sum() / (e * r).sum() / c["batch"]
            loss.backward()
            total += float(loss.detach())
        g = w16.grad
        m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
        w = w - lr * (m / (1 - 0.9 ** t)) / ((v / (1 - 0.999 ** t)).sqrt() + 1e-8)
    return total, w.cpu().numpy()


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind in ("krylov", "direct"):
        faces = learned.tanh_faces(c["nr"])
        f, _ = _rhs(faces, c["nr"], c["nz"], learned.ZMAX, seed)
        return np.ascontiguousarray(_solve_k(faces, c["nz"], learned.ZMAX, f).T)
    if kind == "train":
        return _train_exact(c, seed)
    if kind == "thomas":
        r, a, b, d = (t.cpu().numpy().astype(np.longdouble) for t in _systems(c, seed))
        for k in range(1, c["n"]):
            w = a[:, k] / b[:, k - 1]
            b[:, k] -= w * d[:, k - 1]
            r[:, k] -= w * r[:, k - 1]
        r[:, -1] /= b[:, -1]
        for k in range(c["n"] - 2, -1, -1):
            r[:, k] = (r[:, k] - d[:, k] * r[:, k + 1]) / b[:, k]
        return r.astype(np.float64)
    return None  # a time step has no plain restatement apart from the whole solver


# ---- what a pass cannot do without -------------------------------------------------
def _step_work(cells, mixed):
    """Per time step: the state (q, ru, pres, prg) read and written in each of
    three substeps; the stencils, substitutions and transforms of each."""
    words = 6 * 8 + 14 * (4 if mixed else 8)
    return dict(bytes=3 * words * cells, flops=3 * 500 * cells)


def _part_work(n, words, substeps):
    return dict(bytes=2 * 8 * words * n, flops=3600 * substeps * n)


def _sum(*ws, times=1):
    return {k: float(times * sum(w[k] for w in ws)) for k in ("bytes", "flops")}


def work(case):
    c, kind = case, case["kind"]
    if kind in ("ring", "routines"):
        cells = c["nth"] * c["nr"] * c["nz"]
        return _sum(_step_work(cells, c.get("precision") == "mixed"), _part_work(c.get("tracers", 0), 45, 5),
                    _part_work(c.get("inertial", 0), 117, 20), times=c["steps"])
    if kind == "ensemble":
        return _sum(*[_step_work(s["nth"] * s["nr"] * s["nz"], True) for s in _ensemble_specs(c)],
                    _part_work(c["rings"] * c["tracers"], 45, 5), times=c["steps"])
    n = c.get("nr", 0) * c.get("nz", 0)
    if kind == "krylov":  # the vectors fit the chip: only the products with the operator and the dots count
        its = {"cg": 20, "pcg": 8, "bicgstab": 8, "fcg_jacobi": 5, "learned": 1}[c["method"]] * max(c["nr"], c["nz"]) / 2
        per = 50 if c["method"] != "learned" else 50 + 2 * 9 * sum(a * b for a, b in _layers(dict(c0=16, c1=32, c2=48, c3=64))[-2:])
        return dict(bytes=3.0 * 8 * n, flops=float(per * n * its))
    if kind == "direct":  # both transforms by their fast form, one division-free substitution
        return dict(bytes=2.0 * 8 * n, flops=float(n * (2 * 2.5 * math.log2(c["nz"]) + 6)))
    if kind == "train":
        lev, macs = [0, 0, 1, 1, 2, 2, 3, 3, 2, 2, 1, 1, 0, 0], 0.0
        for (ci, co), l in zip(_layers(c), lev):
            macs += 9 * ci * co * n / c["pool"] ** (2 * l)
        return dict(bytes=8.0 * n * c["batch"], flops=3 * 2 * macs * c["batch"])
    return dict(bytes=5.0 * 8 * c["n"] * c["nbatch"], flops=9.0 * c["n"] * c["nbatch"])

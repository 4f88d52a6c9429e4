"""The work that programs have this framework do, as cases that can be timed.

A case is one call (or one short sequence of calls) of the public Python
binding, with inputs of a size and distribution that the path meets in use:
one force evaluation of the leapfrog schedule through the drop-in call, the
device-resident call or the per-phase calls, whole schedules, many systems in
one context, a serving tick, particle text in and out, and the direct sum
that force errors are measured against.

``listed()`` names the cases, ``draw(rng)`` gives more of the same ranges,
``prepare`` makes what a program holds before the call, ``run`` is one pass,
``work`` the bytes and flops a pass cannot do without, and ``exact`` what the
pass computes in plain 64-bit torch, where that is affordable.
"""
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "amt-bh-benchmark_b200"))
import bhg  # noqa: E402

DEV = "cuda:0"
G = 1.0
RMAX = 10.0  # spheres are truncated at ten scale radii


# ---- the cases ---------------------------------------------------------------


def listed():
    return [
        # The drop-in call of a small simulation, host vectors in and out, at
        # the reference's default leaf, group and target sizes: all latency.
        dict(name="dropin-1k", kind="dropin", n=1021, dist="sphere", theta=0.5, eps=0.01, leaf=8, target=32, dt=1 / 128),
        # A whole leapfrog schedule of an ordinary small system without
        # softening (the masked self term), resident between its evaluations.
        dict(name="schedule-16k", kind="schedule", n=16411, dist="sphere", theta=0.5, eps=0.0, leaf=16, target=16,
             dt=1 / 1024, steps=8),
        # One resident evaluation at the benchmark's small size.
        dict(name="step-65k", kind="step", n=65536, dist="sphere", theta=0.5, eps=0.01, leaf=16, target=16, quad=True,
             dt=1 / 128),
        # The plain 64-bit path, phase by phase, accelerations returned to the host.
        dict(name="forces64-40k", kind="forces", n=40009, dist="sphere", theta=0.5, eps=0.01, leaf=16, target=16),
        # Monopoles only, at the reference's default leaf and target sizes, an odd million.
        dict(name="mono-1m", kind="step", n=1000003, dist="sphere", theta=0.6, eps=0.01, leaf=8, target=32, quad=False,
             dt=1 / 256),
        # One evaluation of the headline workload.
        dict(name="step-4m", kind="step", n=4194304, dist="sphere", theta=0.5, eps=0.005, leaf=16, target=16, quad=True,
             dt=1 / 256),
        # The largest configured system: two spheres on their way to each other.
        dict(name="merger-16m", kind="step", n=16777216, dist="merger", theta=0.6, eps=0.002, leaf=16, target=16,
             quad=True, dt=1 / 256),
        # Independent systems of uneven size advanced together, at the leaf
        # size the autotuner picks for them.
        dict(name="ensemble-256", kind="ensemble", systems=256, nmin=1024, nmax=262144, leaf=48, dt=1 / 1024),
        # One tick of the server: a request leaves with its particles, another
        # joins (generated on the device), all the resident ones take a step.
        dict(name="serve-tick-48", kind="serve", systems=48, nmin=4096, nmax=262144, leaf=32, dt=1 / 1024),
        # Particles arriving as text in host memory.
        dict(name="csv-131k", kind="csv", n=131071),
        # Particles leaving as text into pinned host memory.
        dict(name="vtk-500k", kind="vtk", n=500009),
        # The error check of the benchmark and the autotuner: sampled rows
        # of the 64-bit direct sum.
        dict(name="direct-1m", kind="direct", n=1048576, rows=4096, eps=0.005),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choice(["dropin", "schedule", "step", "step", "step", "forces", "ensemble", "serve", "csv", "vtk", "direct"])
    theta = rng.choice([0.4, 0.5, 0.6, 0.7])
    eps = rng.choice([0.0, 0.002, 0.005, 0.01, 0.01])
    dist = rng.choice(["sphere", "sphere", "merger", "cube"])
    leaf = rng.choice([8, 16, 16, 24, 32, 48])
    target = rng.choice([leaf, leaf, 32])
    if kind == "dropin":
        return dict(kind=kind, n=_log_int(rng, 200, 50000), dist=dist, theta=theta, eps=eps, leaf=leaf, target=target,
                    dt=1 / 128)
    if kind == "schedule":
        return dict(kind=kind, n=_log_int(rng, 1000, 120000), dist="sphere", theta=theta, eps=eps, leaf=leaf,
                    target=target, dt=1 / 1024, steps=rng.randint(2, 12))
    if kind == "step":
        return dict(kind=kind, n=_log_int(rng, 1000, 6000000), dist=dist, theta=theta, eps=eps, leaf=leaf, target=target,
                    quad=rng.random() < 0.8, dt=1 / 256)
    if kind == "forces":
        return dict(kind=kind, n=_log_int(rng, 2000, 120000), dist=dist, theta=theta, eps=eps, leaf=leaf, target=target)
    if kind == "ensemble":
        return dict(kind=kind, systems=rng.randint(8, 256), nmin=1024, nmax=rng.choice([16384, 65536, 262144]),
                    leaf=rng.choice([16, 32, 48]), dt=1 / 1024)
    if kind == "serve":
        return dict(kind=kind, systems=rng.randint(8, 64), nmin=4096, nmax=rng.choice([65536, 262144]),
                    leaf=rng.choice([16, 32]), dt=1 / 1024)
    if kind == "csv":
        return dict(kind=kind, n=_log_int(rng, 1000, 200000))
    if kind == "vtk":
        return dict(kind=kind, n=_log_int(rng, 1000, 1000000))
    return dict(kind=kind, n=_log_int(rng, 20000, 1500000), rows=_log_int(rng, 256, 4096), eps=rng.choice([0.002, 0.005, 0.01]))


# ---- inputs --------------------------------------------------------------------


def _directions(n, gen):
    z = torch.rand(n, generator=gen, device=DEV, dtype=torch.float64) * 2 - 1
    phi = torch.rand(n, generator=gen, device=DEV, dtype=torch.float64) * (2 * math.pi)
    s = torch.sqrt(1 - z * z)
    return torch.stack((s * torch.cos(phi), s * torch.sin(phi), z), 1)


def _sphere(n, gen, a=1.0):
    """Positions and velocities of a Plummer sphere of mass 1 and scale radius
    a: radii from the cumulative mass, speeds (in units of the escape speed)
    from the cumulative distribution of q^2 (1 - q^2)^(7/2)."""
    u = torch.rand(n, generator=gen, device=DEV, dtype=torch.float64) * (1 + RMAX**-2) ** -1.5
    r = (u.clamp_min(1e-14) ** (-2 / 3) - 1) ** -0.5
    qn = np.linspace(0, 1, 8193)
    cdf = np.cumsum(qn * qn * (1 - qn * qn) ** 3.5)  # on the host: the same bits every time
    q, cdf = torch.from_numpy(qn).to(DEV), torch.from_numpy(cdf / cdf[-1]).to(DEV)
    v = torch.rand(n, generator=gen, device=DEV, dtype=torch.float64)
    k = torch.searchsorted(cdf, v).clamp(1, 8192)
    frac = ((v - cdf[k - 1]) / (cdf[k] - cdf[k - 1]).clamp_min(1e-300)).clamp(0, 1)
    speed = (q[k - 1] + frac / 8192) * math.sqrt(2 / a) * (1 + r * r) ** -0.25
    return _directions(n, gen) * (a * r)[:, None], _directions(n, gen) * speed[:, None]


def _state(n, dist, seed):
    """mass [n], pos [n, 3] and vel [n, 3] of one system."""
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed)
    if dist == "cube":
        pos = torch.rand(n, 3, generator=gen, device=DEV, dtype=torch.float64) * 2 - 1
        vel = torch.randn(n, 3, generator=gen, device=DEV, dtype=torch.float64) * 0.3
        return torch.full((n,), 1.0 / n, device=DEV, dtype=torch.float64), pos, vel
    if dist == "merger":
        h = n // 2
        p1, v1 = _sphere(h, gen, 1.0)
        p2, v2 = _sphere(n - h, gen, 0.5)
        p1[:, 0] -= 5.0
        p2[:, 0] += 5.0
        v1[:, 0] += 0.15
        v2[:, 0] -= 0.15
        return (torch.full((n,), 1.0 / h, device=DEV, dtype=torch.float64), torch.cat((p1, p2)), torch.cat((v1, v2)))
    pos, vel = _sphere(n, gen)
    return torch.full((n,), 1.0 / n, device=DEV, dtype=torch.float64), pos, vel


def _records(mass, pos, vel):
    """bh::Particle records (64 bytes) as an [n, 8] float64 device tensor."""
    n = len(mass)
    rec = torch.zeros(n, 8, device=DEV, dtype=torch.float64)
    rec.view(torch.int32).view(n, 16)[:, 0] = torch.arange(n, device=DEV, dtype=torch.int32)
    rec[:, 1] = mass
    rec[:, 2:5] = pos
    rec[:, 5:8] = vel
    return rec


def _fields(rec):
    """A record tensor's fields, as views of it."""
    n = len(rec)
    return dict(id=rec.view(torch.int32).view(n, 16)[:, 0], mass=rec[:, 1], pos=rec[:, 2:5], vel=rec[:, 5:8])


def _host_records(rec):
    return np.ascontiguousarray(rec.cpu().numpy()).view(bhg.PARTICLE).reshape(-1)


def _sizes(case):
    """The systems' sizes: evenly spread over the logarithm of the range, in a
    mixed order."""
    k, lo, hi = case["systems"], math.log(case["nmin"]), math.log(case["nmax"])
    n = [int(round(math.exp(lo + (hi - lo) * (i + 0.5) / k))) for i in range(k)]
    random.Random(k).shuffle(n)
    return n


_THETAS = (0.4, 0.5, 0.7)  # the serving stream's opening angles


class _State:
    """What a program holds: a context, and its buffers."""

    def __init__(self, case):
        self.case = case
        self.ctx = bhg.Context(device=0)

    def __del__(self):
        ctx = getattr(self, "ctx", None)
        if ctx is not None:
            ctx.close()


def prepare(case, seed):
    st = _State(case)
    kind = case["kind"]
    if kind in ("ensemble", "serve"):
        sizes = _sizes(case)
        st.sizes = sizes
        st.handles = [st.ctx.add_generated([dict(n=n, a=1.0, mass=1.0)], seed=seed * 1000003 + s) for s, n in enumerate(sizes)]
        st.theta = [0.5] * len(sizes) if kind == "ensemble" else [_THETAS[s % 3] for s in range(len(sizes))]
        st.next_seed = seed * 1000003 + len(sizes)
        st.out = torch.empty(sum(sizes), 8, device=DEV, dtype=torch.float64)
        st.ctx.set_system_params(theta=st.theta, eps2=[1e-4] * len(sizes), kick_dt=[case["dt"]] * len(sizes),
                                 drift_dt=[case["dt"]] * len(sizes))
        st.fp = bhg.Context.params(0.5, 1e-4, G)
        return st
    n = case["n"]
    rec = _records(*_state(n, case.get("dist", "sphere"), seed))
    if kind == "csv":
        rows = rec[:, 1:].cpu().numpy().tolist()
        line = ",".join(["%d"] + ["%.17g"] * 7)
        st.text = ("id,mass,x,y,z,vx,vy,vz\n" + "\n".join(line % (i, *r) for i, r in enumerate(rows)) + "\n").encode()
        st.out = torch.empty(n, 8, device=DEV, dtype=torch.float64)
        return st
    if kind == "dropin":
        st.parts = _host_records(rec)
        return st
    st.rec = rec
    st.out = torch.empty_like(rec)
    if kind == "vtk":
        st.ctx.upload_device(rec.data_ptr(), n)
        st.text = torch.zeros(st.ctx.snapshot_vtk_bound(), dtype=torch.uint8, pin_memory=True).numpy()
        return st
    if kind == "direct":
        st.ctx.upload_device(rec.data_ptr(), n)
        st.idx = _rows(case, seed)
        return st
    st.fp = bhg.Context.params(case["theta"], case["eps"] ** 2, G, case.get("quad", True),
                               bhg.PRECISION_FP64 if kind == "forces" else bhg.PRECISION_SPLIT)
    return st


def _rows(case, seed):
    return np.sort(np.random.default_rng(seed).choice(case["n"], case["rows"], replace=False)).astype(np.uint32)


# ---- one pass --------------------------------------------------------------------


def run(st):
    case, ctx = st.case, st.ctx
    kind = case["kind"]
    if kind == "dropin":
        p = bhg.step_particles(st.parts, case["theta"], case["eps"] ** 2, G, True, case["leaf"], 256, case["target"],
                               case["dt"] / 2, case["dt"], workspace=ctx)
        return dict(id=p["id"], mass=p["mass"], pos=p["pos"], vel=p["vel"])
    if kind == "step":
        ctx.upload_device(st.rec.data_ptr(), case["n"])
        ctx.step(st.fp, case["leaf"], 256, case["target"], case["dt"] / 2, case["dt"])
        _download(ctx, st.out)
        return _fields(st.out)
    if kind == "schedule":
        ctx.upload_device(st.rec.data_ptr(), case["n"])
        ctx.run_schedule(st.fp, case["leaf"], 256, case["target"], case["dt"], case["steps"])
        _download(ctx, st.out)
        return _fields(st.out)
    if kind == "forces":
        ctx.upload_device(st.rec.data_ptr(), case["n"])
        ctx.build_tree(case["leaf"], 256)
        ctx.compute_multipoles()
        acc = ctx.walk_forces(st.fp, case["target"])
        return dict(acc=acc)
    if kind == "ensemble":
        ctx.step_systems(st.fp, case["leaf"], 256, case["leaf"])
        _download(ctx, st.out)
        return _fields(st.out)
    if kind == "serve":
        # the oldest request leaves, one of its size joins at the end
        n, theta = st.sizes.pop(0), st.theta.pop(0)
        gone = ctx.remove_systems([st.handles.pop(0)], want=True, sizes=[n])[0]
        st.handles.append(ctx.add_generated([dict(n=n, a=1.0, mass=1.0)], seed=st.next_seed))
        st.next_seed += 1
        st.sizes.append(n)
        st.theta.append(theta)
        k = len(st.sizes)
        ctx.set_system_params(theta=st.theta, eps2=[1e-4] * k, kick_dt=[case["dt"]] * k, drift_dt=[case["dt"]] * k)
        ctx.step_systems(st.fp, case["leaf"], 256, case["leaf"])
        _download(ctx, st.out)
        return dict(_fields(st.out), gone=dict(id=gone["id"], mass=gone["mass"], pos=gone["pos"], vel=gone["vel"]))
    if kind == "csv":
        ctx.upload_csv(st.text)
        _download(ctx, st.out)
        return _fields(st.out)
    if kind == "vtk":
        return dict(bytes=ctx.snapshot_vtk_into(st.text), text=st.text)
    return ctx.direct_sum(st.idx, case["eps"] ** 2, G)


def _download(ctx, out):
    """The state into a device tensor (the C entry point has no method of its own)."""
    r = ctx.L.bhg_download_device(ctx.h, out.data_ptr())
    if r:
        raise bhg.BhgError(r, ctx.last_error())


# ---- what a pass cannot do without -----------------------------------------------


# Interactions per particle of a sphere at theta 0.5 and leaf 16, counted by
# the walk (bhg_get_stats): particles, particle-cell, particle-particle.
_COUNTED = ((1021, 81, 553), (4096, 381, 762), (16411, 878, 774), (65536, 1291, 667), (262144, 1604, 496),
            (1000003, 1793, 512), (4194304, 1985, 459), (16777216, 2180, 440))


def _flops(n, leaf, theta, quad):
    """Flops of one evaluation's interactions: 20 per particle pair (and per
    monopole), 60 per particle-cell quadrupole, the counts interpolated from
    the table above (within about a third of the walk's own counts)."""
    x = math.log(max(n * 16 / leaf, 1))
    at = [(math.log(m), c, p) for m, c, p in _COUNTED]
    x = min(max(x, at[0][0]), at[-1][0])
    k = max(i for i in range(len(at) - 1) if at[i][0] <= x)
    f = (x - at[k][0]) / (at[k + 1][0] - at[k][0])
    pc = (at[k][1] + f * (at[k + 1][1] - at[k][1])) * (0.5 / theta) ** 2.2
    pp = (at[k][2] + f * (at[k + 1][2] - at[k][2])) * (0.5 / theta) ** 2.6 * (leaf / 16) ** 1.1
    return n * (min(pc, n) * (60.0 if quad else 20.0) + min(pp, n) * 20.0)


def work(case):
    kind = case["kind"]
    if kind in ("ensemble", "serve"):
        sizes = _sizes(case)
        return dict(bytes=128.0 * sum(sizes), flops=sum(_flops(n, case["leaf"], 0.5, True) for n in sizes))
    n = case["n"]
    if kind == "csv":
        return dict(bytes=(146 + 64.0) * n, flops=0.0)
    if kind == "vtk":
        return dict(bytes=(64 + 72.0) * n, flops=0.0)
    if kind == "direct":
        return dict(bytes=32.0 * n + 28.0 * case["rows"], flops=20.0 * n * case["rows"])
    evals = case["steps"] + 1 if kind == "schedule" else 1
    return dict(bytes=128.0 * n * evals, flops=evals * _flops(n, case["leaf"], case["theta"], case.get("quad", True)))


# ---- the same in plain 64-bit torch ----------------------------------------------


def _direct(pos, mass, rows, eps2):
    """Softened direct-sum accelerations of the given rows (a body exerts none on itself)."""
    out = torch.empty(len(rows), 3, device=DEV, dtype=torch.float64)
    step = max(1, (1 << 27) // len(pos))
    for b in range(0, len(rows), step):
        d = pos[None, :, :] - pos[rows[b:b + step], None, :]
        r2 = (d * d).sum(2)
        w = (r2 + eps2) ** -1.5 * mass
        w = torch.where(r2 > 0, w, torch.zeros_like(w))
        out[b:b + step] = (d * w[:, :, None]).sum(1)
    return out * G


def _morton_order(pos):
    """Indices that put the particles in Morton order: 21 bits per axis over
    the bounding cube, x in the lowest bit."""
    lo, hi = pos.min(0).values, pos.max(0).values
    hw = 0.5 * (hi - lo).max()
    if not hw > 0:
        hw = torch.ones_like(hw)
    hw = hw * (1.0 + 1e-9)
    q = torch.floor((pos - (0.5 * (lo + hi) - hw)) * (float(1 << 21) / (2.0 * hw))).clamp(0, (1 << 21) - 1).to(torch.int64)
    key = torch.zeros(len(pos), device=DEV, dtype=torch.int64)
    for bit in range(21):
        for axis in range(3):
            key |= ((q[:, axis] >> bit) & 1) << (3 * bit + axis)
    return torch.sort(key, stable=True).indices


def exact(case, seed):
    kind, n = case["kind"], case.get("n", 0)
    if kind == "csv":
        return _fields(_records(*_state(n, "sphere", seed)))
    if kind == "direct":
        mass, pos, _ = _state(n, "sphere", seed)
        rows = torch.from_numpy(_rows(case, seed).astype(np.int64)).to(DEV)
        return _direct(pos, mass, rows, case["eps"] ** 2)
    if kind not in ("dropin", "step", "forces") or n > 150000:
        return None
    mass, pos, vel = _state(n, case["dist"], seed)
    order = _morton_order(pos)
    acc = _direct(pos, mass, torch.arange(n, device=DEV), case["eps"] ** 2)
    if kind == "forces":
        return dict(acc=acc[order])
    vel = vel + (case["dt"] / 2) * acc
    pos = pos + case["dt"] * vel
    return dict(id=order.to(torch.int32), mass=mass[order], pos=pos[order], vel=vel[order])

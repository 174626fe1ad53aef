"""The workloads this framework's speed is measured on.

Each case goes through the public entry points a program calls: the pipeline
driver (`pipeline.run`), the batch call (`gpu.batch_run`), the stage calls of
`gpu.Context`, and the torch wrappers.  The framework's data boundary is the
host: snapshots, groupings and catalogues are host arrays, as a snapshot file
or a simulation hands them over, so a pass includes their copies.  The torch
wrapper takes tensors on the GPU.

Sizes follow the repository's own configurations (the 2^21 clustered box, the
uneven sub-volumes, the 2^20 adjoint workload, the mixed-species generator),
its tests (a few thousand particles, ragged counts, open boxes) and sizes
between them.
"""
from __future__ import annotations

import dataclasses
import math

import numpy as np
import torch

from skid_gb300 import autograd, gpu, pipeline, synth, tipsy
from skid_gb300.options import PLUMMER, SPLINE, Options

# Largest counts an FP64 all-pairs evaluation is done for.
EXACT_POINTS = 140_000
EXACT_PAIRS = 3.0e10


def listed():
    return [
        # A few thousand dark particles, the size of a test snapshot or one
        # zoomed halo: launches and host round trips count here.
        dict(name="run_small", kind="run", n=5003, k=32, box="periodic", mixed=False),
        # The headline workload: the 2^21 clustered periodic box, host buffers
        # in, catalogue out.
        dict(name="run_box_2e21", kind="run", n=1 << 21, k=64, box="periodic", mixed=False),
        # Gas and dark matter together with -gd at z = 0.5 on a Gaussian
        # random field background, with the .stat columns.
        dict(name="run_mixed", kind="run", n=150_001, k=64, box="periodic", mixed=True),
        # Uneven independent sub-volumes of a survey or a zoom suite, several
        # at once.
        dict(name="batch_uneven", kind="batch", volumes=12, lo=14, hi=18, workers=8),
        # The density stage alone (`-den`): tree, neighbours, density.
        dict(name="density_box", kind="density", n=1 << 20, k=64, box="periodic"),
        # The same for an isolated (open) region, a ragged count, k = 32.
        dict(name="density_open", kind="density", n=70_001, k=32, box="open"),
        # Neighbour radii of a point set, with the largest usual k.
        dict(name="knn_k128", kind="knn", n=131_071, k=128, box="periodic"),
        # The density field's gradient at positions of the caller's choice.
        dict(name="field", kind="field", n=131_072, nm=100_003, k=64, box="periodic"),
        # Friends-of-friends over a point set.
        dict(name="fof", kind="fof", n=1 << 20, box="periodic"),
        # Unbinding of a grouping found elsewhere (`-unbind`): groups over
        # three decades of size, spline softening.
        dict(name="unbind", kind="unbind", n=400_000, groups=300, soft="spline"),
        # Density and its gradient with respect to positions, as a fit over
        # particle positions asks for it: new positions every step.
        dict(name="density_grad", kind="density_grad", n=100_000, k=64, box="periodic"),
        # Potential energies of chosen groups and their gradient, through the
        # torch wrapper.
        dict(name="potential_grad", kind="potential_grad", n=200_000, groups=24, soft="spline"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run", "run", "batch", "density", "knn", "field", "fof", "unbind",
                       "density_grad", "potential_grad"])
    box = rng.choice(["periodic", "periodic", "open"])
    if kind == "run":
        return dict(kind=kind, n=_log_int(rng, 4096, 1 << 20), k=rng.choice([32, 48, 64]),
                    box=box, mixed=rng.random() < 0.3)
    if kind == "batch":
        lo = rng.randint(13, 15)
        return dict(kind=kind, volumes=rng.randint(3, 12), lo=lo, hi=rng.randint(lo + 1, 18),
                    workers=rng.choice([1, 4, 8, 12]))
    if kind == "density":
        return dict(kind=kind, n=_log_int(rng, 4096, 1 << 20), k=rng.choice([16, 32, 64, 100, 128]),
                    box=box)
    if kind == "knn":
        return dict(kind=kind, n=_log_int(rng, 1000, 1 << 20), k=rng.choice([8, 24, 32, 64, 128]),
                    box=box)
    if kind == "field":
        return dict(kind=kind, n=_log_int(rng, 4096, 1 << 18), nm=_log_int(rng, 1000, 1 << 19),
                    k=rng.choice([32, 64]), box=box)
    if kind == "fof":
        return dict(kind=kind, n=_log_int(rng, 2048, 1 << 21), box=box)
    soft = rng.choice(["spline", "spline", "plummer"])
    if kind == "unbind":
        n = _log_int(rng, 8192, 1 << 19)
        return dict(kind=kind, n=n, groups=_log_int(rng, 3, max(4, n // 1000)), soft=soft)
    if kind == "density_grad":
        return dict(kind=kind, n=_log_int(rng, 4096, 1 << 19), k=rng.choice([32, 64]), box=box)
    return dict(kind=kind, n=_log_int(rng, 8192, 1 << 18), groups=rng.randint(4, 64), soft=soft)


# ---------------------------------------------------------------------------
# inputs

def _tau(n):
    return 0.5 * n ** (-1.0 / 3.0)


def _snapshot(case, seed):
    """The clustered box of this size: NFW halos in proportion to the count
    over a uniform background, or the mixed-species generator's gas and dark
    matter over a Gaussian random field."""
    n = case["n"]
    if case.get("mixed"):
        spec = dataclasses.replace(synth.CONFIG4_SLICE, n=n, n_halo=max(2, n * 6000 // (1 << 24)),
                                   r200_max=0.03, seed=seed)
        return synth.make_snapshot(spec, time=1.0 / 1.5)
    return synth.make_snapshot(dataclasses.replace(synth.config1_spec(n), seed=seed))


def _options(case):
    f = ["-tau", repr(0.004 if case["n"] == 1 << 21 else _tau(case["n"])), "-s", str(case["k"]),
         "-m", "16", "-O", "0.3", "-Lambda", "0.7", "-H", f"{synth.hubble_for(0.3):.6g}"]
    if case["box"] == "periodic":
        f += ["-p", "1"]
    if case["mixed"]:
        f += ["-gd", "-z", "0.5", "-stats"]
    return Options.parse(f)


def _period(case):
    return 1.0 if case["box"] == "periodic" else None


def _clumps(n, n_groups, seed):
    """Isolated clumps with a known grouping: group sizes log-uniform over
    three decades hold 70 % of the particles, radii after Hernquist (1990)
    inside eight scale lengths, isotropic Gaussian velocities near the virial
    dispersion (so a tail is unbound); the rest is uniform background, some
    of it (2 %) wrongly counted into groups, as linking does.
    Returns (snapshot, group ids with 0 = none)."""
    rng = np.random.default_rng(seed)
    w = 10.0 ** rng.uniform(0.0, 3.0, n_groups)
    counts = np.maximum(8, np.floor(0.7 * n * w / w.sum())).astype(np.int64)
    while counts.sum() > 0.9 * n:
        counts = np.maximum(2, counts // 2)
    gid = np.repeat(np.arange(n_groups), counts)
    nc = len(gid)
    r200 = 0.03 * (counts / counts.max()) ** (1.0 / 3.0)
    s = np.sqrt(rng.uniform(0.0, 0.79, nc))
    r = (r200[gid] / 8.0) * s / (1.0 - s)
    d = rng.normal(size=(nc, 3))
    d /= np.linalg.norm(d, axis=1)[:, None]
    centres = rng.uniform(-0.5, 0.5, (n_groups, 3))
    sig = np.sqrt(counts / n / (2.0 * r200))
    pos = np.concatenate([centres[gid] + r[:, None] * d, rng.uniform(-0.5, 0.5, (n - nc, 3))])
    vel = np.concatenate([rng.normal(0.0, 0.1, (n_groups, 3))[gid] +
                          rng.normal(size=(nc, 3)) * sig[gid][:, None],
                          rng.normal(0.0, 0.05, (n - nc, 3))])
    grp = np.concatenate([gid + 1, np.zeros(n - nc, np.int64)])
    stray = nc + np.flatnonzero(rng.random(n - nc) < 0.02)
    grp[stray] = rng.integers(1, n_groups + 1, len(stray))
    p = rng.permutation(n)
    pos = pos - np.floor(pos + 0.5)
    pos = np.clip(pos[p].astype(np.float32), np.float32(-0.5), np.float32(0.49999997))
    snap = tipsy.Snapshot(1.0, 0, n, 0, pos, vel[p].astype(np.float32),
                          np.full(n, 1.0 / n, np.float32),
                          np.full(n, 0.02 * n ** (-1.0 / 3.0), np.float32),
                          np.zeros(n, np.float32))
    return snap, grp[p].astype(np.int32)


def _cotangent(n, seed):
    return np.random.default_rng(seed + 77).normal(size=n).astype(np.float32)


def _field_positions(case, pos, seed):
    """Positions a step or so off particles, as movers are."""
    rng = np.random.default_rng(seed + 5)
    at = pos[rng.integers(0, len(pos), case["nm"])]
    y = at + (rng.normal(size=at.shape) * 0.2 * _tau(case["n"])).astype(np.float32)
    return np.clip(y, np.float32(-0.5), np.float32(0.49999997)).astype(np.float32)


def _volumes(case, seed):
    """Counts log-uniform in [2^lo, 2^hi], the same for every seed."""
    rng = np.random.default_rng([synth.SEED_BASE, case["volumes"], case["lo"], case["hi"]])
    out = []
    for i in range(case["volumes"]):
        n = int(round(2.0 ** rng.uniform(case["lo"], case["hi"])))
        spec = dataclasses.replace(synth.config1_spec(n), seed=seed * 1000 + i)
        out.append((synth.make_snapshot(spec), int(rng.choice([32, 64, 128])), _tau(n)))
    return out


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case, kind=kind)
    if kind == "run":
        s["snap"], s["opts"] = _snapshot(case, seed), _options(case)
        s["ctx"] = gpu.Context(period=_period(case), nSmooth=case["k"])
    elif kind == "batch":
        s["volumes"] = _volumes(case, seed)
        s["opts"] = Options.parse(list(synth.WORKLOAD_FLAGS[1]))
    elif kind in ("density", "density_grad"):
        s["snap"] = _snapshot(case, seed)
        s["w"] = _cotangent(case["n"], seed)
        s["ctx"] = gpu.Context(period=_period(case), nSmooth=case["k"])
    elif kind in ("knn", "fof"):
        s["pos"] = _snapshot(case, seed).pos
        s["ctx"] = gpu.Context(period=_period(case))
    elif kind == "field":
        snap = _snapshot(case, seed)
        s["y"] = _field_positions(case, snap.pos, seed)
        s["ctx"] = ctx = gpu.Context(period=_period(case), nSmooth=case["k"])
        ctx.set_particles(snap)
        ctx.scatter_active()
        ctx.density()
    elif kind == "unbind":
        s["snap"], s["grp"] = _clumps(case["n"], case["groups"], seed)
        s["opts"] = Options.parse(list(synth.WORKLOAD_FLAGS[1]) +
                                  (["-plummer"] if case["soft"] == "plummer" else []))
        s["ctx"] = ctx = gpu.Context(period=1.0)
        ctx.set_particles(s["snap"])
    else:
        snap, grp = _clumps(case["n"], case["groups"], seed)
        s["pos"] = torch.from_numpy(snap.pos).cuda().requires_grad_(True)
        s["mass"] = torch.from_numpy(snap.mass).cuda()
        s["soft"] = torch.from_numpy(snap.soft).cuda()
        s["grp"] = torch.from_numpy(grp).cuda()
        s["sel"] = torch.arange(1, case["groups"] + 1, dtype=torch.int32)
        s["v"] = torch.from_numpy(_cotangent(case["groups"], seed).astype(np.float64)).cuda()
    return s


# ---------------------------------------------------------------------------
# one pass

def _columns(rec, n):
    """A catalogue's columns in arrays as long as any catalogue of n particles
    in groups of 16 or more can need (rows past its end are zero; row 0, the
    ungrouped particles', is not part of a catalogue)."""
    out = np.zeros(n // 16 + 2, rec.dtype)
    out[1:len(rec)] = rec[1:]
    return {f: out[f] for f in rec.dtype.names}


def run(state):
    kind, case, ctx = state["kind"], state["case"], state.get("ctx")
    if kind == "run":
        r = pipeline.run(state["snap"], state["opts"], ctx=ctx)
        out = dict(grp=r.grp, groups=_columns(r.groups, case["n"]),
                   counts={k: r.counts[k] for k in ("nExtraScat", "nMove", "nGroupFoF", "nUnbound",
                                                    "nGroup")})
        if r.stats is not None:
            out["stats"] = _columns(r.stats, case["n"])
        return out
    if kind == "batch":
        res = gpu.batch_run(state["volumes"], state["opts"], n_workers=case["workers"])
        out = []
        for r in res:
            c = _columns(r["groups"], len(r["grp"]))
            out.append(dict(grp=r["grp"], centre=c["rCenter"], mass=c["fMass"],
                            members=c["nMembers"], unbound=r["nUnbound"]))
        return out
    if kind == "density":
        ctx.set_particles(state["snap"])
        ctx.scatter_active()
        ctx.density()
        rho, ball2 = ctx.get_density()
        return dict(rho=rho, ball2=ball2)
    if kind == "density_grad":
        ctx.set_particles(state["snap"])
        ctx.scatter_active()
        ctx.density()
        rho, _ = ctx.get_density()
        return dict(rho=rho, grad=ctx.density_adjoint(state["w"], gpu.ADJ_AUTO))
    if kind == "knn":
        return ctx.knn_ball2(state["pos"], case["k"])
    if kind == "field":
        return ctx.field(state["y"])
    if kind == "fof":
        grp, ng = ctx.fof_points(state["pos"], _tau(case["n"]))
        return dict(grp=grp, n=ng)
    if kind == "unbind":
        o = state["opts"]
        ctx.set_groups(state["grp"])
        nu = ctx.unbind(o.iSoftType, o.fScoop, o.bGasAndDark, o.bNoUnbind, o.nMaxMembers, o.G, o.z,
                        o.a_shift, o.a_hubble)
        ng = ctx.too_small(o.nMembers)
        grp, rec = ctx.get_groups(ng)
        return dict(grp=grp, groups=_columns(rec, case["n"]), unbound=nu)
    pos = state["pos"]
    E = autograd.group_potential(pos, state["mass"], state["soft"], state["grp"], state["sel"],
                                 soft_type=PLUMMER if case["soft"] == "plummer" else SPLINE,
                                 period=1.0)
    (grad,) = torch.autograd.grad(E, pos, state["v"])
    return dict(E=E, grad=grad)


# ---------------------------------------------------------------------------
# what a pass cannot do without

def work(case):
    """Compulsory bytes: host inputs read once, outputs written once.
    Operations: pair terms the definition asks for, about 10 operations a
    distance and 20 a kernel, field or potential term."""
    kind, n, k = case["kind"], case.get("n", 0), case.get("k", 64)
    if kind == "run":
        # neighbours and both density halves; about 30 move steps' worth of
        # full field sums over the run
        return dict(bytes=36 * n + 4 * n, flops=n * k * (30.0 + 30 * 30.0))
    if kind == "batch":
        mid = (2.0 ** case["hi"] - 2.0 ** case["lo"]) / ((case["hi"] - case["lo"]) * math.log(2.0))
        m = case["volumes"] * mid
        return dict(bytes=40 * m, flops=m * 75 * (30.0 + 30 * 30.0))
    if kind == "density":
        return dict(bytes=36 * n + 8 * n, flops=30.0 * n * k)
    if kind == "density_grad":
        return dict(bytes=36 * n + 4 * n + 16 * n, flops=90.0 * n * k)
    if kind == "knn":
        return dict(bytes=16 * n, flops=10.0 * n * k)
    if kind == "field":
        return dict(bytes=24 * case["nm"] + 20 * n, flops=30.0 * case["nm"] * k)
    if kind == "fof":
        return dict(bytes=16 * n, flops=10.0 * n * 8)
    # sum of squared group sizes, log-uniform over three decades, 70 % of n
    g = case["groups"]
    pairs = (0.7 * n) ** 2 / g * 3.46
    if kind == "unbind":
        return dict(bytes=(4 + 36 + 4) * n, flops=0.5 * 30.0 * pairs)
    return dict(bytes=(12 + 4 + 4 + 4 + 12) * n, flops=0.5 * 40.0 * pairs)


# ---------------------------------------------------------------------------
# the same in 64 bits, plain torch

def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _t64(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to(_dev(), torch.float64)


def _delta(a, b, periodic):
    d = a - b
    return d - torch.round(d) if periodic else d


def _neighbours(x, k, periodic):
    """Indices of the k nearest points of every point, itself included,
    nearest first."""
    n = len(x)
    out = torch.empty((n, k), dtype=torch.int64, device=x.device)
    step = max(1, int(3e8 // n))
    for i in range(0, n, step):
        d2 = torch.zeros((min(step, n - i), n), dtype=torch.float64, device=x.device)
        for c in range(3):
            d2 += _delta(x[i:i + step, None, c], x[None, :, c], periodic) ** 2
        out[i:i + step] = torch.topk(d2, k, dim=1, largest=False, sorted=True).indices
    return out


def _w_m4(q2):
    q = torch.sqrt(torch.clamp(q2, min=1e-30))
    return torch.where(q2 < 1.0, 1.0 - 0.75 * (2.0 - q) * q2, 0.25 * (2.0 - q) ** 3)


def _density64(x, mass, idx, periodic):
    """Symmetric SPH density with the neighbour sets idx; ball2 too."""
    n, k = idx.shape
    d2 = (_delta(x[:, None, :], x[idx], periodic) ** 2).sum(-1)
    b = d2[:, -1]
    ih2 = 4.0 / b
    w = 0.5 / math.pi * (ih2 ** 1.5)[:, None] * _w_m4(d2 * ih2[:, None])
    rho = (mass[idx] * w).sum(1)
    rho = rho.index_add(0, idx.reshape(-1), (mass[:, None] * w).reshape(-1))
    return rho, b


def _exact_field(case, seed):
    snap = _snapshot(case, seed)
    per = case["box"] == "periodic"
    x, mass = _t64(snap.pos), _t64(snap.mass)
    idx = _neighbours(x, case["k"], per)
    b = _density64(x, mass, idx, per)[1]
    y = _t64(_field_positions(case, snap.pos, seed))
    ih2 = 4.0 / b
    coef = mass * ih2 ** 2.5 / math.pi
    acc = torch.empty_like(y)
    step = max(1, int(1e8 // len(x)))
    for i in range(0, len(y), step):
        d = [_delta(x[None, :, c], y[i:i + step, None, c], per) for c in range(3)]
        d2 = d[0] ** 2 + d[1] ** 2 + d[2] ** 2
        q2 = d2 * ih2
        q = torch.sqrt(torch.clamp(q2, min=1e-30))
        f = torch.where(q2 < 1.0, 2.25 * q - 3.0, 3.0 - 0.75 * q - 3.0 / q) * coef
        f = torch.where(d2 < b, f, torch.zeros((), dtype=f.dtype, device=f.device))
        for c in range(3):
            acc[i:i + step, c] = (f * d[c]).sum(1)
    return acc.cpu().numpy()


def _psi64(r, e, plummer):
    """The pair potential per unit G m m' (Hernquist & Katz 1989 spline, or
    Plummer), e the sum of the two softenings."""
    if plummer:
        return 1.0 / torch.sqrt(r * r + 0.25 * e * e)
    u = 2.0 * r / e
    inner = 1.4 - (2.0 / 3.0) * u ** 2 + 0.3 * u ** 4 - 0.1 * u ** 5
    outer = -1.0 / (15.0 * u) + 1.6 - (4.0 / 3.0) * u ** 2 + u ** 3 - 0.3 * u ** 4 + u ** 5 / 30.0
    return torch.where(u < 1.0, 2.0 / e * inner, torch.where(u < 2.0, 2.0 / e * outer, 1.0 / r))


def _exact_potential(case, seed):
    snap, grp = _clumps(case["n"], case["groups"], seed)
    v = _cotangent(case["groups"], seed).astype(np.float64)
    x, mass, soft = _t64(snap.pos), _t64(snap.mass), _t64(snap.soft)
    E = torch.zeros(case["groups"], dtype=torch.float64, device=x.device)
    grad = torch.zeros_like(x)
    g = torch.from_numpy(grp).to(x.device)
    # coordinates are taken relative to the group's last member and wrapped,
    # so a pair is not always at its nearest image
    for s in range(case["groups"]):
        m = torch.nonzero(g == s + 1).reshape(-1)
        xr = _delta(x[m], x[m[-1]], True)
        step = max(1, int(1e8 // max(1, len(m))))
        for i in range(0, len(m), step):
            a = xr[i:i + step].clone().requires_grad_(True)
            d2 = ((a[:, None, :] - xr[None, :, :]) ** 2).sum(-1)
            own = torch.zeros_like(d2, dtype=torch.bool)
            own[torch.arange(len(a)), torch.arange(i, i + len(a))] = True
            r = torch.sqrt(torch.where(own, torch.ones_like(d2), d2))
            psi = _psi64(r, soft[m][i:i + step, None] + soft[m][None, :], case["soft"] == "plummer")
            psi = torch.where(own, torch.zeros_like(psi), psi)
            e = -0.5 * (mass[m][i:i + step] * (psi * mass[m][None, :]).sum(1)).sum()
            (ga,) = torch.autograd.grad(e, a)
            E[s] += e.detach()
            grad[m[i:i + step]] = 2.0 * float(v[s]) * ga     # both ends of every pair
    return dict(E=E.cpu().numpy(), grad=grad.cpu().numpy())


def exact(case, seed):
    kind = case["kind"]
    if kind in ("density", "density_grad", "knn", "field") and case["n"] > EXACT_POINTS:
        return None
    if kind in ("density", "density_grad", "knn"):
        snap = _snapshot(case, seed)
        per = case["box"] == "periodic"
        x, mass = _t64(snap.pos), _t64(snap.mass)
        x.requires_grad_(kind == "density_grad")
        idx = _neighbours(x.detach(), case["k"], per)
        rho, b = _density64(x, mass, idx, per)
        if kind == "knn":
            return b.cpu().numpy()
        if kind == "density":
            return dict(rho=rho.cpu().numpy(), ball2=b.cpu().numpy())
        (grad,) = torch.autograd.grad(rho, x, _t64(_cotangent(case["n"], seed)))
        return dict(rho=rho.detach().cpu().numpy(), grad=grad.cpu().numpy())
    if kind == "field" and float(case["n"]) * case["nm"] <= EXACT_PAIRS:
        return _exact_field(case, seed)
    if kind == "potential_grad" and work(case)["flops"] <= 3e11:
        return _exact_potential(case, seed)
    return None      # catalogues are whole numbers and what follows from them

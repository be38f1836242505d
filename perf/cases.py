"""The work whose speed matters to a user of this package, as measurable cases.

Each case is one call pattern of the public API at one size: the resident
`System` in its mixed and plain FP64 forms (a frame every few tens of steps),
a `Batch` of replicas, the reference-layout drop-ins on host arrays, the
trajectory gradient, and the analysis of a state.  `exact` restates the same
physics in plain torch FP64 for checking.
"""
import math

import numpy as np
import torch

import proteinsim2015_gb300 as psim
from proteinsim2015_gb300 import adjoint as padj, batch as pbatch, init

LJ_KT, LJ_RC, LJ_DT = 1.5, 2.5, 0.002          # the rho = 0.8 liquid of the benchmark
PLUGIN_CFG = "force = LennardJones\nkT = 1\n"   # the LennardJones plugin's own defaults
ADJ_BINS, ADJ_RANGE = 100, (0.8, 3.0)


def listed():
    return [
        # the reference's own 4000-particle AO case (L = 21, 7 cells a side): the
        # smallest system anyone runs, a frame every 100 steps
        dict(name="ao_4000_mixed", kind="system", force="AO", n=4000, phi=0.2262, form="mixed",
             skin=-1.0, steps=100),
        # the same in the plain FP64 form, with the whole state read back
        dict(name="ao_4000_fp64", kind="system", force="AO", n=4000, phi=0.2262, form="fp64",
             skin=0.0, steps=40),
        # the LennardJones plugin as it comes (2n-n with n = 18 and a Yukawa tail),
        # loaded from its shared object: a mid-sized run of odd size
        dict(name="plugin_lj18_50k_mixed", kind="system", force="PLUGIN", n=50001, phi=0.2,
             form="mixed", skin=-1.0, steps=60),
        # the benchmark's headline: the 2^20-particle liquid with a pair list
        dict(name="lj_1m_mixed", kind="system", force="LJ", n=1 << 20, phi=0.0, form="mixed",
             skin=0.4, steps=40),
        # its plain FP64 form, with the whole state read back
        dict(name="lj_1m_fp64", kind="system", force="LJ", n=1 << 20, phi=0.0, form="fp64",
             skin=0.0, steps=5),
        # the aggregating gel with its cell list rebuilt every step
        dict(name="gel_2m_mixed", kind="system", force="GEL", n=1 << 21, phi=0.30, form="mixed",
             skin=0.0, steps=20),
        # a parameter sweep: independent AO replicas of uneven size in one batch
        dict(name="batch_64_mixed", kind="batch", replicas=64, sweep=2015, form="mixed", skin=0.3,
             steps=40),
        # a reference host that calls the three drop-ins on its own arrays, with
        # the library's defaults (FP64, every call alone)
        dict(name="host_ao_20k_fp64", kind="host", force="AO", n=20001, phi=0.2, form="fp64",
             skin=0.0, pinned=False, steps=4),
        # the same loop on a million-particle liquid (63^3 cells) in the mixed form,
        # its pair list kept
        dict(name="host_lj_1m_mixed", kind="host", force="LJ", n=4 * 63 ** 3, phi=0.0, form="mixed",
             skin=-1.0, pinned=True, steps=6),
        # gradient of a g(r) loss with respect to every parameter: a small fit
        dict(name="grad_4096", kind="grad", n=4096, phi=0.15, lj=True, steps=60, every=20),
        # and the differentiable workload's size (AO + Yukawa)
        dict(name="grad_32768", kind="grad", n=32768, phi=0.15, lj=False, steps=60, every=20),
        # the analysis of one stored state: energy, g(r), contacts, clusters
        dict(name="analysis_131k", kind="analysis", n=1 << 17, phi=0.30),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["system", "system", "system", "batch", "host", "grad", "analysis"])
    if kind in ("system", "host"):
        form = rng.choice(["mixed", "fp64"])
        force = rng.choice(["AO", "LJ", "PLUGIN", "GEL"] if kind == "system" else ["AO", "LJ"])
        n = _log_int(rng, 1000, 1 << 20) | 1
        phi = 0.0 if force == "LJ" else round(rng.uniform(0.08, 0.3), 3)
        skin = 0.0 if form == "fp64" else rng.choice([0.0, -1.0])
        c = dict(kind=kind, force=force, n=n, phi=phi, form=form, skin=skin)
        if kind == "host":
            c["n"] = n - n % 4 + 1
            return dict(c, pinned=rng.choice([False, True]), steps=rng.randint(2, 4))
        most = (5 << 20) // n if form == "fp64" else (20 << 20) // n
        return dict(c, steps=max(2, min(most, rng.randint(10, 60))))
    if kind == "batch":
        return dict(kind=kind, replicas=rng.randint(4, 48), sweep=rng.randint(1, 9999), form="mixed",
                    skin=rng.choice([0.0, 0.3]), steps=rng.randint(10, 40))
    if kind == "grad":
        n = _log_int(rng, 1000, 32768)
        return dict(kind=kind, n=n, phi=round(rng.uniform(0.08, 0.16), 3),
                    lj=rng.choice([False, True]), steps=rng.randint(20, 50),
                    every=rng.choice([7, 10, 25]))
    return dict(kind=kind, n=_log_int(rng, 2000, 1 << 17) | 1, phi=round(rng.uniform(0.1, 0.3), 3))


# ------------------------------------------------------------------ inputs

def _ao_cell(c):
    box = 21.0 if (c["n"], c["phi"]) == (4000, 0.2262) else (c["n"] * math.pi / 6.0 / c["phi"]) ** (1 / 3)
    return box, init.rsa_native(c["n"], box, 1.0, seed=c["seed"]).reshape(-1)


def _force(c):
    """The force, kT, dt and preferred skin of a case."""
    if c["force"] == "LJ":
        return psim.make_force("LJ", LJ_RC, kT=LJ_KT, well_depth=1.0 / LJ_KT, lj_num=6), LJ_KT, LJ_DT
    if c["force"] == "GEL":
        return pbatch.ao_params(psim, 6.0, 0.08), 1.0, 0.001
    if c["force"] == "PLUGIN":
        return psim.load_plugin(psim.Config(PLUGIN_CFG)), 1.0, 0.001
    return psim.make_force("AO", 1.1, kT=1.0, well_depth=0.25), 1.0, 0.001


def _single(c):
    """box, cells a side, positions and velocities of a one-system case.  The
    liquid starts as an FCC lattice with every site displaced (and, for a size
    that is no 4 k^3, random vacancies); the colloids by random sequential
    addition."""
    n, rng = c["n"], np.random.default_rng(c["seed"])
    force, kT, _ = _force(c)
    rc = force.max_cutoff()
    if c["force"] == "LJ":
        k = int(math.ceil((n / 4.0) ** (1 / 3) - 1e-9))
        a = (4.0 / 0.8) ** (1 / 3)
        box = k * a
        pos = init.fcc(k, a).reshape(-1, 3)
        if len(pos) > n:
            pos = pos[np.sort(rng.permutation(len(pos))[:n])]
        pos = np.mod(pos + rng.uniform(-0.1, 0.1, pos.shape), box).reshape(-1)
    else:
        box, pos = _ao_cell(c)
    want = 0.4 if c["skin"] < 0 else c["skin"]
    edge = max(rc + want, 1.2 if c["force"] == "GEL" else rc)
    scale = min(256, max(3, int(box / edge)))
    vel = init.maxwell(n, kT, seed=c["seed"]).reshape(-1)
    return box, scale, pos, vel


def _pinned(n, dtype=torch.float64):
    return torch.empty(n, dtype=dtype, pin_memory=True).numpy()


def _grad_inputs(c):
    box = (c["n"] * math.pi / 6.0 / c["phi"]) ** (1 / 3)
    pos = init.rsa_native(c["n"], box, 1.0, seed=c["seed"]).reshape(-1)
    vel = init.maxwell(c["n"], 1.0, seed=c["seed"]).reshape(-1)
    scale = max(3, int(box / 3.1))
    p, _ = padj.plugin_params(3.0, 0.1, 10.0, 4.0, **(dict(lj_epsilon=0.5, lj_sigma=0.97, lj_n=6,
                                                           lj_cutoff=2.5) if c["lj"] else {}))
    r = ADJ_RANGE[0] + (np.arange(ADJ_BINS) + 0.5) * (ADJ_RANGE[1] - ADJ_RANGE[0]) / ADJ_BINS
    target = (1.0 - np.exp(-(r / 1.05) ** 12)) * (1.0 + 0.4 * np.exp(-((r - 1.15) / 0.2) ** 2))
    return box, scale, pos, vel, p, target


def _replicas(c):
    draws = [dict(d, seed=(c["seed"] + 7 * k) & 0x3fffffff)
             for k, d in enumerate(pbatch.c2_draws(c["replicas"], seed=c["sweep"]))]
    pos, vel = pbatch.states(draws)
    return draws, pos, vel


def prepare(case, seed):
    c = dict(case, seed=1 + seed % (1 << 30))
    prec = psim.PRECISION_MIXED if c.get("form") == "mixed" else psim.PRECISION_FP64
    if c["kind"] == "system":
        force, kT, dt = _force(c)
        box, scale, pos, vel = _single(c)
        g = psim.geometry(c["n"], box, box / scale, scale)
        s = psim.System(g, force, gamma=1.0, dt=dt, kT=kT, seed=c["seed"], precision=prec,
                        skin="auto" if c["skin"] < 0 else c["skin"])
        s.upload(pos, np.full(c["n"], 0.5), vel=vel)
        return dict(c, s=s, frame=_pinned(3 * c["n"]))
    if c["kind"] == "batch":
        draws, pos, vel = _replicas(c)
        b = psim.Batch(pbatch.replicas(psim, draws, skin=c["skin"]), gamma=1.0, dt=0.001, kT=1.0,
                       precision=prec, skin=c["skin"])
        b.upload(pos, np.full(b.n, 0.5), vel=vel)
        return dict(c, s=b, frame=_pinned(3 * b.n))
    if c["kind"] == "host":
        force, kT, dt = _force(c)
        box, scale, pos, vel = _single(c)
        n, cells = c["n"], scale ** 3
        new = _pinned if c["pinned"] else (lambda m, t=torch.float64: torch.empty(m, dtype=t).numpy())
        st = {k: new(3 * n) for k in ("pos", "pos0", "vel", "frc", "frc0", "f")}
        st["pos"][:], st["pos0"][:], st["vel"][:] = pos, pos, vel
        for k in ("frc", "frc0", "f"):
            st[k][:] = 0.0
        mass, rad = new(n), new(n)
        mass[:], rad[:] = 1.0, 0.5
        out = (new(2 * n, torch.int32), new(2 * cells, torch.int32).view(np.uint32), new(4 * n))
        g = psim.geometry(n, box, box / scale, scale)
        psim.set_force_list_skin(c["skin"])
        psim.cells_build(g, st["pos"], rad, out=out)
        return dict(c, st=st, mass=mass, rad=rad, cells=out, g=g, p=force, prec=prec, dt=dt, t=0.0,
                    it=psim.Integrator(n, gamma=1.0, dt=dt, kT=kT, seed=c["seed"]))
    if c["kind"] == "grad":
        box, scale, pos, vel, p, target = _grad_inputs(c)
        a = padj.Adjoint(psim.geometry(c["n"], box, box / scale, scale), c["steps"], dt=0.001,
                         seed=c["seed"], checkpoint_every=c["every"], sample_every=10,
                         r_min=ADJ_RANGE[0], r_max=ADJ_RANGE[1], n_bins=ADJ_BINS)
        return dict(c, a=a, p=p, pos=pos, vel=vel, target=target)
    box, pos = _ao_cell(c)
    force = pbatch.ao_params(psim, 6.0, 0.08)
    scale = min(256, int(box / 1.5))
    s = psim.System(psim.geometry(c["n"], box, box / scale, scale), force, seed=c["seed"],
                    precision=psim.PRECISION_MIXED, skin="auto")
    s.upload(pos, np.full(c["n"], 0.5), vel=init.maxwell(c["n"], 1.0, seed=c["seed"]).reshape(-1))
    return dict(c, s=s)


# ------------------------------------------------------------------ one pass

def run(state):
    c = state
    if c["kind"] in ("system", "batch"):
        s = c["s"]
        if c["form"] == "fp64":
            s.step(c["steps"])
            return s.download()
        s.step_async(c["steps"])
        s.snapshot_async(c["frame"])
        s.sync()
        s.snapshot_wait()
        return {"pos": c["frame"]}
    if c["kind"] == "host":
        st, out, box = c["st"], c["cells"], c["g"].box_size
        for _ in range(c["steps"]):
            psim.force_evaluate(c["p"], c["g"], out[2], out[0], out[1], precision=c["prec"],
                                out=st["f"])
            c["it"].next_system(c["t"], box, st["pos"], st["pos0"], st["vel"], st["frc"],
                                st["frc0"], c["mass"], particle_force=st["f"])
            psim.cells_build(c["g"], st["pos"], c["rad"], out=out)
            c["t"] += c["dt"]
        return {"pos": st["pos"], "pos0": st["pos0"], "frc": st["frc"], "frc0": st["frc0"],
                "hash_index": out[0], "cells": out[1].view(np.int32), "sorted": out[2]}
    if c["kind"] == "grad":
        loss, g, grad, gp = c["a"].gradient(c["p"], c["pos"], c["target"], vel0=c["vel"], wrt_pos=True)
        return {"loss": loss, "g": g, "grad": grad, "grad_pos": gp}
    s = c["s"]
    u, w = s.energy()
    coor, total = s.interactions(1.2)
    root, groups, _ = s.clusters(1.2, 4)
    return {"energy": u, "virial": w, "g": s.rdf(0.8, 1.48, 100), "coor": coor, "total": total,
            "root": root, "clusters": len(groups), "temperature": s.temperature()}


def work(case):
    """Bytes: every state array of a step read and written once (host arrays
    included).  Flops: 30 per ordered pair in range and 60 per update."""
    c = case
    if c["kind"] in ("system", "host"):
        rc, rho = {"LJ": (2.5, 0.8), "PLUGIN": (2.5, 6 / math.pi * c["phi"]),
                   "GEL": (1.08, 6 / math.pi * c["phi"]), "AO": (1.1, 6 / math.pi * c["phi"])}[c["force"]]
        pairs = 4 / 3 * math.pi * rc ** 3 * rho
        # device state: x, x0, noise memory, force in and out, tag and 1/m; the
        # host loop: cells, positions and forces over the link (bench.py's count)
        per = 204 if c["kind"] == "system" else 112 + 96 + 24 + 96 + 40 + 32
        return {"bytes": per * c["n"] * c["steps"], "flops": (30 * pairs + 60) * c["n"] * c["steps"]}
    if c["kind"] == "batch":
        n = sum(d["n"] for d in pbatch.c2_draws(c["replicas"], seed=c["sweep"]))
        return {"bytes": 204 * n * c["steps"], "flops": (30 * 2.5 + 60) * n * c["steps"]}
    rho = 6 / math.pi * c["phi"]
    if c["kind"] == "grad":
        # the forward twice (checkpoints) and the reverse once: positions, forces
        # and multipliers in and out; 50 flops a pair forward, 150 back
        pairs = 4 / 3 * math.pi * 27 * rho
        return {"bytes": (2 * 144 + 168) * c["n"] * c["steps"],
                "flops": (2 * 50 + 150) * pairs * c["n"] * c["steps"]}
    pairs = 4 / 3 * math.pi * 1.48 ** 3 * rho
    return {"bytes": 4 * 28 * c["n"], "flops": 4 * 10 * pairs * c["n"]}


# ------------------------------------------- the same physics in plain FP64

def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _pairs(x, L, r):
    """Unordered pairs (i, j) closer than r of positions x (n, 3) in a periodic
    box: a cell grid's half stencil, candidates tested offset by offset."""
    n, s = len(x), int(L / r)
    if s < 3:
        i, j = torch.triu_indices(n, n, 1, device=x.device)
        d = x[j] - x[i]
        d -= L * torch.round(d / L)
        k = (d * d).sum(1) < r * r
        return i[k], j[k]
    w = torch.remainder(x, L)
    c = torch.clamp((w * (s / L)).long(), max=s - 1)
    key = c[:, 0] + s * (c[:, 1] + s * c[:, 2])
    order = torch.argsort(key)
    count = torch.bincount(key, minlength=s ** 3)
    start = torch.cumsum(count, 0) - count
    idx = torch.arange(n, device=x.device)
    found = []
    for dx, dy, dz in [(0, 0, 0)] + [(a, b, e) for e in (-1, 0, 1) for b in (-1, 0, 1)
                                     for a in (-1, 0, 1) if (e, b, a) > (0, 0, 0)]:
        o = torch.remainder(c + torch.tensor([dx, dy, dz], device=x.device), s)
        k = o[:, 0] + s * (o[:, 1] + s * o[:, 2])
        m = count[k]
        i = torch.repeat_interleave(idx, m)
        first = torch.repeat_interleave(start[k] - (torch.cumsum(m, 0) - m), m)
        j = order[first + torch.arange(len(i), device=x.device)]
        if (dx, dy, dz) == (0, 0, 0):
            keep = i < j
            i, j = i[keep], j[keep]
        d = w[j] - w[i]
        d -= L * torch.round(d / L)
        keep = (d * d).sum(1) < r * r
        found.append((i[keep], j[keep]))
    return torch.cat([f[0] for f in found]), torch.cat([f[1] for f in found])


def _mulhilo(a, b):
    t = a * (b >> 16) + ((a * (b & 0xffff)) >> 16)
    return t >> 16, (a * b) & 0xffffffff


def _gauss6(seed, tag, step):
    """Philox4x32-10 (Salmon et al., SC'11) and the Box-Muller transform."""
    def four(group):
        c = [torch.full_like(tag, step), torch.full_like(tag, group), tag, torch.zeros_like(tag)]
        k0, k1 = seed, 0x5053494D
        for _ in range(10):
            h0, l0 = _mulhilo(0xD2511F53, c[0])
            h1, l1 = _mulhilo(0xCD9E8D57, c[2])
            c = [h1 ^ c[1] ^ k0, l1, h0 ^ c[3] ^ k1, l0]
            k0, k1 = (k0 + 0x9E3779B9) & 0xffffffff, (k1 + 0xBB67AE85) & 0xffffffff
        return c

    def two(a, b):
        rad = torch.sqrt(-2.0 * torch.log(((a >> 8) + 1).double() / (1 << 24)))
        ang = 2.0 * math.pi * (b >> 8).double() / (1 << 24)
        return [rad * torch.cos(ang), rad * torch.sin(ang)]

    a, b = four(0), four(1)
    return torch.stack(two(a[0], a[1]) + two(a[2], a[3]) + two(b[0], b[1]), 1)


def _vgb(dt, kT, y_gamma=1.0):
    """van Gunsteren & Berendsen's coefficients at friction gamma (>= 0.05)."""
    y = y_gamma * dt
    e0, ep = math.exp(-y), math.exp(y)
    a1 = 1 - e0
    s1 = math.sqrt(kT * (2 * y - 3 + 4 * e0 - math.exp(-2 * y))) / y_gamma
    s2 = math.sqrt(-kT * (-2 * y - 3 + 4 * ep - math.exp(2 * y))) / y_gamma
    corr = kT / y_gamma ** 2 * (ep - 2 * y - e0) / (s1 * s2)
    return dict(e0=e0, c1=a1 / y, c2=(0.5 * y * (1 + e0) - a1) / (y * y), c3=(y - a1) / (y * y),
                s1=s1, s2=s2, corr=corr, dev=math.sqrt(1 - corr * corr))


def _ao_c(kT, wd, rc):
    a1 = -kT * wd * (rc / (rc - 1)) ** 3
    return a1 * 3 / (2 * rc), -3 * a1 / (2 * rc ** 3)


def _ao_f(r, c1, c2):
    return -(36 * r ** -38 + c1 / r + c2 * r)


def _lj_f(r, eps, n, yuk, lam):
    L = r ** -n
    return -eps * ((2 * L - 1) * 4 * n * L / r + yuk * torch.exp(-r / lam) * (lam + r) / r ** 2)


def _trajectory(x, v, box, seeds, tags, steps, dt, kT, listing, fnet, rcut, skin=0.3):
    """`steps` vGB steps in wrapped coordinates: x, x0, F and F0 at the end.
    box, seeds: a number or one per particle; listing(x, r): pairs within r."""
    c = _vgb(dt, kT)
    one = not torch.is_tensor(box)
    x0, F0, mem, built = x.clone(), torch.zeros_like(x), torch.zeros_like(x), None
    F = F0
    for t in range(steps):
        if built is not None:
            m = x - built
            m -= box * torch.round(m / box)
        if built is None or float((m * m).sum(1).max()) > (0.5 * skin) ** 2:
            i, j = listing(x, skin)
            built = x.clone()
        d = x[j] - x[i]
        bp = box if one else box[i]
        d -= bp * torch.round(d / bp)
        r = torch.sqrt((d * d).sum(1))
        rc = rcut if not torch.is_tensor(rcut) else rcut[i]
        f = torch.where(r < rc, fnet(r, i), torch.zeros_like(r)) / r
        d = d * f[:, None]
        F0, F = F, torch.zeros_like(x).index_add_(0, i, d).index_add_(0, j, -d)
        xi = _gauss6(seeds, tags, t)
        if t == 0:
            mem = xi[:, :3]
            nw = x + v * c["c1"] * dt + F * c["c3"] * dt * dt + c["s1"] * mem
        else:
            mc = c["s2"] * (c["corr"] * mem + c["dev"] * xi[:, :3])
            mem = xi[:, 3:]
            nw = x + c["e0"] * (x - x0) + dt * dt * (c["c1"] * F + c["c2"] * (F - F0)) + c["s1"] * mem + c["e0"] * mc
        xn = torch.where(nw < 0, nw + box, torch.where(nw >= box, nw - box, nw))
        m = xn - x
        x0 = torch.where(m.abs() > box / 2, torch.where(m < 0, x - box, x + box), x)
        x = xn
    return x, x0, F, F0


def _exact_single(c):
    box, scale, pos, vel = _single(c)
    force, kT, dt = _force(c)
    p, rc = force.as_dict(), force.max_cutoff()
    x = torch.tensor(pos, device=_dev()).reshape(-1, 3)
    v = torch.tensor(vel, device=_dev()).reshape(-1, 3)
    if p["kind"] == "AO":
        c1, c2 = _ao_c(p["kT"], p["well_depth"], p["cutoff"])
        fnet = lambda r, i: _ao_f(r, c1, c2)  # noqa: E731
    else:
        fnet = lambda r, i: _lj_f(r, p["kT"] * p["well_depth"], p["lj_num"], p["yukawa_strength"],  # noqa: E731
                                  p["debye_length"])
    out = _trajectory(x, v, box, c["seed"], torch.arange(c["n"], device=x.device), c["steps"], dt, kT,
                      lambda y, s: _pairs(y, box, rc + s), fnet, rc)
    return [a.reshape(-1).cpu().numpy() for a in out] + [vel]


def _exact_batch(c):
    draws, pos, vel = _replicas(c)
    dev = _dev()
    n = [d["n"] for d in draws]
    off = np.concatenate([[0], np.cumsum(n)])
    rep = torch.repeat_interleave(torch.arange(len(n), device=dev), torch.tensor(n, device=dev))
    col = lambda f: torch.tensor([f(d) for d in draws], device=dev, dtype=torch.float64)[rep]  # noqa: E731
    wd = lambda d: d["contact_kT"] * d["q"] / (1.5 + d["q"])  # noqa: E731
    c1 = col(lambda d: _ao_c(1.0, wd(d), 1 + d["q"])[0])
    c2 = col(lambda d: _ao_c(1.0, wd(d), 1 + d["q"])[1])
    x = torch.tensor(pos, device=dev).reshape(-1, 3)

    def listing(y, s):
        got = [_pairs(y[off[k]:off[k + 1]], d["box"], 1 + d["q"] + s) for k, d in enumerate(draws)]
        return [torch.cat([g[a] + int(off[k]) for k, g in enumerate(got)]) for a in (0, 1)]

    seeds = torch.tensor([d["seed"] & 0xffffffff for d in draws], device=dev)[rep]
    tags = torch.arange(len(rep), device=dev) - torch.tensor(off[:-1], device=dev)[rep]
    got = _trajectory(x, torch.tensor(vel, device=dev).reshape(-1, 3), col(lambda d: d["box"])[:, None],
                      seeds, tags, c["steps"], 0.001, 1.0, listing,
                      lambda r, i: _ao_f(r, c1[i], c2[i]), col(lambda d: 1 + d["q"]))
    return got[0].reshape(-1).cpu().numpy()


def _exact_grad(c):
    box, _, pos, vel, p, target = _grad_inputs(c)
    dev, dt, n, T = _dev(), 0.001, c["n"], c["steps"]
    leaf = lambda v: torch.tensor(v, device=dev, dtype=torch.float64, requires_grad=True)  # noqa: E731
    th = [leaf(v) for v in (p.ao_well_depth, p.ao_range, p.yuk_amplitude, p.yuk_length, p.lj_epsilon, p.lj_sigma)]
    c1, c2 = _ao_c(1.0, th[0], th[1])
    x = x_first = torch.tensor(pos, device=dev).reshape(-1, 3).requires_grad_(True)
    v = torch.tensor(vel, device=dev).reshape(-1, 3)
    q, tags = _vgb(dt, 1.0), torch.arange(n, device=dev)
    dr = (ADJ_RANGE[1] - ADJ_RANGE[0]) / ADJ_BINS
    sig, reach = dr, 4 * dr + ADJ_RANGE[1]
    rb = ADJ_RANGE[0] + (torch.arange(ADJ_BINS, device=dev, dtype=torch.float64) + 0.5) * dr
    hist = torch.zeros(ADJ_BINS, device=dev, dtype=torch.float64)
    xp, F, mem, built = x, torch.zeros_like(x), None, None
    for t in range(T + 1):
        if built is None or float((x.detach() - built).square().sum(1).max()) > 0.15 ** 2:
            built = x.detach().clone()
            i, j = _pairs(built, box, reach + 0.3)
        d = x[j] - x[i]
        d = d - box * torch.round(d.detach() / box)
        r = torch.sqrt((d * d).sum(1))
        if t > 0 and t % 10 == 0:
            near = r < reach
            rr = r[near]
            b0 = torch.floor((rr.detach() - ADJ_RANGE[0]) / dr).long()
            for k in range(-5, 6):
                b = b0 + k
                ok = (b >= 0) & (b < ADJ_BINS)
                z = (rr[ok] - rb[b[ok]]) / sig
                hist = hist.index_add(0, b[ok], 2 * dr / (math.sqrt(2 * math.pi) * sig) * torch.exp(-0.5 * z * z))
        if t == T:
            break
        f = -th[2] * torch.exp(-r / th[3]) * (th[3] + r) / r ** 2 * (r < p.yuk_cutoff)
        k = (r < p.ao_cutoff).nonzero()[:, 0]
        f = f.index_add(0, k, _ao_f(r[k], c1, c2))
        if p.lj_cutoff > 0:
            L = (th[5] / r) ** p.lj_n
            f = f - th[4] * (2 * L - 1) * 4 * p.lj_n * L / r * (r < p.lj_cutoff)
        d = d * (f / r)[:, None]
        F0, F = F, torch.zeros_like(x).index_add(0, i, d).index_add(0, j, -d)
        xi = _gauss6(c["seed"], tags, t)
        if t == 0:
            mem = xi[:, :3]
            xn = x + v * q["c1"] * dt + F * q["c3"] * dt * dt + q["s1"] * mem
        else:
            mc = q["s2"] * (q["corr"] * mem + q["dev"] * xi[:, :3])
            mem = xi[:, 3:]
            xn = (1 + q["e0"]) * x - q["e0"] * xp + dt * dt * ((q["c1"] + q["c2"]) * F - q["c2"] * F0) \
                + q["s1"] * mem + q["e0"] * mc
        xp, x = x, xn
    g = hist / ((T // 10) * n * (n / box ** 3) * 4 * math.pi * rb * rb * dr)
    loss = (g - torch.tensor(target, device=dev)).square().sum()
    used = th if p.lj_cutoff > 0 else th[:4]
    got = torch.autograd.grad(loss, used + [x_first])
    grad = np.zeros(6)
    grad[:len(used)] = [float(a) for a in got[:len(used)]]
    return {"loss": loss.item(), "g": g.detach().cpu().numpy(), "grad": grad,
            "grad_pos": got[-1].reshape(-1).cpu().numpy()}


def _exact_analysis(c):
    box, pos = _ao_cell(c)
    n, p = c["n"], pbatch.ao_params(psim, 6.0, 0.08).as_dict()
    x = torch.tensor(pos, device=_dev()).reshape(-1, 3)
    i, j = _pairs(x, box, 1.5)
    d = x[j] - x[i]
    d -= box * torch.round(d / box)
    r = torch.sqrt((d * d).sum(1))
    rc = p["cutoff"]
    c1, c2 = _ao_c(p["kT"], p["well_depth"], rc)
    s = r[r < rc]
    u = 36 / 37 * (s ** -37 - rc ** -37) + c1 * torch.log(rc / s) + 0.5 * c2 * (rc * rc - s * s)
    lo, hi = 0.8, 1.48
    h = torch.histc(r[(r >= lo) & (r < hi)], 100, lo, hi)
    e = lo + (hi - lo) / 100 * torch.arange(101, device=x.device, dtype=torch.float64)
    g = 2 * h / (n * n / box ** 3 * 4 / 3 * math.pi * (e[1:] ** 3 - e[:-1] ** 3))
    v = init.maxwell(n, 1.0, seed=c["seed"])
    return {"energy": float(u.sum()) / n, "virial": -float((_ao_f(s, c1, c2) * s).sum()) / n,
            "g": g.cpu().numpy(), "coor": None, "total": None, "root": None, "clusters": None,
            "temperature": float((v * v).sum() / (3 * n))}


def exact(case, seed):
    c = dict(case, seed=1 + seed % (1 << 30))
    if c["kind"] == "grad":
        return _exact_grad(c)
    if c["kind"] == "analysis":
        return _exact_analysis(c)
    if c["kind"] == "batch":
        return {"pos": _exact_batch(c)}
    pos, pos0, frc, frc0, vel = _exact_single(c)
    if c["kind"] == "host":
        return {"pos": pos, "pos0": pos0, "frc": frc, "frc0": frc0, "hash_index": None, "cells": None,
                "sorted": None}
    if c["form"] == "mixed":
        return {"pos": pos}
    return {"pos": pos, "pos0": pos0, "vel": vel, "frc": frc, "frc0": frc0}

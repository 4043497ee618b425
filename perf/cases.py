"""Timed cases: the evaluations, MD steps and served requests that users of this library run.

``listed()`` names them, ``draw(rng)`` gives further ones of the same ranges, ``prepare`` makes a case's
inputs and handles, ``run`` is one pass through the public API and ``exact`` its outputs in FP64 from a
direct Ewald sum (and a velocity-Verlet loop over it) that shares no code with the library.

Systems are the library's two workloads: rock-salt ions on a jittered lattice (spacing 1, r_c 3, list skin
0.4) and rigid three-site water (33.4 molecules per nm^3, r_c 0.9 nm, skin 0.1). Kinds:

  eval   one system, forces and totals over a caller's HOOMD-layout neighbour list (FP32 or FP64)
  hoomd  the HOOMD ForceCompute contract (per-particle virial, external terms) with excluded pairs
  md     a batch of systems: pair-list build, one evaluation and NVE steps (rigid molecules for water)
  md64   one FP64 system with the Lennard-Jones core: list build, one evaluation and NVE steps
  serve  a burst of requests in host memory through the continuous-batching server

The FP32 mode's totals are FP64 accumulators of FP32 terms; ``run`` returns them in FP32, the precision of
what they sum.
"""
import math
import random

import numpy as np
import torch

from esp_hoomd_b200 import native

INV_4PI = 1.0 / (4.0 * math.pi)
RS_RCUT, RS_SKIN, RS_CAP = 3.0, 0.4, 256
W_RCUT, W_SKIN, W_CAP = 0.9, 0.1, 640
W_DENSITY, W_QO, W_OH, W_ANGLE = 33.4, -0.8476, 0.1, 109.47
W_HH = 2.0 * W_OH * math.sin(math.radians(W_ANGLE / 2.0))
LJ = (1.0, 0.9, 2.5)
DT = 0.002
DEV = "cuda"
# support -> relative force error target, the pairs in use (6/8/10 are the water accuracy sweep's)
TARGET = {6: 1e-3, 7: 1e-4, 8: 1e-5, 9: 1e-6, 10: 1e-7}


def listed():
    return [
        # the smallest call: one evaluation of 512 ions, latency bound (the plain path on a small box)
        {"name": "ions-512", "kind": "eval", "system": "rocksalt", "ex": 8, "ey": 8, "ez": 8, "order": 8,
         "precision": "f32", "virial": True},
        # a non-cubic box, an odd support and meshes of mixed radix, forces and energy only
        {"name": "ions-ragged", "kind": "eval", "system": "rocksalt", "ex": 18, "ey": 26, "ez": 34, "order": 7,
         "precision": "f32", "virial": False},
        # the water accuracy sweep (32,768 molecules): a coarse target, the usual one, and FP64 at 1e-7
        {"name": "water-1e-3", "kind": "eval", "system": "water", "molecules": 32768, "order": 6, "precision": "f32",
         "virial": False},
        {"name": "water-1e-5", "kind": "eval", "system": "water", "molecules": 32768, "order": 8, "precision": "f32",
         "virial": True},
        {"name": "water-f64", "kind": "eval", "system": "water", "molecules": 32768, "order": 10, "precision": "f64",
         "virial": True},
        # a HOOMD force compute on a molecular system: intramolecular exclusions, per-particle virial
        {"name": "hoomd-water", "kind": "hoomd", "system": "water", "molecules": 4321, "order": 8},
        # the plain FP64 case with the Lennard-Jones core, between two list rebuilds
        {"name": "md-f64-1000", "kind": "md64", "edge": 10, "mesh": 32, "steps": 10},
        # many small systems: few particles per launch, every stage short
        {"name": "md-small", "kind": "md", "system": "rocksalt", "systems": 32, "lo": 8, "hi": 14, "order": 8,
         "steps": 10},
        # rigid water replicas (SETTLE / RATTLE in the steps)
        {"name": "md-water", "kind": "md", "system": "water", "systems": 6, "lo": 1000, "hi": 6000, "order": 8,
         "steps": 10},
        # the headline batch: 256 rock-salt systems, n even in 8..40
        {"name": "md-batch256", "kind": "md", "system": "rocksalt", "systems": 256, "lo": 8, "hi": 40, "order": 8,
         "steps": 10},
        # the scale-up: one system of 10^6 ions (mesh 200^3, the per-line FFT passes)
        {"name": "md-million", "kind": "md", "system": "rocksalt", "systems": 1, "lo": 100, "hi": 100, "order": 8,
         "steps": 10},
        # served requests, half rock-salt and half rigid water, host memory in and out
        {"name": "serve-burst", "kind": "serve", "requests": 40, "lo": 8, "hi": 48, "mol_lo": 1000, "mol_hi": 12000,
         "steps": 10},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["eval", "eval", "eval", "hoomd", "md64", "md", "md", "serve"])
    if kind == "eval":
        f64 = rng.random() < 0.3
        c = {"kind": "eval", "system": rng.choice(["rocksalt", "water"]), "order": rng.choice([6, 7, 8, 9, 10]),
             "precision": "f64" if f64 else "f32", "virial": rng.random() < 0.5}
        if c["system"] == "water":
            c["molecules"] = _log_int(rng, 1000, 32768)
        else:
            for a in ("ex", "ey", "ez"):
                c[a] = 2 * _log_int(rng, 4, 28)
        return c
    if kind == "hoomd":
        return {"kind": "hoomd", "system": "water", "molecules": _log_int(rng, 1000, 20000),
                "order": rng.choice([6, 8, 8])}
    if kind == "md64":
        return {"kind": "md64", "edge": 2 * rng.randint(4, 8), "mesh": rng.choice([27, 30, 32, 36, 40]),
                "steps": rng.randint(5, 20)}
    if kind == "md":
        if rng.random() < 0.35:
            return {"kind": "md", "system": "water", "systems": _log_int(rng, 1, 12), "lo": 1000,
                    "hi": _log_int(rng, 1200, 9000), "order": rng.choice([6, 8, 8]), "steps": rng.randint(3, 12)}
        return {"kind": "md", "system": "rocksalt", "systems": _log_int(rng, 1, 160), "lo": 8,
                "hi": 2 * rng.randint(5, 18), "order": rng.choice([6, 8, 8, 8]), "steps": rng.randint(3, 12)}
    return {"kind": "serve", "requests": _log_int(rng, 4, 40), "lo": 8, "hi": 2 * rng.randint(6, 24), "mol_lo": 1000,
            "mol_hi": _log_int(rng, 1200, 12000), "steps": rng.randint(2, 10)}


# ------------------------------------------------------------------------------------------------ systems
def _sizes(case):
    """The sizes of a batch's (or a burst's) systems: fixed by the case, not by the seed of its inputs."""
    rng = random.Random(1004)
    if case["kind"] == "serve":
        out = []
        for i in range(case["requests"]):
            out.append(("rocksalt", 2 * rng.randint(case["lo"] // 2, case["hi"] // 2)) if i % 2 == 0 else
                       ("water", rng.randint(case["mol_lo"], case["mol_hi"])))
        return out
    if case["system"] == "water":
        return [("water", rng.randint(case["lo"], case["hi"])) for _ in range(case["systems"])]
    return [("rocksalt", 2 * rng.randint(case["lo"] // 2, case["hi"] // 2)) for _ in range(case["systems"])]


def _rocksalt(shape, g):
    """Jittered simple-cubic lattice of alternating unit charges: positions, charges, velocities, box."""
    ix = torch.stack(torch.meshgrid(*[torch.arange(n, device=DEV) for n in shape], indexing="ij"), -1).reshape(-1, 3)
    jit = torch.rand(ix.shape, generator=g, device=DEV, dtype=torch.float64) * 0.2 - 0.1
    pos = ix.double() + 0.5 + jit
    q = 1.0 - 2.0 * (ix.sum(1) % 2).double()
    vel = torch.randn(ix.shape, generator=g, device=DEV, dtype=torch.float64)
    vel -= vel.mean(0)
    return pos, q, vel, tuple(float(n) for n in shape)


def _water(n_mol, g):
    """Rigid water on a jittered cubic lattice, random orientations, at rest: positions, charges, velocities, box."""
    m = int(math.ceil(n_mol ** (1.0 / 3.0) - 1e-9))
    L = (n_mol / W_DENSITY) ** (1.0 / 3.0)
    a = L / m
    site = torch.sort(torch.randperm(m ** 3, generator=g, device=DEV)[:n_mol])[0]
    c = torch.stack([site // (m * m), (site // m) % m, site % m], -1).double().add(0.5).mul(a)
    c += (torch.rand(c.shape, generator=g, device=DEV, dtype=torch.float64) - 0.5) * 0.1 * a
    half = math.radians(W_ANGLE) / 2.0
    body = torch.tensor([[0.0, 0.0, 0.0], [W_OH * math.sin(half), 0.0, W_OH * math.cos(half)],
                         [-W_OH * math.sin(half), 0.0, W_OH * math.cos(half)]], dtype=torch.float64, device=DEV)
    body -= body.mean(0)
    qt = torch.randn((n_mol, 4), generator=g, device=DEV, dtype=torch.float64)
    qt /= qt.norm(dim=1, keepdim=True)
    w, v = qt[:, None, :1], qt[:, None, 1:].expand(-1, 3, -1)
    b = body[None].expand(n_mol, -1, -1)
    t = 2.0 * torch.cross(v, b, dim=2)
    pos = c[:, None, :] + b + w * t + torch.cross(v, t, dim=2)
    pos = torch.remainder(pos.reshape(-1, 3), L)
    q = torch.tensor([W_QO, -W_QO / 2, -W_QO / 2], dtype=torch.float64, device=DEV).repeat(n_mol)
    return pos, q, torch.zeros_like(pos), (L, L, L)


def _system(kind, size, g):
    return _water(size, g) if kind == "water" else _rocksalt(size if isinstance(size, tuple) else (size,) * 3, g)


def _cutoffs(system):
    return (W_RCUT, W_SKIN, W_CAP) if system == "water" else (RS_RCUT, RS_SKIN, RS_CAP)


def _generator(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _vec4(xyz, w, dtype):
    out = torch.empty((xyz.shape[0], 4), dtype=dtype, device=DEV)
    out[:, :3] = xyz
    out[:, 3] = w
    return out


def _masses(system, n):
    return torch.tensor([16.0, 1.0, 1.0], device=DEV).repeat(n // 3) if system == "water" else torch.ones(n, device=DEV)


def _inputs(case, seed):
    """What prepare() and exact() share: the systems of the case as FP64 tensors, rounded as the mode stores them."""
    g = _generator(seed)
    if case["kind"] in ("md", "serve"):
        systems = [(k, _system(k, n, g)) for k, n in _sizes(case)]
    elif case["kind"] == "md64":
        systems = [("rocksalt", _rocksalt((case["edge"],) * 3, g))]
    elif case["system"] == "water":
        systems = [("water", _water(case["molecules"], g))]
    else:
        systems = [("rocksalt", _rocksalt((case["ex"], case["ey"], case["ez"]), g))]
    if case["kind"] == "md64" or case.get("precision") == "f64":
        return systems
    return [(k, (p.float().double(), q.float().double(), v.float().double(), box)) for k, (p, q, v, box) in systems]


def _neighbours(params, pos32, box, rlist, cap, exclusions=None):
    n = pos32.shape[0]
    b = native.Batch(params, [n], [box])
    if exclusions is not None:
        b.set_exclusions(*exclusions, 2)
    head = torch.zeros(n, dtype=torch.int32, device=DEV)
    nn = torch.zeros(n, dtype=torch.int32, device=DEV)
    nl = torch.zeros(n * cap, dtype=torch.int32, device=DEV)
    b.build_nlist(pos32, rlist, cap, head, nn, nl)
    b.nlist_check()
    return b, (head, nn, nl)


def _exclusions(n):
    """Intramolecular exclusions of (O, H, H) triples: each atom excludes the other two."""
    i = torch.arange(n, device=DEV)
    base, k = i - i % 3, i % 3
    ex = torch.stack([base + (k + 1) % 3, base + (k + 2) % 3], 1).sort(1)[0]
    return torch.full((n,), 2, dtype=torch.int32, device=DEV), ex.int().contiguous()


# ------------------------------------------------------------------------------------------------ passes
def prepare(case, seed):
    systems = _inputs(case, seed)
    kind = case["kind"]
    st = {"kind": kind, "case": case}
    if kind in ("eval", "hoomd"):
        name, (pos, q, _, box) = systems[0]
        rcut, skin, cap = _cutoffs(name)
        f64 = case.get("precision") == "f64"
        dt = torch.float64 if f64 else torch.float32
        n = pos.shape[0]
        order = case["order"]
        exclusions = _exclusions(n) if kind == "hoomd" else None
        builder, nlist = _neighbours(native.make_params(order=8, rcut=rcut), _vec4(pos, 0.0, torch.float32), box,
                                     rcut + skin, cap, exclusions)
        builder.close()
        ctx = native.Context(native.make_params(order=order, rcut=rcut, target_error=TARGET[order],
                                                precision=int(f64)), box, n)
        st.update(ctx=ctx, nlist=nlist, f64=f64, pos=_vec4(pos, 0.0, dt), q=q.to(dt),
                  force=torch.zeros((n, 4), dtype=dt, device=DEV))
        if kind == "hoomd":
            ctx.set_exclusions(*exclusions, 2)
            st.update(virial=torch.zeros((6, n), device=DEV), ext=torch.zeros(7, dtype=torch.float64, device=DEV))
        else:
            tot = torch.zeros(7, dtype=torch.float64, device=DEV)
            st.update(tot=tot if case["virial"] else tot[:1], energy=tot[:1],
                      virial=tot[1:7] if case["virial"] else None)
        return st
    if kind == "md64":
        _, (pos, q, vel, box) = systems[0]
        n = pos.shape[0]
        mesh = (case["mesh"],) * 3
        lister, nlist = _neighbours(native.make_params(rcut=RS_RCUT), _vec4(pos, 0.0, torch.float32), box,
                                    RS_RCUT + RS_SKIN, RS_CAP)
        b = native.Batch(native.make_params(order=8, rcut=RS_RCUT, mesh=mesh, precision=1), [n], [box])
        pos0, vel0 = _vec4(pos, 0.0, torch.float64), _vec4(vel, 1.0, torch.float64)
        st.update(b=b, lister=lister, nlist=nlist, pos0=pos0, vel0=vel0, pos=pos0.clone(), vel=vel0.clone(), q=q,
                  force=torch.zeros_like(pos0), energy=torch.zeros(1, dtype=torch.float64, device=DEV),
                  e_lj=torch.zeros(1, dtype=torch.float64, device=DEV))
        return st
    if kind == "md":
        rcut, skin, cap = _cutoffs(case["system"])
        N = [s[0].shape[0] for _, s in systems]
        b = native.Batch(native.make_params(order=case["order"], rcut=rcut, target_error=TARGET[case["order"]]), N,
                         [s[3] for _, s in systems])
        if case["system"] == "water":
            b.set_rigid_water([0] * len(N), [n // 3 for n in N], W_OH, W_HH)
        pos0 = _vec4(torch.cat([s[0] for _, s in systems]), 0.0, torch.float32)
        vel0 = _vec4(torch.cat([s[2] for _, s in systems]), _masses(case["system"], sum(N)), torch.float32)
        st.update(b=b, rlist=rcut + skin, cap=cap, pos0=pos0, vel0=vel0, pos=pos0.clone(), vel=vel0.clone(),
                  q=torch.cat([s[1] for _, s in systems]).float(), force=torch.zeros_like(pos0),
                  energy=torch.zeros(len(N), dtype=torch.float64, device=DEV))
        return st
    # serve: page-locked host inputs, one output array of each kind that the requests' ranges share
    N = [s[0].shape[0] for _, s in systems]
    off = np.concatenate([[0], np.cumsum(N)]).tolist()
    pos = _vec4(torch.cat([s[0] for _, s in systems]), 0.0, torch.float32).cpu().pin_memory()
    mass = torch.cat([_masses(k, n) for (k, _), n in zip(systems, N)])
    vel = _vec4(torch.cat([s[2] for _, s in systems]), mass, torch.float32).cpu().pin_memory()
    q = torch.cat([s[1] for _, s in systems]).float().cpu().pin_memory()
    out_vel = torch.zeros((off[-1], 4)).pin_memory()
    out_force = torch.zeros((off[-1], 4)).pin_memory()
    out_energy = torch.zeros(len(N), dtype=torch.float64).pin_memory()
    srv = native.Server(native.make_params(order=8, target_error=1e-5), hbm_budget=6 << 30, max_systems=64,
                        max_particles=262144)
    srv.start()
    reqs = []
    for i, (k, s) in enumerate(systems):
        a, e = off[i], off[i + 1]
        rcut, skin, _ = _cutoffs(k)
        reqs.append(((pos[a:e], q[a:e], s[3], rcut),
                     dict(vel4=vel[a:e], nsteps=case["steps"], dt=DT, skin=skin, out_vel4=out_vel[a:e],
                          out_force4=out_force[a:e], out_energy=out_energy[i:i + 1],
                          rigid_water=(W_OH, W_HH) if k == "water" else None)))
    st.update(srv=srv, reqs=reqs, out=(out_vel, out_force, out_energy))
    return st


def run(st):
    kind, case = st["kind"], st["case"]
    if kind == "eval":
        if st["f64"]:
            st["ctx"].compute_f64(st["pos"], st["q"], st["force"], st["energy"], st["virial"], nlist=st["nlist"])
            return st["force"], st["tot"]
        st["ctx"].compute(st["pos"], st["q"], st["force"], st["energy"], st["virial"], nlist=st["nlist"])
        return st["force"], st["tot"].float()
    if kind == "hoomd":
        st["ctx"].compute_hoomd(st["pos"], st["q"], st["force"], st["virial"], st["ext"], nlist=st["nlist"])
        return st["force"], st["virial"], st["ext"].float()
    if kind == "md64":
        pos, vel, q, force, energy, e_lj, nl = (st[k] for k in ("pos", "vel", "q", "force", "energy", "e_lj", "nlist"))
        pos.copy_(st["pos0"])
        vel.copy_(st["vel0"])
        st["lister"].build_nlist(pos.float(), RS_RCUT + RS_SKIN, RS_CAP, *nl)
        st["b"].compute_f64(pos, q, force, energy, None, nlist=nl)
        e_lj.zero_()
        st["b"].lj(pos, nl, *LJ, force, e_lj)
        st["b"].md_run_f64(pos, vel, q, force, energy, None, nl, case["steps"], DT, lj=LJ)
        return pos, vel, force, energy
    if kind == "md":
        b, pos, vel, q, force, energy = (st[k] for k in ("b", "pos", "vel", "q", "force", "energy"))
        pos.copy_(st["pos0"])
        vel.copy_(st["vel0"])
        b.build_pairlist(pos, st["rlist"], st["cap"])
        b.compute(pos, q, force, energy, None)
        b.md_run(pos, vel, q, force, energy, None, None, case["steps"], DT)
        # positions are wrapped into the box: an atom at a face may come out at either end. The lattice keeps
        # the ions off the faces; water's positions show in its forces and velocities
        return (vel, force, energy.float()) if case["system"] == "water" else (pos, vel, force, energy.float())
    for args, kw in st["reqs"]:
        st["srv"].submit(*args, **kw)
    st["srv"].wait_all(60.0)
    out_vel, out_force, out_energy = st["out"]
    return out_vel, out_force, out_energy.float()


# ------------------------------------------------------------------------------------------------ work
def _mesh_points(box, rcut, order, mesh=None):
    """Mesh points of the planner's rule: h = pi r_c / kappa_N, the next 2/3/5-smooth length."""
    if mesh:
        return float(mesh) ** 3
    kn = {6: 11.5, 7: 14.0, 8: 18.5, 9: 22.0, 10: 26.0}[order]
    m = 1.0
    for L in box:
        n = max(order, math.ceil(L * kn / (math.pi * rcut)))
        while True:
            k = n
            for p in (2, 3, 5):
                while k % p == 0:
                    k //= p
            if k == 1:
                break
            n += 1
        m *= n
    return m


def _eval_work(kind, size, order, f64, virial, mesh=None, listed_rows=False):
    """(bytes, flops) of one evaluation: positions, charges and a caller's list read, the influence table read,
    forces written; arithmetic of the pairs inside r_c, the 2 P^3 taps and the two transforms."""
    rcut, skin, _ = _cutoffs(kind)
    if kind == "water":
        n = 3 * size
        box = ((size / W_DENSITY) ** (1.0 / 3.0),) * 3
    else:
        box = tuple(float(x) for x in (size if isinstance(size, tuple) else (size,) * 3))
        n = int(box[0] * box[1] * box[2])
    w = 8 if f64 else 4
    dens = n / (box[0] * box[1] * box[2])
    sphere = 4.0 / 3.0 * math.pi * dens
    m = _mesh_points(box, rcut, order, mesh)
    byts = n * 9 * w + m / 2 * w
    if listed_rows:
        byts += n * (8 + 4 * sphere * (rcut + skin) ** 3)
    flops = n * sphere * rcut ** 3 * (60 if virial else 45) + n * order ** 3 * 10 + 2 * 2.5 * m * math.log2(max(m, 2))
    return byts, flops


def work(case):
    kind = case["kind"]
    if kind in ("eval", "hoomd"):
        size = case["molecules"] if case["system"] == "water" else (case["ex"], case["ey"], case["ez"])
        b, f = _eval_work(case["system"], size, case["order"], case.get("precision") == "f64",
                          kind == "hoomd" or case["virial"], listed_rows=True)
        return {"bytes": b + (24 * 3 * case["molecules"] if kind == "hoomd" else 0), "flops": f}
    evals = case["steps"] + 1
    if kind == "md64":
        b, f = _eval_work("rocksalt", case["edge"], 8, True, False, case["mesh"])
        return {"bytes": evals * b, "flops": evals * f}
    b = f = 0.0
    for k, n in _sizes(case):
        bb, ff = _eval_work(k, n, case.get("order", 8), False, False)
        b, f = b + evals * bb, f + evals * ff
    return {"bytes": b, "flops": f}


# ------------------------------------------------------------------------------------------------ FP64 reference
def _ewald(pos, q, box):
    """Ewald sum of point charges, E = q_i q_j / 4 pi r: (forces, per-particle energies, virial). alpha r_e = 5.2 and
    the reciprocal sphere at exp(-27): truncation near 1e-12."""
    n, X = pos.shape[0], 5.2
    L = torch.tensor(box, dtype=torch.float64, device=pos.device)
    V, lmin = float(L.prod()), float(L.min())
    # cutoff by cost: candidates of the cell list against the reciprocal vectors
    best = None
    for frac in np.linspace(0.05, 0.5, 46):
        re = frac * lmin
        nk = np.prod([2 * X * X / re * x / math.pi + 1 for x in box]) / 2
        nc = [int(x / re) for x in box]
        cand = 27.0 * n / np.prod(nc) if min(nc) >= 3 else float(n)
        cost = n * (cand * 60.0 + 4.0 * nk)
        if best is None or cost < best[0]:
            best = (cost, re, nc)
    _, re, nc = best
    al = X / re
    F = torch.zeros_like(pos)
    phi = torch.zeros_like(q)
    W = torch.zeros((3, 3), dtype=torch.float64, device=pos.device)
    # real space: the particles of the 27 surrounding cells (or all)
    if min(nc) >= 3:
        nct = torch.tensor(nc, device=pos.device)
        ci = torch.minimum((pos / (L / nct)).long(), nct - 1)
        cell = (ci[:, 0] * nc[1] + ci[:, 1]) * nc[2] + ci[:, 2]
        order = torch.argsort(cell, stable=True)
        count = torch.bincount(cell, minlength=int(np.prod(nc)))
        first = torch.cumsum(count, 0) - count
        table = torch.full((count.numel(), int(count.max())), -1, dtype=torch.long, device=pos.device)
        table[cell[order], torch.arange(n, device=pos.device) - first[cell[order]]] = order
        r3 = torch.arange(-1, 2, device=pos.device)
        off = torch.stack(torch.meshgrid(r3, r3, r3, indexing="ij"), -1).reshape(27, 3)
        width = 27 * table.shape[1]
    else:
        table, width = None, n
    step = max(1, int(2.5e7 // width))
    for s in range(0, n, step):
        t = torch.arange(s, min(n, s + step), device=pos.device)
        if table is None:
            j = torch.arange(n, device=pos.device)[None].expand(t.numel(), n)
        else:
            c = torch.remainder(ci[t][:, None] + off[None], nct)
            j = table[(c[..., 0] * nc[1] + c[..., 1]) * nc[2] + c[..., 2]].reshape(t.numel(), -1)
        ok = (j >= 0) & (j != t[:, None])
        j = j.clamp_min(0)
        d = pos[t][:, None] - pos[j]
        d -= L * torch.round(d / L)
        r2 = (d * d).sum(-1)
        ok &= r2 < re * re
        r2 = torch.where(ok, r2, 1.0)
        r = r2.sqrt()
        qj = torch.where(ok, q[j], 0.0)
        ec = qj * torch.erfc(al * r) / r
        f = (ec + qj * (2 * al / math.sqrt(math.pi)) * torch.exp(-al * al * r2)) / r2 * q[t][:, None]
        phi[t] += ec.sum(1)
        F[t] += (f[..., None] * d).sum(1)
        W += 0.5 * torch.einsum("ij,ija,ijb->ab", f, d, d)
    F, phi, W = F * INV_4PI, phi * INV_4PI, W * INV_4PI
    # reciprocal space: half of the sphere (m_x >= 0, planes m_x > 0 doubled), one matrix product per plane
    kmax = 2 * al * X
    M = [int(kmax * x / (2 * math.pi)) for x in box]
    kv = [2 * math.pi / box[a] * torch.arange(0 if a == 0 else -M[a], M[a] + 1, dtype=torch.float64,
                                              device=pos.device) for a in range(3)]
    ph = [torch.polar(torch.ones((), dtype=torch.float64, device=pos.device), -pos[:, a:a + 1] * kv[a][None])
          for a in range(3)]
    KY, KZ = torch.meshgrid(kv[1], kv[2], indexing="ij")
    for m in range(M[0] + 1):
        kx = kv[0][m]
        k2 = kx * kx + KY * KY + KZ * KZ
        g = torch.where((k2 > 0) & (k2 < kmax * kmax), torch.exp(-k2 / (4 * al * al)) / k2, 0.0)
        g *= (1.0 if m == 0 else 2.0) / V
        A = ph[0][:, m:m + 1] * ph[1]
        S = (A * q[:, None]).T @ ph[2]
        gS = g * S.conj()
        T = [torch.einsum("ny,yz,nz->n", A, h, ph[2]) if n < 512 else ((A @ h) * ph[2]).sum(1)
             for h in (gS, kx * gS, KY * gS, KZ * gS)]
        phi += T[0].real
        for a in range(3):
            F[:, a] -= q * T[1 + a].imag
        e = 0.5 * g * (S.real ** 2 + S.imag ** 2)
        k2s = torch.where(k2 > 0, k2, 1.0)
        b = 2.0 * (1.0 / k2s + 1.0 / (4 * al * al))
        K = (kx.expand_as(KY), KY, KZ)
        W += torch.stack([torch.stack([(e * ((1.0 if a == c else 0.0) - b * K[a] * K[c])).sum() for c in range(3)])
                          for a in range(3)])
    phi -= 2 * al / math.sqrt(math.pi) * q * INV_4PI
    return F, 0.5 * q * phi, torch.stack([W[0, 0], W[0, 1], W[0, 2], W[1, 1], W[1, 2], W[2, 2]])


def _lj(pos, box):
    eps, sig, rc = LJ
    L = torch.tensor(box, dtype=torch.float64, device=pos.device)
    d = pos[:, None] - pos[None]
    d -= L * torch.round(d / L)
    r2 = (d * d).sum(-1)
    ok = (r2 < rc * rc) & (r2 > 0)
    r2 = torch.where(ok, r2, 1.0)
    s6 = torch.where(ok, (sig * sig / r2) ** 3, 0.0)
    F = ((24 * eps * (2 * s6 * s6 - s6) / r2)[..., None] * d).sum(1)
    return F, (2 * eps * (s6 * s6 - s6)).sum(1)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("eval", "hoomd"):
        n = 3 * case["molecules"] if case["system"] == "water" else case["ex"] * case["ey"] * case["ez"]
        if n > 110000:
            return None
        _, (pos, q, _, box) = _inputs(case, seed)[0]
        F, e, W = _ewald(pos, q, box)
        if kind == "eval":
            return torch.cat([F, e[:, None]], 1), torch.cat([e.sum()[None], W]) if case["virial"] else e.sum()[None]
        L = torch.tensor(box, dtype=torch.float64, device=pos.device)
        ex = _exclusions(n)[1].long()
        d = pos[:, None] - pos[ex]
        d -= L * torch.round(d / L)
        r2 = (d * d).sum(-1)
        u = INV_4PI * q[:, None] * q[ex] / r2.sqrt()
        F = F - ((u / r2)[..., None] * d).sum(1)
        # the per-particle virial and the external terms depend on where the method splits 1/r
        return torch.cat([F, (e - 0.5 * u.sum(1))[:, None]], 1), None, None
    if kind == "serve" or case.get("system") == "water":
        return None  # constrained dynamics of many systems: no quick FP64 value
    if kind == "md64":
        (_, (pos, q, vel, box)), = _inputs(case, seed)
        return _verlet(pos, q, vel, box, case["steps"], True)
    sizes = [n for _, n in _sizes(case)]
    if max(sizes) > 16 or len(sizes) * (case["steps"] + 1) > 700:
        return None
    out = [_verlet(*s, case["steps"], False) for _, s in _inputs(case, seed)]
    return tuple(torch.cat([o[k] for o in out]) for k in range(4))


def _verlet(pos, q, vel, box, steps, lj):
    """Velocity Verlet with unit masses: the positions, velocities, forces and energy after `steps`."""
    L = torch.tensor(box, dtype=torch.float64, device=pos.device)

    def forces(p):
        F, e, _ = _ewald(p, q, box)
        if lj:
            F2, e2 = _lj(p, box)
            F, e = F + F2, e + e2
        return F, e

    F, e = forces(pos)
    for _ in range(steps):
        vel = vel + 0.5 * DT * F
        pos = torch.remainder(pos + DT * vel, L)
        F, e = forces(pos)
        vel = vel + 0.5 * DT * F
    w0, w1 = torch.zeros_like(q)[:, None], torch.ones_like(q)[:, None]
    return torch.cat([pos, w0], 1), torch.cat([vel, w1], 1), torch.cat([F, e[:, None]], 1), e.sum()[None]

"""The calls that users of the engine wait for, as timed passes with FP64 answers beside them.

A case names one family of calls and its sizes:

* ``force``   -- ``ForceCalculator.compute_device`` on a kept pair list (the step between two searches),
                or, with ``search``, ``md_step_device`` on a search step (gridding, search, prune, forces);
* ``host``    -- nblib's own call, ``ForceCalculator.compute`` on numpy arrays;
* ``md``      -- ``MdRunner.run``: forces with searches and pruning, PME, leap-frog;
* ``pme``     -- ``Pme.compute_device``, the reciprocal half of the Ewald sum;
* ``batch``   -- ``BatchForceCalculator.compute_device``, an ensemble of uneven boxes in one launch;
* ``adjoint`` -- ``DifferentiableNonbonded``: one force-matching gradient step through autograd;
* ``match``   -- ``BatchForceMatcher``: the same over a batch of liquids.

Energies, virials, losses and parameter gradients are FP64 sums of single-precision pair terms; they
are returned as single-precision values, as the reference's energy file stores them.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from gmxapi_gb300 import adjoint, batch, md, nblib, pme, systems

DEV = "cuda:0"
RC, RLIST, RINNER = 0.9, 1.0, 0.95
DRIFT = 0.002  # nm per coordinate between the list's coordinates and the evaluated ones
KE = 138.93545764438198  # kJ mol^-1 nm e^-2
WATER_VOLUME = 0.0299  # nm^3 per molecule
LIQUID_DENSITY = 100.0  # atoms per nm^3
LATTICE, MASS, TEMPERATURE = 0.5256, systems.ARGON_MASS, 120.0


def listed():
    return [
        # the reference's own benchmark box (3,000 atoms): one MD step's forces, all latency and launches
        dict(name="water-3k-force", kind="force", molecules=1000, coulomb="ewald", vdw="shift", energy=False,
             search=False),
        # nblib's default call on an ordinary box with numpy arrays: copies in and out, energies, virial
        dict(name="water-24k-host", kind="host", molecules=8011, energy=True),
        # the benchmark box of bench.py: a step that reports energies and the virial
        dict(name="water-288k-energy", kind="force", molecules=96000, coulomb="ewald", vdw="shift", energy=True,
             search=False),
        # a large box on a search step: gridding, pair search, balancing, fresh prune and the forces
        dict(name="water-960k-search", kind="force", molecules=320000, coulomb="ewald", vdw="shift", energy=False,
             search=True),
        # an ordinary box of odd size with reaction field, on a search step with energies
        dict(name="water-45k-rf-search", kind="force", molecules=14999, coulomb="rf", vdw="shift", energy=True,
             search=True),
        # force-switched Lennard-Jones (the modifier of CHARMM-type force fields), forces of an MD step
        dict(name="water-96k-fswitch", kind="force", molecules=32000, coulomb="ewald", vdw="fswitch", energy=False,
             search=False),
        # 20 GPU-resident MD steps of a charged argon crystal with PME, two searches among them
        dict(name="md-32k-20steps", kind="md", cells=20, steps=20),
        # the reciprocal half for the small box: launches and a small grid
        dict(name="pme-3k-force", kind="pme", molecules=1000, energy=False),
        # and for the benchmark box with energy and virial
        dict(name="pme-288k-energy", kind="pme", molecules=96000, energy=True),
        # 64 uneven boxes of an ensemble in one launch
        dict(name="batch-64-energy", kind="batch", systems=64, n_min=500, n_max=20000),
        # a force-matching gradient step of one liquid (8 types) through autograd
        dict(name="adjoint-24k", kind="adjoint", atoms=24000, types=8),
        # a force-matching gradient step over 16 liquids of uneven size
        dict(name="match-16", kind="match", systems=16, n_min=2000, n_max=50000, types=8),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["force", "force", "force", "host", "md", "pme", "pme", "batch", "adjoint", "match"])
    if kind == "force":
        return dict(kind=kind, molecules=_log(rng, 400, 300000), coulomb=rng.choice(["ewald", "ewald", "rf"]),
                    vdw=rng.choice(["shift", "shift", "fswitch", "pswitch"]), energy=rng.random() < 0.5,
                    search=rng.random() < 0.3)
    if kind == "host":
        return dict(kind=kind, molecules=_log(rng, 400, 60000), energy=rng.random() < 0.5)
    if kind == "md":
        return dict(kind=kind, cells=rng.randint(9, 24), steps=rng.randint(11, 25))
    if kind == "pme":
        return dict(kind=kind, molecules=_log(rng, 400, 200000), energy=rng.random() < 0.5)
    if kind == "batch":
        return dict(kind=kind, systems=_log(rng, 8, 96), n_min=500, n_max=_log(rng, 2000, 20000))
    if kind == "adjoint":
        return dict(kind=kind, atoms=_log(rng, 2000, 50000), types=rng.randint(1, 15))
    return dict(kind=kind, systems=_log(rng, 2, 16), n_min=2000, n_max=_log(rng, 5000, 50000), types=rng.randint(2, 12))


# ---- inputs ----


def _water(molecules, seed):
    return systems.spc_water(molecules, (molecules * WATER_VOLUME) ** (1.0 / 3.0), seed)


def _liquid(n, ntypes, seed, sigma, epsilon):
    """A multi-type LJ + Coulomb liquid at 100 atoms/nm^3: jittered cubic lattice sites, random types."""
    rng = np.random.default_rng(seed)
    edge = (n / LIQUID_DENSITY) ** (1.0 / 3.0)
    m = int(math.ceil(n ** (1.0 / 3.0) - 1e-9))
    sites = rng.choice(m**3, size=n, replace=False)
    ijk = np.stack((sites // (m * m), sites // m % m, sites % m), axis=1)
    x = (ijk + 0.5) * (edge / m) + rng.uniform(-0.012, 0.012, size=(n, 3))
    q = rng.normal(0.0, 0.4, size=n)
    sij = 0.5 * (sigma[:, None] + sigma[None, :])
    eij = np.sqrt(epsilon[:, None] * epsilon[None, :])
    return systems.System(
        x=x.astype(np.float32), box=np.full(3, edge, np.float32), q=(q - q.mean()).astype(np.float32),
        type=rng.integers(0, ntypes, size=n).astype(np.int32), ntypes=ntypes,
        nbfp=systems.nbfp_from_c6c12(4.0 * eij * sij**6, 4.0 * eij * sij**12),
        excl_index=np.arange(n + 1, dtype=np.int32), excl_list=np.arange(n, dtype=np.int32), name=f"liquid{n}",
        sigma=sigma, epsilon=epsilon)


def _types(ntypes, rng):
    return rng.uniform(0.25, 0.40, size=ntypes), rng.uniform(0.1, 1.0, size=ntypes)


def _liquids(case, seed):
    rng = np.random.default_rng(seed)
    sigma, epsilon = _types(case["types"], rng)
    if case["kind"] == "adjoint":
        return [_liquid(case["atoms"], case["types"], seed, sigma, epsilon)]
    lo, hi = math.log(case["n_min"]), math.log(case["n_max"])
    # sizes spread evenly over the logarithm, so that every seed has the same amount of work
    sizes = np.exp(lo + (hi - lo) * (np.arange(case["systems"]) + 0.5) / case["systems"]).astype(int)
    return [_liquid(int(n), case["types"], seed * 1000 + k, sigma, epsilon) for k, n in enumerate(sizes)]


def _ensemble(case, seed):
    lo, hi = math.log(case["n_min"] / 3), math.log(case["n_max"] / 3)
    sizes = np.exp(lo + (hi - lo) * (np.arange(case["systems"]) + 0.5) / case["systems"])
    return [_water(int(round(m)), seed * 1000 + k) for k, m in enumerate(np.random.default_rng(seed).permutation(sizes))]


def _moved(x, seed):
    g = torch.Generator(device=DEV).manual_seed(int(seed) + 17)
    x0 = torch.from_numpy(np.ascontiguousarray(x, np.float32).reshape(-1)).to(DEV)
    return x0, x0 + DRIFT * torch.randn(x0.shape, generator=g, device=DEV)


def _targets(n, seed):
    """Force-matching targets (kJ/mol/nm) and parameter-like scales are plain seeded numbers."""
    g = torch.Generator(device=DEV).manual_seed(int(seed) + 23)
    return 200.0 * torch.randn((n, 3), generator=g, device=DEV)


def _options(case):
    vdw = {"shift": nblib.VdwModifier.PotShift, "fswitch": nblib.VdwModifier.ForceSwitch,
           "pswitch": nblib.VdwModifier.PotSwitch}[case["vdw"]]
    coulomb = nblib.CoulombType.ReactionField if case["coulomb"] == "rf" else nblib.CoulombType.Pme
    return nblib.NBKernelOptions(coulomb_type=coulomb, pairlist_cutoff=RLIST, rcoulomb=RC, rlist_inner=RINNER,
                                 nstlist=100, nstlist_prune=10, epsilon_rf=78.0, vdw_modifier=vdw,
                                 rvdw_switch=0.8 if case["vdw"] != "shift" else 0.0)


def _crystal(case, seed):
    s = systems.lj_fcc(cells=case["cells"], lattice=LATTICE, charge=0.1, seed=seed)
    rng = np.random.default_rng(seed + 5)
    s.x = (s.x + rng.uniform(-0.01, 0.01, size=s.x.shape)).astype(np.float32)
    v = rng.standard_normal((s.n, 3)) * math.sqrt(0.00831446 * TEMPERATURE / MASS)
    return s, v.astype(np.float32)


def prepare(case, seed):
    stream = torch.cuda.current_stream(DEV).cuda_stream
    kind = case["kind"]
    st = {"case": case}
    if kind in ("force", "host", "pme"):
        s = _water(case["molecules"], seed)
        x0, x = _moved(s.x, seed)
    if kind == "force":
        c = st["calc"] = nblib.ForceCalculator(s, _options(case))
        c.set_stream(stream)
        st["x"], st["f"] = x, torch.zeros_like(x)
        st["ev"] = torch.zeros(11, dtype=torch.float64, device=DEV)
    elif kind == "host":
        st["calc"] = nblib.ForceCalculator(s, nblib.NBKernelOptions(compute_virial_and_energy=case["energy"]))
        st["x"] = x.cpu().numpy().reshape(-1, 3)
        st["f"] = np.zeros_like(st["x"])
    elif kind == "md":
        s, v = _crystal(case, seed)
        opts = nblib.NBKernelOptions(pairlist_cutoff=RLIST, rcoulomb=RC, rlist_inner=0.92, nstlist=10,
                                     nstlist_prune=4, compute_virial_and_energy=True)
        st["md"] = md.MdRunner(s, np.full(s.n, MASS, np.float32), opts, dt=0.002, velocities=v)
        st["x0"], st["v0"] = st["md"].x.clone(), st["md"].v.clone()
    elif kind == "pme":
        p = st["pme"] = pme.Pme([float(b) for b in s.box], rcoulomb=RC)
        p.set_stream(stream)
        st["n"], st["x"], st["f"] = s.n, x, torch.zeros_like(x)
        st["q"] = torch.from_numpy(s.q).to(DEV)
        st["ev"] = torch.zeros(10, dtype=torch.float64, device=DEV)
    elif kind == "batch":
        ens = _ensemble(case, seed)
        b = st["batch"] = batch.BatchForceCalculator(ens, nblib.NBKernelOptions(
            pairlist_cutoff=RLIST, rcoulomb=RC, rlist_inner=RINNER, nstlist=100, nstlist_prune=10,
            compute_virial_and_energy=True))
        b.set_stream(stream)
        x0, st["x"] = _moved(np.concatenate([s.x for s in ens]), seed)
        b.search_device(x0.data_ptr())
        st["f"] = torch.zeros_like(x0)
        st["e"] = torch.zeros((len(ens), 2), dtype=torch.float64, device=DEV)
        st["v"] = torch.zeros((len(ens), 9), dtype=torch.float64, device=DEV)
    else:
        ens = _liquids(case, seed)
        n = sum(s.n for s in ens)
        target = _targets(n, seed)
        st["q"] = torch.from_numpy(np.concatenate([s.q for s in ens])).to(DEV).requires_grad_(True)
        st["sigma"] = torch.tensor(ens[0].sigma, dtype=torch.float64, device=DEV, requires_grad=True)
        st["epsilon"] = torch.tensor(ens[0].epsilon, dtype=torch.float64, device=DEV, requires_grad=True)
        if kind == "adjoint":
            st["x"] = torch.from_numpy(ens[0].x).to(DEV).requires_grad_(True)
            st["target"] = target
            st["engine"] = adjoint.DifferentiableNonbonded(ens[0])
            st["engine"].search(st["x"])
        else:
            st["matcher"] = adjoint.BatchForceMatcher(ens, target)
    return st


# ---- one pass ----


def _single(t):
    return t.to(torch.float32)


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "force":
        ev = st["ev"]
        e, v = (ev.data_ptr(), ev[2:].data_ptr()) if case["energy"] else (None, None)
        if case["search"]:
            st["calc"].md_step_device(0, st["x"].data_ptr(), st["f"].data_ptr(), e, v)
        else:
            st["calc"].compute_device(st["x"].data_ptr(), st["f"].data_ptr(), e, v)
        if not case["energy"]:
            return {"f": st["f"]}
        ev = _single(ev)
        return {"f": st["f"], "e": ev[:2], "vir": ev[2:]}
    if kind == "host":
        c = st["calc"]
        c.compute(st["x"], st["f"])
        if not case["energy"]:
            return {"f": st["f"]}
        return {"f": st["f"], "e": c.energies.astype(np.float32), "vir": c.virial.reshape(-1).astype(np.float32)}
    if kind == "md":
        r = st["md"]
        r.x.copy_(st["x0"])
        r.v.copy_(st["v0"])
        r.step = 0
        rows = r.run(case["steps"], nstcalcenergy=10)
        return {"x": r.x, "v": r.v, "f": r.f, "e": rows.astype(np.float32)}
    if kind == "pme":
        ev = st["ev"]
        st["f"].zero_()
        e, v = (ev.data_ptr(), ev[1:].data_ptr()) if case["energy"] else (None, None)
        st["pme"].compute_device(st["n"], st["x"].data_ptr(), st["q"].data_ptr(), st["f"].data_ptr(), e, v)
        if not case["energy"]:
            return {"f": st["f"]}
        ev = _single(ev)
        return {"f": st["f"], "e": ev[:1], "vir": ev[1:]}
    if kind == "batch":
        st["batch"].compute_device(st["x"].data_ptr(), st["f"].data_ptr(), st["e"].data_ptr(), st["v"].data_ptr())
        return {"f": st["f"], "e": _single(st["e"]), "vir": _single(st["v"])}
    for k in ("x", "q", "sigma", "epsilon"):
        if k in st:
            st[k].grad = None
    table = adjoint.lorentz_berthelot_nbfp(st["sigma"], st["epsilon"])
    if kind == "adjoint":
        f, _ = st["engine"](st["x"], st["q"], table, search=False)
        loss = adjoint.force_matching_loss(f, st["target"])
    else:
        loss = st["matcher"](st["q"], table)
    loss.backward()
    out = {"loss": _single(loss.detach()), "gq": st["q"].grad, "gsigma": _single(st["sigma"].grad),
           "gepsilon": _single(st["epsilon"].grad)}
    if kind == "adjoint":
        out["f"], out["gx"] = f.detach(), st["x"].grad
    return out


# ---- what a pass cannot do without ----

#: flops of one pair within the cut-off: the reference's own counts (forces; forces and energies), and
#: for the gradient pass the pair terms and their derivatives once more
FLOPS_F, FLOPS_VF, FLOPS_GRAD = 70, 107, 250


def _pairs(n, density, rc=RC):
    return 0.5 * n * density * 4.0 / 3.0 * math.pi * rc**3


def work(case):
    kind = case["kind"]
    water = 3.0 / WATER_VOLUME
    if kind in ("force", "host"):
        n = 3 * case["molecules"]
        # positions, charges and types in, forces out
        return {"bytes": 32 * n, "flops": _pairs(n, water, RC if kind == "force" else 1.0)
                * (FLOPS_VF if case["energy"] else FLOPS_F)}
    if kind == "md":
        n = 4 * case["cells"] ** 3
        points = math.prod(pme.grid_size([case["cells"] * LATTICE] * 3))
        # per step: positions and velocities in and out, charges; the real grid written and read once
        flops = _pairs(n, 4.0 / LATTICE**3) * FLOPS_F + n * 64 * 10 + points * 5 * math.log2(points)
        return {"bytes": case["steps"] * (56 * n + 8 * points), "flops": case["steps"] * flops}
    if kind == "pme":
        n = 3 * case["molecules"]
        points = math.prod(pme.grid_size([(case["molecules"] * WATER_VOLUME) ** (1.0 / 3.0)] * 3))
        return {"bytes": 28 * n + 8 * points, "flops": n * 64 * 10 + points * 5 * math.log2(points)}
    if kind == "batch":
        sizes = np.exp(np.linspace(math.log(case["n_min"]), math.log(case["n_max"]), 2 * case["systems"] + 1)[1::2])
        return {"bytes": 32 * float(sizes.sum()), "flops": float(_pairs(sizes, water).sum()) * FLOPS_VF}
    if kind == "adjoint":
        n = case["atoms"]
        return {"bytes": 60 * n, "flops": _pairs(n, LIQUID_DENSITY) * (FLOPS_VF + FLOPS_GRAD)}
    sizes = np.exp(np.linspace(math.log(case["n_min"]), math.log(case["n_max"]), 2 * case["systems"] + 1)[1::2])
    return {"bytes": 40 * float(sizes.sum()), "flops": float(_pairs(sizes, LIQUID_DENSITY).sum())
            * (FLOPS_VF + FLOPS_GRAD)}


# ---- the same in 64 bits ----


def _bisect(f, target):
    lo, hi = 0.0, 100.0
    for _ in range(200):
        mid = 0.5 * (lo + hi)
        lo, hi = (mid, hi) if f(mid) > target else (lo, mid)
    return 0.5 * (lo + hi)


def _beta(rc):
    return _bisect(lambda b: math.erfc(b * rc), 1e-5)


def _near(x, box, rc):
    """Chunks (i, j, dx) of the unordered pairs within rc, dx = x_i - x_j in the nearest images."""
    n = x.shape[0]
    dev = x.device
    ncell = int(box // rc)
    x = x - box * torch.floor(x / box)
    if ncell < 3:
        step = max(1, 20_000_000 // n)
        for a in range(-1, 2):
            for b in range(-1, 2):
                for c in range(-1, 2):
                    shift = box * torch.tensor([a, b, c], dtype=torch.float64, device=dev)
                    for i0 in range(0, n, step):
                        d = x[i0 : i0 + step, None, :] - x[None, :, :] + shift
                        i, j = torch.nonzero((d * d).sum(-1) < rc * rc, as_tuple=True)
                        keep = i + i0 < j
                        i, j = i[keep], j[keep]
                        yield i + i0, j, d[i, j]
        return
    at = torch.clamp((x * (ncell / box)).long(), max=ncell - 1)
    cell = (at[:, 0] * ncell + at[:, 1]) * ncell + at[:, 2]
    order = torch.argsort(cell)
    counts = torch.bincount(cell, minlength=ncell**3)
    starts = torch.cumsum(counts, 0) - counts
    most = int(counts.max())
    lane = torch.arange(most, device=dev)
    table = torch.where(lane[None, :] < counts[:, None],
                        order[torch.clamp(starts[:, None] + lane[None, :], max=n - 1)], -1)
    ids = torch.arange(ncell**3, device=dev)
    cx, cy, cz = ids // ncell**2, ids // ncell % ncell, ids % ncell
    step = max(1, 30_000_000 // most**2)
    for a in range(-1, 2):
        for b in range(-1, 2):
            for c in range(-1, 2):
                if (a, b, c) < (0, 0, 0):
                    continue
                other = ((cx + a) % ncell * ncell + (cy + b) % ncell) * ncell + (cz + c) % ncell
                for c0 in range(0, ncell**3, step):
                    ti, tj = table[c0 : c0 + step], table[other[c0 : c0 + step]]
                    d = x[ti][:, :, None, :] - x[tj][:, None, :, :]
                    d = d - box * torch.round(d / box)
                    ok = ((d * d).sum(-1) < rc * rc) & (ti[:, :, None] >= 0) & (tj[:, None, :] >= 0)
                    if (a, b, c) == (0, 0, 0):
                        ok &= ti[:, :, None] < tj[:, None, :]
                    k, p, q = torch.nonzero(ok, as_tuple=True)
                    yield ti[k, p], tj[k, q], d[k, p, q]


def _lj(r, c6, c12, vdw, rc, rs=0.8):
    """Energy and force / r of 12-6 pairs with the modifier."""
    v6, v12 = r**-6, r**-12
    if vdw == "shift":
        return c12 * (v12 - rc**-12) - c6 * (v6 - rc**-6), (12 * c12 * v12 - 6 * c6 * v6) / (r * r)
    t = torch.clamp(r - rs, min=0.0)
    if vdw == "pswitch":
        u, w = t / (rc - rs), rc - rs
        sw = 1 - 10 * u**3 + 15 * u**4 - 6 * u**5
        dsw = (-30 * u**2 + 60 * u**3 - 30 * u**4) / w
        e = c12 * v12 - c6 * v6
        return sw * e, (sw * (12 * c12 * v12 - 6 * c6 * v6) / r - dsw * e) / r

    def term(p, v):
        a = -p * ((p + 4) * rc - (p + 1) * rs) / (rc ** (p + 2) * (rc - rs) ** 2)
        b = p * ((p + 3) * rc - (p + 1) * rs) / (rc ** (p + 2) * (rc - rs) ** 3)
        c = rc**-p - a / 3 * (rc - rs) ** 3 - b / 4 * (rc - rs) ** 4
        return v - a / 3 * t**3 - b / 4 * t**4 - c, p * v / r + a * t**2 + b * t**3

    (e6, f6), (e12, f12) = term(6, v6), term(12, v12)
    return c12 * e12 - c6 * e6, (c12 * f12 - c6 * f6) / r


def _nonbonded(x, q, types, nbfp, nt, mol, box, rc=RC, coulomb="ewald", vdw="shift"):
    """(forces, {E_lj, E_coulomb}, virial) of the real-space half, all in 64 bits."""
    f = torch.zeros_like(x)
    e = torch.zeros(2, dtype=torch.float64, device=x.device)
    vir = torch.zeros(3, 3, dtype=torch.float64, device=x.device)
    beta = _beta(rc)
    krf = (78.0 - 1.0) / ((2 * 78.0 + 1.0) * rc**3)
    crf = 1.0 / rc + krf * rc**2
    tab = nbfp.reshape(nt, nt, 2)
    for i, j, d in _near(x, box, rc):
        r = d.norm(dim=-1)
        apart = (mol[i] != mol[j]).double()
        par = tab[types[i], types[j]]
        el, fl = _lj(torch.where(apart > 0, r, torch.full_like(r, 0.5)), par[:, 0] / 6, par[:, 1] / 12, vdw, rc)
        qq = KE * q[i] * q[j]
        if coulomb == "ewald":
            br = beta * r
            ec = qq * (apart - torch.erf(br)) / r
            fc = (ec / r + qq * beta * 2 / math.sqrt(math.pi) * torch.exp(-br * br) / r) / r
        else:
            ec = qq * (apart / r + krf * r * r - crf)
            fc = qq * (apart / r**3 - 2 * krf)
        fv = (fl * apart + fc)[:, None] * d
        f.index_add_(0, i, fv)
        f.index_add_(0, j, -fv)
        e += torch.stack(((el * apart).sum(), ec.sum()))
        vir -= 0.5 * d.T @ fv
    self_term = beta / math.sqrt(math.pi) if coulomb == "ewald" else 0.5 * crf
    e[1] -= KE * self_term * (q * q).sum()
    return f, e, vir


def _spline(n, x, box):
    """Grid indices (N, 4), fourth-order B-spline weights and their derivatives along one axis."""
    t = x / box
    t = (t - torch.floor(t)) * n
    i = torch.floor(t)
    u = (t - i)[:, None]
    w = torch.cat(((1 - u) ** 3, 3 * u**3 - 6 * u**2 + 4, -3 * u**3 + 3 * u**2 + 3 * u + 1, u**3), 1) / 6
    dw = torch.cat((-3 * (1 - u) ** 2, 9 * u**2 - 12 * u, -9 * u**2 + 6 * u + 3, 3 * u**2), 1) / 6
    return (i.long()[:, None] + torch.arange(4, device=x.device)) % n, w, dw


def _reciprocal(x, q, box, grid, beta):
    """(forces, energy, virial) of smooth PME of order 4 on the given grid, in 64 bits."""
    dev = x.device
    nx, ny, nz = grid
    ax = [_spline(grid[d], x[:, d], box) for d in range(3)]
    point = ((ax[0][0][:, :, None, None] * ny + ax[1][0][:, None, :, None]) * nz + ax[2][0][:, None, None, :])

    def weights(a, b, c):
        return a[:, :, None, None] * b[:, None, :, None] * c[:, None, None, :]

    w = weights(ax[0][1], ax[1][1], ax[2][1])
    g = torch.zeros(nx * ny * nz, dtype=torch.float64, device=dev)
    g.index_add_(0, point.reshape(-1), (w * q[:, None, None, None]).reshape(-1))
    h = torch.fft.fftn(g.reshape(nx, ny, nz))
    m, moduli = [], []
    for n in grid:
        k = torch.arange(n, dtype=torch.float64, device=dev)
        k = torch.where(k < (n + 1) // 2, k, k - n)
        m.append(k / box)
        phase = 2 * math.pi * k / n
        moduli.append(((4 + 2 * torch.cos(phase)) / 6) ** 2)
    mx, my, mz = m[0][:, None, None], m[1][None, :, None], m[2][None, None, :]
    m2 = mx * mx + my * my + mz * mz
    bb = moduli[0][:, None, None] * moduli[1][None, :, None] * moduli[2][None, None, :]
    m2[0, 0, 0] = 1.0
    term = KE * torch.exp(-((math.pi / beta) ** 2) * m2) / (math.pi * box**3 * m2 * bb)
    term[0, 0, 0] = 0.0
    s = term * (h.real**2 + h.imag**2)
    vf = s * 2 * ((math.pi / beta) ** 2 + 1 / m2)
    vir = torch.zeros(3, 3, dtype=torch.float64, device=dev)
    for a, ma in enumerate((mx, my, mz)):
        for b, mb in enumerate((mx, my, mz)):
            vir[a, b] = 0.25 * ((vf * ma * mb).sum() - (s.sum() if a == b else 0.0))
    phi = (torch.fft.ifftn(term * h).real * (nx * ny * nz)).reshape(-1)[point]
    f = torch.stack([-(q * grid[d] / box) * (phi * weights(*[ax[k][2 if k == d else 1] for k in range(3)])).sum((1, 2, 3))
                     for d in range(3)], dim=1)
    return f, 0.5 * s.sum(), vir


def _on(a, dtype=torch.float64):
    return torch.as_tensor(np.asarray(a), device=DEV).to(dtype)


def _exact_water(s, x, rc=RC, coulomb="ewald", vdw="shift"):
    x = torch.as_tensor(x, device=DEV).double().reshape(-1, 3)
    mol = torch.arange(s.n, device=DEV) // 3
    return _nonbonded(x, _on(s.q), _on(s.type, torch.long), _on(s.nbfp), s.ntypes, mol, float(s.box[0]), rc, coulomb,
                      vdw)


def _exact_md(case, seed):
    s, v = _crystal(case, seed)
    box = float(s.box[0])
    x, v, q = _on(s.x), _on(v), _on(s.q)
    types, nbfp, mol = _on(s.type, torch.long), _on(s.nbfp), torch.arange(s.n, device=DEV)
    grid, beta, dt, rows = pme.grid_size([box] * 3), _beta(RC), 0.002, []
    dt = float(np.float32(dt))
    inverse = float(np.float32(1.0 / MASS))
    for k in range(case["steps"]):
        f, e, _ = _nonbonded(x, q, types, nbfp, 1, mol, box)
        fr, er, _ = _reciprocal(x, q, box, grid, beta)
        f = f + fr
        new = v + f * dt * inverse
        if k % 10 == 0:
            kin = 0.25 / inverse * ((v * v).sum() + (new * new).sum())
            rows.append(torch.stack((e[0], e[1], er, kin)))
        v = new
        x = x + v * dt
        if (k + 1) % 10 == 0:  # put back in the box on the update before a search step
            x = x - box * torch.floor(x / box)
    return {"x": x.reshape(-1), "v": v.reshape(-1), "f": f.reshape(-1), "e": torch.stack(rows)}


def _exact_match(case, seed):
    """Loss and gradients by autograd through explicit pair sums."""
    ens = _liquids(case, seed)
    target = _targets(sum(s.n for s in ens), seed).double()
    sigma = _on(ens[0].sigma).requires_grad_(True)
    epsilon = _on(ens[0].epsilon).requires_grad_(True)
    beta, first, total, gq, out = _beta(RC), 0, 0.0, [], {}
    for s in ens:
        box = float(s.box[0])
        x, q = _on(s.x).requires_grad_(True), _on(s.q).requires_grad_(True)
        types = _on(s.type, torch.long)
        found = [(i, j, d - (x.detach()[i] - x.detach()[j])) for i, j, d in _near(x.detach(), box, RC)]
        i, j, shift = (torch.cat(c) for c in zip(*found))
        r = (x[i] - x[j] + shift).norm(dim=-1)
        sij = 0.5 * (sigma[types[i]] + sigma[types[j]])
        eij = torch.sqrt(epsilon[types[i]] * epsilon[types[j]])
        s6 = (sij / r) ** 6
        energy = (4 * eij * (s6 * s6 - s6) + KE * q[i] * q[j] * torch.erfc(beta * r) / r).sum()
        f = -torch.autograd.grad(energy, x, create_graph=True)[0]
        loss = ((f - target[first : first + s.n]) ** 2).sum()
        loss.backward()
        first, total = first + s.n, total + loss.detach()
        gq.append(q.grad)
        if case["kind"] == "adjoint":
            out["f"], out["gx"] = f.detach(), x.grad
    out.update(loss=total, gq=torch.cat(gq), gsigma=sigma.grad, gepsilon=epsilon.grad)
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "md":
        return _exact_md(case, seed)
    if kind in ("adjoint", "match"):
        return _exact_match(case, seed)
    if kind == "batch":
        ens = _ensemble(case, seed)
        _, x = _moved(np.concatenate([s.x for s in ens]), seed)
        got, first = [], 0
        for s in ens:
            got.append(_exact_water(s, x[3 * first : 3 * (first + s.n)]))
            first += s.n
        return {"f": torch.cat([g[0].reshape(-1) for g in got]), "e": torch.stack([g[1] for g in got]),
                "vir": torch.stack([g[2].reshape(-1) for g in got])}
    s = _water(case["molecules"], seed)
    _, x = _moved(s.x, seed)
    if kind == "pme":
        box = float(s.box[0])
        grid = pme.grid_size([box] * 3)
        f, e, vir = _reciprocal(x.double().reshape(-1, 3), _on(s.q), box, grid, _beta(RC))
        e = e.reshape(1)
    elif kind == "host":
        f, e, vir = _exact_water(s, x, rc=1.0)
    else:
        f, e, vir = _exact_water(s, x, coulomb=case["coulomb"], vdw=case["vdw"])
    out = {"f": f if kind == "host" else f.reshape(-1)}
    if case["energy"]:
        out["e"], out["vir"] = e, vir.reshape(-1)
    return out

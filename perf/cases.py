"""
Performance cases of taichimps_gb300: what its users have it do.

Single runs through ``Simulation.run`` (small and large, dilute and contact-dense, plain FP64 and mixed
precision, with and without the pressure servo), a whole job from page-locked host arrays, a run between walls,
a batched ensemble, and the gradient of a stress curve.  Sizes and parameters follow this repository's
benchmark configurations and tests; packings are synthetic and made from the seed.

``exact`` restates the same runs in plain PyTorch FP64 (half pair list, index_add), without the package's code.
"""

from __future__ import annotations

import math

import numpy as np
import torch

DENSITY = 2.5
CELL_N = 15625                      # spheres of the compressed cell that dense packings are tiled from
LEGACY = dict(kn=2.0e5, kt=2.0e5 * 2.0 / 7.0, gamman=50.0, gammat=25.0, xmu=0.5)
GAS_HOOKE = dict(kn=2000.0, kt=2000.0 * 2.0 / 7.0, gamman=50.0, gammat=25.0, xmu=0.5)
# hertz/material with the elastic stiffness of LEGACY (4/3 E* = 2e5), coeff_restitution 0.5, Poisson 0.3
EMOD, COR, POISSON = 2.0e5 * 1.5 * (1.0 - 0.3 ** 2), 0.5, 0.3
ROLLING = (1.0e3, 50.0, 0.1)
ISO = dict(style=("pressure",) * 3, ptarget=1.0, pgain=1.0e-3, rate=0.0, couple=True, max_rate=1.0e-4)
TRIAXIAL = dict(style=("pressure", "pressure", "erate"), ptarget=1.0, pgain=0.1, rate=-1.0e-3, couple=False,
                max_rate=1.0e-2)
SERVOS = {"iso": ISO, "triaxial": TRIAXIAL}
DRUM = dict(kn=2.0e4, kt=2.0e4 * 2.0 / 7.0, gamman=50.0, gammat=25.0, xmu=0.5)


def listed():
    run = dict(kind="run", cundall=False, speed=0.0)
    return [
        # the small plain run of the configurations: a collisional gas, where latency and launches count
        dict(run, name="gas_4k_fp64", packing="gas", n=4000, pair="hooke", precision="fp64", servo="none",
             speed=0.1, steps=500, dt=1.0e-4),
        # spheres inside a rotating-drum style cylinder: walls, a few thousand particles
        dict(name="drum_3k_fp64", kind="drum", n=3001, steps=200, dt=1.0e-4, speed=0.5),
        # the headline run: isotropic compression of a million spheres, both precisions
        dict(run, name="compress_1m_mixed", packing="gas", n=1_000_000, pair="hertz", precision="mixed",
             servo="iso", cundall=True, steps=200, dt=5.0e-5),
        dict(run, name="compress_1m_fp64", packing="gas", n=1_000_000, pair="hertz", precision="fp64",
             servo="iso", cundall=True, steps=100, dt=5.0e-5),
        # the same physics where the packing is jammed (four touching neighbours per sphere)
        dict(run, name="jammed_1m_mixed", packing="dense", n=1_000_000, pair="hertz", precision="mixed",
             servo="iso", cundall=True, steps=50, dt=5.0e-5),
        dict(run, name="jammed_110k_fp64", packing="dense", n=109_301, pair="hertz", precision="fp64",
             servo="iso", cundall=True, steps=50, dt=5.0e-5),
        # one logging interval of a triaxial test: pair granular with rolling resistance
        dict(run, name="triaxial_250k_mixed", packing="dense", n=250_000, pair="granular", precision="mixed",
             servo="triaxial", steps=100, dt=5.0e-5),
        # a fast gas from device arrays, list rebuilds along the way; a fresh system each time
        dict(name="job_flow_65k_mixed", kind="job", packing="gas", n=65_537, pair="hertz", precision="mixed",
             servo="none", cundall=False, speed=6.0, steps=300, dt=5.0e-5, source="device"),
        # a whole job from page-locked host arrays, as the end-to-end benchmark line runs it
        dict(name="job_500k_mixed", kind="job", packing="gas", n=499_999, pair="hertz", precision="mixed",
             servo="iso", cundall=True, speed=0.0, steps=20, dt=5.0e-5, source="pinned"),
        # a parameter study: independent packings of uneven size advanced together
        dict(name="ensemble_24", kind="ensemble", instances=24, nmin=500, nmax=16000, steps=1024, dt=5.0e-5,
             precision="mixed"),
        # gradients of a stress curve, at the size of the checks and at calibration size
        dict(name="gradient_2k", kind="gradient", n=2048, steps=100, every=20, checkpoint=50, dt=5.0e-5),
        dict(name="gradient_31k", kind="gradient", n=31_250, steps=100, every=50, checkpoint=100, dt=5.0e-5),
    ]


def draw(rng):
    log = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    dense_n = lambda cells: CELL_N * cells - rng.randrange(0, 40 * cells)
    kind = rng.choice(["gas", "gas", "compress", "jammed", "jammed", "triaxial", "drum", "job", "ensemble", "gradient"])
    prec = rng.choice(["fp64", "mixed"])
    base = dict(kind="run", precision=prec, cundall=False, speed=0.0, dt=5.0e-5)
    if kind == "gas":
        return dict(base, packing="gas", n=log(500, 200_000), pair=rng.choice(["hooke", "hertz"]), servo="none",
                    speed=0.1, steps=rng.randrange(100, 400), dt=1.0e-4)
    if kind == "compress":
        return dict(base, packing="gas", n=log(4000, 1_000_000), pair="hertz", servo="iso", cundall=True,
                    steps=rng.randrange(50, 101))
    if kind == "jammed":
        top = 64 if prec == "mixed" else 8
        return dict(base, packing="dense", n=dense_n(log(1, top)), pair=rng.choice(["hertz", "granular"]),
                    servo="iso", cundall=True, steps=rng.randrange(20, 51))
    if kind == "triaxial":
        top = 16 if prec == "mixed" else 4
        return dict(base, packing="dense", n=dense_n(log(1, top)), pair="granular", servo="triaxial",
                    steps=rng.randrange(30, 101))
    if kind == "drum":
        return dict(kind="drum", n=log(500, 20_000), steps=rng.randrange(50, 201), dt=1.0e-4, speed=0.5)
    if kind == "job":
        return dict(kind="job", packing="gas", n=log(10_000, 500_000), pair="hertz", precision=prec, servo="iso",
                    cundall=True, speed=0.0, steps=rng.randrange(10, 41), dt=5.0e-5,
                    source=rng.choice(["pinned", "device"]))
    if kind == "ensemble":
        return dict(kind="ensemble", instances=rng.randrange(4, 25), nmin=500, nmax=log(2000, 16000),
                    steps=64 * rng.randrange(4, 17), dt=5.0e-5, precision="mixed")
    n = rng.choice([log(600, 6000), dense_n(1), dense_n(2)])
    every = rng.choice([10, 20, 25])
    return dict(kind="gradient", n=n, steps=every * rng.randrange(2, 5), every=every, checkpoint=rng.choice([20, 50, 100]),
                dt=5.0e-5)


# ------------------------------------------------------------------ packings


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) & 0x7FFFFFFF)
    return g


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64)


def _normal(g, sigma, n):
    return sigma * torch.randn(n, 3, generator=g, device="cuda", dtype=torch.float64)


def gas(g, n, spread, speed, jitter=0.004):
    """n spheres, diameters U[1 - spread, 1 + spread], on randomly chosen FCC sites of a periodic cube whose nearest
    sites lie just further apart than the largest diameter (solid fraction about 0.4), jittered by up to `jitter`
    lattice constants: a few of the largest neighbours touch."""
    m = max(2, math.ceil((n / 4.0) ** (1.0 / 3.0) - 1e-9))
    while 4 * m ** 3 < n:
        m += 1
    a = 1.004 * (1.0 + spread) * math.sqrt(2.0)
    cells = torch.stack(torch.meshgrid(*[torch.arange(m, device="cuda")] * 3, indexing="ij"), -1).reshape(-1, 1, 3)
    base = torch.tensor([[0.0, 0, 0], [0.5, 0.5, 0], [0.5, 0, 0.5], [0, 0.5, 0.5]], device="cuda", dtype=torch.float64)
    sites = (cells.double() + base).reshape(-1, 3)
    pick = torch.randperm(len(sites), generator=g, device="cuda")[:n]
    x = (sites[pick] + 0.25 + jitter * (2.0 * _rand(g, n, 3) - 1.0)) * a
    radius = 0.5 * (1.0 - spread + 2.0 * spread * _rand(g, n))
    return dict(x=x, radius=radius, v=_normal(g, speed, n), lo=[0.0] * 3, L=[m * a] * 3)


def _cell(g):
    """The compressed cell under a random symmetry (axes permuted, mirrored, shifted around the period)."""
    from taichimps_gb300.packing import dense_cell
    c = dense_cell()
    perm = torch.randperm(3, generator=g, device="cuda").tolist()
    L = torch.tensor([float(c["L"][k]) for k in perm], device="cuda", dtype=torch.float64)
    x = torch.as_tensor(c["x"] - c["lo"], device="cuda")[:, perm].contiguous()
    flip = _rand(g, 3) < 0.5
    x = torch.where(flip, L - x, x)
    x = torch.remainder(x + _rand(g, 3) * L, L)
    return x, torch.as_tensor(c["radius"], device="cuda"), L


def dense(g, n, speed=1.0e-4):
    """A jammed packing at p = 1: the compressed cell tiled in a periodic box, the few spheres past n left out, in a
    random order.  Below one cell: a block cut out of it, spheres that overlap across the new period left out."""
    x, r, L = _cell(g)
    if n < CELL_N // 2:
        side = L * (1.12 * n / CELL_N) ** (1.0 / 3.0)
        while True:
            keep = (x < side).all(1).nonzero().flatten()
            xs, rs = x[keep], r[keep]
            d = xs[:, None] - xs[None]
            d = d - side * torch.round(d / side)
            over = (rs[:, None] + rs[None]) - d.norm(dim=2) > 2e-3
            bad = torch.triu(over, 1).any(0)
            xs, rs = xs[~bad], rs[~bad]
            if len(xs) >= n:
                break
            side = side * 1.01
        L = side
    else:
        cells = -(-n // CELL_N)
        reps = min(((a, b, cells // (a * b)) for a in range(1, cells + 1) if cells % a == 0
                    for b in range(1, cells // a + 1) if (cells // a) % b == 0), key=lambda t: max(t) / min(t))
        off = torch.stack(torch.meshgrid(*[torch.arange(k, device="cuda") for k in reps], indexing="ij"), -1)
        xs = (x[None] + (off.reshape(-1, 1, 3) * L)).reshape(-1, 3)
        rs = r.repeat(cells)
        L = L * torch.tensor(reps, device="cuda")
    pick = torch.randperm(len(xs), generator=g, device="cuda")[:n]
    return dict(x=xs[pick].contiguous(), radius=rs[pick].contiguous(), v=_normal(g, speed, n), lo=[0.0] * 3, L=L.tolist())


def drum(g, n, speed):
    """FCC sites inside a cylinder along z as long as it is wide (z periodic, x and y open)."""
    a = 1.02 * 1.1 * math.sqrt(2.0)
    m = 2
    while True:
        R = 0.5 * m * a
        cells = torch.stack(torch.meshgrid(*[torch.arange(m, device="cuda")] * 3, indexing="ij"), -1).reshape(-1, 1, 3)
        base = torch.tensor([[0.0, 0, 0], [0.5, 0.5, 0], [0.5, 0, 0.5], [0, 0.5, 0.5]], device="cuda", dtype=torch.float64)
        s = ((cells.double() + base).reshape(-1, 3) + 0.25) * a
        s[:, :2] -= R
        s = s[(s[:, 0] ** 2 + s[:, 1] ** 2).sqrt() < R - 0.53]
        if len(s) >= n:
            break
        m += 1
    pick = torch.randperm(len(s), generator=g, device="cuda")[:n]
    x = s[pick] + 0.004 * (2.0 * _rand(g, n, 3) - 1.0)
    return dict(x=x, radius=0.5 * (0.9 + 0.2 * _rand(g, n)), v=_normal(g, speed, n), lo=[-R - 1.0, -R - 1.0, 0.0],
                L=[2.0 * R + 2.0, 2.0 * R + 2.0, m * a], R=R)


def packing(case, seed):
    g = _gen(seed)
    if case["kind"] == "drum":
        return drum(g, case["n"], case["speed"])
    if case["kind"] == "gradient":
        return dense(g, case["n"], speed=0.02)
    if case["packing"] == "gas":
        if case["servo"] == "iso":
            return gas(g, case["n"], 0.2, case["speed"])
        return gas(g, case["n"], 0.1, case["speed"], jitter=0.012)
    return dense(g, case["n"])


def ensemble_members(case, seed):
    """The instances: sphere counts spread over the logarithm of the range, kn log-uniform [1e4, 1e6], xmu
    U[0.1, 0.8]."""
    rng = np.random.default_rng(int(seed))
    lo, hi, m = math.log(case["nmin"]), math.log(case["nmax"]), case["instances"]
    out = []
    for k in range(m):
        n = int(round(math.exp(lo + (hi - lo) * ((k * 0.6180339887498949) % 1.0))))
        kn, xmu = float(math.exp(rng.uniform(math.log(1e4), math.log(1e6)))), float(rng.uniform(0.1, 0.8))
        p = gas(_gen(int(seed) * 1009 + k), n, 0.2, 0.0)
        out.append((p, dict(kn=kn, kt=kn * 2.0 / 7.0, gamman=50.0, gammat=25.0, xmu=xmu)))
    return out


# ------------------------------------------------------------------ the framework


def _sim(p, pair, precision, servo, cundall, dt, walls=None, slots=None, host=None):
    import taichimps_gb300 as G
    n = len(p["radius"])
    src = p if host is None else host
    periodic = ("p", "p", "p") if walls is None else ("f", "f", "p")
    dom = G.Domain(boxlo=p["lo"], boxhi=[a + b for a, b in zip(p["lo"], p["L"])], boundary=periodic)
    atom = G.AtomSystem(max_atoms=n)
    atom.add_particles(x=src["x"], radius=src["radius"], density=DENSITY, v=src["v"])
    nl = G.NeighborList(domain=dom, skin=0.1, max_atoms=n, max_neighbors_per_atom=16, slots=slots)
    hist = G.ContactHistory(max_atoms=n, max_neighbors=16)
    if pair == "granular":
        law = G.PairGranular(domain=dom, normal="hertz/material", normal_coeffs=[EMOD, COR, POISSON],
                             damping="coeff_restitution", tangential="mindlin", tangential_coeffs=[None, 1.0, 0.5],
                             rolling="epsd", rolling_coeffs=list(ROLLING))
    elif isinstance(pair, dict):
        law = G.GranHertzHistory(domain=dom, dampflag=1, **pair)
    elif pair == "hertz":
        law = G.GranHertzHistory(domain=dom, dampflag=1, **LEGACY)
    else:
        law = G.GranHookeHistory(domain=dom, dampflag=1, **(DRUM if walls is not None else GAS_HOOKE))
    sim = G.Simulation(domain=dom, atom=atom, neighbor=nl, history=hist, pair=law, dt=dt, precision=precision)
    sim.add_fix(G.FixNVESphere(domain=dom))
    if cundall:
        sim.add_fix(G.FixDampingCundall(domain=dom, gamma_lin=0.7, gamma_ang=0.7))
    if walls is not None:
        sim.add_fix(G.FixWallGranRegion(domain=dom, axis=2, radius=walls, side="in", fstyle="hooke/history",
                                        max_atoms=n, **DRUM))
    if servo in SERVOS:
        s = SERVOS[servo]
        axes = {d: {"style": "pressure", "ptarget": s["ptarget"], "pgain": s["pgain"]} if st == "pressure"
                else {"style": "erate", "rate": s["rate"]} for d, st in zip("xyz", s["style"])}
        sim.add_fix(G.FixDeformPressure(domain=dom, axes=axes, couple="xyz" if s["couple"] else "none",
                                        max_rate=s["max_rate"], remap="x"))
    return sim


def prepare(case, seed):
    import taichimps_gb300 as G
    kind = case["kind"]
    if kind == "ensemble":
        sims = [_sim(p, c, case["precision"], "iso", False, case["dt"], slots="auto")
                for p, c in ensemble_members(case, seed)]
        return dict(case=case, sims=sims, engine=G.BatchedEngine(sims, precision=case["precision"]))
    p = packing(case, seed)
    if kind == "gradient":
        from taichimps_gb300.adjoint import AdjointRun
        axes = {"x": {"style": "pressure", "ptarget": 1.0, "pgain": 0.1},
                "y": {"style": "pressure", "ptarget": 1.0, "pgain": 0.1}, "z": {"style": "erate", "rate": -1.0e-3}}
        job = AdjointRun(p["x"], p["radius"].cpu().numpy(), DENSITY, p["lo"], [a + b for a, b in zip(p["lo"], p["L"])],
                         dt=case["dt"], steps=case["steps"], axes=axes, max_rate=1.0e-2, sample_every=case["every"],
                         checkpoint_every=case["checkpoint"], v=p["v"].cpu().numpy())
        leaf = lambda a: torch.tensor(a, dtype=torch.float64, requires_grad=True)
        return dict(case=case, job=job, params={k: leaf(v) for k, v in LEGACY.items()},
                    radius=p["radius"].clone().requires_grad_(True))
    if kind == "job":
        src = {k: p[k] for k in ("x", "radius", "v")}
        if case["source"] == "pinned":
            src = {k: a.cpu().pin_memory() for k, a in src.items()}
        return dict(case=case, p=p, src=src)
    if kind == "drum":
        return dict(case=case, sim=_sim(p, "hooke", "fp64", "none", False, case["dt"], walls=p["R"]))
    sim = _sim(p, case["pair"], case["precision"], case["servo"], case["cundall"], case["dt"])
    if case["servo"] == "triaxial":
        sim.fixes[-1].record_pressure(8)
        return dict(case=case, sim=sim, coordination=G.ComputeContactAtom(max_atoms=case["n"]))
    return dict(case=case, sim=sim)


def _fields(sim, names):
    return {k: getattr(sim.atom, k).to_numpy() for k in names}


def _box(sim):
    return np.concatenate([sim.domain.boxlo, sim.domain.boxhi])


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "ensemble":
        state["engine"].run(case["steps"])
        out = [_fields(s, ("x", "v")) for s in state["sims"]]
        return dict({k: np.concatenate([o[k] for o in out]) for k in ("x", "v")},
                    box=np.stack([_box(s) for s in state["sims"]]))
    if kind == "gradient":
        from taichimps_gb300.adjoint import stress_curve
        P, r = state["params"], state["radius"]
        for t in (*P.values(), r):
            t.grad = None
        q = stress_curve(state["job"], P["kn"], P["kt"], P["gamman"], P["gammat"], P["xmu"], r)
        (q ** 2).sum().backward()
        return dict({k: t.grad for k, t in P.items()}, q=q.detach(), radius=r.grad)
    if kind == "job":
        sim = _sim(state["p"], case["pair"], case["precision"], case["servo"], case["cundall"], case["dt"],
                   host=state["src"])
        sim.run(case["steps"])
        return dict(_fields(sim, ("x", "v")), box=_box(sim))
    sim = state["sim"]
    sim.run(case["steps"])
    out = dict(_fields(sim, ("x", "v", "f")), box=_box(sim))
    if "coordination" in state:
        # the log line of a triaxial test
        out["contacts"] = state["coordination"].compute(sim.atom, sim.domain, sim.neighbor)
    return out


def work(case):
    """Per step and atom: position, velocity and angular velocity read and written, radius and mass read; per
    touching pair: its index and its shear, read and written.  A gradient runs the steps twice forward and once
    back.  Arithmetic: about 60 operations per atom and step, 250 per contact."""
    kind, steps = case["kind"], case["steps"]
    if kind == "ensemble":
        lo, hi = case["nmin"], case["nmax"]
        n = case["instances"] * ((hi - lo) / math.log(hi / lo))
    else:
        n = case["n"]
    contacts = n * (2.05 if kind == "gradient" or case.get("packing") == "dense" else 0.05)
    pair = 104.0 if case.get("pair") == "granular" else 56.0
    step = n * 160.0 + contacts * pair
    if kind == "gradient":
        steps, contacts = 4 * steps, 1.5 * contacts
    out = n * (48.0 if kind in ("job", "ensemble") else 72.0)
    return {"bytes": steps * step + out + (56.0 * n if kind == "job" else 0.0),
            "flops": steps * (60.0 * n + 250.0 * contacts)}


# ------------------------------------------------------------------ the same in plain PyTorch, 64 bits


def _image(d, prd, per):
    return d - per * torch.round(d / prd) * prd


def _pairs(x, r, lo, prd, per, skin):
    """Half list (i < j, sorted) of the pairs within ri + rj + skin."""
    n = len(x)
    cut = 2.0 * float(r.max()) + skin
    g = [max(1, min(160, int(float(prd[k]) / cut))) for k in range(3)]
    gt = torch.tensor(g, device=x.device)
    c = torch.minimum(((x - lo) / prd * gt).floor().long().clamp(min=0), gt - 1)
    lin = (c[:, 0] * g[1] + c[:, 1]) * g[2] + c[:, 2]
    order = torch.argsort(lin)
    count = torch.bincount(lin, minlength=g[0] * g[1] * g[2])
    start = torch.cumsum(count, 0) - count
    most = int(count.max())
    ids = torch.arange(n, device=x.device)
    found = []
    for o in range(27):
        off = torch.tensor([o // 9 - 1, o // 3 % 3 - 1, o % 3 - 1], device=x.device)
        q = c + off
        ok = ((per > 0) | ((q >= 0) & (q < gt))).all(1)
        q = torch.remainder(q, gt)
        ql = (q[:, 0] * g[1] + q[:, 1]) * g[2] + q[:, 2]
        for k in range(most):
            i = ids[ok & (count[ql] > k)]
            j = order[start[ql[i]] + k]
            i, j = i[j > i], j[j > i]
            d = _image(x[i] - x[j], prd, per)
            near = (d * d).sum(1) < (r[i] + r[j] + skin) ** 2
            found.append(i[near] * n + j[near])
    key = torch.unique(torch.cat(found))
    return key // n, key % n, key


def _dot(a, b):
    return (a * b).sum(1)


def _root(a):
    """sqrt with a zero (not infinite) slope at zero."""
    pos = a > 0
    return torch.where(pos, torch.sqrt(torch.where(pos, a, torch.ones_like(a))), torch.zeros_like(a))


def _legacy(P, hertz, dt, update, d, rsq, r, ra, rb, ma, mb, va, vb, wa, wb, h):
    """gran/hooke/history and gran/hertz/history: force on a, torque of a and of b, history."""
    delta = ra + rb - r
    poly = torch.sqrt(ra * rb / (ra + rb) * delta) if hertz else torch.ones_like(r)
    meff = ma * mb / (ma + mb)
    vr = va - vb
    vn = _dot(vr, d)
    vtr = vr - d * (vn / rsq)[:, None] + torch.linalg.cross(d, (ra[:, None] * wa + rb[:, None] * wb) / r[:, None])
    ccel = (P["kn"] * delta / r - meff * P["gamman"] * vn / rsq) * poly
    geff = (meff * P["gammat"])[:, None]
    sh = h + vtr * dt if update else h
    moved = _dot(sh, sh).detach() > 0
    if update:
        sh = sh - (_dot(sh, d) / rsq)[:, None] * d
    fs = -poly[:, None] * (P["kt"] * sh + geff * vtr)
    mag = _root(_dot(fs, fs))
    cap = P["xmu"] * torch.abs(ccel * r)
    slip = mag > cap
    ratio = torch.where(slip & moved, cap / torch.where(slip, mag, torch.ones_like(mag)), torch.ones_like(mag))[:, None]
    dc = geff * vtr / P["kt"]
    sh = torch.where((slip & moved)[:, None], ratio * (sh + dc) - dc, sh)
    fs = torch.where((slip & ~moved)[:, None], torch.zeros_like(fs), ratio * fs)
    tor = torch.linalg.cross(d, fs) / r[:, None]
    return d * ccel[:, None] + fs, -ra[:, None] * tor, -rb[:, None] * tor, sh


def _granular(dt, update, d, rsq, r, ra, rb, ma, mb, va, vb, wa, wb, h):
    """hertz/material + coeff_restitution + mindlin + rolling resistance; history = shear and rolling (6)."""
    kn = 4.0 / 3.0 * EMOD / (2.0 * (1.0 - POISSON ** 2))
    kt = 8.0 * EMOD / (4.0 * (2.0 - POISSON) * (1.0 + POISSON))
    logc = math.log(COR)
    damp = -2.0 * math.sqrt(5.0 / 6.0) * math.sqrt(1.5) * logc / math.sqrt(math.pi ** 2 + logc ** 2)
    nv = d / r[:, None]
    delta = ra + rb - r
    reff, meff = ra * rb / (ra + rb), ma * mb / (ma + mb)
    a = torch.sqrt(delta * reff)
    vr = va - vb
    vn = _dot(vr, nv)
    vtr = vr - vn[:, None] * nv - torch.linalg.cross(ra[:, None] * wa + rb[:, None] * wb, nv)
    fne = kn * a * delta
    dpf = damp * torch.sqrt((meff * fne / delta).clamp(min=0.0))
    fn = fne - dpf * vn
    cap = 0.5 * torch.abs(fn)
    keff = (kt * a)[:, None]
    sh, rl = h[:, :3], h[:, 3:]
    wrel = wa - wb
    if update:
        hn = _dot(sh, nv)
        o = sh - hn[:, None] * nv
        om = _root(_dot(o, o))
        scale = torch.where(om > 0, _root(_dot(sh, sh)) / torch.where(om > 0, om, torch.ones_like(om)), om)
        sh = torch.where((torch.abs(hn) * kt * a > 1e-10 * cap)[:, None], o * scale[:, None], sh) + vtr * dt
        rl = rl + wrel * dt
    fd = -dpf[:, None] * vtr
    fs = -keff * sh + fd
    mag = _root(_dot(fs, fs))
    slip = mag > cap
    some = _dot(sh, sh) > 0
    fs = torch.where((slip & some)[:, None], fs * (cap / torch.where(slip, mag, torch.ones_like(mag)))[:, None], fs)
    sh = torch.where((slip & some)[:, None], -(fs - fd) / keff, sh)
    fs = torch.where((slip & ~some)[:, None], torch.zeros_like(fs), fs)
    k_roll, g_roll, mu_roll = ROLLING
    tr = k_roll * _root(_dot(rl, rl))
    top = mu_roll * reff * torch.abs(fn)
    over = ((tr > top) & (tr > 1e-12))[:, None]
    unit = rl / torch.where(tr > 0, tr, torch.ones_like(tr))[:, None]
    troll = torch.where(over, -top[:, None] * unit, -k_roll * rl - g_roll * wrel)
    rl = torch.where(over, top[:, None] / k_roll * unit, rl)
    c = -torch.linalg.cross(nv, fs)
    return (fn[:, None] * nv + fs, (ra - 0.5 * delta)[:, None] * c + troll, (rb - 0.5 * delta)[:, None] * c - troll,
            torch.cat([sh, rl], 1))


def _wall(R, dt, update, x, r, m, v, w, h, touch):
    """The inside of a cylinder along z, hooke with history: force, torque, history."""
    rho = torch.sqrt(x[:, 0] ** 2 + x[:, 1] ** 2)
    nv = torch.stack([-x[:, 0] / rho, -x[:, 1] / rho, torch.zeros_like(rho)], 1)
    delta = r - (R - rho)
    on = (delta > 0)[:, None]
    vr = v - r[:, None] * torch.linalg.cross(w, nv)
    vn = _dot(vr, nv)
    vt = vr - vn[:, None] * nv
    fn = DRUM["kn"] * delta - m * DRUM["gamman"] * vn
    h = torch.where(touch[:, None], h, torch.zeros_like(h))
    if update:
        h = h + vt * dt
    some = _dot(h, h) != 0
    if update:
        h = h - _dot(h, nv)[:, None] * nv
    fd = -(m * DRUM["gammat"])[:, None] * vt
    fs = -DRUM["kt"] * h + fd
    mag, cap = _root(_dot(fs, fs)), DRUM["xmu"] * torch.abs(fn)
    slip = mag > cap
    fs = torch.where((slip & some)[:, None], fs * (cap / torch.where(slip, mag, torch.ones_like(mag)))[:, None], fs)
    h = torch.where((slip & some)[:, None], -(fs - fd) / DRUM["kt"], h)
    fs = torch.where((slip & ~some)[:, None], torch.zeros_like(fs), fs)
    zero = torch.zeros_like(fs)
    return (torch.where(on, fn[:, None] * nv + fs, zero), torch.where(on, -r[:, None] * torch.linalg.cross(nv, fs), zero),
            torch.where(on, h, zero), on[:, 0])


def _restate(p, pair, coeffs, dt, steps, servo=None, cundall=False, walls=None, radius=None):
    """The run's final state and the deviatoric stress of each step; radius and coefficients may require grad."""
    x, v = p["x"].double(), p["v"].double()
    dev, n = x.device, len(x)
    vec = lambda a: torch.tensor(a, dtype=torch.float64, device=dev)
    r = p["radius"].double() if radius is None else radius
    m = 4.0 / 3.0 * math.pi * r ** 3 * DENSITY
    inertia = 0.4 * m * r * r
    w = torch.zeros_like(x)
    lo, prd = vec(p["lo"]), vec(p["L"])
    per = vec([1.0, 1.0, 1.0] if walls is None else [0.0, 0.0, 1.0])
    lo_s, prd_s, cum = lo.clone(), prd.clone(), torch.zeros_like(lo)
    skin, width = 0.1, 6 if pair == "granular" else 3
    wrap = lambda x: x - per * torch.floor((x - lo) / prd) * prd
    x = wrap(x)
    i, j, key = _pairs(x.detach(), r.detach(), lo.detach(), prd.detach(), per, skin)
    xb = x.detach()
    h = torch.zeros(len(i), width, dtype=torch.float64, device=dev)
    hw, tw = torch.zeros_like(x), torch.zeros(n, dtype=torch.bool, device=dev)

    def forces(update):
        nonlocal h, hw, tw
        d = _image(x[i] - x[j], prd, per)
        rsq = _dot(d, d)
        on = (rsq < (r[i] + r[j]) ** 2).nonzero().flatten()
        a, b, d, rsq = i[on], j[on], d[on], rsq[on]
        args = (dt, update, d, rsq, torch.sqrt(rsq), r[a], r[b], m[a], m[b], v[a], v[b], w[a], w[b], h[on])
        F, Ta, Tb, hn = _granular(*args) if pair == "granular" else _legacy(coeffs, pair == "hertz", *args)
        h = torch.zeros_like(h).index_copy(0, on, hn)
        f = torch.zeros_like(x).index_add(0, a, F).index_add(0, b, -F)
        t = torch.zeros_like(x).index_add(0, a, Ta).index_add(0, b, Tb)
        vir = (d * F).sum(0)
        if walls is not None:
            fw, tq, hw, tw = _wall(walls, dt, update, x, r, m, v, w, hw, tw)
            f, t = f + fw, t + tq
        if cundall:
            f = f * torch.where(f * v >= 0, vec(1.0 - 0.7), vec(1.0 + 0.7))
            t = t * torch.where(t * w >= 0, vec(1.0 - 0.7), vec(1.0 + 0.7))
        return f, t, vir

    f, t, _ = forces(False)
    stress = []
    for s in range(1, steps + 1):
        v = v + 0.5 * dt * f / m[:, None]
        x = x + dt * v
        w = w + 0.5 * dt * t / inertia[:, None]
        if float(((x.detach() - xb) ** 2).sum(1).max()) > 0.25 * skin * skin:
            x = wrap(x)
            xb = x.detach()
            i, j, new = _pairs(xb, r.detach(), lo.detach(), prd.detach(), per, skin)
            at = torch.searchsorted(key, new).clamp(max=len(key) - 1)
            h = torch.where((key[at] == new)[:, None], h[at], torch.zeros(1, dtype=torch.float64, device=dev))
            key = new
        f, t, vir = forces(True)
        v = v + 0.5 * dt * f / m[:, None]
        w = w + 0.5 * dt * t / inertia[:, None]
        if servo is None:
            continue
        P = (vir + (m[:, None] * v * v).sum(0)) / prd.prod()
        stress.append(P[2] - 0.5 * (P[0] + P[1]))
        P = P.mean().repeat(3) if servo["couple"] else P
        rate = servo["pgain"] * (P - servo["ptarget"])
        rate = torch.where(torch.abs(rate) > servo["max_rate"], servo["max_rate"] * torch.sign(rate.detach()), rate)
        held = torch.tensor([st == "pressure" for st in servo["style"]], device=dev)
        cum = torch.where(held, cum + dt * rate * prd, s * dt * servo["rate"] * prd_s)
        lo_n, prd_n = lo_s - 0.5 * cum, prd_s + cum
        x = lo_n + prd_n * ((x - lo) / prd)
        lo, prd = lo_n, prd_n
    return x, v, f, torch.cat([lo, lo + prd]), stress


def _host(*a):
    return [t.detach().cpu().numpy() for t in a]


def exact(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        if case["instances"] * case["steps"] > 3000:
            return None     # one small step after another: over 20 seconds
        xs, vs, bs = [], [], []
        for p, c in ensemble_members(case, seed):
            x, v, _, box, _ = _restate(p, "hertz", c, case["dt"], case["steps"], servo=ISO)
            x, v, box = _host(x, v, box)
            xs.append(x), vs.append(v), bs.append(box)
        return dict(x=np.concatenate(xs), v=np.concatenate(vs), box=np.stack(bs))
    p = packing(case, seed)
    if kind == "gradient":
        leaf = lambda a: torch.tensor(a, dtype=torch.float64, device="cuda", requires_grad=True)
        P = {k: leaf(v) for k, v in LEGACY.items()}
        r = p["radius"].clone().requires_grad_(True)
        stress = _restate(p, "hertz", P, case["dt"], case["steps"], servo=TRIAXIAL, radius=r)[4]
        q = torch.stack(stress[case["every"] - 1::case["every"]])
        (q ** 2).sum().backward()
        return dict({k: t.grad.cpu() for k, t in P.items()}, q=q.detach().cpu(), radius=r.grad.cpu())
    if kind == "drum":
        x, v, f, box, _ = _restate(p, "hooke", DRUM, case["dt"], case["steps"], walls=p["R"])
    else:
        x, v, f, box, _ = _restate(p, case["pair"], LEGACY if case["pair"] == "hertz" else GAS_HOOKE, case["dt"],
                                   case["steps"], servo=SERVOS.get(case["servo"]), cundall=case["cundall"])
    x, v, f, box = _host(x, v, f, box)
    if kind == "job":
        return dict(x=x, v=v, box=box)
    out = dict(x=x, v=v, f=f, box=box)
    if case.get("servo") == "triaxial":
        out["contacts"] = None
    return out

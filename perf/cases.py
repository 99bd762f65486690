"""The framework's work at the sizes and options its users run it with.

Every case is one pass through public entry points: a packing job on the
engine (state in, steps, observables and state out), an adjoint window, the
reference's own step loop through the compatible wrappers, its radix sort.
Each pass starts from the same inputs, so a pass is repeatable.

Kinds
  run      upload -> step(steps) -> scalars -> download.  io "host": pinned
           host arrays, particles in the caller's arbitrary order (the engine
           sorts them); io "device": torch tensors, kept in the caller's order
           (here cell order, as a program that keeps its state on the GPU has
           it).
  watch    run, observing every single step: step(1) + scalars, steps times.
  pour     run, with layers joining while it steps (dem_set_pour).
  adjoint  upload -> adjoint(steps, every): the potential energy's gradients
           with respect to the contact parameters and all radii.
  compat   dempacking.cu's loop through the compatible wrappers: the re-list
           chain, then `steps` steps of force, gather, walls, update.
  sort     the compatible RadixSort of (key, value) records.

States
  gas      spheres placed at random without overlap, solid fraction ~0.07 (as
           the 500,000-sphere lognormal and the 4,000,000-sphere bidisperse
           configurations), at rest under gravity.
  lattice  the 2,000-sphere configuration: cubic lattice, spacing 1.1 d, jitter.
  bed      a settled bed: jammed random packing (solid fraction ~0.64, ~3
           contacts per sphere, overlaps of a few thousandths of d) on the floor and
           between the walls, spheres moving slowly.
"""
import ctypes
import importlib.util
import math
import pathlib
import sys

import numpy as np
import torch
import torch.utils.checkpoint

ROOT = pathlib.Path(__file__).resolve().parents[1]
PKG_DIR = ROOT / "discrete-element-method-for-packing-cuda-c-code_b200"


def package():
    """The framework's package, imported under its short name."""
    if "dem_b200" not in sys.modules:
        spec = importlib.util.spec_from_file_location("dem_b200", PKG_DIR / "__init__.py",
                                                      submodule_search_locations=[str(PKG_DIR)])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["dem_b200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["dem_b200"]


# Reduced units of the reference: length 1 mm, time sqrt(1 mm / g).
D_REF, G, RHO, E_MOD, NU = 1e-3, 9.81, 2500.0, 1e7, 0.29
DT = 5e-7 / math.sqrt(D_REF / G)
SKIN = 0.05
RELIST = 20


def contact_constants(mu=0.3, roll_rel=0.002, e=0.5):
    """Contact parameters of E = 1e7 Pa, nu = 0.29, rho = 2500 kg/m^3 and
    restitution e, in reduced units."""
    estar = (4.0 / 3.0) * (6.0 * E_MOD / (math.pi * RHO * G * D_REF)) / (2.0 * (1.0 - NU * NU))
    ln = math.log(e)
    c = -2.0 * math.sqrt(5.0 / 18.0) * ln / math.sqrt(ln * ln + math.pi ** 2)
    return dict(estar=estar, mu=mu, nu=NU, damp_n=c, damp_t=c, roll=0.0, roll_rel=roll_rel)


# ------------------------------------------------------------------- cases
def listed():
    return [
        # the smallest configuration as shipped (2,000 spheres, FP64): latency and launches
        dict(name="lattice_2k_fp64", kind="run", state="lattice", n=2000, precision="fp64", mode="pccp", io="host",
             steps=400),
        # a user who records every step's observables of a small bed
        dict(name="watch_3k_fp64", kind="watch", state="bed", n=3001, precision="fp64", mode="pccp", io="host",
             steps=40),
        # a short poured packing (layers join between steps), small
        dict(name="pour_2k_mixed", kind="pour", state="gas", n=2000, precision="mixed", mode="pccp", io="host",
             steps=200),
        # the headline configuration: 500,000 lognormal spheres, mixed, end to end
        dict(name="gas_500k_mixed", kind="run", state="gas", n=500_000, precision="mixed", mode="pccp", io="host",
             steps=400),
        # the same in the plain FP64 form, state kept on the GPU
        dict(name="gas_500k_fp64", kind="run", state="gas", n=500_000, precision="fp64", mode="pccp", io="device",
             steps=200),
        # the memory-scale configuration: 4,000,000 bidisperse spheres, mixed
        dict(name="gas_4m_mixed", kind="run", state="gas", n=4_000_000, precision="mixed", mode="pccp", io="device",
             steps=100),
        # where a packing ends up: the 500,000 spheres as a settled bed, mixed
        dict(name="bed_500k_mixed", kind="run", state="bed", n=500_000, precision="mixed", mode="pccp", io="host",
             steps=100),
        # a settled bed of ragged size in the plain FP64 form
        dict(name="bed_100k_fp64", kind="run", state="bed", n=100_003, precision="fp64", mode="pccp", io="device",
             steps=100),
        # the paper's particle-parallel form on a bed
        dict(name="bed_60k_mixed_pp", kind="run", state="bed", n=60_001, precision="mixed", mode="pp", io="host",
             steps=100),
        # parameter identification on a settled bed: gradients over a window, two checkpoints
        dict(name="adjoint_20k_mixed", kind="adjoint", state="bed", n=20_011, precision="mixed", mode="pccp",
             io="host", steps=200, every=100),
        # the drop-in wrappers under the reference's own loop, one re-list and ten steps
        dict(name="compat_50k", kind="compat", state="bed", n=50_000, precision="fp64", mode="pccp", io="device",
             steps=10),
        # the wrappers' radix sort alone, all 32 key bits
        dict(name="sort_1m", kind="sort", state="keys", n=1_000_000, precision="u32", mode="pccp", io="device",
             steps=1, bits=32),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["run", "run", "run", "run", "run", "watch", "pour", "adjoint", "compat", "sort"])
    c = dict(kind=kind, state="bed", n=0, precision=rng.choice(["mixed", "mixed", "fp64"]), mode="pccp",
             io=rng.choice(["host", "device"]), steps=0)
    if kind == "run":
        c["state"] = rng.choice(["gas", "bed", "bed"])
        c["mode"] = rng.choice(["pccp", "pccp", "pccp", "pp"])
        if c["state"] == "gas":
            c.update(n=size(500, 2_000_000))
            c.update(steps=rng.choice([60, 100, 130]))
        else:
            c.update(n=size(500, 150_000))
            c.update(steps=rng.choice([40, 60, 90, 100]))
    elif kind == "watch":
        c.update(n=size(500, 60_000), steps=rng.choice([25, 40]), io="host")
    elif kind == "pour":
        c.update(state="gas", n=size(500, 20_000), steps=rng.choice([100, 150, 200]), io="host")
    elif kind == "adjoint":
        every = rng.choice([20, 60, 100])
        c.update(n=size(1000, 20_000), every=every, steps=every * rng.choice([1, 2]), io="host")
    elif kind == "compat":
        c.update(n=size(1000, 100_000), steps=rng.choice([1, 5, 10]), precision="fp64", io="device")
    else:
        c.update(state="keys", n=size(1000, 4_000_000), precision="u32", io="device", steps=1,
                 bits=rng.choice([16, 20, 24, 32]))
    return c


# ------------------------------------------------------------------ states
def generator(seed, salt):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed * 1000003 + salt)
    return g


def uniform(g, *shape):
    return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64)


def lognormal_radii(g, n):
    """Median 0.5, sigma 0.2, truncated to [0.3, 0.8]; FP32-representable."""
    r = torch.empty(n, device="cuda", dtype=torch.float64)
    todo = torch.arange(n, device="cuda")
    while todo.numel():
        v = torch.exp(math.log(0.5) + 0.2 * torch.randn(todo.numel(), generator=g, device="cuda", dtype=torch.float64))
        ok = (v >= 0.3) & (v <= 0.8)
        r[todo[ok]] = v[ok]
        todo = todo[~ok]
    return r.float().double()


def cell_ids(x, lo, cs, dims):
    c = ((x - lo) / cs).floor().long()
    c = torch.minimum(c.clamp_(min=0), torch.tensor(dims, device=x.device) - 1)
    return c


def close_pairs(x, rad, gap, queries=None):
    """All pairs (i, j), j != i, with |x_i - x_j| < r_i + r_j + gap, i from
    `queries` (default: every particle, each pair once with i < j)."""
    n = x.shape[0]
    lo = x.min(0).values - 1e-9
    cs = 2.0 * float(rad.max()) + gap + 1e-9
    dims = [int(v) + 1 for v in ((x.max(0).values - lo) / cs).tolist()]
    c = cell_ids(x, lo, cs, dims)
    key = (c[:, 2] * dims[1] + c[:, 1]) * dims[0] + c[:, 0]
    order = torch.argsort(key, stable=True)
    counts = torch.bincount(key, minlength=dims[0] * dims[1] * dims[2])
    start = torch.cumsum(counts, 0) - counts
    q = torch.arange(n, device=x.device) if queries is None else queries
    out_i, out_j = [], []
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                m = c[q] + torch.tensor([dx, dy, dz], device=x.device)
                inside = ((m >= 0) & (m < torch.tensor(dims, device=x.device))).all(1)
                a, m = q[inside], m[inside]
                k = (m[:, 2] * dims[1] + m[:, 1]) * dims[0] + m[:, 0]
                s, cnt = start[k], counts[k]
                top = int(cnt.max()) if cnt.numel() else 0
                for t in range(top):
                    sel = cnt > t
                    i, j = a[sel], order[s[sel] + t]
                    d = x[j] - x[i]
                    near = (d * d).sum(1) < (rad[i] + rad[j] + gap) ** 2
                    near &= (j > i) if queries is None else (j != i)
                    out_i.append(i[near])
                    out_j.append(j[near])
    return torch.cat(out_i), torch.cat(out_j)


def gas_state(n, seed, bidisperse):
    """Spheres at random in a box of solid fraction ~0.07, no overlaps: the
    later of two overlapping spheres is placed again until none overlap."""
    g = generator(seed, 1)
    if bidisperse:
        rad = torch.where(torch.randperm(n, generator=g, device="cuda") % 2 == 0, 0.4, 0.6).double().float().double()
    else:
        rad = lognormal_radii(g, n)
    vol = n * 8.0                                    # one sphere per 8 mm^3
    side = (vol / 4.0) ** (1.0 / 3.0) if n >= 100_000 else (vol / 2.0) ** (1.0 / 3.0)
    side = max(side, 4.0)
    world = (side, side, max(vol / side ** 2, 4.0))
    w = torch.tensor(world, device="cuda", dtype=torch.float64)

    def place(idx):
        r = rad[idx, None]
        lo = torch.cat([r - w[0] / 2, r - w[1] / 2, r], 1)
        hi = torch.cat([w[0] / 2 - r, w[1] / 2 - r, w[2] - r], 1)
        return lo + (hi - lo) * uniform(g, idx.numel(), 3)

    todo = torch.arange(n, device="cuda")
    x = place(todo)
    while todo.numel():
        i, j = close_pairs(x, rad, 1e-3, todo)
        # a sphere that was just placed gives way to one that was not, and the
        # larger index to the smaller
        fresh = torch.zeros(n, dtype=torch.bool, device="cuda")
        fresh[todo] = True
        bad = torch.zeros(n, dtype=torch.bool, device="cuda")
        bad[i[(~fresh[j]) | (j < i)]] = True
        todo = bad.nonzero()[:, 0]
        if todo.numel():
            x[todo] = place(todo)
    v = torch.zeros_like(x)
    return x, v, torch.zeros_like(x), rad, world


def lattice_state(n, seed):
    g = generator(seed, 2)
    k = torch.arange(n, device="cuda")
    per = 18 * 18
    x = torch.stack([(k % 18) - 8.5, ((k // 18) % 18) - 8.5, k // per + 0.5], 1).double() * 1.1
    x += 0.04 * (2.0 * uniform(g, n, 3) - 1.0)
    rad = torch.full((n,), 0.5, device="cuda", dtype=torch.float64)
    return x, torch.zeros_like(x), torch.zeros_like(x), rad, (20.0, 20.0, 100.0)


def jammed_block(g, m, mono):
    """m spheres in a periodic cube at random close packing, pushed apart (with
    momentum, stopped when it goes uphill) until the overlaps are a few
    thousandths of d: ~3 contacts and ~3.7 pairs within the skin per sphere,
    as in a bed settled under gravity."""
    rad = torch.full((m,), 0.5, device="cuda", dtype=torch.float64) if mono else lognormal_radii(g, m)
    solid = 0.635 if mono else 0.64
    L = (float((4.0 / 3.0 * math.pi * rad ** 3).sum()) / solid) ** (1.0 / 3.0)
    x = L * uniform(g, m, 3)
    v = torch.zeros_like(x)
    rr = rad[:, None] + rad[None, :]
    for _ in range(400):
        d = x[:, None, :] - x[None, :, :]
        d -= L * torch.round(d / L)
        dist = torch.sqrt((d * d).sum(2))
        dist.fill_diagonal_(1e9)
        f = torch.einsum("ij,ijk->ik", (rr - dist).clamp_(min=0.0) / dist, d)
        v = 0.92 * v + 0.25 * f
        v = v * ((v * f).sum() >= 0)
        x = torch.remainder(x + v, L)
    return x, rad, L


def bed_state(n, seed, mono=False):
    g = generator(seed, 3)
    m = 1200
    bx, br, L = jammed_block(g, m, mono)
    across = max(1, round((n / m) ** (1.0 / 3.0)))
    up = 1
    while True:
        t = torch.stack(torch.meshgrid(*[torch.arange(k, device="cuda", dtype=torch.float64)
                                         for k in (across, across, up)], indexing="ij"), -1).reshape(-1, 1, 3)
        x = (bx[None] + L * t).reshape(-1, 3)
        r = br.repeat(t.shape[0])
        x[:, :2] -= 0.5 * L * across
        half = 0.5 * L * across
        keep = (x[:, 0].abs() < half - 0.997 * r) & (x[:, 1].abs() < half - 0.997 * r) & (x[:, 2] > 0.997 * r)
        if int(keep.sum()) >= n and (up == 1 or float(x[keep][:, 2].sort().values[n - 1]) < L * up - 1.0):
            break
        up += 1
    x, r = x[keep], r[keep]
    low = torch.argsort(x[:, 2], stable=True)[:n]
    x, r = x[low], r[low]
    x = x + 2e-4 * (2.0 * uniform(g, n, 3) - 1.0)
    v = 0.3 * DT * (2.0 * uniform(g, n, 3) - 1.0)
    a = 0.3 * DT * (2.0 * uniform(g, n, 3) - 1.0)
    world = (2.0 * half, 2.0 * half, float(x[:, 2].max()) + 5.0)
    return x, v, a, r, world


def initial_state(case, seed):
    """Positions, displacements and rotations per step, radii, box; on the GPU
    in 64 bits, in the order the case's user has them."""
    n = case["n"]
    if case["state"] == "gas":
        x, v, a, r, world = gas_state(n, seed, bidisperse=n >= 3_000_000)
    elif case["state"] == "lattice":
        x, v, a, r, world = lattice_state(n, seed)
    else:
        x, v, a, r, world = bed_state(n, seed, mono=case["kind"] == "compat")
    if case["kind"] == "pour":
        order = torch.argsort(x[:, 2], stable=True)      # layers from below
    elif case["io"] == "host":
        order = torch.randperm(n, generator=generator(seed, 4), device="cuda")
    else:
        lo = torch.tensor([-0.5 * world[0], -0.5 * world[1], 0.0], device="cuda", dtype=torch.float64)
        cs = 2.0 * float(r.max()) + SKIN
        dims = [int(s / cs) + 1 for s in world]
        c = cell_ids(x, lo, cs, dims)
        order = torch.argsort((c[:, 2] * dims[1] + c[:, 1]) * dims[0] + c[:, 0], stable=True)
    x, v, a, r = (t[order].contiguous() for t in (x, v, a, r))
    return x, v, a, r, world


def friction(case):
    return dict(mu=0.5, roll_rel=0.005) if case["n"] >= 3_000_000 else dict(mu=0.3, roll_rel=0.002)


def pour_plan(case):
    """Layers of a tenth of the spheres; half are in at the start and a layer
    joins about every 60 steps."""
    per = max(1, case["n"] // 10)
    return per, 60.2 * DT, case["n"] // 2


# ----------------------------------------------------------------- prepare
COMPAT_CUB, COMPAT_ROW = 1.2, 30


class State:
    pass


def pinned(t):
    return t.reshape(-1).cpu().pin_memory().numpy()


def prepare(case, seed):
    s = State()
    s.case = case
    if case["kind"] == "sort":
        g = generator(seed, 5)
        n = case["n"]
        s.records = torch.empty((n, 2), dtype=torch.int32, device="cuda")
        # cell keys: ~1.6 records per key over the low `bits` bits
        top = min(2 ** case["bits"], 2 ** 31) - 1
        s.records[:, 0] = torch.randint(0, top, (n,), generator=g, device="cuda", dtype=torch.int64).int()
        s.records[:, 1] = torch.arange(n, device="cuda", dtype=torch.int32)
        s.work0, s.work1 = torch.empty_like(s.records), torch.empty_like(s.records)
        return s
    dem = package()
    x, v, a, r, world = initial_state(case, seed)
    s.world = world
    if case["kind"] == "compat":
        return prepare_compat(s, x, v, a, r)
    p = contact_constants(**friction(case))
    s.engine = dem.Engine(case["n"], world, DT, SKIN,
                          precision=dem.PREC_MIXED if case["precision"] == "mixed" else dem.PREC_FP64,
                          relist_interval=RELIST, cell=2.0 * float(r.max()) + SKIN + 1e-4,
                          force_mode=dem.FORCE_PP if case["mode"] == "pp" else dem.FORCE_PCCP)
    s.engine.set_material(p, dict(p))
    if case["io"] == "host":
        s.inputs = [pinned(t) for t in (x, r, v, a)]
        s.outputs = [pinned(torch.empty(3 * case["n"], dtype=torch.float64)) for _ in range(3)]
    else:
        s.inputs = [t.reshape(-1) for t in (x, r, v, a)]
        s.outputs = [torch.empty(3 * case["n"], dtype=torch.float64, device="cuda") for _ in range(3)]
    return s


def prepare_compat(s, x, v, a, r):
    dem = package()
    n, c = s.case["n"], 3
    s.state0 = [t.reshape(-1) for t in (x, v, a)]
    s.rad = r
    s.mass = 8.0 * r ** 3
    s.inert = 0.4 * s.mass * r * r
    s.cell = (COMPAT_CUB,) * 3
    s.origin = (-0.5 * s.world[0], -0.5 * s.world[1], 0.0)
    s.grid = tuple(int(w / COMPAT_CUB) + 1 for w in s.world)
    cells = s.grid[0] * s.grid[1] * s.grid[2]
    cap = n * COMPAT_ROW

    def words(k):
        return torch.zeros(k, dtype=torch.int32, device="cuda")

    def reals(k):
        return torch.zeros(k, dtype=torch.float64, device="cuda")

    s.pos, s.pdis, s.angv, s.qi = (reals(c * n) for _ in range(4))
    s.hash0, s.hash1, s.cell_start = words(2 * n), words(2 * n), words(cells)
    s.anei, s.aref = words(cap), words(cap)
    s.njgi, s.njli, s.sjgi, s.oldsjgi, s.contacts = (words(n) for _ in range(5))
    s.lp, s.ln, s.oldln, s.contactpair = (words(cap) for _ in range(4))
    s.hist, s.oldhist, s.fpair, s.ti, s.tj = (reals(c * cap) for _ in range(5))
    s.fric, s.oldfric = reals(cap), reals(cap)
    s.histw, s.fricw, s.fi, s.tq = reals(c * n), reals(n), reals(c * n), reals(c * n)
    p = contact_constants()
    dem.compat.set_cutoff(1.0, COMPAT_CUB)
    dem.compat.set_material(dict(estarp=p["estar"], ufricp=p["mu"], vpois=NU, dampnp=p["damp_n"], damptp=p["damp_t"],
                                 upp=5e-4),
                            dict(estarw=p["estar"], ufricw=p["mu"], vpoisw=NU, dampnw=p["damp_n"],
                                 damptw=p["damp_t"], upw=5e-4))
    return s


# --------------------------------------------------------------------- run
def run(s):
    kind = s.case["kind"]
    if kind == "sort":
        s.work0.copy_(s.records)
        package().compat.RadixSort(s.work0, s.work1, s.case["n"], s.case["bits"])
        return s.work0
    if kind == "compat":
        return run_compat(s)
    dem, e, case = package(), s.engine, s.case
    x, r, v, a = s.inputs
    if case["io"] == "host":
        e.upload(x, r, v, a)
    else:
        e.upload_device(x, r, v, a)
    if kind == "adjoint":
        g = e.adjoint(case["steps"], case["every"], dem.OBJ_POTENTIAL)
        out = {"value": g["value"], "d_radii": g["d_radii"]}
        for side in ("d_pp", "d_pw"):
            out[side] = np.array([g[side][k] for k in PARAMS])
        return out
    if kind == "pour":
        e.set_pour(*pour_plan(case))
    if kind == "watch":
        seen = []
        for _ in range(case["steps"]):
            e.step(1)
            seen.append(e.scalars())
        q = seen[-1]
        watched = {"contacts": np.array([k["contacts"] for k in seen]),
                   "height": np.array([k["maxhz"] for k in seen])}
    else:
        e.step(case["steps"])
        q = e.scalars()
        watched = {"contacts": q["contacts"], "height": q["maxhz"]}
    if case["io"] == "host":
        dem.check(dem.lib().dem_download_state(e.handle, *[o.ctypes.data_as(ctypes.c_void_p) for o in s.outputs]))
    else:
        e.download_device(*s.outputs)
    return {"pos": s.outputs[0], "pdis": s.outputs[1], "angv": s.outputs[2], "pairs": q["pairs"],
            "fraction": q["packing_fraction"], **watched}


def run_compat(s):
    c, n = package().compat, s.case["n"]
    for t, t0 in zip((s.pos, s.pdis, s.angv), s.state0):
        t.copy_(t0)
    for t in (s.qi, s.sjgi, s.histw, s.fricw):
        t.zero_()
    c.calcHash(s.pos, s.hash0, s.grid, s.cell, s.origin, n)
    c.RadixSort(s.hash0, s.hash1, n, 32)
    c.findCellStart(s.hash0, s.cell_start, n, s.cell_start.numel())
    c.neighborarray(s.pos, s.hash0, s.cell_start, s.grid, s.cell, s.origin, COMPAT_ROW, n, s.anei, s.njgi, s.njli)
    total = c.prefixsum(n, s.njgi, s.sjgi, s.oldsjgi)
    c.pairlist(s.sjgi, s.oldsjgi, s.oldln, s.anei, s.njgi, s.njli, s.oldhist, s.oldfric, COMPAT_ROW, COMPAT_ROW, n,
               s.aref, s.lp, s.ln, s.hist, s.fric)
    for _ in range(s.case["steps"]):
        c.calculateforcepair(s.pos, s.pdis, s.angv, s.rad, s.mass, s.lp, s.ln, s.oldln, s.hist, s.fric, s.oldhist,
                             s.oldfric, DT, s.fpair, s.ti, s.tj, s.contactpair, total)
        c.sumallforcei(COMPAT_ROW, n, s.njgi, s.njli, s.fpair, s.ti, s.tj, s.contactpair, s.aref, s.fi, s.tq,
                       s.contacts)
        c.calculateforceiw(s.world, s.pos, s.pdis, s.angv, s.rad, s.mass, DT, total, n, s.histw, s.fricw, s.fi, s.tq)
        moved, height = c.updateposition(s.world, n, s.pos, s.pdis, s.angv, s.mass, s.inert, s.fi, s.tq, s.qi, DT)
    touching = c.outputporositycn(n, s.contacts, height, s.world)
    return {"pos": s.pos, "pdis": s.pdis, "angv": s.angv, "force": s.fi, "torque": s.tq, "contacts": s.contacts,
            "lp": s.lp, "ln": s.ln, "height": height, "touching": touching, "moved": moved}


# -------------------------------------------------------------------- work
def work(case):
    """State read once and written once (positions, displacements, rotations;
    radii), the operations of the steps: about 300 per touching pair, 40 per
    sphere.  Sort: records read and written once."""
    n, steps = case["n"], case["steps"]
    if case["kind"] == "sort":
        return {"bytes": 16.0 * n, "flops": 0.0}
    contacts = 3.0 * n if case["state"] == "bed" else 0.0
    flops = steps * (300.0 * contacts + 40.0 * n)
    b = n * (9 * 8 + 8 + 9 * 8)
    if case["kind"] == "adjoint":
        return {"bytes": float(b), "flops": 5.0 * flops}
    return {"bytes": float(b), "flops": flops}


# ------------------------------------------------------- 64-bit expectation
PARAMS = ("estar", "mu", "damp_n", "damp_t", "roll", "roll_rel")
WALLS = ((0.0, 0.0, -1.0), (-1.0, 0.0, 0.0), (1.0, 0.0, 0.0), (0.0, -1.0, 0.0), (0.0, 1.0, 0.0))


def cross(a, b):
    return torch.linalg.cross(a, b, dim=1)


def safe_sqrt(v):
    """sqrt(v) with a zero derivative at v <= 0."""
    pos = v > 0
    return torch.where(pos, torch.where(pos, v, torch.ones_like(v)).sqrt(), torch.zeros_like(v))


def hertz_mindlin(delta, nrm, rstar, mstar, U, Wr, xi, c):
    """Force on i, its tangential part, the rolling torque on i and the new
    tangential history of touching pairs (the published Hertz-Mindlin law with
    viscous damping, Coulomb limit and rolling resistance)."""
    delta, rstar, mstar = delta[:, None], rstar[:, None], mstar[:, None]
    fe = c["estar"] * rstar.sqrt() * delta * delta.sqrt()
    un = (U * nrm).sum(1, keepdim=True)
    cn = c["damp_n"] * (4.5 * c["estar"] * mstar * (rstar * delta).sqrt()).sqrt()
    fn = fe - cn * un / DT
    ut = U - un * nrm
    xi = xi - (xi * nrm).sum(1, keepdim=True) * nrm + ut
    xmax = c["mu"] * (2.0 - c["nu"]) / (2.0 * (1.0 - c["nu"])) * delta
    length = safe_sqrt((xi * xi).sum(1, keepdim=True))
    rest = 1.0 - torch.minimum(length, xmax) / xmax
    so = safe_sqrt(rest)
    fel = c["mu"] * fe * (1.0 - rest * so)
    ct = c["damp_t"] * safe_sqrt(6.0 * c["mu"] * mstar * fe * so / xmax)
    ft = torch.where(length > 0, fel / torch.where(length > 0, length, torch.ones_like(length)),
                     torch.zeros_like(length)) * xi + ct * ut / DT
    size = safe_sqrt((ft * ft).sum(1, keepdim=True))
    cap = c["mu"] * fe
    ft = torch.where(size > cap, ft * cap / torch.where(size > 0, size, torch.ones_like(size)), ft)
    xi = torch.where(length > xmax, xi * xmax / torch.where(length > 0, length, torch.ones_like(length)), xi)
    w = safe_sqrt((Wr * Wr).sum(1, keepdim=True))
    mr = torch.where(w > 1e-30, -(c["roll"] + c["roll_rel"] * rstar) * fe / torch.where(w > 0, w, torch.ones_like(w)),
                     torch.zeros_like(w)) * Wr
    return ft - fn * nrm, ft, mr, xi


class Reference:
    """The step in 64-bit torch: contacts, walls, gravity, symplectic Euler in
    displacement form; history of a pair kept while it touches."""

    def __init__(self, x, v, a, rad, world, pp, pw):
        self.x, self.v, self.a, self.rad, self.world, self.pp, self.pw = x, v, a, rad, world, pp, pw
        self.m = 8.0 * rad ** 3
        self.inertia = 0.4 * self.m * rad ** 2
        self.hw = torch.zeros_like(x)
        self.key = torch.empty(0, dtype=torch.int64, device=x.device)
        self.h = torch.empty((0, 3), dtype=torch.float64, device=x.device)

    def relist(self, act):
        n = self.x.shape[0]
        i, j = close_pairs(self.x[:act].detach(), self.rad[:act].detach(), SKIN)
        key, order = (i * n + j).sort()
        h = torch.zeros((key.numel(), 3), dtype=torch.float64, device=key.device)
        if self.key.numel() and key.numel():
            at = torch.searchsorted(self.key, key).clamp(max=self.key.numel() - 1)
            h = torch.where((self.key[at] == key)[:, None], self.h[at], h)
        self.key, self.h, self.i, self.j = key, h, i[order], j[order]

    def forces(self, act):
        x, v, a, r, m = self.x, self.v, self.a, self.rad, self.m
        F, T = torch.zeros_like(x), torch.zeros_like(x)
        on = act_mask(x, act)
        F = F - torch.stack([torch.zeros_like(m), torch.zeros_like(m), m * on], 1)
        d = x[self.j] - x[self.i]
        with torch.no_grad():
            t = ((self.rad[self.i] + self.rad[self.j]) - (d * d).sum(1).sqrt() > 0).nonzero()[:, 0]
        i, j = self.i[t], self.j[t]
        self.touching = int(t.numel())
        h = torch.zeros_like(self.h)
        if self.touching:
            d = x[j] - x[i]
            dist = (d * d).sum(1).sqrt()
            nrm = d / dist[:, None]
            ri, rj = r[i], r[j]
            U = v[j] - v[i] - cross(ri[:, None] * a[i] + rj[:, None] * a[j], nrm)
            f, ft, mr, hn = hertz_mindlin(ri + rj - dist, nrm, ri * rj / (ri + rj), m[i] * m[j] / (m[i] + m[j]), U,
                                          a[i] - a[j], self.h[t], self.pp)
            nf = cross(nrm, ft)
            F = F.index_add(0, i, f).index_add(0, j, -f)
            T = T.index_add(0, i, ri[:, None] * nf + mr).index_add(0, j, rj[:, None] * nf - mr)
            h = h.index_copy(0, t, hn)
        self.h = h
        hx, hy = 0.5 * self.world[0], 0.5 * self.world[1]
        over = torch.stack([r - x[:, 2], r - (x[:, 0] + hx), r - (hx - x[:, 0]), r - (x[:, 1] + hy),
                            r - (hy - x[:, 1])], 1)
        first = over.detach().argmax(1)
        hw = torch.zeros_like(self.hw)
        for k in range(5):
            b = ((over[:, k].detach() > 0) & (on > 0)).nonzero()[:, 0]
            if not b.numel():
                continue
            nrm = torch.tensor(WALLS[k], device=x.device, dtype=torch.float64).expand(b.numel(), 3)
            own = (first[b] == k)[:, None]
            U = -v[b] - r[b][:, None] * cross(a[b], nrm)
            f, ft, mr, hn = hertz_mindlin(over[b, k], nrm, r[b], m[b], U, a[b],
                                          torch.where(own, self.hw[b], torch.zeros_like(self.hw[b])), self.pw)
            F = F.index_add(0, b, f)
            T = T.index_add(0, b, r[b][:, None] * cross(nrm, ft) + mr)
            hw = hw.index_add(0, b, torch.where(own, hn, torch.zeros_like(hn)))
        self.hw = hw
        self.F, self.T = F, T
        return F, T

    def step(self, act):
        F, T = self.forces(act)
        on = act_mask(self.x, act)[:, None]
        self.v = self.v + on * F * (DT * DT / self.m[:, None])
        self.a = self.a + on * T * (DT * DT / self.inertia[:, None])
        self.x = self.x + on * self.v

    def height(self, act):
        return max(0.0, float(self.x[:act, 2].detach().max())) if act else 0.0

    def potential(self):
        x, r = self.x, self.rad
        u = (self.m * x[:, 2]).sum()
        d = x[self.j] - x[self.i]
        dist = (d * d).sum(1).sqrt()
        ri, rj = r[self.i], r[self.j]
        over = ri + rj - dist
        t = over.detach() > 0
        over, rs = over[t], (ri * rj / (ri + rj))[t]
        u = u + (0.4 * self.pp["estar"] * rs.sqrt() * over ** 2 * over.sqrt()).sum()
        hx, hy = 0.5 * self.world[0], 0.5 * self.world[1]
        for w in (r - x[:, 2], r - (x[:, 0] + hx), r - (hx - x[:, 0]), r - (x[:, 1] + hy), r - (hy - x[:, 1])):
            t = w.detach() > 0
            u = u + (0.4 * self.pw["estar"] * r[t].sqrt() * w[t] ** 2 * w[t].sqrt()).sum()
        return u


def act_mask(x, act):
    on = torch.ones(x.shape[0], dtype=torch.float64, device=x.device)
    on[act:] = 0.0
    return on


def exact(case, seed):
    """What run returns, from the 64-bit reference above; whole numbers have no
    other value than their own."""
    if case["kind"] == "sort":
        return None
    x, v, a, r, world = initial_state(case, seed)
    n, steps = case["n"], case["steps"]
    if case["kind"] == "compat":
        p = dict(contact_constants(), roll=5e-4, roll_rel=0.0)
        q = Reference(x, v, a, r, world, p, dict(p))
        with torch.no_grad():
            q.relist(n)
            for _ in range(steps):
                q.step(n)
        return {"pos": q.x.reshape(-1), "pdis": q.v.reshape(-1), "angv": q.a.reshape(-1), "force": q.F.reshape(-1),
                "torque": q.T.reshape(-1), "contacts": None, "lp": None, "ln": None, "height": q.height(n),
                "touching": None, "moved": None}
    p = contact_constants(**friction(case))
    if case["kind"] == "adjoint":
        return exact_adjoint(case, x, v, a, r, world, p)
    q = Reference(x, v, a, r, world, p, dict(p))
    act, heights = n, []
    if case["kind"] == "pour":
        per, every, act = pour_plan(case)
    with torch.no_grad():
        since = 0
        for k in range(steps):
            if case["kind"] == "pour" and act < n and DT * (k + 1) > float(np.float32(act)) * every / float(per):
                act, since = min(act + per, n), 0
            if since == 0:
                q.relist(act)
            q.step(act)
            since = (since + 1) % RELIST
            if case["kind"] == "watch":
                heights.append(q.height(n))
    height = q.height(act)
    solid = float((4.0 / 3.0 * math.pi * r[:act] ** 3).sum()) / (world[0] * world[1] * height)
    return {"pos": q.x.reshape(-1), "pdis": q.v.reshape(-1), "angv": q.a.reshape(-1), "pairs": None, "contacts": None,
            "fraction": solid, "height": np.array(heights) if heights else height}


def exact_adjoint(case, x, v, a, r, world, p):
    rad = r.clone().requires_grad_(True)
    sides = []
    for _ in range(2):
        sides.append({k: torch.tensor(val, device="cuda", dtype=torch.float64, requires_grad=k in PARAMS)
                      for k, val in p.items()})
    q = Reference(x, v, a, rad, world, *sides)

    def segment(x, v, a, hw, h, *leaves):
        q.x, q.v, q.a, q.hw, q.h = x, v, a, hw, h
        for _ in range(RELIST):
            q.step(case["n"])
        return q.x, q.v, q.a, q.hw, q.h

    leaves = [rad] + [s[k] for s in sides for k in PARAMS]
    for _ in range(case["steps"] // RELIST):
        q.relist(case["n"])
        i, j, key = q.i, q.j, q.key

        def window(*t, i=i, j=j, key=key):
            q.i, q.j, q.key = i, j, key
            return segment(*t)

        q.x, q.v, q.a, q.hw, q.h = torch.utils.checkpoint.checkpoint(window, q.x, q.v, q.a, q.hw, q.h, *leaves,
                                                                    use_reentrant=False)
    value = q.potential()
    grads = torch.autograd.grad(value, leaves, allow_unused=True)
    g = [0.0 if t is None else t for t in grads]
    k = len(PARAMS)
    return {"value": float(value.detach()), "d_radii": g[0], "d_pp": np.array([float(t) for t in g[1:1 + k]]),
            "d_pw": np.array([float(t) for t in g[1 + k:]])}

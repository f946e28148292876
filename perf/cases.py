"""The workloads this solver's speed is measured on, and their exact answers.

Each case goes through the package's public entry points the way a user's
program does: a handle is made once and kept (``prepare``), a pass is one
piece of the program's work (``run``).

* solve   from rest: init_dist_macro, N lattice steps, the macros read back
          into pinned host memory (and the distributions, where small).
* resume  a checkpoint's distributions up, N steps, the distributions down.
* first   a geometry never seen before: flag grid (or V.bin records) to
          handle, N steps, permeability and macros, handle closed.
* pool    scans of uneven size admitted into a batched pool, some
          intervals stepped, permeabilities and macros read, all released.
* serve   a burst of requests through the continuous-batching server until
          every one has reached its tolerance.
* pack    the device sphere-pack generator, its flag grid on the host.

``exact`` restates the lattice model (D3Q19 BGK with porelb's link
bounce-back or half-way walls) in plain 64-bit torch, and the sphere-pack
rule in numpy, without the package's code.
"""
import math
from statistics import NormalDist
from types import SimpleNamespace

import numpy as np
import torch

import porelb_gb300 as P
from porelb_gb300.batch import Batch
from porelb_gb300.serve import Server

VALUE_BYTES = {"fp64_exact": 8, "fp64": 8, "fp64_fma": 8, "fp32": 4,
               "fp16dev": 2, "bf16dev": 2}
# rough steps per second and node of each form (sizes the drawn cases only)
RATE = {"fp64_exact": 2.0e9, "fp64": 14e9, "fp64_fma": 3e9, "fp32": 26e9,
        "fp16dev": 33e9, "bf16dev": 33e9}
FLOPS_PER_NODE = 250   # adds and multiplies of one collision

# D3Q19 in the reference's order
EX = (0, 1, -1, 0, 0, 0, 0, 0, 0, 0, 0, -1, 1, -1, 1, -1, 1, -1, 1)
EY = (0, 0, 0, 1, -1, 0, 0, 1, -1, -1, 1, 0, 0, 0, 0, 1, -1, -1, 1)
EZ = (0, 0, 0, 0, 0, 1, -1, 1, -1, 1, -1, -1, 1, 1, -1, 0, 0, 0, 0)
W = (1 / 3,) + (1 / 18,) * 6 + (1 / 36,) * 12
OPP = (0,) + tuple(j + 1 if j % 2 else j - 1 for j in range(1, 19))


# ------------------------------------------------------------------ cases

def _solve(name, dims, precision, steps, **kw):
    c = dict(name=name, kind="solve", nx=dims[0], ny=dims[1], nz=dims[2],
             precision=precision, steps=steps, porosity=0.35, rmin=4.0,
             rmax=10.0, tau=0.8, force=5e-7, boundary="reference", num_p=1,
             source="flag", tile=1, with_f=False)
    c.update(kw)
    return c


def listed():
    c1 = dict(porosity=0.40, rmin=6.0, rmax=6.0, tau=1.0, force=1e-6)
    return [
        # the smoke test's domain in the default, bit-exact form: the
        # smallest call a user makes (3.3k nodes, launches and latency)
        _solve("tiny_exact", (24, 20, 16), "fp64_exact", 40, porosity=0.45,
               rmin=3.0, rmax=5.0, force=1e-4, source="table", with_f=True),
        # the 64^3 plain configuration, in the default form
        _solve("cube64_exact", (64, 64, 64), "fp64_exact", 100,
               source="table", with_f=True, **c1),
        # the same in the fast FP64 form, a stretch between two checks
        _solve("cube64_fp64", (64, 64, 64), "fp64", 500, with_f=True, **c1),
        # a decomposed table (4 slabs, mpirun -np 4), ragged box, bit-exact
        _solve("slabs_exact", (129, 127, 124), "fp64_exact", 30, num_p=4,
               source="table"),
        # the headline configuration: 256^3 sphere pack, FP64
        _solve("plain256_fp64", (256, 256, 256), "fp64", 60, tile=2),
        # reduced storage, odd sizes, half-way walls
        _solve("ragged_fp32", (246, 266, 234), "fp32", 60, tile=2,
               boundary="halfway"),
        # the largest: 64M cells in scaled FP16 deviations
        _solve("large400_fp16", (400, 400, 400), "fp16dev", 40, tile=2),
        # restart from a checkpoint, checkpoint again
        _solve("resume96_fp64", (96, 96, 96), "fp64", 20, kind="resume"),
        # a new 160^3 geometry to its first answers
        _solve("first160_fp32", (160, 160, 160), "fp32", 20, kind="first"),
        # the batched workload's shape: uneven samples in one FP32 pool
        dict(name="pool_fp32", kind="pool", precision="fp32", samples=12,
             median=72, sigma=0.5, lo=32, hi=128, check_every=200,
             intervals=2, force=1e-6),
        # the serving workload's shape: a burst of requests to convergence
        dict(name="serve_fp32", kind="serve", precision="fp32", samples=10,
             median=64, sigma=0.4, lo=48, hi=128, check_every=250, tol=1e-6,
             force=1e-6),
        # geometry generation alone
        dict(name="pack200", kind="pack", nx=200, ny=192, nz=210,
             porosity=0.30, rmin=3.0, rmax=8.0),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["solve"] * 6 + ["resume", "first", "pool", "pool",
                                       "serve", "pack"])
    if kind == "pool":
        return dict(kind=kind, precision=rng.choice(["fp32", "fp32", "fp16dev",
                                                     "bf16dev", "fp64"]),
                    samples=rng.randint(2, 14), median=round(_log(rng, 36, 80)),
                    sigma=rng.uniform(0.1, 0.5), lo=32, hi=128,
                    check_every=rng.choice([50, 100, 200]),
                    intervals=rng.randint(1, 3), force=1e-6)
    if kind == "serve":
        return dict(kind=kind, precision="fp32", samples=rng.randint(2, 10),
                    median=round(_log(rng, 48, 68)), sigma=rng.uniform(0.1, 0.4),
                    lo=48, hi=112, check_every=rng.choice([250, 500]),
                    tol=rng.choice([1e-5, 1e-6]), force=1e-6)
    edge = _log(rng, 16, 240 if kind == "solve" else 150)
    dims = [max(10, round(edge * rng.uniform(0.8, 1.25))) for _ in range(3)]
    num_p = rng.choice([1, 1, 1, 2, 4])
    dims[2] = max(num_p, dims[2] // num_p * num_p)
    rmin = min(edge / 6, rng.uniform(2.5, 5.0))
    c = dict(kind=kind, nx=dims[0], ny=dims[1], nz=dims[2],
             porosity=rng.uniform(0.2, 0.5), rmin=rmin,
             rmax=rmin * rng.uniform(1.0, 2.0))
    if kind == "pack":
        return c
    precision = rng.choice(["fp64_exact", "fp64_exact", "fp64", "fp64", "fp32",
                            "fp16dev", "bf16dev", "fp64_fma"])
    nodes = c["porosity"] * dims[0] * dims[1] * dims[2]
    # 1 ms to 25 ms of steps, each step taking 3 us at least
    per_step = max(3e-6, nodes / RATE[precision])
    steps = min(400, max(2, round(_log(rng, 1e-3, 25e-3) / per_step)))
    c.update(precision=precision, steps=steps, tau=rng.uniform(0.6, 1.5),
             force=_log(rng, 2e-7, 2e-5),
             boundary=rng.choice(["reference", "reference", "halfway"]),
             num_p=num_p, source=rng.choice(["flag", "table"]), tile=1,
             with_f=nodes < 2e5)
    return c


# --------------------------------------------------------------- geometry

def _uniforms(seed, count, start=0):
    """Draws start .. start+count-1 of the splitmix64 stream of `seed`
    (Steele, Lea & Flood 2014), as 53-bit uniforms in [0, 1)."""
    with np.errstate(over="ignore"):
        k = np.arange(start + 1, start + count + 1, dtype=np.uint64)
        z = np.uint64(seed & (2 ** 64 - 1)) + k * np.uint64(0x9E3779B97F4A7C15)
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        z = z ^ (z >> np.uint64(31))
    return (z >> np.uint64(11)).astype(np.float64) * 2.0 ** -53


def _near(center, r, n):
    """Cell indices along one axis that a sphere can reach, and their
    squared periodic minimum-image distances."""
    lo, hi = math.floor(center - r) - 1, math.ceil(center + r) + 1
    i = np.arange(lo, hi + 1) % n if hi - lo + 1 <= n else np.arange(n)
    d = np.abs(i - center)
    d = np.minimum(d, n - d)
    return i, d * d


def sphere_flag(seed, dims, rmin, rmax, porosity, trim=False):
    """Periodic sphere pack: uint8 flag[z, y, x], 1 = fluid.  Spheres (centre
    and radius drawn from the seed) are added until the fluid fraction is at
    most `porosity`.  With `trim` the last sphere gives back the cells it took
    too many, so that every seed has the same number of fluid cells."""
    nx, ny, nz = dims
    flag = np.ones((nz, ny, nx), np.uint8)
    total = flag.size
    fluid, at = total, 0
    while fluid / total > porosity:
        u = _uniforms(seed, 4 * 1024, at).reshape(-1, 4)
        at += 4 * 1024
        for a, b, c, s in u:
            r = rmin + (rmax - rmin) * s
            x, dx = _near(a * nx, r, nx)
            y, dy = _near(b * ny, r, ny)
            z, dz = _near(c * nz, r, nz)
            inside = ((dx[None, None, :] + dy[None, :, None]) + dz[:, None, None]) <= r * r
            # a sphere that wraps around no face is a plain sub-box
            box = (tuple(slice(i[0], i[-1] + 1) for i in (z, y, x))
                   if all(i[-1] - i[0] == len(i) - 1 for i in (z, y, x)) else np.ix_(z, y, x))
            old = flag[box].copy()
            flag[box] = old & ~inside
            fluid -= int(np.count_nonzero(old & inside))
            if not fluid / total > porosity:
                break
    if trim:
        last = np.flatnonzero(old & inside)[: int(porosity * total) - fluid]
        part = flag[box].copy()
        part.reshape(-1)[last] = 1
        flag[box] = part
    return flag


def _flag(case, seed):
    """The case's geometry, flat, x fastest; `tile` periodic copies per axis."""
    t = case.get("tile", 1)
    dims = (case["nx"] // t, case["ny"] // t, case["nz"] // t)
    f = sphere_flag(1000 + seed, dims, case["rmin"], case["rmax"], case["porosity"], trim=True)
    return np.tile(f, (t, t, t)).reshape(-1) if t > 1 else f.reshape(-1)


def _samples(case, seed):
    """Uneven samples: edges at the quantiles of a clipped lognormal and
    porosities spread over [0.15, 0.45] (the same for every seed), the rest
    drawn from the seed."""
    rng = np.random.default_rng(seed)
    out = []
    for i in range(case["samples"]):
        z = NormalDist().inv_cdf((i + 0.5) / case["samples"])
        edge = min(case["hi"], max(case["lo"], round(case["median"] * math.exp(case["sigma"] * z))))
        r = float(rng.uniform(4.0, 8.0))
        out.append(SimpleNamespace(
            index=i, edge=edge, porosity=0.15 + 0.30 * ((7 * i + 3) % 11) / 11, rmin=r, rmax=r,
            tau=float(rng.uniform(0.6, 1.2)), force=case["force"],
            tol=case.get("tol", 0.0), seed=int(rng.integers(1, 2 ** 62)), arrival=0.0))
    return out


def _sample_flag(r):
    """A sample's scan, flat."""
    return sphere_flag(r.seed, (r.edge,) * 3, r.rmin, r.rmax, r.porosity, trim=True).reshape(-1)


# ---------------------------------------------------------------- passes

def _simulation(case, flag):
    dims = (case["nx"], case["ny"], case["nz"])
    kw = dict(tau=case["tau"], force=case["force"], precision=case["precision"],
              boundary=case["boundary"])
    if case["source"] == "table":
        V, starts = P.build_table(flag, *dims, case["num_p"])
        return P.Simulation(V, *dims, starts, **kw)
    return P.Simulation.from_flag(flag, *dims, num_p=case["num_p"], **kw)


def _pinned(*shape):
    return torch.empty(shape, dtype=torch.float64, pin_memory=True).numpy()


def _checkpoint(n, seed):
    """A state as a run leaves it: the rest state with a few percent of
    slowly varying density and flow and some noise, AoS."""
    rng = np.random.default_rng(seed)
    f = np.asarray(W) * (1.0 + 0.01 * rng.standard_normal((n, 19)))
    u = 0.02 * np.sin(np.arange(n) * (2 * math.pi / 977.0))
    f *= 1.0 + 3.0 * u[:, None] * np.asarray(EX)[None, :]
    return f.reshape(-1)


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case, kind=kind)
    if kind == "pack":
        s["seed"] = 1000 + seed
    elif kind == "first":
        s["flag"] = _flag(case, seed)
        if case["source"] == "table":
            dims = (case["nx"], case["ny"], case["nz"])
            s["table"] = P.build_table(s["flag"], *dims, case["num_p"])
    elif kind in ("solve", "resume"):
        sim = s["sim"] = _simulation(case, _flag(case, seed))
        if kind == "resume":
            sim.init_dist_macro()
            s["f"] = _checkpoint(sim.N, seed)
        else:
            s["out"] = _pinned(4, sim.N)
    else:
        s["samples"] = _samples(case, seed)
        room = int(sum(r.edge ** 3 * r.porosity + 512 for r in s["samples"]) * 1.02)
        # the launch is the library's default, not a tuning run's outcome
        s["pool"] = Batch(room, len(s["samples"]), case["precision"], case["check_every"],
                          keep_macros=kind == "pool")
        if kind == "serve":
            s["server"] = Server(0, case["precision"], case["check_every"], batch=s["pool"])
        else:
            s["flags"] = [_sample_flag(r) for r in s["samples"]]
    return s


def _rows(macros):
    return dict(zip(("rho", "ux", "uy", "uz"), macros))


def _run_solve(s):
    c, sim = s["case"], s["sim"]
    sim.init_dist_macro()
    sim.step(c["steps"])
    out = _rows(sim.macros(out=s["out"]))
    if c["with_f"]:
        out["f"] = sim.get_f()
    return out


def _run_resume(s):
    sim = s["sim"]
    sim.set_f(s["f"])
    sim.step(s["case"]["steps"], it_begin=1000)
    return {"f": sim.get_f()}


def _run_first(s):
    c = s["case"]
    dims = (c["nx"], c["ny"], c["nz"])
    kw = dict(tau=c["tau"], force=c["force"], precision=c["precision"], boundary=c["boundary"])
    if "table" in s:
        sim = P.Simulation(s["table"][0], *dims, s["table"][1], **kw)
    else:
        sim = P.Simulation.from_flag(s["flag"], *dims, num_p=c["num_p"], **kw)
    with sim:
        sim.init_dist_macro()
        sim.step(c["steps"])
        k = sim.permeability()
        return dict(_rows(sim.macros()), k=np.array(k))


def _run_pool(s):
    c, pool = s["case"], s["pool"]
    ids = [pool.add_flag(f, r.edge, r.edge, r.edge, r.tau, r.force, tol=0.0, max_steps=10 ** 9)
           for r, f in zip(s["samples"], s["flags"])]
    pool.run(c["intervals"])
    res = [pool.result(i) for i in ids]
    macros = [pool.macros(i) for i in ids]
    for i in ids:
        pool.release(i)
    return {"k": np.array([r["k_darcy"] for r in res]),
            "mean_ux": np.array([r["mean_ux"] for r in res]), "macros": macros}


def _run_serve(s):
    done, _ = s["server"].serve(s["samples"])
    done = sorted(done, key=lambda d: d["index"])
    return {"k": np.array([d["k_darcy"] for d in done]),
            "steps": np.array([d["steps"] for d in done]),
            "nodes": np.array([d["nodes"] for d in done]),
            "status": np.array([d["status"] for d in done])}


def _run_pack(s):
    c = s["case"]
    flag, spheres, porosity = P.sphere_pack_device(s["seed"], c["nx"], c["ny"], c["nz"],
                                                   c["rmin"], c["rmax"], c["porosity"])
    return {"flag": flag, "spheres": spheres, "porosity": porosity}


def run(state):
    return {"solve": _run_solve, "resume": _run_resume, "first": _run_first, "pool": _run_pool,
            "serve": _run_serve, "pack": _run_pack}[state["kind"]](state)


# ------------------------------------------------------------------ work

def work(case):
    """A step reads and writes 19 values per node and reads 18 neighbour
    words; what goes up and comes down is counted once."""
    kind = case["kind"]
    if kind == "pack":
        return {"bytes": case["nx"] * case["ny"] * case["nz"], "flops": 0}
    per_step = 38 * VALUE_BYTES[case["precision"]] + 72
    if kind in ("pool", "serve"):
        s = _samples(case, 0)
        nodes = sum(r.edge ** 3 * r.porosity for r in s)
        # a served request runs to its second check at least
        steps = case["check_every"] * (case["intervals"] if kind == "pool" else 2)
        io = 32 * nodes if kind == "pool" else 0
    else:
        cells = case["nx"] * case["ny"] * case["nz"]
        nodes, steps = cells * case["porosity"], case["steps"]
        io = 304 * nodes if kind == "resume" else 32 * nodes
        if kind == "first":
            io += cells + 72 * nodes
        elif case["with_f"]:
            io += 152 * nodes
    return {"bytes": nodes * steps * per_step + io, "flops": nodes * steps * FLOPS_PER_NODE}


# ----------------------------------------------------------------- exact

class _Lattice:
    """The reference's step in 64-bit torch on the fluid cells of a flag."""

    def __init__(self, flag, dims, tau, force, halfway, num_p):
        nx, ny, nz = dims
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        fluid = torch.from_numpy(flag.reshape(nz, ny, nx)).to(dev) == 1
        cell = fluid.reshape(-1).nonzero().reshape(-1)
        self.n = n = cell.numel()
        number = torch.full((nx * ny * nz,), -1, dtype=torch.int64, device=dev)
        number[cell] = torch.arange(n, device=dev)
        x, y, z = cell % nx, cell // nx % ny, cell // (nx * ny)
        me = torch.arange(n, device=dev)
        slab = nz // num_p
        self.tau, self.force, self.cells = tau, force, nx * ny * nz
        # where direction j of a node is pulled from, in the flat state;
        # entry 19 n + j holds the weight of slots that nothing writes
        self.source = [me]
        for j in range(1, 19):
            sz = (z - EZ[j]) % nz
            s = number[(sz * ny + (y - EY[j]) % ny) * nx + (x - EX[j]) % nx]
            t = number[((z + EZ[j]) % nz * ny + (y + EY[j]) % ny) * nx + (x + EX[j]) % nx]
            back = OPP[j] * n + me
            if halfway:
                src = torch.where(s >= 0, j * n + s, back)
            else:
                wins = (s >= 0) & ((t >= 0) | (s > me) | (num_p > 1) & (sz // slab != z // slab))
                src = torch.where(wins, j * n + s, torch.where(t < 0, back, 19 * n + j))
            self.source.append(src)
        self.w = torch.tensor(W, dtype=torch.float64, device=dev)

    def run(self, steps, it=0, f=None):
        n, w = self.n, self.w
        omega = 1.0 / self.tau
        f = w[:, None].expand(19, n) if f is None else f.to(w.device).reshape(n, 19).t()
        state = torch.cat([f.reshape(-1), w])
        for k in range(steps):
            g = [state[src] for src in self.source]
            rho = sum(g[1:], g[0])
            u = [sum((e[j] * g[j] for j in range(1, 19) if e[j]), torch.zeros_like(rho))
                 for e in (EX, EY, EZ)]
            if it + k > 0:
                u[0] = u[0] + 0.5 * self.force
            u = [c / rho for c in u]
            sq = 1.5 * (u[0] * u[0] + u[1] * u[1] + u[2] * u[2])
            new = torch.empty_like(state)
            new[19 * n:] = w
            for j in range(19):
                eu = EX[j] * u[0] + EY[j] * u[1] + EZ[j] * u[2]
                feq = W[j] * rho * (1.0 + 3.0 * eu + 4.5 * eu * eu - sq)
                a = omega + (1.0 - 0.5 * omega) * 3.0 * (EX[j] - u[0]) * self.force
                new[j * n:(j + 1) * n] = (1.0 - omega) * g[j] + a * feq
            state = new
        macros = torch.stack([rho] + u).cpu().numpy()
        return macros, state[:19 * n].reshape(19, n).t()

    def permeability(self, ux):
        nu, total = (self.tau - 0.5) / 3.0, float(np.sum(ux))
        return total / self.cells * nu / self.force, total / self.n * nu / self.force


def exact(case, seed):
    kind = case["kind"]
    if kind == "serve":   # thousands of steps to convergence
        return None
    if kind == "pack":
        flag = sphere_flag(1000 + seed, (case["nx"], case["ny"], case["nz"]), case["rmin"],
                           case["rmax"], case["porosity"])
        return {"flag": None, "spheres": None, "porosity": float(flag.mean(dtype=np.float64))}
    if kind == "pool":
        steps = case["check_every"] * case["intervals"]
        k, mean, macros = [], [], []
        for r in _samples(case, seed):
            lat = _Lattice(_sample_flag(r), (r.edge,) * 3, r.tau, r.force, False, 1)
            macros.append(lat.run(steps)[0])
            k.append(lat.permeability(macros[-1][1])[0])
            mean.append(float(np.sum(macros[-1][1])) / lat.cells)
        return {"k": np.array(k), "mean_ux": np.array(mean), "macros": macros}
    lat = _Lattice(_flag(case, seed), (case["nx"], case["ny"], case["nz"]), case["tau"],
                   case["force"], case["boundary"] == "halfway", case["num_p"])
    if kind == "resume":
        f = torch.from_numpy(_checkpoint(lat.n, seed))
        return {"f": lat.run(case["steps"], 1000, f)[1].reshape(-1)}
    macros, f = lat.run(case["steps"])
    out = _rows(macros)
    if kind == "first":
        out["k"] = np.array(lat.permeability(macros[1]))
    elif case["with_f"]:
        out["f"] = f.reshape(-1)
    return out

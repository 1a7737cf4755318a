"""Performance cases of the N-body step: what a user's program has the library do.

Each case is one call sequence through the public Python entry points over inputs that stand on
the GPU (or, for the batched dwarfs, whose interface takes host arrays, on the host): bodies
are set, the forces evaluated, a number of kick-drift-kick steps taken and the bodies read
back, so that every pass does the same work.  The sizes are this repository's own: the 1,024
bodies of the golden models, the sample workunit's 20,000, the 131,072 of the differentiable
run, the benchmark's 1,048,576 and 8,388,608, and batches of dwarfs with log-uniform sizes.

The forces have a plain restatement in 64-bit torch (class _Tree and the functions after it):
the same octree, opening test and multipoles, with sums in another order.
"""
import functools
import math

import torch

from milkywayathome_client_b200 import adjoint, models
from milkywayathome_client_b200.histogram import HistogramParams, data_from_counts
from milkywayathome_client_b200.nbody import NBodyBatch, NBodyCtx, plummer_dwarf_struct

DEV = torch.device("cuda", 0)
F64 = torch.float64


# ---- the cases ------------------------------------------------------------------------------
def listed():
    return [
        # the golden models' size: a parameter fit runs thousands of steps of it, and each step
        # is latency (launches, one warp's walk)
        dict(name="steps 1k sw93 fp64", kind="steps", n=1024, precision="fp64", criterion="SW93",
             theta=1.0, quad=True, steps=20),
        # the sample workunit, the client's everyday job, in both precisions
        dict(name="steps 20k fp64", kind="steps", n=20000, precision="fp64", criterion="TreeCode",
             theta=1.0, quad=True, steps=10),
        dict(name="steps 20k mixed", kind="steps", n=20000, precision="mixed",
             criterion="TreeCode", theta=1.0, quad=True, steps=10),
        # the benchmark's dwarf in both precisions
        dict(name="steps 1m fp64", kind="steps", n=1048576, precision="fp64",
             criterion="TreeCode", theta=0.5, quad=True, steps=1),
        dict(name="steps 1m mixed", kind="steps", n=1048576, precision="mixed",
             criterion="TreeCode", theta=0.5, quad=True, steps=2),
        # the largest dwarf
        dict(name="steps 8m mixed", kind="steps", n=8388608, precision="mixed",
             criterion="TreeCode", theta=0.5, quad=True, steps=1),
        # the Exact criterion (a direct sum), an odd size
        dict(name="steps 10k exact", kind="steps", n=10007, precision="fp64", criterion="Exact",
             theta=1.0, quad=True, steps=4),
        # batched dwarfs of a parameter search, uneven sizes; and a batch of small ones in FP64
        dict(name="batch 64 mixed", kind="batch", ndwarfs=64, nmin=4096, nmax=65536,
             precision="mixed", theta=1.0, steps=16),
        dict(name="batch 24 fp64", kind="batch", ndwarfs=24, nmin=1000, nmax=10000,
             precision="fp64", theta=0.7, steps=8),
        # a gradient of the differentiable run: forward, recompute and reverse steps
        dict(name="adjoint 131k", kind="adjoint", n=131072, theta=0.5, steps=4, every=2),
        # the dwarfs of a batch sampled on the GPU
        dict(name="sample 8", kind="sample", ndwarfs=8, nmin=4096, nmax=65536),
        # the run loop with its best-likelihood scan, as a golden model runs
        dict(name="run 10k likelihood", kind="run", n=10000, precision="fp64", criterion="SW93",
             theta=1.0, steps=16, scan=0.5),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["steps", "steps", "steps", "steps", "batch", "adjoint", "sample", "run"])
    theta = round(rng.uniform(0.5, 1.0), 3)
    if kind == "steps":
        precision = rng.choice(["fp64", "mixed"])
        criterion = rng.choice(["TreeCode", "TreeCode", "TreeCode", "SW93", "BH86", "Exact"])
        if criterion == "Exact":
            n, precision = _log_int(rng, 500, 30000), "fp64"
        else:
            n = _log_int(rng, 300, 1048576 if precision == "fp64" else 4194304)
        if criterion in ("SW93", "BH86"):
            theta = round(rng.uniform(0.7, 1.0), 3)
        return dict(kind=kind, n=n, precision=precision, criterion=criterion, theta=theta,
                    quad=rng.random() < 0.85, steps=max(1, min(20, rng.randint(150000, 500000) // n)))
    if kind == "batch":
        nd = rng.randint(2, 48)
        nmin = _log_int(rng, 200, 8000)
        return dict(kind=kind, ndwarfs=nd, nmin=nmin, nmax=nmin * rng.randint(1, 8),
                    precision=rng.choice(["fp64", "mixed"]), theta=theta, steps=rng.randint(2, 16))
    if kind == "adjoint":
        return dict(kind=kind, n=_log_int(rng, 500, 131072), theta=theta,
                    steps=rng.randint(1, 4), every=rng.randint(1, 4))
    if kind == "sample":
        nmin = _log_int(rng, 100, 8000)
        return dict(kind=kind, ndwarfs=rng.randint(1, 8), nmin=nmin,
                    nmax=nmin * rng.randint(1, 8))
    return dict(kind=kind, n=_log_int(rng, 500, 40000), precision=rng.choice(["fp64", "mixed"]),
                criterion=rng.choice(["TreeCode", "SW93"]), theta=round(rng.uniform(0.7, 1.0), 3),
                steps=rng.randint(4, 16), scan=0.5)


# ---- inputs ---------------------------------------------------------------------------------
# the sample workunit's dwarf: baryons a = 0.2 kpc, M = 12; dark matter a = 0.8 kpc, M = 48
_A_L, _M_L, _A_D, _M_D = 0.2, 12.0, 0.8, 48.0
_DT = 5.1398e-4


def _eps2(n):
    """eps = 0.98 r_v N^-0.26 of that dwarf (0.0787 kpc at 20,000 bodies)."""
    return (0.0787 * (n / 20000.0) ** -0.26) ** 2


def _dwarf(n, seed):
    """Positions, velocities, masses of a two-component Plummer dwarf on its orbit (torch)."""
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 7919 + n)
    u = lambda *s: torch.rand(*s, generator=g, device=DEV, dtype=F64)
    nb = n // 2
    light = torch.arange(n, device=DEV) < nb
    a = torch.where(light, _A_L, _A_D).to(F64)
    m = torch.where(light, _M_L / max(nb, 1), _M_D / max(n - nb, 1)).to(F64)
    r = a / torch.sqrt((1e-12 + u(n) * ((1.0 + 1.0 / 2500.0) ** -1.5)) ** (-2.0 / 3.0) - 1.0)

    def directions():
        z = 2.0 * u(n) - 1.0
        p = 2.0 * math.pi * u(n)
        s = torch.sqrt(1.0 - z * z)
        return torch.stack([s * torch.cos(p), s * torch.sin(p), z], 1)

    # speed over escape speed: q^2 ~ Beta(3/2, 9/2), from gamma variates
    def gamma_half(k):
        e = -torch.log1p(-u(n, k)).sum(1)
        x = torch.randn(n, generator=g, device=DEV, dtype=F64)
        return e + 0.5 * x * x

    ga, gb = gamma_half(1), gamma_half(4)
    q = torch.sqrt(ga / (ga + gb))
    phi = _M_L / torch.sqrt(r * r + _A_L ** 2) + _M_D / torch.sqrt(r * r + _A_D ** 2)
    x = r[:, None] * directions()
    v = (q * torch.sqrt(2.0 * phi))[:, None] * directions()
    x = x - (m[:, None] * x).sum(0) / m.sum()
    v = v - (m[:, None] * v).sum(0) / m.sum()
    orbit, v0 = models.SAMPLE_ORBIT
    x = x + torch.tensor(models.lbr_to_cartesian(*orbit), device=DEV, dtype=F64)
    v = v + torch.tensor(v0, device=DEV, dtype=F64)
    return x.contiguous(), v.contiguous(), m.contiguous()


def _ctx(case, n):
    return NBodyCtx(timestep=_DT, eps2=_eps2(n), theta=case["theta"],
                    criterion=case.get("criterion", "TreeCode"), useQuad=case.get("quad", True),
                    potential=models.sample_workunit_potential(),
                    precision=case.get("precision", "fp64"))


def _sizes(case):
    """The batch's dwarf sizes: log-uniform between nmin and nmax, in an uneven order."""
    lo, hi, k = math.log(case["nmin"]), math.log(case["nmax"]), case["ndwarfs"]
    return [int(round(math.exp(lo + (hi - lo) * (((i + 1) * 0.6180339887498949) % 1.0))))
            for i in range(k)]


_BATCH_DT = 1.0e-3


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("steps", "run"):
        n = case["n"]
        x, v, m = _dwarf(n, seed)
        s = dict(case=case, ctx=_ctx(case, n), ds=adjoint.DeviceState(n, DEV), x=x, v=v, m=m)
        if kind == "run":
            s["params"], s["data"] = _target(n)
            types = torch.where(torch.arange(n) < n // 2, 1, -1).to(torch.int32).numpy()
            s["ds"].st.set_types(types)
        return s
    if kind == "batch":
        sizes = _sizes(case)
        parts = [_dwarf(n, seed * 1000 + k) for k, n in enumerate(sizes)]
        x, v, m = (torch.cat([p[c] for p in parts]).cpu().numpy() for c in range(3))
        batch = NBodyBatch([(n, _eps2(n), _BATCH_DT, 4.0) for n in sizes])
        return dict(case=case, ctx=_ctx(case, 20000), batch=batch, x=x, v=v, m=m)
    if kind == "adjoint":
        x, v, m = _dwarf(case["n"], seed)
        g = torch.Generator(device=DEV)
        g.manual_seed(int(seed) + 17)
        gx, gv = (torch.randn(case["n"], 3, generator=g, device=DEV, dtype=F64) for _ in range(2))
        leaf = lambda t: t.clone().requires_grad_(True)
        return dict(case=case, ctx=_ctx(case, case["n"]), x=leaf(x), v=leaf(v), m=leaf(m),
                    dt=torch.tensor(_DT, dtype=F64, device=DEV, requires_grad=True), gx=gx, gv=gv)
    sizes = _sizes(case)
    orbit, v0 = models.SAMPLE_ORBIT
    where = models.lbr_to_cartesian(*orbit)
    dwarfs = [plummer_dwarf_struct(n, seed * 1000 + k, None, position=where, velocity=v0)
              for k, n in enumerate(sizes)]
    return dict(case=case, batch=NBodyBatch([(n, _eps2(n), _DT, 4.0) for n in sizes]),
                dwarfs=dwarfs)


@functools.lru_cache(maxsize=None)
def _target(n):
    """Histogram settings and the data histogram a run is compared with: the counts of the
    golden data's shape (34 Lambda bins, beta dispersions), smooth in Lambda."""
    params = HistogramParams(lambdaStart=-150.0, lambdaEnd=150.0, lambdaBins=50)
    lam, _ = params.centres()
    w = torch.exp(-0.5 * ((torch.tensor(lam) - 5.0) / 25.0) ** 2)
    counts = (w * (n // 2) / w.sum()).round().to(torch.int64).numpy().astype("uint32")
    comps = torch.zeros(7, 2, params.nbins, dtype=F64).numpy()
    comps[0, 0], comps[0, 1] = 1.5, 0.4
    return params, data_from_counts(params, counts, n // 2, _M_L / (n // 2), comps)


# ---- one pass -------------------------------------------------------------------------------
def run(s):
    kind = s["case"]["kind"]
    if kind == "steps":
        ds, ctx = s["ds"], s["ctx"]
        ds.set(s["x"], s["v"], s["m"], ctx.treeRSize)
        ds.gravmap(ctx)
        ds.st.check("run_steps", ds.st.run_steps(ctx, s["case"]["steps"]))
        return dict(zip("xva", ds.get()))
    if kind == "run":
        ds, ctx, steps = s["ds"], s["ctx"], s["case"]["steps"]
        ds.set(s["x"], s["v"], s["m"], ctx.treeRSize)
        rc, res = ds.st.run_system(ctx, steps, steps * ctx.timestep, s["params"], s["data"],
                                   use_best_like=True, best_like_start=s["case"]["scan"])
        ds.st.check("run_system", rc)
        out = dict(zip("xva", ds.get()))
        # the terms of the default comparison; those not compared are NaN
        out.update(final=res["final"][[0, 1, 2, 3, 10]], best=res["best"][[0, 1, 2, 3, 10]],
                   best_step=res["best_step"], best_count=res["best_count"])
        return out
    if kind == "batch":
        b, ctx = s["batch"], s["ctx"]
        b.set_bodies(s["x"], s["v"], s["m"])
        b.check("gravMap", b.gravMap(ctx))
        b.check("run_steps", b.run_steps(ctx, s["case"]["steps"]))
        x, v = b.bodies()
        return dict(x=x, v=v, a=b.accels())
    if kind == "adjoint":
        x, v = adjoint.run(s["ctx"], s["x"], s["v"], s["m"], s["dt"], s["case"]["steps"],
                           s["case"]["every"])
        g = torch.autograd.grad([x, v], [s["x"], s["v"], s["m"], s["dt"]], [s["gx"], s["gv"]])
        return dict(x=x.detach(), v=v.detach(), gx=g[0], gv=g[1], gm=g[2], gdt=g[3])
    b = s["batch"]
    b.generate(s["dwarfs"])
    x, v = b.bodies()
    return dict(x=x, v=v)


# ---- work and tolerance ---------------------------------------------------------------------
def _interactions(n, theta, criterion="TreeCode"):
    """Interactions per body of the tree walk (counted on the dwarf above, 1k to 1M bodies)."""
    if criterion == "Exact":
        return float(n)
    i = 232.0 * theta ** -0.95 + 57.0 * theta ** -2.2 * math.log2(max(n, 1024) / 1024.0)
    return min(float(n), i)


def _force_flops(case, n):
    per = 18.0 if case.get("criterion") == "Exact" or not case.get("quad", True) else 56.0
    return n * (per * _interactions(n, case["theta"], case.get("criterion", "TreeCode")) + 60.0)


def work(case):
    """Bytes: bodies in (56 each) and out (72).  Flops: each evaluation's interactions, 56 for a
    quadrupole cell and 18 for a pair (divisions and roots counted as one)."""
    kind = case["kind"]
    if kind in ("steps", "run"):
        n = case["n"]
        return {"bytes": 128.0 * n, "flops": (case["steps"] + 1) * _force_flops(case, n)}
    sizes = _sizes(case) if kind in ("batch", "sample") else None
    if kind == "batch":
        return {"bytes": 128.0 * sum(sizes),
                "flops": (case["steps"] + 1) * sum(_force_flops(case, n) for n in sizes)}
    if kind == "adjoint":
        n, k = case["n"], case["steps"]
        # forward and recomputed steps, and a vector-Jacobian product of about twice a force's
        # flops per step
        return {"bytes": 208.0 * n, "flops": (4.0 * k + 3.0) * _force_flops(case, n)}
    # about 14 evaluations of the distribution function a body, 330 quadrature points each of
    # 15 potential and density values of about 15 flops
    return {"bytes": 48.0 * sum(sizes), "flops": sum(sizes) * 14.0 * 330.0 * 225.0}


def tolerance(case):
    """Measured with the walk's groups and lists of other sizes (other summation orders) and
    against exact() below, about four times the largest difference seen over these ranges."""
    kind = case["kind"]
    if kind == "adjoint":
        # node adjoints are summed with atomics, in any order (gradients 2e-14, largest 1e-13 of
        # 4,000 bodies; more terms a node at 131,072)
        return {"rel": 1e-12, "max": 1e-11}
    if kind == "sample":
        # a body's radius and speed are drawn numbers, accepted or not: the same up to rounding
        return {"rel": 1e-11, "max": 1e-9}
    if case["precision"] == "mixed":
        # accelerations differ by 1e-8 to 4e-8, and by up to 1.3e-6 (largest 7e-4) where a
        # single-precision opening test falls the other way for a cell near its limit
        return {"rel": 5e-6, "max": 3e-3}
    return "exact"      # the reference's own rounding, term by term


# ---- the same in plain 64-bit torch ---------------------------------------------------------
class _Tree:
    """The octree of the bodies (every cell of two or more bodies, and the root), its moments
    and opening radii.  Moments carry gradients with respect to x and m; the tree does not."""

    def __init__(self, x, m, rsize, criterion, theta):
        with torch.no_grad():
            top = float(x.abs().max())
        while rsize < 2.0 * top:
            rsize *= 2.0
        self.rsize = rsize
        n = x.shape[0]
        bodies = torch.arange(n, device=x.device)
        cell = torch.zeros(n, dtype=torch.long, device=x.device)
        centre = torch.zeros(1, 3, dtype=x.dtype, device=x.device)
        size, base = rsize, 0
        com, mass, quad, crit, parents, children = [], [], [], [], [], []
        for _ in range(62):
            k = centre.shape[0]
            xb, mb = x[bodies], m[bodies]
            M = torch.zeros(k, dtype=x.dtype, device=x.device).index_add(0, cell, mb)
            c = torch.zeros(k, 3, dtype=x.dtype, device=x.device).index_add(
                0, cell, mb[:, None] * xb) / M[:, None]
            d = xb - c[cell]
            d2 = (d * d).sum(1)
            t = 3.0 * d[:, [0, 0, 0, 1, 1, 2]] * d[:, [0, 1, 2, 1, 2, 2]]
            trace = torch.tensor([1.0, 0.0, 0.0, 1.0, 0.0, 1.0], dtype=x.dtype, device=x.device)
            t = mb[:, None] * (t - d2[:, None] * trace)
            q = torch.zeros(k, 6, dtype=x.dtype, device=x.device).index_add(0, cell, t)
            with torch.no_grad():
                if criterion == "TreeCode":
                    rc2 = (size / theta + (c - centre).norm(dim=1)) ** 2
                elif criterion == "BH86":
                    rc2 = torch.full((k,), (size / theta) ** 2, dtype=x.dtype, device=x.device)
                else:
                    lo = c - (centre - 0.5 * size)
                    rc2 = (torch.maximum(lo, size - lo) ** 2).sum(1) / (theta * theta)
                right = xb >= centre[cell]
                octant = right[:, 0] * 4 + right[:, 1] * 2 + right[:, 2] * 1
                key, inv, cnt = torch.unique(cell * 8 + octant, return_inverse=True,
                                             return_counts=True)
                many = cnt > 1
                number = torch.cumsum(many, 0) - 1
                one = ~many[inv]
                # children: cells by their number, bodies as -(index + 1)
                child = base + k + number
                child[inv[one]] = -(bodies[one] + 1)
                com.append(c); mass.append(M); quad.append(q); crit.append(rc2)
                parents.append(base + key // 8); children.append(child)
                bit = torch.stack([(key >> 2) & 1, (key >> 1) & 1, key & 1], 1).to(x.dtype)
                nxt = (centre[key // 8] + 0.25 * size * (2.0 * bit - 1.0))[many]
                keep = many[inv]
                bodies, cell = bodies[keep], number[inv[keep]]
                centre, base, size = nxt, base + k, 0.5 * size
            if centre.shape[0] == 0:
                break
        self.com, self.mass = torch.cat(com), torch.cat(mass)
        self.quad, self.crit = torch.cat(quad), torch.cat(crit)
        parents, self.children = torch.cat(parents), torch.cat(children)
        self.count = torch.bincount(parents, minlength=self.com.shape[0])
        self.first = torch.cumsum(self.count, 0) - self.count      # parents are in order


def _terms(dx, m, eps2, q=None):
    s = (dx * dx).sum(1) + eps2
    r = torch.sqrt(s)
    out = (m / (s * r))[:, None] * dx
    if q is not None:
        qd = torch.stack([q[:, 0] * dx[:, 0] + q[:, 1] * dx[:, 1] + q[:, 2] * dx[:, 2],
                          q[:, 1] * dx[:, 0] + q[:, 3] * dx[:, 1] + q[:, 4] * dx[:, 2],
                          q[:, 2] * dx[:, 0] + q[:, 4] * dx[:, 1] + q[:, 5] * dx[:, 2]], 1)
        r5 = 1.0 / (s * s * r)
        out = out + (2.5 * r5 * (qd * dx).sum(1) / s)[:, None] * dx - r5[:, None] * qd
    return out


def _external(x):
    """Miyamoto-Nagai disk, Hernquist bulge and logarithmic halo of the sample workunit."""
    X, Y, Z = x[:, 0], x[:, 1], x[:, 2]
    zp = torch.sqrt(Z * Z + 0.26 ** 2)
    az = 6.5 + zp
    k = -4.45865888e5 / (X * X + Y * Y + az * az) ** 1.5
    a = torch.stack([k * X, k * Y, k * Z * az / zp], 1)
    k = -2.0 * 74.61 ** 2 / (12.0 ** 2 + (x * x).sum(1))
    r = torch.sqrt((x * x).sum(1))
    b = -1.52954402e5 / (r * (0.7 + r) ** 2)
    return a + (k + b)[:, None] * x


def _forces(x, m, eps2, criterion, theta, quad, rsize):
    """Accelerations and the root size."""
    n = x.shape[0]
    acc = torch.zeros_like(x)
    if criterion == "Exact":
        rows = max(1, 30_000_000 // n)
        for lo in range(0, n, rows):
            d = x[None, :, :] - x[lo:lo + rows, None, :]
            s = (d * d).sum(2) + eps2
            acc[lo:lo + rows] = ((m / (s * torch.sqrt(s)))[:, :, None] * d).sum(1)
        return acc + _external(x), rsize
    t = _Tree(x, m, rsize, criterion, theta)
    rows = 16384
    parts = []
    for lo in range(0, n, rows):
        b = torch.arange(lo, min(lo + rows, n), device=x.device)
        a = torch.zeros(b.shape[0], 3, dtype=x.dtype, device=x.device)
        c = torch.zeros_like(b)
        while b.shape[0]:
            dx = t.com[c] - x[b]
            take = (dx * dx).sum(1) >= t.crit[c]
            bt, ct = b[take], c[take]
            a = a.index_add(0, bt - lo, _terms(dx[take], t.mass[ct], eps2,
                                               t.quad[ct] if quad else None))
            b, c = b[~take], c[~take]
            num = t.count[c]
            at = torch.repeat_interleave(t.first[c] - (torch.cumsum(num, 0) - num), num)
            kids = t.children[at + torch.arange(at.shape[0], device=x.device)]
            b = torch.repeat_interleave(b, num)
            body = (kids < 0) & (kids != -(b + 1))
            j = -kids[body] - 1
            bt = b[body]
            a = a.index_add(0, bt - lo, _terms(x[j] - x[bt], m[j], eps2))
            cell = kids >= 0
            b, c = b[cell], kids[cell]
        parts.append(a)
    return torch.cat(parts) + _external(x), t.rsize


def _steps(x, v, m, dt, eps2, case, steps):
    settings = (eps2, case.get("criterion", "TreeCode"), case["theta"], case.get("quad", True))
    a, rsize = _forces(x, m, *settings, 4.0)
    for _ in range(steps):
        v = v + 0.5 * dt * a
        x = x + dt * v
        a, rsize = _forces(x, m, *settings, rsize)
        v = v + 0.5 * dt * a
    return x, v, a


def exact(case, seed):
    kind = case["kind"]
    if kind == "sample":
        return None             # random draws: no value but the sampler's own
    if kind == "batch":
        sizes = _sizes(case)
        if sum(_interactions(n, case["theta"]) * n for n in sizes) * (case["steps"] + 1) > 4e9:
            return None
        outs = []
        for k, n in enumerate(sizes):
            x, v, m = _dwarf(n, seed * 1000 + k)
            outs.append(_steps(x, v, m, _BATCH_DT, _eps2(n), case, case["steps"]))
        return dict(zip("xva", (torch.cat([o[c] for o in outs]) for c in range(3))))
    n = case["n"]
    cost = n * _interactions(n, case["theta"], case.get("criterion", "TreeCode"))
    if kind == "adjoint":
        if cost * (case["steps"] + 1) > 1.2e7:
            return None         # the whole graph is kept
        s = prepare(case, seed)
        x, v, _ = _steps(s["x"], s["v"], s["m"], s["dt"], _eps2(n), case, case["steps"])
        g = torch.autograd.grad([x, v], [s["x"], s["v"], s["m"], s["dt"]], [s["gx"], s["gv"]])
        return dict(x=x.detach(), v=v.detach(), gx=g[0], gv=g[1], gm=g[2], gdt=g[3])
    if cost * (case["steps"] + 1) > 1.2e10:
        return None
    x, v, m = _dwarf(n, seed)
    with torch.no_grad():
        out = dict(zip("xva", _steps(x, v, m, _DT, _eps2(n), case, case["steps"])))
    if kind == "run":
        out.update(final=None, best=None, best_step=None, best_count=None)
    return out

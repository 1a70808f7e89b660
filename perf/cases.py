"""The work whose speed counts: what programs built on this framework have it do.

``listed()`` names twelve cases, ``draw(rng)`` gives further ones from the
same ranges, ``prepare`` builds what a program holds before the call (inputs
and handles), ``run`` makes one pass through the public Python front end, and
``exact`` computes the same outputs in 64 bits with plain torch.

Every case is a dict of plain values.  ``kind`` selects the path:

  operators  one explicit step written with the operator layer (CFL step,
             gradient, Laplacian, stabilisation, update, boundary cells,
             conserved total), as programs that assemble their own equation do
  heat       a heat solve (``heat_run``)
  wave       an acoustic solve (``wave_run``), uniform or distorted mesh,
             FP32 fused or FP64 per-operator path, constant c or a c field
  euler      a compressible solve to an end time (``Euler.run``), totals read
  ensemble   many small problems advanced together (``Batch.run``)
  gradient   the discrete-adjoint gradient of an acoustic solve
  leapfrog   second-order wave steps called one by one (``d2t_step``), the
             loop of a program that looks at the field between steps
"""
from __future__ import annotations

import math

import numpy as np
import torch

import cfdarcov2_b200 as cfdb
from cfdarcov2_b200.api import Batch, Context, Euler, Mesh

DEVICE = "cuda"
GAMMA = 1.4


# ---- the cases ------------------------------------------------------------------
def listed():
    return [
        # a step of a small interactive model: launches and the two host
        # read-backs (dt, total) are all there is
        dict(name="operators_small", kind="operators", nx=32, ny=24, nz=20, dtype="f32", mesh="uniform"),
        # the mesh size of the reference's own heat and Euler benchmark rows,
        # through the operator layer in its precision
        dict(name="operators_200", kind="operators", nx=200, ny=200, nz=200, dtype="f32", mesh="uniform"),
        # a validation run on a distorted mesh: double precision, ragged sizes
        dict(name="operators_f64_vertices", kind="operators", nx=80, ny=72, nz=66, dtype="f64", mesh="vertices"),
        # the benchmark's heat workload, one whole solve
        dict(name="heat_64", kind="heat", nx=64, ny=64, nz=64, steps=200),
        # a heat field far beyond the L2 cache, no dimension a power of two
        dict(name="heat_large", kind="heat", nx=384, ny=400, nz=392, steps=20),
        # the benchmark's headline mesh: the acoustic system at 128^3
        dict(name="wave_128", kind="wave", nx=128, ny=128, nz=128, steps=100, dtype="f32", mesh="uniform", c_field=False),
        # the acoustic system on a jittered mesh
        dict(name="wave_vertices", kind="wave", nx=96, ny=96, nz=96, steps=50, dtype="f32", mesh="vertices", c_field=False),
        # the double-precision run that single-precision results are judged by
        dict(name="wave_f64", kind="wave", nx=100, ny=90, nz=96, steps=20, dtype="f64", mesh="uniform", c_field=False),
        # the benchmark's shock tube, the first part of the run
        dict(name="euler_sod", kind="euler", nx=512, ny=64, nz=64, t_end=0.02, dtype="f32", flow="tube"),
        # a parameter study: heat and wave cubes of mixed sizes, tuned once
        dict(name="ensemble", kind="ensemble", count=96, nmin=16, nmax=96, kinds="mixed", steps=20),
        # one iteration of an inversion: gradient with respect to c and p0
        dict(name="gradient", kind="gradient", nx=96, ny=96, nz=96, steps=48, snapshots=48),
        # the mesh of the reference's wave example with unit cells, step by step
        dict(name="leapfrog_200", kind="leapfrog", nx=200, ny=200, nz=200, steps=20),
    ]


def _log_int(rng, lo, hi, multiple=1):
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(multiple, int(round(v / multiple)) * multiple)


def _dims(rng, lo, hi, cells, zmul):
    """Three sizes of [lo, hi] (nz a multiple of zmul) with at most `cells` cells."""
    while True:
        d = [_log_int(rng, lo, hi), _log_int(rng, lo, hi), _log_int(rng, max(lo, zmul), hi, zmul)]
        if d[0] * d[1] * d[2] <= cells:
            return d


def draw(rng):
    kind = rng.choice(["operators", "operators", "heat", "heat", "wave", "wave", "euler", "ensemble", "gradient", "leapfrog"])
    if kind == "operators":
        mesh = rng.choice(["uniform", "uniform", "vertices"])
        nx, ny, nz = _dims(rng, 8, 256, 8_000_000 if mesh == "uniform" else 400_000, 1)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, dtype=rng.choice(["f32", "f64"]), mesh=mesh)
    if kind == "heat":
        nx, ny, nz = _dims(rng, 16, 512, 60_000_000, 4)
        most = max(8, min(200, 1_200_000_000 // (nx * ny * nz)))
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, steps=_log_int(rng, 5, most))
    if kind == "wave":
        form = rng.choice(["const", "const", "field", "vertices", "f64"])
        cells = {"const": 8_000_000, "field": 4_000_000, "vertices": 700_000, "f64": 2_000_000}[form]
        nx, ny, nz = _dims(rng, 16, 256, cells, 1 if form == "f64" else 4)
        most = max(8, min(200, 200_000_000 // (nx * ny * nz)))
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, steps=_log_int(rng, 5, most), dtype="f64" if form == "f64" else "f32",
                    mesh="vertices" if form == "vertices" else "uniform", c_field=form == "field")
    if kind == "euler":
        f64 = rng.random() < 0.25
        nx, ny, nz = _dims(rng, 16, 512, 300_000 if f64 else 2_000_000, 4)
        # about `steps` steps: dt is near cfl h / 4 with the smallest spacing h = 1 / max(n)
        steps = _log_int(rng, 10, 60)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, t_end=round(0.1 * steps / max(nx, ny, nz), 6), dtype="f64" if f64 else "f32",
                    flow=rng.choice(["tube", "blast"]))
    if kind == "ensemble":
        lo = rng.choice([16, 16, 20, 31])
        return dict(kind=kind, count=_log_int(rng, 16, 96), nmin=lo, nmax=rng.randint(lo + 8, 96),
                    kinds=rng.choice(["mixed", "mixed", "heat", "wave"]), steps=_log_int(rng, 4, 40))
    if kind == "gradient":
        nx, ny, nz = _dims(rng, 16, 128, 1_000_000, 4)
        steps = _log_int(rng, 8, 48)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, steps=steps, snapshots=rng.choice([steps, steps, max(2, steps // 6)]))
    nx, ny, nz = _dims(rng, 24, 400, 16_000_000, 4)
    return dict(kind=kind, nx=nx, ny=ny, nz=nz, steps=_log_int(rng, 4, 40))


# ---- inputs -----------------------------------------------------------------------
def _real(case):
    return torch.float64 if case.get("dtype") == "f64" else torch.float32


def _spacing(case):
    """The longest side of the box is 1 (cubic cells)."""
    return 1.0 / max(case["nx"], case["ny"], case["nz"])


def _centres(nx, ny, nz, h):
    ax = [(torch.arange(m, device=DEVICE, dtype=torch.float64) + 0.5) * h for m in (nx, ny, nz)]
    return ax[0][:, None, None], ax[1][None, :, None], ax[2][None, None, :]


def _pulse(nx, ny, nz, h, rng, sigma):
    x, y, z = _centres(nx, ny, nz, h)
    c = [rng.uniform(0.3, 0.7) * m * h for m in (nx, ny, nz)]
    return torch.exp(-((x - c[0]) ** 2 + (y - c[1]) ** 2 + (z - c[2]) ** 2) / (2 * sigma ** 2))


def _smooth(nx, ny, nz, h, rng):
    """A smooth field of unit amplitude: a few long cosine modes."""
    x, y, z = _centres(nx, ny, nz, h)
    out = torch.zeros(nx, ny, nz, device=DEVICE, dtype=torch.float64)
    for _ in range(3):
        k = rng.uniform(1.0, 5.0, size=3)
        out += torch.cos(k[0] * x + rng.uniform(0, 6)) * torch.cos(k[1] * y + rng.uniform(0, 6)) * torch.cos(k[2] * z + rng.uniform(0, 6))
    return out / 3


def _vertices(nx, ny, nz, h, rng):
    """Lattice vertices jittered by up to a fifth of a cell; walls stay flat."""
    ax = [np.arange(m + 1) * h for m in (nx, ny, nz)]
    v = np.stack(np.meshgrid(*ax, indexing="ij"), axis=-1)
    j = rng.uniform(-0.2, 0.2, size=v.shape) * h
    j[[0, -1], :, :, 0] = 0.0
    j[:, [0, -1], :, 1] = 0.0
    j[:, :, [0, -1], 2] = 0.0
    return v + j


def _problems(case, rng):
    probs = []
    for i in range(case["count"]):
        n = int(math.floor(math.exp(rng.uniform(math.log(case["nmin"]), math.log(case["nmax"] + 1)))))
        n = min(max(n, case["nmin"]), case["nmax"])
        kind = {"heat": 0, "wave": 1}.get(case["kinds"], i % 2)
        h = 1.0 / n
        param = float(rng.uniform(1e-3, 1e-2)) if kind == 0 else float(rng.uniform(0.5, 2.0))
        dt = 0.1 * h * h / param if kind == 0 else 0.4 * h / (3 * param)
        probs.append(dict(n=n, kind=kind, param=param, dt=dt))
    return probs


def _inputs(case, seed):
    """The inputs of a case, made from the seed alone (device tensors in the
    case's precision; vertices and problem lists on the host)."""
    rng = np.random.Generator(np.random.PCG64(seed))
    kind = case["kind"]
    if kind == "ensemble":
        # sizes and parameters belong to the study, not to the seed of a pass
        probs = _problems(case, np.random.Generator(np.random.PCG64(11)))
        fields = []
        for p in probs:
            q = torch.zeros((4 if p["kind"] else 1,) + (p["n"],) * 3, device=DEVICE, dtype=torch.float64)
            q[0] = _pulse(p["n"], p["n"], p["n"], 1.0 / p["n"], rng, 0.1)
            fields.append(q.float())
        return dict(probs=probs, fields=fields)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    R = _real(case)
    h = 1.0 if kind == "leapfrog" else _spacing(case)
    d = dict(h=h)
    if case.get("mesh") == "vertices":
        # the mesh belongs to the case, the fields to the seed
        d["vertices"] = _vertices(nx, ny, nz, h, np.random.Generator(np.random.PCG64(2)))
    if kind == "operators":
        d["T"] = (1 + _smooth(nx, ny, nz, h, rng)).to(R)
        d["p"] = (1 + 0.4 * _smooth(nx, ny, nz, h, rng)).to(R)
        d["rho"] = (1 + 0.4 * _smooth(nx, ny, nz, h, rng)).to(R)
        for name in ("u", "v", "w"):
            d[name] = (0.3 * _smooth(nx, ny, nz, h, rng)).to(R)
    elif kind == "heat":
        d["k"] = 0.01
        d["dt"] = 0.1 * h * h / d["k"]
        g = torch.Generator(device=DEVICE).manual_seed(seed)
        noise = torch.rand((nx, ny, nz), generator=g, device=DEVICE, dtype=torch.float64) - 0.5
        d["T"] = (_pulse(nx, ny, nz, h, rng, 0.1) + 2e-3 * noise).float()
    elif kind in ("wave", "gradient"):
        q = torch.zeros((4, nx, ny, nz), device=DEVICE, dtype=torch.float64)
        q[0] = _pulse(nx, ny, nz, h, rng, 0.05 + h)
        d["q"] = q.to(R)
        cmax = 1.0
        if kind == "gradient" or case["c_field"]:
            d["c"] = torch.exp(0.2 * _smooth(nx, ny, nz, h, rng)).to(R)
            cmax = math.exp(0.2)
        if kind == "gradient":
            d["target"] = (0.5 * q[0] + 0.1 * _smooth(nx, ny, nz, h, rng)).to(R)
        d["dt"] = (0.3 if "vertices" in d else 0.4) * h / (3 * cmax)
    elif kind == "euler":
        x = _centres(nx, ny, nz, h)[0]
        ones = torch.ones((nx, ny, nz), device=DEVICE, dtype=torch.float64)
        if case["flow"] == "tube":
            left = (x < 0.5 * nx * h) * ones
            rho, p = 0.125 + 0.875 * left, 0.1 + 0.9 * left
        else:
            rho, p = 1.0 * ones, 0.1 + 2.0 * _pulse(nx, ny, nz, h, rng, 0.15)
        rho = rho * (1 + 0.02 * _smooth(nx, ny, nz, h, rng))
        u = [0.05 * _smooth(nx, ny, nz, h, rng) for _ in range(3)]
        E = p / (GAMMA - 1) + 0.5 * rho * (u[0] ** 2 + u[1] ** 2 + u[2] ** 2)
        d["U"] = torch.stack([rho, rho * u[0], rho * u[1], rho * u[2], E]).to(R)
    else:  # leapfrog: unit cells, dt c < 1 / sqrt(2)
        x, y, z = _centres(nx, ny, nz, 1.0)
        c = [rng.uniform(0.3, 0.7) * m for m in (nx, ny, nz)]
        s = 0.06 * max(nx, ny, nz)
        d["u"] = torch.exp(-((x - c[0]) ** 2 + (y - c[1]) ** 2 + (z - c[2]) ** 2) / (2 * s * s)).float()
        d["k"], d["dt"] = 1.0, 0.4
    return d


# ---- one pass ---------------------------------------------------------------------
def prepare(case, seed):
    d = _inputs(case, seed)
    ctx = Context(0)
    s = dict(case=case, ctx=ctx)
    if case["kind"] == "ensemble":
        probs = d["probs"]
        b = Batch(ctx, probs)
        a0 = torch.zeros(b.pool_elems, device=DEVICE)
        for off, q in zip(b.offsets, d["fields"]):
            a0[off: off + q.numel()] = q.reshape(-1)
        a, other = a0.clone(), torch.empty_like(a0)
        b.tune(a, other)
        last = b.offsets[-1] + d["fields"][-1].numel()
        s.update(batch=b, a0=a0, a=a, b=other, cells=slice(b.offsets[0], last))
        return s
    nx, ny, nz, h = case["nx"], case["ny"], case["nz"], d["h"]
    if "vertices" in d:
        mesh = Mesh.from_vertices(ctx, nx, ny, nz, h, h, h, d["vertices"])
    else:
        mesh = Mesh.structured(ctx, nx, ny, nz, h, h, h)
    flat = {k: v.reshape(-1).contiguous() for k, v in d.items() if torch.is_tensor(v)}
    s.update(mesh=mesh, **flat)
    kind = case["kind"]
    if kind == "heat":
        s.update(k=d["k"], dt=d["dt"], a=torch.empty_like(flat["T"]), b=torch.empty_like(flat["T"]))
    elif kind == "wave":
        s.update(dt=d["dt"], a=torch.empty_like(flat["q"]), b=torch.empty_like(flat["q"]))
    elif kind == "gradient":
        s.update(dt=d["dt"], gc=torch.empty_like(flat["c"]), gp=torch.empty_like(flat["c"]))
    elif kind == "euler":
        f64 = case["dtype"] == "f64"
        s.update(a=torch.empty_like(flat["U"]), b=torch.empty_like(flat["U"]),
                 solver=Euler(ctx, mesh, cfdb.F64 if f64 else cfdb.F32, cfdb.PLAIN if f64 else cfdb.FUSED, GAMMA, 0.4,
                              case["t_end"], 100000))
    elif kind == "leapfrog":
        s.update(k=d["k"], dt=d["dt"], bufs=[torch.empty_like(flat["u"]) for _ in range(3)])
    return s


def run(s):
    case, ctx, kind = s["case"], s["ctx"], s["case"]["kind"]
    if kind == "operators":
        m = s["mesh"]
        dt = ctx.cfl_dt(m, 0.1, GAMMA, s["p"], s["rho"], s["u"], s["v"], s["w"])
        grad = ctx.grad(m, s["T"])
        lapl = ctx.lapl(m, s["T"])
        stab = ctx.stab(m, s["T"])
        rhs = ctx.binary(cfdb.capi.OP_SUB, ctx.scalar(cfdb.capi.OP_MUL, lapl, 1e-3), grad)
        new = ctx.d1t(rhs, s["T"], dt)
        ctx.boundary_set(m, new, s["T"])
        return dict(dt=dt, grad=grad, lapl=lapl, stab=stab, new=new, total=ctx.total_fp64(m, new))
    if kind == "heat":
        s["a"].copy_(s["T"])
        return ctx.heat_run(s["mesh"], s["a"], s["b"], s["k"], s["dt"], case["steps"])
    if kind == "wave":
        s["a"].copy_(s["q"])
        path = cfdb.PLAIN if case["dtype"] == "f64" else cfdb.FUSED
        return ctx.wave_run(s["mesh"], s["a"], s["b"], s["dt"], case["steps"], c=s.get("c"), c_const=1.0, path=path)
    if kind == "euler":
        s["a"].copy_(s["U"])
        s["solver"].begin(s["a"])
        _, in_b = s["solver"].run(s["a"], s["b"])
        return dict(state=s["b"] if in_b else s["a"], totals=s["solver"].totals()[-1])
    if kind == "ensemble":
        s["a"].copy_(s["a0"])
        return s["batch"].run(s["a"], s["b"], case["steps"])[s["cells"]]
    if kind == "gradient":
        J, _ = ctx.wave_gradient(s["mesh"], s["q"], s["c"], s["target"], case["steps"], s["dt"], case["snapshots"], s["gc"], s["gp"])
        return dict(J=J, grad_c=s["gc"], grad_p0=s["gp"])
    prev, cur, nxt = s["bufs"]
    prev.copy_(s["u"])
    masks = [1, 2]
    ctx.d2t_step(s["mesh"], prev, None, cur, s["k"], masks, s["dt"], first_step=True)
    for _ in range(case["steps"] - 1):
        ctx.d2t_step(s["mesh"], cur, prev, nxt, s["k"], masks, s["dt"])
        prev, cur, nxt = cur, nxt, prev
    return dict(u=cur, u_prev=prev)


# ---- what a pass cannot do without ------------------------------------------------
# Fields that come in once and go out once, and the additions and
# multiplications of the scheme per cell and step.
_FLOPS = {"heat": 15, "wave": 64, "euler": 260, "gradient": 64 + 190, "leapfrog": 14}


def work(case):
    kind = case["kind"]
    if kind == "ensemble":
        probs = _problems(case, np.random.Generator(np.random.PCG64(11)))
        b = sum(8 * p["n"] ** 3 * (4 if p["kind"] else 1) for p in probs)
        f = case["steps"] * sum(p["n"] ** 3 * _FLOPS["wave" if p["kind"] else "heat"] for p in probs)
        return {"bytes": b, "flops": f}
    n = case["nx"] * case["ny"] * case["nz"]
    es = 8 if case.get("dtype") == "f64" else 4
    vert = case.get("mesh") == "vertices"
    geom = 24 * n if vert else 0  # three doubles per vertex, about one vertex per cell
    if kind == "operators":
        return {"bytes": (6 + 4) * es * n + geom, "flops": (20 + 24 + 15 + 80 + 5) * n}
    if kind == "euler":
        steps = max(1, round(case["t_end"] / (0.4 * _spacing(case) / 4.2)))
        return {"bytes": 2 * 5 * es * n, "flops": steps * _FLOPS["euler"] * n}
    if kind == "gradient":
        return {"bytes": (4 + 1 + 1 + 2) * es * n, "flops": case["steps"] * _FLOPS["gradient"] * n}
    fields = {"heat": 2, "wave": 8 + (1 if case.get("c_field") else 0), "leapfrog": 3}[kind]
    return {"bytes": fields * es * n + geom, "flops": case["steps"] * (2 if vert else 1) * _FLOPS[kind] * n}


# ---- the same in 64 bits, plain torch ---------------------------------------------
def _nb(a, dim, side):
    """The neighbour along `dim` (side 0: -, 1: +); a wall cell sees itself."""
    n = a.shape[dim]
    lo, hi = a.narrow(dim, 0, 1), a.narrow(dim, n - 1, 1)
    if side:
        return torch.cat([a.narrow(dim, 1, n - 1), hi], dim)
    return torch.cat([lo, a.narrow(dim, 0, n - 1)], dim)


def _wall(shape, dim, side):
    w = torch.zeros(shape, device=DEVICE, dtype=torch.bool)
    w.narrow(dim, shape[dim] - 1 if side else 0, 1).fill_(True)
    return w


def _heat_step(T, c):
    out = T.clone()
    for d in range(3):
        out += c * ((_nb(T, d, 1) - T) + (_nb(T, d, 0) - T))
    return out


def _reflect(q, d, side):
    """Neighbour state of the acoustic system, a wall mirrors the velocity."""
    g = _nb(q, d + 1, side)
    n = q.shape[d + 1]
    sign = torch.ones(n, device=DEVICE, dtype=torch.float64)
    sign[n - 1 if side else 0] = -1
    shape = [1, 1, 1]
    shape[d] = n
    fields = [g[f] * sign.reshape(shape) if f == 1 + d else g[f] for f in range(4)]
    return torch.stack(fields)


def _wave_step(q, c, h, dt, mode):
    """One Rusanov step on cubic cells; c a number or a field."""
    field = torch.is_tensor(c)
    rhs = [0.0, 0.0, 0.0, 0.0]
    for d in range(3):
        m, p = _reflect(q, d, 0), _reflect(q, d, 1)
        if field:
            cm, cp = _nb(c, d, 0), _nb(c, d, 1)
            fm, fp = (torch.maximum(c, cm), torch.maximum(c, cp)) if mode == 0 else (0.5 * (c + cm), 0.5 * (c + cp))
        else:
            fm = fp = c
        for f in range(4):
            rhs[f] = rhs[f] + (0.5 * fp * (p[f] - q[f]) + 0.5 * fm * (m[f] - q[f])) / h
        rhs[0] = rhs[0] - c * c * 0.5 * (p[1 + d] - m[1 + d]) / h
        rhs[1 + d] = rhs[1 + d] - 0.5 * (p[0] - m[0]) / h
    return q + dt * torch.stack(rhs)


def _euler_prim(U):
    u = U[1:4] / U[0]
    p = (GAMMA - 1) * (U[4] - 0.5 * (U[1:4] * u).sum(0))
    return u, p, torch.sqrt(GAMMA * p / U[0])


def _euler(U, h, t_end):
    t = 0.0
    while t < t_end:
        u, p, a = _euler_prim(U)
        dt = 0.4 / sum(float((u[d].abs() + a).max()) / h for d in range(3))
        last = dt >= t_end - t
        dt = t_end - t if last else dt
        new = U.clone()
        for d in range(3):
            for side in (0, 1):
                N = _nb(U, d + 1, side)
                if d > 0:
                    N[1 + d].narrow(d, U.shape[d + 1] - 1 if side else 0, 1).neg_()
                un, pn, an = _euler_prim(N)
                s = 1.0 if side else -1.0
                lam = torch.maximum(u[d].abs() + a, un[d].abs() + an)
                F = 0.5 * s * (U * u[d] + N * un[d])
                F[1 + d] += 0.5 * s * (p + pn)
                F[4] += 0.5 * s * (p * u[d] + pn * un[d])
                new -= dt / h * (F - 0.5 * lam * (N - U))
        U = new
        t = t_end if last else t + dt
    return U


def _geometry(case, d):
    """Faces in the order z-, z+, y-, y+, x-, x+ as a function giving (unit
    normal along the axis, outward sign, area, centre), with cell centres and volumes."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    if "vertices" in d:
        V = torch.from_numpy(d["vertices"]).to(DEVICE)
    else:
        ax = [torch.arange(m + 1, device=DEVICE, dtype=torch.float64) * d["h"] for m in (nx, ny, nz)]
        V = torch.stack(torch.meshgrid(*ax, indexing="ij"), -1)
    V = V.movedim(-1, 0)

    def corner(a, b, c):
        return V[:, a: a + nx, b: b + ny, c: c + nz]

    cc = sum(corner(a, b, c) for a in (0, 1) for b in (0, 1) for c in (0, 1)) / 8

    def face(f):
        s, dim = f % 2, 2 - f // 2
        other = [e for e in range(3) if e != dim]

        def at(i, j):
            o = [0, 0, 0]
            o[dim], o[other[0]], o[other[1]] = s, i, j
            return corner(*o)
        A, B, C, D = at(0, 0), at(1, 0), at(1, 1), at(0, 1)
        S = 0.5 * torch.linalg.cross(C - A, D - B, dim=0)
        area = S.norm(dim=0)
        n = S / area
        n = torch.where(n[dim] < 0, -n, n)  # along +axis
        return n, (1.0 if s else -1.0), area, (A + B + C + D) / 4, dim, s
    vol = 0.0
    for f in range(6):
        n, sg, area, fc, _, _ = face(f)
        vol = vol + sg * ((fc - cc) * n).sum(0) * area
    return cc, vol / 3, face


def _operators(case, d):
    f64 = {k: v.double() for k, v in d.items() if torch.is_tensor(v)}
    T = f64["T"]
    cc, vol, face = _geometry(case, d)
    speed = torch.sqrt(GAMMA * f64["p"] / f64["rho"]) + torch.sqrt(f64["u"] ** 2 + f64["v"] ** 2 + f64["w"] ** 2)
    dt = float(0.1 * (d["h"] / speed).min())
    g = [0.0, 0.0, 0.0]
    lapl = 0.0
    for f in range(6):
        n, sg, area, fc, dim, s = face(f)
        N = _nb(T, dim, s)
        for e in range(3):
            g[e] = g[e] + 0.5 * (T + N) * sg * n[e] * area / vol
        dist = ((_nb(cc, dim + 1, s) - cc) * n).sum(0).abs()
        alpha = torch.where(dist > 0, 1 / dist, 0.0)  # a wall face has N = T
        lapl = lapl + (N - T) * alpha * n.sum(0) * area / vol
    stab = 0.0
    for f in range(6):
        n, sg, area, fc, dim, s = face(f)
        nf, sgf, _, fcf, _, _ = face(f ^ 1)
        length, other = (fc - cc).norm(dim=0), (fcf - cc).norm(dim=0)
        for e in range(3):
            mine = T + length * g[e] * sg * n[e]
            # the neighbour's value on its face towards this cell; a wall cell takes its own opposite face
            opp = _nb(T + other * g[e] * sgf * nf[e], dim, s)
            stab = stab + 0.5 * (mine - opp) * n[e] * area / vol
    grad = g[0] + g[1] + g[2]
    new = dt * (1e-3 * lapl - grad) + T
    inner = (slice(1, -1),) * 3
    out = T.clone()
    out[inner] = new[inner]
    return dict(dt=dt, grad=grad.reshape(-1), lapl=lapl.reshape(-1), stab=stab.reshape(-1), new=out.reshape(-1),
                total=float((out * vol).sum()))


def _wave_vertices(case, d, q):
    _, vol, face = _geometry(case, d)
    faces = []
    for f in range(6):
        n, sg, area, _, dim, s = face(f)
        faces.append((sg * n, area, dim, s, _wall(vol.shape, dim, s)))
    for _ in range(case["steps"]):
        rhs = torch.zeros_like(q)
        for n, area, dim, s, wall in faces:
            un = (q[1:] * n).sum(0)
            ghost = torch.cat([q[:1], q[1:] - 2 * un * n])
            N = torch.where(wall, ghost, _nb(q, dim + 1, s))
            unN = (N[1:] * n).sum(0)
            F = -0.5 * (N - q)
            F[0] += 0.5 * (un + unN)
            F[1:] += 0.5 * (q[0] + N[0]) * n
            rhs -= F * area
        q = q + d["dt"] * rhs / vol
    return q


def exact(case, seed):
    d = _inputs(case, seed)
    kind = case["kind"]
    if kind == "operators":
        return _operators(case, d)
    if kind == "heat":
        T = d["T"].double()
        for _ in range(case["steps"]):
            T = _heat_step(T, d["dt"] * d["k"] / d["h"] ** 2)
        return T.reshape(-1)
    if kind == "wave":
        q = d["q"].double()
        if "vertices" in d:
            return _wave_vertices(case, d, q).reshape(-1)
        c = d["c"].double() if "c" in d else 1.0
        for _ in range(case["steps"]):
            q = _wave_step(q, c, d["h"], d["dt"], 0)
        return q.reshape(-1)
    if kind == "euler":
        U = _euler(d["U"].double(), d["h"], case["t_end"])
        return dict(state=U.reshape(-1), totals=np.array([float(U[0].sum()), float(U[4].sum())]) * d["h"] ** 3)
    if kind == "ensemble":
        out = []
        for p, q in zip(d["probs"], d["fields"]):
            q, h = q.double(), 1.0 / p["n"]
            for _ in range(case["steps"]):
                if p["kind"] == 0:
                    q = _heat_step(q[0], p["dt"] * p["param"] / h ** 2)[None]
                else:
                    q = _wave_step(q, p["param"], h, p["dt"], 0)
            out.append(q.reshape(-1))
        return torch.cat(out)
    if kind == "gradient":
        from torch.utils.checkpoint import checkpoint
        c = d["c"].double().requires_grad_()
        p0 = d["q"][0].double().requires_grad_()
        q = torch.cat([p0[None], d["q"][1:].double()])
        for _ in range(case["steps"]):
            q = checkpoint(_wave_step, q, c, d["h"], d["dt"], 1, use_reentrant=False)
        J = 0.5 * ((q[0] - d["target"].double()) ** 2).sum()
        gc, gp = torch.autograd.grad(J, (c, p0))
        return dict(J=float(J.detach()), grad_c=gc.reshape(-1), grad_p0=gp.reshape(-1))
    prev = d["u"].double()

    def rate(u):
        return d["k"] * sum((_nb(u, e, 1) - u) + (_nb(u, e, 0) - u) for e in (0, 1))
    cur = d["dt"] * rate(prev) + prev
    for _ in range(case["steps"] - 1):
        prev, cur = cur, d["dt"] ** 2 * rate(cur) + 2 * cur - prev
    return dict(u=cur.reshape(-1), u_prev=prev.reshape(-1))
